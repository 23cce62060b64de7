"""The search tree's entry grid against brute force, bit for bit, where a cell could
list too few nodes: points on the cells' borders and just beside them, on and outside
the bounding box, flat scenes, and scenes far from the origin, tiny and huge."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLACES = ["unit", "flat", "offset", "tiny", "huge", "long"]


def _place(V, place):
    V = V.astype(np.float64)
    if place == "flat":
        V[:, -1] = 0.25
    elif place == "offset":
        V = V + 1000.0
    elif place == "tiny":
        V = V * 1e-12
    elif place == "huge":
        V = V * 1e12
    elif place == "long":
        V[:, 0] *= 1000.0
    return V.astype(np.float32)


def _points(V, rng):
    lo, hi = V.min(0), V.max(0)
    ext = np.maximum(hi - lo, (hi - lo).max() * np.float32(1e-3))
    inside = lo + ext * rng.uniform(0, 1, (3000, V.shape[1]))
    # borders of the cells at every power of two, and their neighbours
    border = (lo + ext * (rng.integers(0, 129, (1500, V.shape[1])) / 128.0)).astype(np.float32)
    near = np.nextafter(border, np.where(rng.uniform(size=border.shape) < 0.5, -np.inf, np.inf).astype(np.float32))
    outside = lo + ext * rng.uniform(-1, 2, (500, V.shape[1]))
    on = V[rng.integers(0, len(V), 500)]
    return np.concatenate([inside, border, near, outside, on, lo[None], hi[None]]).astype(np.float32)


@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("dim,size", [(2, 40), (2, 1024), (2, 5000), (3, 1), (3, 3), (3, 4)])
def test_grid_equals_brute_force(cuda, dim, size, place):
    import wos
    from wos.native import NativeScene
    V, F = wos.shapes.star(size) if dim == 2 else wos.shapes.icosphere(size)
    V = np.asarray(V) * (1.0 if dim == 2 else np.array([1.0, 0.8, 0.6]))
    V = _place(V, place)
    rng = np.random.default_rng(size + dim)
    ns = NativeScene(V, F, np.zeros(len(V), np.float32))
    for W in (V, (V * np.float32(0.75)).copy()):  # as built, and after a move
        ns.update_vertices(W)
        P = _points(W, rng)
        a, b = ns.closest(P, use_bvh=True), ns.closest(P, use_bvh=False)
        for k in ("prim", "dist", "tuv", "pt"):
            assert np.array_equal(a[k].cpu().numpy(), b[k].cpu().numpy(), equal_nan=True), k
