"""Scenes so small that squared distances, or the products in a triangle's barycentric
coordinates, are denormal floats, where rounding is a step and not a fraction: the tree
against brute force, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def clean_status(cuda):
    """Queries that find no primitive (every distance NaN) say so in the device's status."""
    import wos
    yield
    wos.device_status(reset=True)


@pytest.mark.parametrize("scale", [1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-13, 1e-16, 1e-17, 1e-18, 1e-19, 1e-20, 1e-21,
                                   1e-22, 1e-23, 1e-25, 1e-30])
@pytest.mark.parametrize("dim,size", [(2, 40), (2, 1024), (3, 2), (3, 4)])
def test_small_scene_equals_brute_force(cuda, dim, size, scale):
    import wos
    from wos.native import NativeScene
    V, F = wos.shapes.star(size) if dim == 2 else wos.shapes.icosphere(size)
    V = (np.asarray(V, np.float64) * scale).astype(np.float32)
    rng = np.random.default_rng(size)
    P = np.concatenate([rng.uniform(-1, 1, (6000, dim)), rng.uniform(-5, 5, (1000, dim)),
                        rng.uniform(-300, 300, (1000, dim))]) * scale
    P = np.concatenate([P.astype(np.float32), V[rng.integers(0, len(V), 500)]])
    ns = NativeScene(V, F, np.zeros(len(V), np.float32))
    x, y = ns.closest(P, use_bvh=True), ns.closest(P, use_bvh=False)
    for k in ("prim", "dist"):
        a, b = x[k].cpu().numpy(), y[k].cpu().numpy()
        assert np.array_equal(a, b), (k, np.count_nonzero(a != b))
