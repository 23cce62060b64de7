"""Searches that a warp's lanes finish together against brute force, bit for bit:
points at nearly or exactly the same distance from much of the scene, alone and
several to a warp, with ties between equal primitives."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,size", [(2, 4096), (3, 3), (3, 5)])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 200, 5000])
def test_shared_searches_equal_brute_force(cuda, dim, size, n):
    import wos
    from wos.native import NativeScene
    if dim == 2:
        t = 2 * np.pi * np.arange(size) / size
        V, F = np.stack([np.cos(t), np.sin(t)], 1), np.stack([np.arange(size), (np.arange(size) + 1) % size], 1)
    else:
        V, F = wos.shapes.icosphere(size)
        V = np.asarray(V)
    F = np.concatenate([F, F[::3]])  # equal primitives
    rng = np.random.default_rng(n)
    P = rng.normal(size=(n, dim)) * np.where(rng.uniform(size=(n, 1)) < 0.7, 1e-3, 0.4)
    P[0] = 0.0
    V, F, P = V.astype(np.float32), F.astype(np.int32), P.astype(np.float32)
    ns = NativeScene(V, F, np.zeros(len(V), np.float32))
    a, b = ns.closest(P, use_bvh=True), ns.closest(P, use_bvh=False)
    for k in ("prim", "dist", "tuv", "pt"):
        assert np.array_equal(a[k].cpu().numpy(), b[k].cpu().numpy(), equal_nan=True), k
