"""Scenes with vertices that are not finite, or so far apart that the box's extent is
not: queries and walks by the tree against brute force, bit for bit, also where the
tree lacks some of its last nodes, and after a move to finite vertices and back."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def clean_status(cuda):
    """Queries that find no primitive say so in the device's status word."""
    import wos
    yield
    wos.device_status(reset=True)


@pytest.mark.parametrize("what", ["inf", "-inf", "nan", "all_nan", "far", "huge"])
@pytest.mark.parametrize("dim,n", [(2, 1), (2, 5), (2, 40), (2, 300), (3, 1), (3, 3), (3, 40), (3, 300)])
def test_nonfinite_scene_equals_brute_force(cuda, dim, n, what):
    from wos.native import NativeScene, WalkSettings
    rng = np.random.default_rng(n)
    V = (rng.uniform(-1, 1, (n, 1, dim)) + 0.1 * rng.normal(size=(n, dim, dim))).reshape(-1, dim).astype(np.float32)
    F = np.arange(n * dim, dtype=np.int32).reshape(n, dim)
    W = V.copy()
    if what == "all_nan":
        W[:] = np.nan
    elif what == "far":
        W[0], W[-1] = -3e38, 3e38
    elif what == "huge":
        W *= np.float32(1e38)
    else:
        W[len(W) // 2, rng.integers(dim)] = float(what)
        if n > 5:
            W[:3] = float(what)
    P = np.concatenate([rng.uniform(-1.5, 1.5, (500, dim)), V, 1e37 * rng.normal(size=(50, dim))]).astype(np.float32)
    ns = NativeScene(W, F, rng.uniform(-1, 1, len(V)).astype(np.float32))
    s = dict(nwalks=2, nsteps=8, epsilon=1e-2, double_sided=True)
    for X in (W, V, W):
        ns.update_vertices(X)
        a, b = ns.closest(P, use_bvh=True), ns.closest(P, use_bvh=False)
        for k in ("prim", "dist"):
            assert np.array_equal(a[k].cpu().numpy(), b[k].cpu().numpy(), equal_nan=True), k
        u, v = (ns.values(P[:500], WalkSettings(use_bvh=t, **s)).cpu().numpy() for t in (True, False))
        assert np.array_equal(u, v, equal_nan=True)
