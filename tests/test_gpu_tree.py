"""The search tree against brute force, bit for bit, at the sizes where its shape
changes: one primitive, whole and broken leaves and nodes, and the segment sizes
of the mesh order's median splits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 63, 64, 65, 127, 129, 511, 513, 1023, 1024, 1025, 2047, 2048, 2049, 4097]


def _soup(dim, n, seed):
    """n primitives of uneven sizes, scattered or chained, some of them equal and
    some degenerate."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, dim))
    V = c + rng.uniform(-1, 1, (n, dim, dim)) * np.exp(rng.uniform(-5, 0, (n, 1, 1)))
    if n > 4:
        V[1] = V[0]  # ties
        V[n // 2, 1:] = V[n // 2, :1]  # a point
        V[n - 1] = V[n // 3]
    F = np.arange(n * dim).reshape(n, dim)
    return V.reshape(-1, dim).astype(np.float32), F.astype(np.int32)


def _check(ns, P):
    a, b = ns.closest(P, use_bvh=True), ns.closest(P, use_bvh=False)
    for k in ("prim", "dist", "tuv", "pt"):
        x, y = a[k].cpu().numpy(), b[k].cpu().numpy()
        assert np.array_equal(x, y, equal_nan=True), k


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", SIZES)
def test_tree_equals_brute_force(cuda, dim, n):
    from wos.native import NativeScene
    V, F = _soup(dim, n, 17 * n + dim)
    rng = np.random.default_rng(n)
    P = np.concatenate([rng.uniform(-2, 2, (500, dim)), V[rng.integers(0, len(V), 40)], V.mean(0)[None],
                        rng.uniform(-50, 50, (20, dim))]).astype(np.float32)
    ns = NativeScene(V, F, np.zeros(len(V), np.float32))
    _check(ns, P)
    # moved vertices: the mesh keeps its order, the bounds are new
    ns.update_vertices((V[:, ::-1] * np.float32(0.5) + np.float32(0.1)).copy())
    _check(ns, P)


@pytest.mark.parametrize("dim", [2, 3])
def test_ball_search_equals_brute_force(cuda, dim):
    """The largest inscribed ball at closest-point records, tree against brute force."""
    from wos.native import NativeScene
    V, F = _soup(dim, 333, 5)
    ns = NativeScene(V, F, np.zeros(len(V), np.float32))
    P = np.random.default_rng(1).uniform(-1.5, 1.5, (257, dim)).astype(np.float32)
    o = ns.closest(P)
    valid = np.ones(len(P), np.uint8)
    valid[::7] = 0
    a = ns.inscribed_ball(valid, o["pt"], o["n"], 1e-3, use_bvh=True).cpu().numpy()
    b = ns.inscribed_ball(valid, o["pt"], o["n"], 1e-3, use_bvh=False).cpu().numpy()
    assert np.array_equal(a, b, equal_nan=True)
