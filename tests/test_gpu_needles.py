"""Needle triangles, whose barycentric coordinates (and with them the closest point
and its distance) are inexact in float: the tree against brute force, bit for bit,
where such a needle is the only near primitive of a cell of the entry grid."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _needle(rng, length, aspect):
    d = rng.normal(size=3)
    d /= np.linalg.norm(d)
    e = np.cross(d, rng.normal(size=3))
    e /= np.linalg.norm(e)
    f = np.cross(d, e)
    a = rng.uniform(-0.05, 0.05, 3) - 0.5 * length * d
    w = length * aspect
    return np.stack([a, a + length * d + w * rng.uniform(-1, 1) * f, a + rng.uniform(0.2, 1) * length * d + w * e])


@pytest.mark.parametrize("level", [2, 4, 5])
@pytest.mark.parametrize("aspect", [1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
def test_needles_equal_brute_force(cuda, level, aspect):
    import wos
    from wos.native import NativeScene
    V, F = wos.shapes.icosphere(level)
    V, F = np.asarray(V, np.float64), np.asarray(F)
    for trial in range(6):
        rng = np.random.default_rng(100 * level + trial)
        T = [_needle(rng, 1.8, aspect) for _ in range(1 + trial % 3)]
        W = np.concatenate([V] + T).astype(np.float32)
        G = np.concatenate([F, len(V) + np.arange(3 * len(T)).reshape(-1, 3)]).astype(np.int32)
        ns = NativeScene(W, G, np.zeros(len(W), np.float32))
        # beside the needles, all along them
        b = rng.dirichlet([1, 1, 1], 20000)
        P = (np.stack(T)[rng.integers(0, len(T), 20000)] * b[:, :, None]).sum(1)
        P = (P + rng.normal(size=P.shape) * np.exp(rng.uniform(-9, -2.5, (len(P), 1)))).astype(np.float32)
        x, y = ns.closest(P, use_bvh=True), ns.closest(P, use_bvh=False)
        for k in ("prim", "dist", "tuv", "pt"):
            a, c = x[k].cpu().numpy(), y[k].cpu().numpy()
            assert np.array_equal(a, c), (k, trial, np.count_nonzero(a != c))


@pytest.mark.parametrize("n", [100, 1000, 10000])
def test_fan_equals_brute_force(cuda, n):
    """A cylinder whose caps are fans about one vertex."""
    from wos.native import NativeScene
    t = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(t), np.sin(t)], 1)
    V = np.concatenate([np.c_[ring, np.full(n, -0.5)], np.c_[ring, np.full(n, 0.5)], [[0, 0, -0.5], [0, 0, 0.5]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    F = np.concatenate([np.stack(f, 1) for f in ((i, j, n + i), (j, n + j, n + i), (j, i, 0 * i + 2 * n),
                                                (n + i, n + j, 0 * i + 2 * n + 1))])
    V, F = V.astype(np.float32), F.astype(np.int32)
    rng = np.random.default_rng(n)
    P = rng.uniform(-1, 1, (20000, 3)) * [1, 1, 0.7]
    P[::2, 2] = np.where(P[::2, 2] > 0, 0.5, -0.5) + rng.normal(size=10000) * np.exp(rng.uniform(-12, -3, 10000))
    ns = NativeScene(V, F, np.zeros(len(V), np.float32))
    x, y = ns.closest(P.astype(np.float32), use_bvh=True), ns.closest(P.astype(np.float32), use_bvh=False)
    for k in ("prim", "dist", "tuv", "pt"):
        assert np.array_equal(x[k].cpu().numpy(), y[k].cpu().numpy()), k
