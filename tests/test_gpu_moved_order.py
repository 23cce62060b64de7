"""Search work on meshes whose vertices were moved: at most twice that of a scene
made anew from the same vertices, however far they moved."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _loose(rng, n=20480, size=0.02):
    """n triangles that share no vertex, on a sphere."""
    c = rng.normal(size=(n, 1, 3))
    c /= np.linalg.norm(c, axis=2, keepdims=True)
    V = c + size * rng.normal(size=(n, 3, 3))
    return V, np.arange(3 * n, dtype=np.int32).reshape(n, 3)


def _moves(kind, rng):
    """(faces, vertices of the scene at first, vertices moved to in turn)"""
    import wos
    if kind.startswith("loose"):
        V, F = _loose(rng)
        step = float(kind.split("_")[1])
        there = V + step * rng.uniform(-1, 1, (len(F), 1, 3))
        return F, V.reshape(-1, 3), [there.reshape(-1, 3)]
    V, F = wos.shapes.icosphere(5)
    V = np.asarray(V, np.float64)
    if kind == "zero":
        return F, 0.0 * V, [V]
    if kind == "line":
        return F, V * [1.0, 0.0, 0.0], [V]
    if kind == "flat":
        return F, V * [1.0, 1.0, 0.0], [V]
    if kind == "shuffled":
        return F, V[rng.permutation(len(V))], [V]
    if kind == "nan":
        return F, V * np.nan, [V]
    if kind == "points":  # triangles collapsed to points, scattered, then put in place
        T = np.repeat(rng.uniform(-1, 1, (len(F), 1, 3)), 3, 1).reshape(-1, 3)
        return np.arange(3 * len(F), dtype=np.int32).reshape(-1, 3), T, [V[F].reshape(-1, 3)]
    if kind == "slowly":  # in steps, each of which is small
        a = rng.normal(size=(len(F), 1, 3))
        T = V[F]
        return (np.arange(3 * len(F), dtype=np.int32).reshape(-1, 3), T.reshape(-1, 3),
                [(T + 0.02 * k * a).reshape(-1, 3) for k in range(1, 16)])
    raise ValueError(kind)


def _steps(ns, P):
    """Node and leaf steps of a solve."""
    import wos
    from wos.native import WalkSettings
    wos.work_counters(reset=True)
    wos.set_work_counting(True)
    try:
        u = ns.values(P, WalkSettings(nwalks=4, nsteps=16, epsilon=1e-3, double_sided=True))
    finally:
        wos.set_work_counting(False)
    c = wos.work_counters(reset=True)
    return u, list(c.values())[1:] if isinstance(c, dict) else list(c)[1:]


@pytest.mark.parametrize("kind", ["loose_0.02", "loose_0.05", "loose_0.2", "loose_0.5", "loose_2", "zero", "line",
                                  "flat", "shuffled", "nan", "points", "slowly"])
def test_moved_mesh_searches_like_a_new_one(cuda, kind):
    from wos.native import NativeScene
    rng = np.random.default_rng(7)
    F, V, moves = _moves(kind, rng)
    g = rng.uniform(-1, 1, len(V)).astype(np.float32)
    ns = NativeScene(V.astype(np.float32), F, g)
    for W in moves:
        ns.update_vertices(W.astype(np.float32))
    fresh = NativeScene(moves[-1].astype(np.float32), F, g)
    P = rng.uniform(-0.6, 0.6, (2000, 3)).astype(np.float32)
    (u, moved), (v, anew) = _steps(ns, P), _steps(fresh, P)
    assert np.array_equal(u.cpu().numpy(), v.cpu().numpy())
    assert sum(moved) <= 2 * sum(anew), (moved, anew)
