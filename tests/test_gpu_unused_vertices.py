"""Scenes most of whose vertices belong to no face: how those lie among the others
makes no difference to the time a scene takes, and their normals are zero."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_runs_of_unused_vertices(cuda, dim):
    import torch
    from wos.native import NativeScene
    nV, k = 20_000_000, 1000
    V, g = torch.rand(nV, dim, device="cuda"), torch.zeros(nV, device="cuda")
    i = torch.arange(k, device="cuda")
    near = torch.stack([i, (i + 1) % k, (i + 7) % k][:dim], 1)

    def best(F):
        t = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            ns = NativeScene(V, F, g)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
            ns.close()
        return min(t)

    together, spread = best(near.int()), best((near * (nV // k)).int())
    assert together < 2 * spread, (together, spread)


@pytest.mark.parametrize("dim", [2, 3])
def test_normals_beside_unused_vertices(cuda, dim):
    import wos
    from wos.native import NativeScene
    V, F = wos.shapes.star(50) if dim == 2 else wos.shapes.icosphere(1)
    V, F = np.asarray(V, np.float32), np.asarray(F)
    want = NativeScene(V, F, V[:, 0].copy()).normals().cpu().numpy()
    at = np.sort(np.random.default_rng(0).choice(1000, len(V), replace=False)) + 3
    W = np.full((1100, dim), 0.1, np.float32)
    W[at] = V
    got = NativeScene(W, at[F].astype(np.int32), W[:, 0].copy()).normals().cpu().numpy()
    assert np.array_equal(got[at], want)
    rest = np.delete(got, at, 0)
    assert np.array_equal(np.nan_to_num(rest), 0 * rest)
