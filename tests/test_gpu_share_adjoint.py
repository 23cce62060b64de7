"""Adjoint samples whose warps share their last searches (meshes of more than 2,048
triangles, few samples): normal derivatives bit for bit and gradients against brute
force, alone and in a batch, where balls touch the mesh in much of it; and the time of
such a call."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind):
    import wos
    from wos.native import NativeScene
    if kind == "sphere":
        V, F = wos.shapes.icosphere(4)
    elif kind == "waves":
        V, F = wos.shapes.displaced_icosphere(4, 0.15, 1)
    else:  # two spheres, one in the other, and equal triangles
        V, F = wos.shapes.icosphere(4)
        V, F = np.concatenate([V, 0.5 * V]), np.concatenate([F, F + len(V), F[::5]])
    V = np.asarray(V, np.float32)
    return NativeScene(V, np.asarray(F, np.int32), (V[:, 0] * V[:, 1] + V[:, 2]).astype(np.float32))


@pytest.mark.parametrize("kind", ["sphere", "waves", "shells"])
@pytest.mark.parametrize("n", [1, 2, 7, 33, 250])
def test_normal_derivatives_equal_brute_force(cuda, kind, n):
    from wos.native import AdjointSettings, WalkSettings
    ns = _scene(kind)
    P = np.random.default_rng(n).uniform(-0.25, 0.25, (n, 3)).astype(np.float32)
    o = ns.records(P, WalkSettings(nwalks=1, nsteps=64, double_sided=kind == "shells"))
    rec = dict(valid=o["valid"], pt=o["pt"], n=o["n"], tuv=o["tuv"], prim=o["prim"])
    s = dict(nwalks=1, nsteps=16, double_sided=kind == "shells", seed=3)
    a = AdjointSettings()
    x, y = (ns.normal_derivative(rec, WalkSettings(use_bvh=b, **s), a).cpu().numpy() for b in (True, False))
    assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("n", [1, 40, 300])
def test_gradients_equal_brute_force(cuda, n):
    import torch
    import wos
    from wos.native import AdjointSettings, WalkSettings
    ns = _scene("sphere")
    P = torch.tensor(np.random.default_rng(n).uniform(-0.3, 0.3, (n, 3)).astype(np.float32), device="cuda")
    a = AdjointSettings(want_dV=True, want_dg=True)
    s = dict(nwalks=2, nsteps=16, seed=5)
    x, y = (ns.solve_adjoint(P, WalkSettings(use_bvh=b, **s), a) for b in (True, False))
    dL = torch.ones(n, device="cuda")
    u, v = (ns.adjoint(P, WalkSettings(use_bvh=b, **s), a, dL) for b in (True, False))
    pairs = [(x["dV"], y["dV"]), (x["dg"], y["dg"]), (u[0], v[0]), (u[1], v[1])]
    plan = wos.BatchPlan([wos.BatchItem(ns, P, WalkSettings(**s), loss_kind=1),
                          wos.BatchItem(_scene("waves"), P, WalkSettings(**s), loss_kind=1)], a)
    plan.run()
    pairs += [(plan.outputs(0)["dV"], y["dV"]), (plan.outputs(0)["dg"], y["dg"])]
    for p, q in pairs:
        p, q = p.cpu().numpy(), q.cpu().numpy()
        np.testing.assert_allclose(p, q, rtol=1e-5, atol=1e-6 * max(np.abs(q).max(), 1e-30))


def test_samples_in_a_sphere_take_little_longer(cuda):
    """1,000 samples in a sphere of 81,920 triangles against one displaced in waves."""
    import torch
    import wos
    from wos.native import AdjointSettings, NativeScene, WalkSettings
    P = torch.tensor(np.random.default_rng(0).uniform(-0.4, 0.4, (1000, 3)).astype(np.float32), device="cuda")
    dL, times = torch.ones(1000, device="cuda"), []
    s, a = WalkSettings(nwalks=1, nsteps=64), AdjointSettings()
    for V, F in (wos.shapes.icosphere(6), wos.shapes.displaced_icosphere(6, 0.15, 0)):
        V = np.asarray(V, np.float32)
        ns = NativeScene(V, F, V[:, 0].copy())
        rec = ns.solve_records(P, s)[2]
        t = []
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            ns.adjoint_records(P, s, a, dL, rec, None)
            e1.record()
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        times.append(min(t))
    assert times[0] < 4 * times[1], times
