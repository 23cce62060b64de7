"""Records handed to adjoint_records and tangent_records that are not those of the call:
too few, of the wrong kind, or of another scene."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(dim, size):
    import wos
    from wos.native import NativeScene
    V, F = wos.shapes.star(size) if dim == 2 else wos.shapes.icosphere(size)
    V = np.asarray(V, np.float32)
    return NativeScene(V, F, V[:, 0].copy(), *((1, [0.1, -0.2, 0.3, 1.5, 0.0]) if dim == 2 else ()))


def _calls(ns, P, s, a, rec, dc):
    import torch
    dV = torch.ones((ns.nV, ns.dim), device="cuda")
    dL = torch.ones(len(P), device="cuda")
    ds = torch.ones(5, device="cuda") if a.want_dsrc else None
    return (lambda: ns.adjoint_records(P, s, a, dL, rec, dc), lambda: ns.tangent_records(P, s, a, rec, dc, dV=dV,
                                                                                          dsrc=ds))


@pytest.mark.parametrize("dim", [2, 3])
def test_short_records_are_refused(cuda, dim):
    import torch
    from wos.native import AdjointSettings, WalkSettings
    ns = _scene(dim, 64 if dim == 2 else 1)
    P = torch.tensor(np.random.default_rng(0).uniform(-0.2, 0.2, (100, dim)).astype(np.float32), device="cuda")
    s = WalkSettings(nwalks=4, include_source=dim == 2)
    a = AdjointSettings(want_dV=True, want_dsrc=dim == 2)
    _, _, rec, dc = ns.solve_records(P, s, want_dcontrib=dim == 2)
    few = ns.solve_records(P, WalkSettings(nwalks=3, include_source=dim == 2), want_dcontrib=dim == 2)
    bad = [(few[2], dc), (rec[:-1], dc), (torch.stack([rec, rec], 1)[:, 0], dc)]
    if dim == 2:
        bad += [(rec, few[3]), (rec, dc.double()), (rec, dc[:-1])]
    for r, d in bad:
        for call in _calls(ns, P, s, a, r, d):
            with pytest.raises(ValueError):
                call()
    for call in _calls(ns, P, s, a, rec, dc):
        call()


@pytest.mark.parametrize("dim,sizes", [(2, (4096, 16)), (3, (4, 0))])
def test_records_of_another_scene_are_passed_over(cuda, dim, sizes):
    """The kernel looks no primitive up that the scene does not have."""
    import torch
    import wos
    from wos.native import AdjointSettings, WalkSettings
    large, small = (_scene(dim, n) for n in sizes)
    P = torch.tensor(np.random.default_rng(0).uniform(-0.2, 0.2, (300, dim)).astype(np.float32), device="cuda")
    s = WalkSettings(nwalks=4, nsteps=64)
    a = AdjointSettings(want_dV=True, want_dg=True)
    rec = large.solve_records(P, s)[2]
    for call in _calls(small, P, s, a, rec, None):
        wos.device_status(reset=True)
        out = call()
        for x in out if isinstance(out, tuple) else (out,):
            assert x is None or bool(torch.isfinite(x).all())
        assert wos.device_status(reset=True) & wos._lib.STATUS_BAD_PRIM
