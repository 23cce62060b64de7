"""Tangents from the forward's records (wos_tangent_records) against walking again
(wos_solve_tangent): the same walks, so the same values, for every subset of the
directions (only a moving boundary orders the samples)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,nwalks", [(2, 1, 1), (2, 33, 7), (2, 700, 8), (3, 5, 3), (3, 257, 8)])
@pytest.mark.parametrize("which", ["V", "g", "s", "Vg", "Vgs"])
def test_records_tangent_equals_solve_tangent(cuda, dim, n, nwalks, which):
    import torch
    import wos
    from wos.native import AdjointSettings, NativeScene, WalkSettings
    if dim == 3:
        which = which.replace("s", "") or "g"
    V, F = wos.shapes.star(96) if dim == 2 else wos.shapes.icosphere(2)
    V = np.asarray(V, np.float32)
    rng = np.random.default_rng(n)
    ns = NativeScene(V, F, rng.uniform(-1, 1, len(V)).astype(np.float32))
    if "s" in which:
        ns.set_source(1, [0.1, -0.2, 0.3, 1.5, 0.0])
    P = rng.uniform(-0.3, 0.3, (n, dim)).astype(np.float32)
    s = WalkSettings(nwalks=nwalks, nsteps=32, epsilon=1e-3, include_source="s" in which)
    a = AdjointSettings(want_dV="V" in which, want_dg="g" in which, want_dsrc="s" in which)
    d = dict(dV=torch.tensor(rng.normal(size=V.shape).astype(np.float32), device="cuda") if "V" in which else None,
             dg=torch.tensor(rng.normal(size=len(V)).astype(np.float32), device="cuda") if "g" in which else None,
             dsrc=torch.tensor(rng.normal(size=5).astype(np.float32), device="cuda") if "s" in which else None)
    ref = ns.solve_tangent(P, s, a, **d)
    mean, _, rec, dc = ns.solve_records(P, s, want_dcontrib="s" in which)
    assert torch.equal(mean, ref["mean"])
    assert torch.equal(ns.tangent_records(P, s, a, rec, dc, **d), ref["tangent"])
