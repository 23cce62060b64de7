"""Walks by brute force in the persistent kernel against one thread per walk, where few
lanes search: the segments' loads are all there is to wait for, and the persistent
kernel keeps as many in flight."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nwalks", [1, 8])
def test_brute_force_walks_keep_loads_in_flight(cuda, nwalks):
    import torch
    import wos
    from wos.native import NativeScene, WalkSettings
    V, F = wos.shapes.star(8192)
    V = np.asarray(V, np.float32)
    ns = NativeScene(V, F, V[:, 0].copy())
    P = torch.tensor(np.random.default_rng(3).uniform(-0.3, 0.3, (1, 2)).astype(np.float32), device="cuda")
    s = WalkSettings(nwalks=nwalks, nsteps=64, use_bvh=False)
    times = []
    for plain in (False, True):
        t = []
        for _ in range(10):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            v = ns.values(P, s, plain=plain)
            e1.record()
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        times.append((min(t), v))
    assert torch.equal(times[0][1], times[1][1])
    assert times[0][0] < 0.85 * times[1][0], [t for t, _ in times]
