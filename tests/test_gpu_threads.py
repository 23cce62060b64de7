"""Calls from several host threads at once: a deep and a shallow scene solved and
differentiated by the same kernels, whose shared memory differs."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_with_scenes_of_different_depth(cuda):
    import torch
    import wos
    from wos.native import AdjointSettings, NativeScene, WalkSettings
    a = AdjointSettings(want_dV=True, want_dg=True)
    s = WalkSettings(nwalks=2, nsteps=4)

    def scene(level):
        V, F = wos.shapes.icosphere(level)
        V = np.asarray(V, np.float32)
        P = torch.tensor(0.9 * V[:8].copy(), device="cuda")
        return NativeScene(V, F, V[:, 0].copy()), P

    scenes = [scene(3), scene(6)]
    want = [ns.solve_adjoint(P, s, a)["mean"] for ns, P in scenes]
    torch.cuda.synchronize()
    wrong, stop = [], threading.Event()

    def work(i):
        ns, P = scenes[i]
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(400):
                    out = ns.solve_adjoint(P, s, a)
                    if stop.is_set():
                        return
                torch.cuda.current_stream().synchronize()
                assert torch.equal(out["mean"], want[i])
        except Exception as e:  # noqa: BLE001
            wrong.append(repr(e))
            stop.set()

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 0, 1, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not wrong, wrong
