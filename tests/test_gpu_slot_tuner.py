"""The batch's slot tuner over a part of every item's points (candidates whose chunks need
no more walks than that): the next step's results are those of a plan never tuned."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sample", [0.01, 0.3, 1.0])
@pytest.mark.parametrize("mode", [0, 1])
def test_tuning_on_a_part_leaves_results_alone(cuda, mode, sample):
    import wos
    from wos.native import AdjointSettings, NativeScene, WalkSettings

    def items():
        out = []
        for i, (dim, size, n) in enumerate([(2, 64, 700), (3, 2, 300), (2, 3000, 1), (3, 4, 900), (2, 700, 1500)]):
            V, F = wos.shapes.star(size) if dim == 2 else wos.shapes.icosphere(size)
            V = np.asarray(V, np.float32)
            src = (1, [0.1, -0.2, 0.3, 1.5, 0.0]) if i == 4 else ()
            ns = NativeScene(V, F, V[:, 0].copy(), *src)
            P = np.random.default_rng(i).uniform(-0.3, 0.3, (n, dim)).astype(np.float32)
            out.append(wos.BatchItem(ns, P, WalkSettings(nwalks=3 + i, nsteps=32, seed=i, include_source=i == 4)))
        return out

    wos.set_sample_order(mode)
    try:
        a = AdjointSettings(want_dV=True, want_dg=True, want_dsrc=True)
        tuned, plain = wos.BatchPlan(items(), a), wos.BatchPlan(items(), a)
        shapes = [(32, 1, 1), (64, 1, 2), (128, 2, 1)]
        best, ms = tuned.autotune_slots(shapes, repeats=2, sample=sample)
        assert set(best) == {(2, 0), (2, 1), (3, 0), (3, 1)}
        assert all(np.isfinite(t) and t > 0 for slot in ms.values() for t in slot.values())
        for graph in (False, True):
            tuned.run(use_graph=graph)
            plain.run(use_graph=graph)
            for i in range(5):
                x, y = tuned.outputs(i), plain.outputs(i)
                for k in ("mean", "var", "loss"):
                    assert np.array_equal(x[k].cpu().numpy(), y[k].cpu().numpy()), (i, k)
                for k in ("dV", "dg", "dsrc"):
                    u, v = x[k].cpu().numpy(), y[k].cpu().numpy()
                    np.testing.assert_allclose(u, v, rtol=1e-5, atol=1e-6 * max(np.abs(v).max(), 1e-30))
    finally:
        wos.set_sample_order(1)
