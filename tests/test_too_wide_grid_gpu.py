"""A grid wider than the launch was sized for, in the one-CTA kernels of the float-float form and of the
adjoint: NaN for that instance and the others' results, as in the FP64 and the cluster kernels
(tests/test_tdse_cluster_gpu.py has those)."""
import numpy as np
import pytest
import torch

from tests.tdse_cases import A_CONFIG

pytestmark = pytest.mark.gpu
PARAMS = [dict(num_r=n, dx=0.2, trg_a=A_CONFIG) for n in (500, 2600, 1300)]


def _field(n=40):
    t = 0.25 * np.arange(1, n + 1)
    return torch.tensor(0.05 * np.sin(np.pi * t / t[-1]) ** 2 * np.cos(0.3 * t), device="cuda")


def test_df64_one_cta(gpu_lib):
    from mma_gb300.tdse_batch import TDSEBatchPlan, TDSEGrids

    grids = TDSEGrids(PARAMS, dt=0.25, df64=True)
    outs = []
    for cap in (None, int(grids.m[2])):
        plan = TDSEBatchPlan(grids, [40] * 3, 0.25, grid_ids=[0, 1, 2], precision="df64", grid_ctas=1)
        if cap:
            plan.launches[0]["max_m"] = cap
        plan.load_fields([_field()] * 3)
        plan.launch()
        torch.cuda.synchronize()
        outs.append(plan.result())
    for i in (0, 2):
        assert torch.equal(outs[1].series(i)["sourceterm"], outs[0].series(i)["sourceterm"])
    assert torch.isnan(outs[1].series(1)["sourceterm"]).all() and torch.isfinite(outs[0].series(1)["sourceterm"]).all()


class _Narrow:
    """The library with one CTA by default and an adjoint sweep sized for at most max_m rows of 256 sites."""

    def __init__(self, lib, max_m):
        self._lib, self._max_m = lib, max_m

    def __getattr__(self, name):
        if name == "mma_tdse_default_ctas":
            return lambda *a: 1
        call = getattr(self._lib, name)
        return (lambda *a: call(*a[:8], min(a[8], self._max_m), *a[9:])) if name == "mma_tdse_adjoint" else call


def test_adjoint_one_cta(gpu_lib, monkeypatch):
    import mma_gb300.tdse_adjoint as ta
    from mma_gb300.tdse_batch import TDSEGrids

    grids = TDSEGrids(PARAMS, dt=0.25, adjoint=True)
    lib, outs = ta._adj_sig(), []
    for cap in (1000, int(grids.m[2])):
        monkeypatch.setattr(ta, "_adj_sig", lambda: _Narrow(lib, cap))
        outs.append(ta.yield_and_grad(grids, torch.stack([_field()] * 3), 0.25, (0.2, 5.0), grid_ids=[0, 1, 2],
                                      ckpt_every=8)[1])
    assert torch.isfinite(outs[0]).all()
    assert torch.equal(outs[0][[0, 2]], outs[1][[0, 2]])
    live = outs[0][1] != 0  # samples the zero gate lets through
    assert torch.isnan(outs[1][1][live]).all() and int(live.sum()) > 10
