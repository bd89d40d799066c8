"""The one-CTA float-float kernel's chunk frames (tdse_df64.cu): grids with one and with many sites per
thread (the phase table in one and in two levels), blocks of steps that end before, at and after the
pulse, snapshots and final states (turned back from the frames), a complex start state.  Batches limited
to one CTA take this kernel.  Against the FP64 one-CTA kernel: 1e-9, the form's stated distance."""
import ctypes

import numpy as np
import pytest
import torch

from tests.tdse_cases import A_CONFIG, rel_l2

pytestmark = pytest.mark.gpu
SERIES = ("sourceterm", "PopTot", "PopInt", "expval")


def _fields(n, k):
    t = 0.25 * np.arange(1, n + 1)
    env = np.sin(np.pi * t / (t[-1] + 0.25)) ** 2
    return torch.tensor(np.stack([(0.08 - 0.03 * j) * env * np.cos((0.3 + 0.2 * j) * t + j) for j in range(k)]), device="cuda")


@pytest.mark.parametrize("num_r, dx, n_f", [(5, 0.4, 70), (255, 0.3, 66), (256, 0.3, 67), (300, 0.3, 190), (8000, 0.1, 50),
                                            (131071, 0.01, 12), (131072, 0.01, 12), (150000, 0.01, 25)])
def test_frames_match_fp64(gpu_lib, num_r, dx, n_f):
    from mma_gb300.tdse_batch import TDSEGrids, run_batch

    fields = _fields(n_f, 2)
    grids = TDSEGrids([dict(num_r=num_r, dx=dx, trg_a=A_CONFIG, CV=1e-13)], dt=0.25, df64=True)
    got, ref = (run_batch(grids, fields, 0.25, precision=p, psi_final=True, snap_every=7, grid_ctas=1)
                for p in ("df64", "fp64"))
    torch.cuda.synchronize()
    for k in SERIES:
        assert rel_l2(got[k].cpu().numpy(), ref[k].cpu().numpy()) < 1e-9, k
    assert torch.equal(got["tgrid"], ref["tgrid"]) and torch.equal(got["Efield"], ref["Efield"])
    for k in ("psi_final", "snapshots"):
        assert rel_l2(got[k].cpu().numpy(), ref[k].cpu().numpy()) < 1e-9, k


def test_frames_complex_start_state(gpu_lib):
    """psi0 turned and boosted in the grid's tables: the projection takes both parts of psi0."""
    from mma_gb300.tdse_batch import GridRec, TDSEGrids, _sig, _stream_ptr, run_batch

    fields = _fields(90, 2)
    grids = TDSEGrids([dict(num_r=700, dx=0.3, trg_a=A_CONFIG)], dt=0.25, df64=True)
    p = grids.psi0(0)
    p *= torch.exp(0.4j * grids.x(0)) * (0.6 - 0.8j)
    lib = _sig()
    assert lib.mma_tdse_build_grids(ctypes.c_void_p(grids.dev_recs.data_ptr()), ctypes.addressof(grids.host_recs), 1, 1,
                                    _stream_ptr()) == 0
    assert lib.mma_tdse_build_df_tables(ctypes.c_void_p(grids.dev_recs.data_ptr()), ctypes.addressof(grids.host_recs), 1,
                                        _stream_ptr()) == 0
    got, ref = (run_batch(grids, fields, 0.25, precision=q, psi_final=True, grid_ctas=1) for q in ("df64", "fp64"))
    torch.cuda.synchronize()
    for k in SERIES:
        assert rel_l2(got[k].cpu().numpy(), ref[k].cpu().numpy()) < 1e-9, k
    assert rel_l2(got["psi_final"].cpu().numpy(), ref["psi_final"].cpu().numpy()) < 1e-9
