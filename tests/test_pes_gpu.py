"""The photoelectron spectrum's two schemes (a pair of threads per energy, a warp per energy) where
their splits can go wrong: grids of fewer rows than lanes, chunks partly or not filled, a single row
per side, an energy beyond full waves, a partly filled group, the least workspace that the entry point
takes.  Against the oracle: 1e-9 of the largest value, the analysis functions' stated bound."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _psi(num_r, dx, seed=0):
    rng = np.random.default_rng(seed)
    x = np.arange(num_r + 1) * dx - 0.5 * num_r * dx
    return np.exp(-np.abs(x)) + 0.2 * (rng.standard_normal(x.size) + 1j * rng.standard_normal(x.size)) * np.exp(-(x / 20) ** 2)


@pytest.mark.parametrize("num_r, num_E", [(1, 3), (2, 5), (3, 40), (30, 7), (31, 33), (32, 1), (63, 64), (64, 65),
                                          (100, 6000), (97, 5837), (40, 9728), (41, 9729), (33, 16000), (800, 100)])
def test_pes_sizes(gpu_lib, num_r, num_E):
    import oracle.analysis as oa
    from mma_gb300 import analysis

    psi = _psi(num_r, 0.3)
    kw = dict(E_start=-0.5, num_E=num_E, epsilon=4e-3, Estep=2e-4)
    _, P = analysis.pes(torch.tensor(psi, device="cuda"), num_r, 0.3, 1.1, **kw)
    ref = oa.pes(psi, num_r, 0.3, 1.1, num_E, 4e-3, 2e-4, -0.5)
    assert np.abs(P.cpu().numpy() - ref).max() <= 1e-9 * np.abs(ref).max()


def test_pes_workspaces(gpu_lib):
    """Any accepted workspace gives the same spectrum: the least one (the call then takes its own), one
    for a few energies and one for all."""
    from mma_gb300 import analysis

    lib = analysis._sig()
    num_r, num_E, n = 200, 9800, 201
    psi = torch.tensor(_psi(num_r, 0.3), device="cuda")
    fixed = (8 * (n + 1) + 255) // 256 * 256 + (16 * n + 255) // 256 * 256
    st = torch.cuda.current_stream().cuda_stream
    outs = []
    for nb in (fixed + 32 * n, fixed + 32 * n * 700, int(lib.mma_tdse_pes_scratch_bytes(num_r, num_E))):
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        out = torch.full((num_E,), float("nan"), dtype=torch.float64, device="cuda")
        assert lib.mma_tdse_pes(psi.data_ptr(), num_r, 0.3, 1.1, num_E, 4e-3, 2e-4, -0.5, out.data_ptr(), ws.data_ptr(),
                                nb, st) == 0
        torch.cuda.synchronize()
        outs.append(out)
    for o in outs[:2]:
        assert float((o - outs[2]).abs().max()) <= 1e-9 * float(outs[2].abs().max())
    assert lib.mma_tdse_pes(psi.data_ptr(), num_r, 0.3, 1.1, num_E, 4e-3, 2e-4, -0.5, out.data_ptr(), ws.data_ptr(),
                            fixed + 32 * n - 1, st) == 1
