"""Which of the photoelectron spectrum's two schemes a call takes (tdse_analysis.cu, pes_by_pairs): on grids
of few rows the pairs serve any number of energies from some hundred on, since a warp per energy pays for
its lanes' reductions."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _psi(num_r, dx):
    x = np.arange(num_r + 1) * dx - 0.5 * num_r * dx
    return np.exp(-np.abs(x)) * (1 + 0.3j * np.cos(x))


@pytest.mark.parametrize("num_r, num_E", [(3, 1), (3, 200), (3, 3000), (4, 9800), (5, 40), (30, 500), (31, 12000), (50, 1100),
                                          (50, 3000), (50, 12000), (200, 6500), (601, 300)])
def test_route_boundaries_match_oracle(gpu_lib, num_r, num_E):
    """1e-9 of the largest value, the analysis functions' stated bound."""
    import oracle.analysis as oa
    from mma_gb300 import analysis

    psi = _psi(num_r, 0.3)
    _, P = analysis.pes(torch.tensor(psi, device="cuda"), num_r, 0.3, 1.1, E_start=-0.5, num_E=num_E, epsilon=4e-3,
                        Estep=2e-4)
    ref = oa.pes(psi, num_r, 0.3, 1.1, num_E, 4e-3, 2e-4, -0.5)
    assert np.abs(P.cpu().numpy() - ref).max() <= 1e-9 * np.abs(ref).max()


@pytest.mark.parametrize("num_r", [3, 50])
def test_fewer_energies_take_no_longer(gpu_lib, num_r):
    """3000 energies against a full wave of 9728: the same chain on fewer threads.  A fifth for the clock;
    by a warp per energy it is 1.8 times the wave's time (50 rows) and 3 (3 rows)."""
    from mma_gb300 import analysis

    psi = torch.tensor(_psi(num_r, 0.3), device="cuda")

    def ms(num_E):
        best = 1e9
        for _ in range(30):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            analysis.pes(psi, num_r, 0.3, 1.1, num_E=num_E)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    wave = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    ms(wave)
    assert ms(3000) <= 1.2 * ms(wave)
