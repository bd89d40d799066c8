"""The fused Gabor rows (dft.cu windowed_smem): lengths whose last pass has each radix, with and without
Bluestein's convolution, odd and even; one bin, a few, and every bin; rows too long for shared memory
(the separate passes).  Against the oracle: 1e-9 of the largest value, the analysis functions' bound."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 8, 14, 16, 18, 30, 49, 98, 441, 500, 1018, 1025, 1458, 2206, 4410, 4412, 16384])
@pytest.mark.parametrize("bins", ["one", "some", "all"])
def test_gabor_lengths(gpu_lib, N, bins):
    import oracle.analysis as oa
    from mma_gb300 import analysis

    dt = 0.3
    rng = np.random.default_rng(N)
    sig = rng.standard_normal((2, N))
    top = 2 * np.pi * np.fft.fftfreq(N, dt)[: N // 2].max()
    om_max = {"one": 0.0, "some": 0.2 * top, "all": 2 * top + 1.0}[bins]
    tg, om, G = analysis.gabor(torch.tensor(sig, device="cuda"), dt, om_max, 0.0, N * dt, 3, a=5.0)
    assert G.shape == (2, 3, len(om))
    for s in range(2):
        ref = oa.gabor(sig[s], dt, N, len(om), 3, 0.0, N * dt, 5.0)
        assert np.abs(G[s].cpu().numpy() - ref).max() <= 1e-9 * max(np.abs(ref).max(), 1e-300)
