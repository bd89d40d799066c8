"""The FP64 far field at the ends of its ranges: distances whose squares leave the range of doubles (the far
zone, up to infinity), where the series has no reference distance; more frequencies than one pass of the
series holds.  Against the oracle, 1e-12 of the largest value as in tests/test_hankel_plain_gpu.py."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
OMEGA0 = 0.057 / 2.4188843265857e-17


@pytest.mark.parametrize("distance", [1e90, 1e120, 1e154, 1e155, 1e200, np.inf])
@pytest.mark.parametrize("planes", [(), (0, -1), (0, 1, 2)])
def test_far_zone(gpu_lib, distance, planes):
    import oracle.hankel as oh
    from mma_gb300 import hankel as H

    rng = np.random.default_rng(5)
    no, nz, nr, nrho = 3, 24, 70, 21
    om, r, z = np.linspace(11, 41, no) * OMEGA0, np.linspace(0.0, 2e-4, nr), np.linspace(-5e-3, 5e-3, nz)
    rho = np.linspace(0.0, 5e-3, nrho)
    S = rng.standard_normal((nz, no, nr)) + 1j * rng.standard_normal((nz, no, nr))
    P = np.stack([oh.hankel_plane(om, r, S[k], distance - z[k], rho, None, True).T for k in range(nz)])
    ref = np.einsum("k,kjo->jo", oh.trapz_weights(z), P)
    ff, pl, _ = H.far_field(om, r, z, rho, torch.tensor(S, device="cuda"), distance, None, True, planes=planes, form="plain")
    scale = np.abs(P).max()
    assert np.isfinite(scale) and np.abs(ff.cpu().numpy() - ref).max() <= 1e-12 * scale * (z[-1] - z[0])
    for k, v in pl.items():
        assert np.abs(v.cpu().numpy() - P[k]).max() <= 1e-12 * scale


@pytest.mark.parametrize("planes", [(), (0, -1)])
def test_frequency_blocks(gpu_lib, planes):
    """More (frequency, radius) pairs than one pass of the series holds (64 MB of contracted sources, 131072
    pairs): the first and last frequencies of both passes."""
    import oracle.hankel as oh
    from mma_gb300 import hankel as H

    no, nz, nr, nrho = 300, 16, 513, 33
    block = (64 << 20) // (nr * 32 * 16)
    assert block < no and no % block
    rng = np.random.default_rng(6)
    om, r, z = np.linspace(11, 41, no) * OMEGA0, np.linspace(0.0, 2e-4, nr), np.linspace(-5e-3, 5e-3, nz)
    rho = np.linspace(0.0, 2e-3, nrho)
    S = torch.tensor(rng.standard_normal((nz, no, nr)) + 1j * rng.standard_normal((nz, no, nr)), device="cuda")
    pre = np.exp(1j * rng.uniform(0, 6, (nz, no)))
    ff, pl, _ = H.far_field(om, r, z, rho, S, 1.0, pre, True, planes=planes, form="plain")
    for o in (0, 1, block - 1, block, block + 1, no - 1):
        P = np.stack([oh.hankel_plane(om[o:o + 1], r, S[k, o:o + 1].cpu().numpy(), 1.0 - z[k], rho, pre[k, o:o + 1],
                                      True).T for k in range(nz)])
        ref, scale = np.einsum("k,kjo->jo", oh.trapz_weights(z), P), np.abs(P).max()
        assert np.abs(ff[:, o:o + 1].cpu().numpy() - ref).max() <= 1e-12 * scale * (z[-1] - z[0]), o
        for k, v in pl.items():
            assert np.abs(v[:, o:o + 1].cpu().numpy() - P[k]).max() <= 1e-12 * scale, (o, k)
