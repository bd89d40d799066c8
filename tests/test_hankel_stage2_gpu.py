"""Stage 2 of the fast far field at the edges of its tiles of radii and blocks of observation points.

The fast form (float32) is held against the plain form (float64) at the fast form's stated bound, a
per-harmonic relative L2 error of 2e-5, for the far field and the planes (as in test_hankel_gpu.py).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAST_TOL = 2e-5


def per_harmonic(a, b):
    return float(np.max(np.linalg.norm(a - b, axis=0) / np.linalg.norm(b, axis=0)))


def _case(n_z, n_omega, n_r, n_rho, seed):
    rng = np.random.default_rng(seed)
    w0 = 2.0 * np.pi * 299792458.0 / 800e-9
    og = w0 * np.linspace(10.0, 42.0, n_omega)
    rg = np.linspace(0.0, 200e-6, n_r)
    zg = np.linspace(-5e-3, 5e-3, n_z)
    rho = np.linspace(0.0, 5e-3, n_rho)
    smooth = np.exp(-((rg / 90e-6) ** 2))[None, None, :]
    S = smooth * (1.0 + 0.3 * rng.standard_normal((n_z, n_omega, n_r)) + 0.3j * rng.standard_normal((n_z, n_omega, n_r)))
    return zg, rg, og, rho, S.astype(np.complex64)


@pytest.mark.parametrize("n_r,n_rho", [(486, 40), (510, 33), (511, 257), (512, 129), (258, 128), (33, 1)])
def test_tiles_of_radii(gpu_lib, n_r, n_rho):
    """Radii that fill one tile, that halve to an odd count, that are odd; blocks of rho that end early."""
    import torch
    from mma_gb300 import hankel as H

    zg, rg, og, rho, S = _case(12, 5, n_r, n_rho, seed=n_r)
    S = torch.tensor(S, device="cuda")
    last = len(zg) - 1
    plain, p_pl, _ = H.far_field(og, rg, zg, rho, S, 1.0, None, True, planes=(0, -1), form="plain")
    fast, f_pl, plan = H.far_field(og, rg, zg, rho, S, 1.0, None, True, planes=(0, -1), form="fast",
                                   planes_via="direct")
    assert plan["planes_via"] == "series"
    assert per_harmonic(fast.cpu().numpy(), plain.cpu().numpy()) < FAST_TOL
    for k in (0, last):
        assert per_harmonic(f_pl[k].cpu().numpy(), p_pl[k].cpu().numpy()) < FAST_TOL
