"""The FP64 far field (hankel_plain.cu) where its branches change: the z-first series and the direct
sum, radii and screen points that leave a tile partly filled, arguments beyond the table of Bessel
nodes, distances too different for the series, no / one / two / more planes, both source types, no
near field, a radial pre-factor, strided sources.

Against the oracle (numpy, scipy's j0): 1e-12 of the largest value.  Both sum at most a few hundred
terms whose J0 and arguments are off by 1e-15; arguments of several thousand carry y 2^-53 = 1e-12
each, so the case beyond the table takes 1e-10, the form's stated bound.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
OMEGA0 = 0.057 / 2.4188843265857e-17


def _run(no, nz, nr, nrho, planes, c64=False, near=True, radial=False, pre=True, rho_max=5e-3, z_half=5e-3, tol=1e-12,
         distance=1.0, negative=False):
    import oracle.hankel as oh
    from mma_gb300 import hankel as H

    rng = np.random.default_rng(no * 1000 + nz * 100 + nr)
    om = np.linspace(11, 41, no) * OMEGA0
    r = np.linspace(0.0, 200e-6, nr)
    z = np.linspace(-z_half, z_half, nz) if nz > 1 else np.zeros(1)
    rho = np.linspace(-rho_max if negative else 0.0, rho_max, nrho)
    S = np.exp(-(r / 5e-5) ** 2)[None, None] * (rng.standard_normal((nz, no, 1)) + 1j * rng.standard_normal((nz, no, 1)))
    if c64:
        S = S.astype(np.complex64)
    tab = None
    if pre:
        tab = np.exp(1j * rng.uniform(0, 6, (nz, no, nr) if radial else (nz, no)))
    P = np.stack([oh.hankel_plane(om, r, S[k], distance - z[k], rho, None if tab is None else tab[k], near).T
                  for k in range(nz)])
    ff_ref = np.einsum("k,kjo->jo", oh.trapz_weights(z) if nz > 1 else np.zeros(1), P)
    src = torch.tensor(S, device="cuda")
    ff, pl, _ = H.far_field(om, r, z, rho, src, distance, tab, near, planes=planes, form="plain")
    scale = np.abs(P).max()
    zscale = scale * (z[-1] - z[0]) if nz > 1 else 1.0
    assert np.abs(ff.cpu().numpy() - ff_ref).max() <= tol * zscale
    assert sorted(pl) == sorted(set(p % nz for p in planes))
    for k, v in pl.items():
        assert np.abs(v.cpu().numpy() - P[k]).max() <= tol * scale, k


@pytest.mark.parametrize("no, nz, nr, nrho", [(1, 2, 2, 1), (1, 17, 64, 8), (3, 16, 65, 9), (2, 33, 31, 33), (5, 40, 130, 70),
                                              (40, 20, 33, 128), (1, 300, 96, 7)])
@pytest.mark.parametrize("planes", [(), (0,), (0, -1), (-1,)])
def test_series_and_direct_tiles(gpu_lib, no, nz, nr, nrho, planes):
    _run(no, nz, nr, nrho, planes)


@pytest.mark.parametrize("kw", [dict(c64=True), dict(near=False), dict(radial=True), dict(pre=False), dict(negative=True),
                                dict(planes=(0, 3, 7)), dict(planes=tuple(range(24))), dict(z_half=0.12),
                                dict(z_half=0.4), dict(rho_max=2e-2), dict(rho_max=0.2, tol=1e-10),
                                dict(rho_max=0.2, planes=(0, 1, 2), tol=1e-10)])
def test_options_and_ranges(gpu_lib, kw):
    kw = dict(kw)
    _run(3, 24, 70, 21, kw.pop("planes", (0, -1)), **kw)


def test_single_plane(gpu_lib):
    _run(2, 1, 64, 12, (0,))


def test_workspace_entry_points_agree(gpu_lib):
    """The stream-allocating entry point and the one with the caller's workspace give the same bits;
    too small a workspace is refused."""
    import ctypes

    from mma_gb300 import hankel as H

    lib = H._sig()
    dev = "cuda"
    og = torch.linspace(11, 41, 3, dtype=torch.float64, device=dev) * OMEGA0
    rg = torch.linspace(0, 2e-4, 65, dtype=torch.float64, device=dev)
    zg = torch.linspace(-5e-3, 5e-3, 20, dtype=torch.float64, device=dev)
    rh = torch.linspace(0, 5e-3, 40, dtype=torch.float64, device=dev)
    S = torch.randn(20, 3, 65, dtype=torch.complex128, device=dev)
    p = H.HankelProblem(3, 65, 20, 40, 1.0, 1, 1, 3 * 65, 65, 0)
    a, b = (torch.zeros(40, 3, dtype=torch.complex128, device=dev) for _ in range(2))
    st = torch.cuda.current_stream().cuda_stream
    args = [ctypes.byref(p), og.data_ptr(), rg.data_ptr(), zg.data_ptr(), rh.data_ptr(), S.data_ptr(), None]
    nb = lib.mma_hankel_plain_scratch_bytes(ctypes.byref(p))
    ws = torch.empty(nb, dtype=torch.uint8, device=dev)
    assert lib.mma_hankel_plain(*args, a.data_ptr(), None, 0, None, st) == 0
    assert lib.mma_hankel_plain_ws(*args, b.data_ptr(), None, 0, None, ws.data_ptr(), nb, st) == 0
    assert lib.mma_hankel_plain_ws(*args, b.data_ptr(), None, 0, None, ws.data_ptr(), nb - 1, st) == 1
    torch.cuda.synchronize()
    assert torch.equal(a, b) and float(a.abs().max()) > 0
