"""The cumulative results' kernel and the device evaluation of a uniform medium's pre-factor: sizes that
leave a block of loads or a CTA partly filled, either output alone, planes in separate allocations.

The running sums against torch's in FP64: the same additions in the same order up to one rounding each,
1e-13 of the largest value.  The tables against pre_factor_table: exponents of up to a few hundred
radians carry 1e-16 of themselves, 1e-12."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz, nrho, no", [(2, 1, 1), (3, 5, 7), (9, 16, 16), (10, 3, 257), (40, 33, 65), (1026, 4, 4)])
@pytest.mark.parametrize("norm, run, apart", [(True, False, False), (False, True, False), (True, True, True)])
def test_cumulative(gpu_lib, nz, nrho, no, norm, run, apart):
    from mma_gb300 import hankel as H

    g = torch.Generator(device="cuda").manual_seed(nz)
    P = torch.randn(nz, nrho, no, dtype=torch.complex128, device="cuda", generator=g)
    z = np.sort(np.random.default_rng(nz).uniform(-1, 1, nz))
    rn = torch.rand(nz, no, dtype=torch.float64, device="cuda", generator=g) if norm else None
    planes = [P[k].clone() for k in range(nz)] if apart else [P[k] for k in range(nz)]
    a, b = H._cumulative(z, planes, rn, run)
    dz = torch.tensor(np.diff(z), device="cuda")
    ref = torch.cumsum(0.5 * dz[:, None, None] * (P[:-1] + P[1:]), dim=0)
    assert (a is not None) == norm and (b is not None) == run
    if run:
        assert float((b - ref).abs().max()) <= 1e-13 * float(ref.abs().max())
    if norm:
        ref = rn[:nz - 1, None, :] * ref
        assert float((a - ref).abs().max()) <= 1e-13 * float(ref.abs().max())


@pytest.mark.parametrize("kw", [dict(), dict(include_absorption=False), dict(include_dispersion=False),
                                dict(pressure=0.37), dict(effective_IR_refrective_index=1.0003)])
def test_uniform_tables(gpu_lib, kw):
    from mma_gb300 import hankel as H

    H.XUV_index.set_constant_index(complex(1 - 1e-5, 1e-7))
    z = np.linspace(-4e-3, 5e-3, 19)
    w = np.linspace(11, 41, 37) * 0.057 / 2.4188843265857e-17
    ref, rn_ref = H.pre_factor_table(z, w, "Ar", **kw)
    kw = dict(kw)
    pre, rn = H._uniform_tables_on_device(
        z, w, "cuda", kw.pop("pressure", 1.0), True, gas="Ar", absorption_tables="Henke", dispersion_tables="Henke",
        n_ir=kw.pop("effective_IR_refrective_index", 1.0), include_absorption=kw.get("include_absorption", True),
        include_dispersion=kw.get("include_dispersion", True))
    assert np.abs(pre.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.abs(rn.cpu().numpy() - rn_ref).max() <= 1e-12 * np.abs(rn_ref).max()
    assert H._uniform_tables_on_device(z, w, "cuda", 1.0, True, gas="Ar", absorption_tables="Henke",
                                       dispersion_tables="Henke", n_ir=1.0 + 1e-6j, include_absorption=True,
                                       include_dispersion=True) is None
