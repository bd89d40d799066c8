"""The propagation that spreads an instance over a thread-block cluster (tdse_cluster.cu) and the
parallel factorisation of the grids' tables, at the sizes where the split can go wrong: fewer sites
than threads, chunks of one site, sites just below, at and above a multiple of the threads, a solve
that decays slowly from site to site (carries that reach over many warps), odd cluster sizes, more
instances than resident clusters.

Against the oracle: relative L2 <= 1e-8, the framework's parity bound.  Against the one-CTA kernels,
which a batch limited to one CTA still takes: the same recurrences in another order of additions, so
FP64 within 1e-10 (4e3 steps of 1e-14) and float-float within 1e-9 (its stated distance from FP64).
"""
import numpy as np
import pytest
import torch

from tests.tdse_cases import A_CONFIG, rel_l2, sin2_pulse

pytestmark = pytest.mark.gpu
SERIES = ("sourceterm", "PopTot", "PopInt", "expval")


def _field(n, seed=0):
    t = 0.25 * np.arange(1, n + 1)
    T = t[-1] + 0.25
    rng = np.random.default_rng(seed)
    return t, 0.06 * np.sin(np.pi * t / T) ** 2 * np.cos(0.3 * t + rng.uniform(0, 1))


@pytest.mark.parametrize("num_r, dx", [(4, 0.4), (126, 0.3), (127, 0.3), (128, 0.3), (255, 0.2), (2046, 0.2),
                                       (2047, 0.2), (2048, 0.2), (4097, 0.1), (1500, 0.02)])
@pytest.mark.parametrize("precision", ["fp64", "df64"])
def test_cluster_matches_oracle_at_chunk_edges(gpu_lib, oracle_built, num_r, dx, precision):
    import oracle.tdse as ot
    from mma_gb300.tdse_batch import TDSEGrids, run_batch

    t, E = _field(61)  # an odd number of steps: 61 + 2, not a multiple of the 8-step sums
    p = dict(num_r=num_r, dx=dx, trg_a=A_CONFIG)
    grids = TDSEGrids([p], dt=0.25, df64=precision == "df64")
    res = run_batch(grids, torch.tensor(E[None], device="cuda"), 0.25, precision=precision, psi_final=True)
    torch.cuda.synchronize()
    x, psi0, e, _ = ot.ground_state(num_r, dx, A_CONFIG, -1.0, 1e-15)
    # the oracle on the GPU's own ground state: on tiny grids the two inverse iterations stop 1e-11 apart
    o = ot.propagate(x, grids.psi0(0).cpu().numpy(), t, E, dx, A_CONFIG)
    for k in SERIES:
        assert rel_l2(res[k][0].cpu().numpy(), o[k]) < 1e-8, k
    psi = res["psi_final"].cpu().numpy()
    assert rel_l2(psi[0::2] + 1j * psi[1::2], o["psi"]) < 1e-8
    assert rel_l2(res["Fsourceterm"][0].cpu().numpy(), o["Fsourceterm"]) < 1e-8


@pytest.mark.parametrize("precision, tol", [("fp64", 1e-10), ("df64", 1e-9)])
@pytest.mark.parametrize("num_r, n_inst", [(601, 2), (1203, 5), (6000, 2), (10000, 2), (12500, 3), (8000, 9), (8000, 41),
                                            (30000, 2)])
def test_cluster_matches_one_cta_kernel(gpu_lib, precision, tol, num_r, n_inst):
    from mma_gb300.tdse_batch import TDSEGrids, run_batch

    t, E = _field(100)
    fields = torch.tensor(np.stack([(0.4 + 0.1 * i) * E for i in range(n_inst)]), device="cuda")
    grids = TDSEGrids([dict(num_r=num_r, dx=0.1, trg_a=A_CONFIG)], dt=0.25, df64=precision == "df64")
    got, ref = (run_batch(grids, fields, 0.25, precision=precision, psi_final=True, snap_every=30, grid_ctas=c)
                for c in (0, 1))
    torch.cuda.synchronize()
    for k in SERIES:
        assert rel_l2(got[k].cpu().numpy(), ref[k].cpu().numpy()) < tol, k
    assert torch.equal(got["tgrid"], ref["tgrid"]) and torch.equal(got["Efield"], ref["Efield"])
    for k in ("psi_final", "snapshots"):
        assert rel_l2(got[k].cpu().numpy(), ref[k].cpu().numpy()) < tol, k


def test_cluster_complex_start_state(gpu_lib, oracle_built):
    """The legacy call accepts any psi0: a complex one takes the projection's imaginary part too."""
    import ctypes

    import oracle.tdse as ot
    from mma_gb300.structures import inputs_def, outputs_def
    from mma_gb300.tdse import TDSE_DLL, init_time_and_field

    dll, num_r, dx = TDSE_DLL(), 700, 0.3
    t, E = sin2_pulse(1.0, skip_first=True)
    inp, out = inputs_def(), outputs_def()
    inp.init_default_inputs(num_r=num_r, dx=dx, dt=0.25, trg_a=A_CONFIG, CV=1e-15)
    init_time_and_field(dll, inp, t, E)
    dll.init_GS(inp)
    x, psi = inp.get_xgrid(), inp.get_GS()
    psi = psi * np.exp(0.3j * x) * (0.8 + 0.6j)
    ctypes.memmove(inp.psi0, np.ascontiguousarray(psi).ctypes.data, psi.nbytes)
    dll.call1DTDSE(inp, out)
    o = ot.propagate(x, psi, t, E, dx, A_CONFIG)
    for k, v in (("sourceterm", out.get_sourceterm()), ("PopTot", out.get_PopTot()), ("PopInt", out.get_PopInt()),
                 ("expval", out.get_expval())):
        assert rel_l2(v, o[k]) < 1e-8, k
    dll.free_outputs(out.ptr)
    dll.free_inputs(inp.ptr)


def test_cluster_uneven_batch_with_too_wide_grid(gpu_lib):
    """Grids of several widths in one launch; an instance wider than the launch was sized for gives
    NaN outputs and the others their results."""
    from mma_gb300.tdse_batch import TDSEBatchPlan, TDSEGrids

    t, E = _field(80)
    params = [dict(num_r=n, dx=0.2, trg_a=A_CONFIG) for n in (500, 1300, 2600)]
    grids = TDSEGrids(params, dt=0.25)
    fields = [torch.tensor(E, device="cuda")] * 3
    outs = []
    for cap in (None, int(grids.m[1])):
        plan = TDSEBatchPlan(grids, [len(E)] * 3, 0.25, grid_ids=[0, 1, 2])
        if cap:
            plan.launches[0]["max_m"] = cap
        plan.load_fields(fields)
        plan.launch()
        torch.cuda.synchronize()
        outs.append(plan.result())
    for i in (0, 1):  # the launch sized for narrower grids splits them otherwise: another order of additions
        for k in SERIES:
            assert rel_l2(outs[1].series(i)[k].cpu().numpy(), outs[0].series(i)[k].cpu().numpy()) < 1e-10
    assert torch.isnan(outs[1].series(2)["sourceterm"]).all()


class _OneCta:
    """The library with a default of one CTA: batches of two then keep the one-CTA kernels."""

    def __init__(self, lib):
        self._lib = lib

    def __getattr__(self, name):
        return (lambda *a: 1) if name == "mma_tdse_default_ctas" else getattr(self._lib, name)


@pytest.mark.parametrize("num_r, dx, K", [(4, 0.4, 8), (127, 0.3, 7), (128, 0.3, 1), (640, 0.2, 64), (2047, 0.2, 9),
                                          (8000, 0.1, 32), (1500, 0.02, 16), (3000, 0.1, 20), (6000, 0.1, 16),
                                          (10000, 0.1, 16), (13000, 0.1, 16)])
def test_adjoint_cluster_matches_one_cta_kernel(gpu_lib, monkeypatch, num_r, dx, K):
    """The cluster form of the adjoint sweep (segments that end inside a batch of phases or of collected
    sums, chunks of one site, threads without sites): 1e-10, as for the propagation."""
    import mma_gb300.tdse_adjoint as ta
    from mma_gb300.tdse_batch import TDSEGrids

    t, E = _field(75)
    fields = torch.tensor(np.stack([E, 0.7 * E[::-1].copy()]), device="cuda")
    grids = TDSEGrids([dict(num_r=num_r, dx=dx, trg_a=A_CONFIG)], dt=0.25, adjoint=True)
    band = (0.2, 1.5)
    L, g = ta.yield_and_grad(grids, fields, 0.25, band, ckpt_every=K)
    lib = ta._adj_sig()
    monkeypatch.setattr(ta, "_adj_sig", lambda: _OneCta(lib))
    L1, g1 = ta.yield_and_grad(grids, fields, 0.25, band, ckpt_every=K)
    torch.cuda.synchronize()
    assert rel_l2(L.cpu().numpy(), L1.cpu().numpy()) < 1e-10
    for i in range(2):
        assert rel_l2(g[i].cpu().numpy(), g1[i].cpu().numpy()) < 1e-10, i


@pytest.mark.parametrize("num_r, dx", [(2, 0.4), (40, 0.4), (127, 0.3), (128, 0.3), (513, 0.3), (2048, 0.2), (8000, 0.1),
                                       (12001, 0.1), (33000, 0.05), (6000, 0.1), (4100, 0.1), (10000, 0.1), (14000, 0.1)])
def test_ground_state_cluster(gpu_lib, oracle_built, num_r, dx):
    """One grid (a cluster) against the oracle and against the same grid among 40 (a CTA per grid).  The
    iterations stop on |dE| <= 1e-15: on small grids two orders of summation leave the energies 1e-11
    apart (tests/test_edges_gpu.py), and one iteration more or less changes psi0 by 1e-11."""
    import oracle.tdse as ot
    from mma_gb300.tdse_batch import TDSEGrids

    p = dict(num_r=num_r, dx=dx, trg_a=A_CONFIG)
    one = TDSEGrids([p], dt=0.25)
    x, psi0, e, _ = ot.ground_state(num_r, dx, A_CONFIG, -1.0, 1e-15)
    assert abs(one.Einit[0] - e) < 1e-10 * abs(e)
    assert rel_l2(one.psi0(0).cpu().numpy(), psi0) < 1e-9
    assert np.array_equal(one.x(0).cpu().numpy(), x)
    if num_r <= 2048:
        many = TDSEGrids([p] * 40, dt=0.25)
        assert abs(one.Einit[0] - many.Einit[17]) < 1e-10 * abs(e)
        assert rel_l2(one.psi0(0).cpu().numpy(), many.psi0(17).cpu().numpy()) < 1e-9


def test_ground_state_cluster_iteration_cap(gpu_lib):
    from mma_gb300.tdse_batch import MMAStatusError, TDSEGrids

    with pytest.raises(MMAStatusError, match="not converged"):
        TDSEGrids([dict(num_r=600, dx=0.4, trg_a=A_CONFIG, max_iter=3)], dt=0.25)


@pytest.mark.parametrize("num_r,dx", [(255, 0.4), (256, 0.4), (777, 0.2), (1023, 0.1), (2400, 0.2), (8000, 0.1)])
def test_few_grids_and_many_give_the_same_bits(gpu_lib, num_r, dx):
    """One grid (a cluster per grid) against the same grid among as many as a CTA each serves: ground
    state, energy, iterations and tables are the same bits, since both run the same operations."""
    import torch
    from mma_gb300.tdse_batch import TDSEGrids

    p = dict(num_r=num_r, dx=dx, trg_a=A_CONFIG)
    one = TDSEGrids([p], dt=0.25)
    many = TDSEGrids([p] * (torch.cuda.get_device_properties(0).multi_processor_count // 4 + 1), dt=0.25)
    for name in ("x", "psi0", "cn_tab", "gs_tab", "result"):
        (o, cnt), (q, _) = one.views[0][name], many.views[-1][name]
        assert torch.equal(one.buf[o:o + cnt].view(torch.int64), many.buf[q:q + cnt].view(torch.int64)), name
