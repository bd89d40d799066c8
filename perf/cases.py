"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case goes through a public entry point:

* ``call``      one TDSE through the reference's own call sequence (``run_single``: grid and ground
                state, propagation, spectra, host arrays out);
* ``batch``     a macroscopic (r, z) map of TDSE instances through ``TDSEBatchPlan`` (FP64,
                float-float or complex64), fields in, every series and spectrum out;
* ``adjoint``   the gradient of a harmonic yield with respect to every field sample;
* ``long``      ``Hankel_long`` as the far-field driver calls it (the default, FP64 form), or with
                ``fast`` and the cumulative results (every plane transformed);
* ``far_field`` the fast far field with the entry and exit planes on a device source;
* ``pes``, ``gabor``  the analysis functions.

``listed`` spans one short pulse on a small grid to the benchmark maps; ``draw`` gives more of the
same kinds.  ``exact`` restates each path in 64 bits with torch alone (dense or banded operators,
direct Bessel sums, torch.fft).
"""
import math

import numpy as np
import torch

from mma_gb300 import analysis
from mma_gb300 import hankel as H
from mma_gb300.tdse import TDSE_DLL, run_single
from mma_gb300.tdse_adjoint import yield_and_grad
from mma_gb300.tdse_batch import TDSEBatchPlan, TDSEGrids

OMEGA0 = 0.057  # 800 nm in atomic units
OMEGA0_SI = OMEGA0 / 2.4188843265857e-17
A_CONFIG = math.sqrt(1.68)
C_LIGHT = 299792458.0
DT = 0.25
BAND = (21 * OMEGA0, 31 * OMEGA0)


def listed():
    return [
        # one short pulse on a small grid: the quick look, where launches and set-up count
        dict(name="call_small", kind="call", num_r=600, dx=0.4, cycles=2.0, dt_field=DT),
        # the benchmark's single instance: 8001 sites, 10 cycles, the call of the reference's notebooks
        dict(name="call_config0", kind="call", num_r=8000, dx=0.1, cycles=10.0, dt_field=DT),
        # a macroscopic map in the plain FP64 form: 16 r x 16 z points on a 4001-site grid
        dict(name="batch_fp64_map", kind="batch", precision="fp64", n_r=16, n_z=16, num_r=4000, dx=0.2, cycles=4.0),
        # an intensity scan: a few instances of the benchmark grid in the float-float form
        dict(name="batch_df64_scan", kind="batch", precision="df64", n_r=24, n_z=1, num_r=8000, dx=0.1, cycles=10.0),
        # the benchmark map (64 r x 32 z, 8001 sites) in its headline form, few-cycle pulses
        dict(name="batch_df64_map", kind="batch", precision="df64", n_r=64, n_z=32, num_r=8000, dx=0.1, cycles=4.0),
        # the uneven complex64 batch: own grid (half-width 200..600 a.u.), length and intensity per instance
        dict(name="batch_c64_uneven", kind="uneven", precision="c64", n_inst=1024, dx=0.1, lo=200.0, hi=600.0,
             c_lo=6, c_hi=12),
        # pulse shaping: gradient of the H21-H31 yield for 64 points of the benchmark grid, 3 cycles
        dict(name="adjoint_64", kind="adjoint", n_inst=64, num_r=8000, dx=0.1, cycles=3.0, ckpt=256),
        # the far-field driver's default call: FP64, entry and exit planes, complex128 source
        dict(name="long_plain", kind="long", form="plain", n_omega=64, n_z=65, n_r=512, n_rho=128, cumulative=False),
        # the cumulative results (every plane) of a quarter of the benchmark's frequencies, fast form
        dict(name="long_cumulative", kind="long", form="fast", n_omega=512, n_z=256, n_r=512, n_rho=256,
             cumulative=True),
        # the benchmark far field: 2048 omega x 255 planes x 512 r -> 256 rho, entry and exit planes
        dict(name="far_field_config3", kind="far_field", n_omega=2048, n_z=255, n_r=512, n_rho=256),
        # photoelectron spectrum of one wavefunction on the reference's default energy grid
        dict(name="pes_default", kind="pes", num_r=8000, dx=0.1, num_E=10000, Estep=5e-4),
        # Gabor maps of a batch of dipole signals
        dict(name="gabor_512", kind="gabor", n_sig=512, cycles=10.0, n_windows=100, omega_max=2.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "fp64", "df64", "uneven", "adjoint", "long", "cumulative", "far_field", "pes", "gabor"])
    if kind == "call":
        return dict(kind="call", num_r=_log(rng, 300, 8000), dx=rng.choice([0.1, 0.2, 0.4]),
                    cycles=round(rng.uniform(1.0, 10.0), 2), dt_field=rng.choice([DT, DT, 2 * DT]))
    if kind in ("fp64", "df64"):
        num_r, cycles = _log(rng, 500, 12000), round(rng.uniform(1.0, 6.0), 2)
        work = 2.0e9 if kind == "fp64" else 1.2e10  # site-steps
        most = int(work / (num_r * cycles * 441.0))
        n = min(_log(rng, 1, 2048), max(1, most))
        n_r = max(1, int(math.sqrt(n * rng.uniform(1.0, 4.0))))
        return dict(kind="batch", precision=kind, n_r=n_r, n_z=max(1, n // n_r), num_r=num_r,
                    dx=rng.choice([0.1, 0.2]), cycles=cycles)
    if kind == "uneven":
        return dict(kind="uneven", precision=rng.choice(["c64", "df64", "fp64"]), n_inst=_log(rng, 3, 96), dx=0.1,
                    lo=round(rng.uniform(60.0, 200.0), 1), hi=round(rng.uniform(210.0, 600.0), 1), c_lo=2,
                    c_hi=rng.randint(3, 8))
    if kind == "adjoint":
        num_r, cycles = _log(rng, 300, 8000), round(rng.uniform(1.0, 4.0), 2)
        n = min(_log(rng, 1, 256), max(1, int(4.0e8 / (num_r * cycles * 441.0))))
        return dict(kind="adjoint", n_inst=n, num_r=num_r, dx=rng.choice([0.1, 0.2]), cycles=cycles,
                    ckpt=rng.choice([64, 100, 256]))
    if kind == "long":
        n_z, n_r, n_rho = _log(rng, 3, 200), _log(rng, 33, 700), _log(rng, 16, 256)
        n_omega = min(_log(rng, 4, 512), max(1, int(5.0e8 / (n_z * n_r * n_rho))))
        return dict(kind="long", form="plain", n_omega=n_omega, n_z=n_z, n_r=n_r, n_rho=n_rho,
                    cumulative=rng.random() < 0.25)
    if kind == "cumulative":
        return dict(kind="long", form="fast", n_omega=_log(rng, 16, 400), n_z=_log(rng, 20, 250),
                    n_r=_log(rng, 64, 512), n_rho=_log(rng, 16, 256), cumulative=True)
    if kind == "far_field":
        return dict(kind="far_field", n_omega=_log(rng, 16, 2048), n_z=_log(rng, 8, 255), n_r=_log(rng, 64, 512),
                    n_rho=_log(rng, 16, 256))
    if kind == "pes":
        return dict(kind="pes", num_r=_log(rng, 400, 8000), dx=rng.choice([0.1, 0.2, 0.4]), num_E=_log(rng, 50, 10000),
                    Estep=rng.choice([5e-4, 2e-3]))
    return dict(kind="gabor", n_sig=_log(rng, 1, 512), cycles=round(rng.uniform(1.0, 10.0), 2),
                n_windows=rng.randint(10, 100), omega_max=rng.choice([1.0, 2.0, 3.0]))


# ------------------------------------------------------------------------------- inputs
def _pulse_grid(cycles, dt=DT, exact_dt=False):
    T = cycles * 2 * np.pi / OMEGA0
    n = int(T / dt) + 1
    n += n % 2
    return T, (dt * np.arange(n) if exact_dt else np.linspace(0.0, T, n))


def _envelope(t, T):
    return np.sin(np.pi * np.clip(t / T, 0.0, 1.0)) ** 2


def _call_inputs(c, seed):
    """One pulse, sampled from one step after t = 0 on (the field is then not exactly 0 there)."""
    rng = np.random.default_rng(seed)
    T, t = _pulse_grid(c["cycles"], c["dt_field"], exact_dt=c["dt_field"] != DT)
    t = np.append(t, 2 * t[-1] - t[-2])[1:]  # an even count without the t = 0 sample
    E0 = float(np.exp(rng.uniform(np.log(0.04), np.log(0.08))))
    cep = float(rng.uniform(-0.5, 0.5))
    return t, E0 * _envelope(t, T) * np.cos(OMEGA0 * t + cep)


def _map_fields(n_r, n_z, cycles, seed):
    """Fields of a Gaussian focus (w0 = 100 um, z in [-5, 5] mm), instance n = kr + kz n_r."""
    rng = np.random.default_rng(seed)
    T, t = _pulse_grid(cycles)
    w0, lam = 100e-6, 800e-9
    r = np.linspace(0.0, 2 * w0, n_r)
    z = np.linspace(-5e-3, 5e-3, n_z) if n_z > 1 else np.zeros(1)
    zR, k0 = np.pi * w0 ** 2 / lam, 2 * np.pi / lam
    zz, rr = np.meshgrid(z, r, indexing="ij")
    w = w0 * np.sqrt(1 + (zz / zR) ** 2)
    amp = rng.uniform(0.045, 0.06) * (w0 / w) * np.exp(-(rr / w) ** 2)
    ph = -0.5 * k0 * rr ** 2 * zz / (zR ** 2 + zz ** 2) + np.arctan(zz / zR) + rng.uniform(-0.5, 0.5)
    f = amp.reshape(-1, 1) * _envelope(t, T)[None, :] * np.cos(OMEGA0 * t[None, :] + ph.reshape(-1, 1))
    return t, f


def _uneven_inputs(c, seed):
    rng = np.random.default_rng(0)  # the grids and lengths are the case's own
    n = c["n_inst"]
    half = rng.uniform(c["lo"], c["hi"], n)
    half[:2] = c["lo"], c["hi"]
    cyc = rng.integers(c["c_lo"], c["c_hi"] + 1, n)
    rng = np.random.default_rng(seed)
    E0 = np.exp(rng.uniform(np.log(0.02), np.log(0.075), n))
    cep = rng.uniform(0.0, 2 * np.pi, n)
    params = [dict(num_r=int(round(2 * h / c["dx"])), dx=c["dx"], trg_a=A_CONFIG) for h in half]
    fields = []
    for i in range(n):
        T = cyc[i] * 2 * np.pi / OMEGA0
        m = int(T / DT)
        m += m % 2
        t = DT * np.arange(1, m + 1)
        fields.append(torch.tensor(E0[i] * _envelope(t, T) * np.cos(OMEGA0 * t + cep[i]), device="cuda"))
    return params, fields


def _source(c, n_z, seed, dtype):
    """|S| ~ exp(-r^2/(50 um)^2) times a comb of odd harmonics with random phases per plane."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = np.linspace(0.0, 200e-6, c["n_r"])
    z = np.linspace(-5e-3, 5e-3, c["n_z"])
    om = np.linspace(10 * OMEGA0_SI, 42 * OMEGA0_SI, c["n_omega"])
    rho = np.linspace(0.0, 5e-3, c["n_rho"])
    q = torch.arange(11, 42, 2, device="cuda", dtype=torch.float64)
    ph = 2 * math.pi * torch.rand(n_z, len(q), generator=g, device="cuda", dtype=torch.float64)
    o = torch.tensor(om / OMEGA0_SI, device="cuda")
    comb = torch.polar(torch.ones_like(ph), ph) @ (1.0 / (1.0 + ((o[None] - q[:, None]) / 0.3) ** 2)).to(torch.complex128)
    prof = torch.exp(-(torch.tensor(r, device="cuda") / 50e-6) ** 2)
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    return z, r, om, rho, comb.to(dtype)[:, :, None] * prof.to(real)[None, None, :]


def _medium(z, om):
    """Pre-factors [Nz, No] of a uniform medium with index 1 - 1e-5 + 1e-7i, and their renormalisation."""
    disp, ab = 1j * (1.0 - (1 - 1e-5)) / C_LIGHT, 1e-7 / C_LIGHT
    pre = np.exp(om[None, :] * (z[:, None] * disp + (z[:, None] - z[-1]) * ab))
    return pre, np.exp((z[-1] - z[:, None]) * (om * ab)[None, :])


def _psi(c, seed):
    """A bound core with an outgoing wave packet and some noise, and its grid."""
    rng = np.random.default_rng(seed)
    x = np.arange(c["num_r"] + 1) * c["dx"] - 0.5 * c["num_r"] * c["dx"]
    psi = (np.exp(-np.abs(x)) + 0.3 * np.exp(-((x - 20.0) / 8.0) ** 2) * np.exp(1j * rng.uniform(0.5, 1.0) * x)
           + 0.01 * rng.standard_normal(x.size) * np.exp(-(x / 30.0) ** 2))
    return x, psi


def _signals(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, t = _pulse_grid(c["cycles"])
    tt = torch.tensor(t, device="cuda")
    E0 = 0.02 + 0.05 * torch.rand(c["n_sig"], 1, generator=g, device="cuda", dtype=torch.float64)
    cep = 6.28 * torch.rand(c["n_sig"], 1, generator=g, device="cuda", dtype=torch.float64)
    noise = torch.randn(c["n_sig"], len(t), generator=g, device="cuda", dtype=torch.float64)
    env = torch.tensor(_envelope(t, T), device="cuda")
    return t, E0 * env * (torch.cos(OMEGA0 * tt + cep) + 0.05 * torch.cos(15 * OMEGA0 * tt + 3 * cep) + 1e-3 * noise)


# ------------------------------------------------------------------------------- the calls
def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "call":
        s["dll"] = TDSE_DLL()
        s["t"], s["E"] = _call_inputs(c, seed)
    elif c["kind"] == "batch":
        t, f = _map_fields(c["n_r"], c["n_z"], c["cycles"], seed)
        dt = float(t[1] - t[0])
        s["fields"] = torch.tensor(f, device="cuda")
        grids = TDSEGrids([dict(num_r=c["num_r"], dx=c["dx"], trg_a=A_CONFIG)], dt=dt, df64=c["precision"] == "df64")
        s["plan"] = TDSEBatchPlan(grids, [f.shape[1]] * f.shape[0], dt, precision=c["precision"], tmax=float(t[-1]))
    elif c["kind"] == "uneven":
        params, s["fields"] = _uneven_inputs(c, seed)
        grids = TDSEGrids(params, dt=DT, c64=c["precision"] == "c64", df64=c["precision"] == "df64")
        s["plan"] = TDSEBatchPlan(grids, [len(f) for f in s["fields"]], DT, grid_ids=np.arange(len(params)),
                                  precision=c["precision"])
    elif c["kind"] == "adjoint":
        t, f = _map_fields(c["n_inst"], 1, c["cycles"], seed)
        s["dt"] = float(t[1] - t[0])
        s["fields"] = torch.tensor(f, device="cuda")
        s["grids"] = TDSEGrids([dict(num_r=c["num_r"], dx=c["dx"], trg_a=A_CONFIG)], dt=s["dt"], adjoint=True)
    elif c["kind"] == "long":
        z, r, om, s["rho"], S = _source(c, c["n_z"], seed, torch.complex64 if c["form"] == "fast" else torch.complex128)
        s["target"] = H.FSources_provider(z, r, om, FSource=S)
    elif c["kind"] == "far_field":
        s["z"], s["r"], s["om"], s["rho"], s["S"] = _source(c, c["n_z"], seed, torch.complex64)
        s["pre"] = torch.tensor(_medium(s["z"], s["om"])[0], device="cuda")
    elif c["kind"] == "pes":
        s["psi"] = torch.tensor(_psi(c, seed)[1], device="cuda")
    else:
        t, s["sig"] = _signals(c, seed)
        s["dt"], s["T"] = float(t[1] - t[0]), float(t[-1])
    return s


def run(state):
    s = state
    c = s["case"]
    if c["kind"] == "call":
        g = run_single(s["dll"], s["t"], s["E"], num_r=c["num_r"], dx=c["dx"], trg_a=A_CONFIG, dt=DT, CV=1e-15)
        return {k: g[k] for k in ("x", "psi0", "Einit", "tgrid", "Efield", "sourceterm", "PopTot", "PopInt", "expval",
                                  "Fsourceterm", "FEfield", "omegagrid")}
    if c["kind"] in ("batch", "uneven"):
        p = s["plan"]
        p.load_fields(s["fields"])
        p.launch()
        res = p.result()
        return {"series": res["outputs"], "F": [g["F"] for g in res["spec_groups"]]}
    if c["kind"] == "adjoint":
        return yield_and_grad(s["grids"], s["fields"], s["dt"], BAND, ckpt_every=c["ckpt"])
    if c["kind"] == "long":
        f = H.Hankel_long(s["target"], 1.0, s["rho"], preset_gas="Ar", form=c["form"], as_numpy=False,
                          store_cumulative_result=c["cumulative"])
        out = {"ff": f.FF_integrated, "entry": f.entry_plane_transform, "exit": f.exit_plane_transform}
        if c["cumulative"]:
            out["cumulative"] = f.cumulative_field
        return out
    if c["kind"] == "far_field":
        ff, planes, _ = H.far_field(s["om"], s["r"], s["z"], s["rho"], s["S"], 1.0, s["pre"], True, planes=(0, -1),
                                    form="fast")
        return {"ff": ff, "planes": [planes[k] for k in sorted(planes)]}
    if c["kind"] == "pes":
        return analysis.pes(s["psi"], c["num_r"], c["dx"], A_CONFIG, E_start=-0.6, num_E=c["num_E"], epsilon=5e-4,
                            Estep=c["Estep"])[1]
    return analysis.gabor(s["sig"], s["dt"], c["omega_max"], 0.0, s["T"], c["n_windows"], a=8.0)[2]


# ------------------------------------------------------------------------------- the work
def _tdse_work(sites_steps, n_inst, steps, sites, n_field):
    """72 flop per site and step; the fields in, six series and a complex spectrum out, one set of tables."""
    return {"bytes": 8.0 * n_inst * (n_field + 6 * (steps + 1) + steps + 2) + 16.0 * 7 * sites,
            "flops": 72.0 * sites_steps}


def work(case):
    c = case
    if c["kind"] == "call":
        nf = len(_call_inputs(c, 0)[0])
        k1 = 1 if c["dt_field"] == DT else 3
        S, n = k1 * nf + 2, c["num_r"] + 1
        return _tdse_work(float(S) * n, 1, S, n, nf)
    if c["kind"] == "batch":
        nf = len(_pulse_grid(c["cycles"])[1])
        n_inst, n = c["n_r"] * c["n_z"], c["num_r"] + 1
        return _tdse_work(float(n_inst) * (nf + 2) * n, n_inst, nf + 2, n, nf)
    if c["kind"] == "uneven":
        n = (c["lo"] + c["hi"]) / c["dx"] + 1
        nf = int((c["c_lo"] + c["c_hi"]) * math.pi / OMEGA0 / DT)
        return _tdse_work(float(c["n_inst"]) * (nf + 2) * n, c["n_inst"], nf + 2, n * c["n_inst"], nf)
    if c["kind"] == "adjoint":  # forward, recompute and adjoint sweep; checkpoints written and read once
        nf, n = len(_pulse_grid(c["cycles"])[1]), c["num_r"] + 1
        w = _tdse_work(3.0 * c["n_inst"] * (nf + 2) * n, c["n_inst"], nf + 2, n, 2 * nf)
        w["bytes"] += 32.0 * c["n_inst"] * n * -(-(nf + 2) // c["ckpt"])
        return w
    if c["kind"] in ("long", "far_field"):
        nz = c["n_z"] - (1 if c["kind"] == "long" else 0)
        el = 16.0 if c.get("form") == "plain" else 8.0
        out = 3 + (nz - 1 if c.get("cumulative") else 0)
        pairs = float(c["n_omega"]) * c["n_r"]
        # 8 flop per term of a plane's transform for the planes asked for, and the contraction over z
        planes = nz if c.get("cumulative") else 3
        return {"bytes": el * pairs * nz + 16.0 * out * c["n_omega"] * c["n_rho"],
                "flops": 8.0 * pairs * c["n_rho"] * planes + 8.0 * pairs * nz}
    if c["kind"] == "pes":
        n = c["num_r"] + 1
        return {"bytes": 16.0 * n + 8.0 * c["num_E"], "flops": 100.0 * n * c["num_E"]}
    n = len(_pulse_grid(c["cycles"])[1])
    rows = float(c["n_sig"]) * c["n_windows"]
    dt = c["cycles"] * 2 * math.pi / OMEGA0 / (n - 1)
    n_freq = min(n // 2, int(c["omega_max"] * n * dt / (2 * math.pi)) + 1)
    return {"bytes": 8.0 * c["n_sig"] * n + 8.0 * rows * n_freq, "flops": rows * (n + 2.5 * n * math.log2(n))}


# ------------------------------------------------------------------------------- 64-bit values
class _Tdse:
    """The Crank-Nicolson-Numerov step psi' = e^{iF dt x} (2 A^-1 M2 - 1) psi of one grid as blocks of
    dense rows: A^-1 decays away from its diagonal, so each block is taken from the inverse of a
    window that reaches 20 decimal digits of that decay beyond it."""

    def __init__(self, num_r, dx, a, dt, adjoint=False):
        dev = "cuda"
        n = num_r + 1
        self.n, self.dt = n, dt
        self.x = torch.tensor(np.arange(n) * dx - 0.5 * num_r * dx, device=dev)
        self.V = -1.0 / torch.sqrt(a * a + self.x ** 2)
        self.dV = self.x * (a * a + self.x ** 2) ** -1.5
        self.dx, tau = dx, 0.5 * dt
        off, diag = complex(1 / 12, -tau * 0.5 / dx ** 2), complex(10 / 12, tau / dx ** 2)
        root = np.roots([off, diag, off])
        h = int(math.ceil(46.0 / -math.log(np.abs(root).min())))
        self.h, self.b = h, max(64, h)
        nb = -(-n // self.b)
        w = self.b + 2 * h
        idx = (torch.arange(nb, device=dev) * self.b - h)[:, None] + torch.arange(w, device=dev)[None, :]
        inside = (idx >= 0) & (idx < n)
        Vw = torch.where(inside, self.V[idx.clamp(0, n - 1)], torch.zeros_like(idx, dtype=torch.float64))
        A = torch.zeros(nb, w, w, dtype=torch.complex128, device=dev)
        M = torch.zeros(nb, w, w, dtype=torch.complex128, device=dev)
        k = torch.arange(w, device=dev)
        both = (inside[:, 1:] & inside[:, :-1]).to(torch.complex128)
        A[:, k, k] = torch.where(inside, diag + 1j * tau * (10 / 12) * Vw, torch.ones_like(Vw, dtype=torch.complex128))
        A[:, k[1:], k[:-1]] = both * (off + 1j * tau / 12 * Vw[:, :-1])
        A[:, k[:-1], k[1:]] = both * (off + 1j * tau / 12 * Vw[:, 1:])
        M[:, k, k] = torch.where(inside, torch.full_like(Vw, 10 / 12), torch.full_like(Vw, 0.5)).to(torch.complex128)
        M[:, k[1:], k[:-1]] = both / 12
        M[:, k[:-1], k[1:]] = both / 12
        U = 2 * torch.linalg.solve(A, M) - torch.eye(w, dtype=torch.complex128, device=dev)
        self.U = U[:, h:h + self.b].contiguous()
        self.UH = U.mH[:, h:h + self.b].contiguous() if adjoint else None
        self.pad = (h, nb * self.b + h - n)

    def apply(self, op, psi):
        """op psi for psi [n, n_inst]."""
        p = torch.nn.functional.pad(torch.view_as_real(psi).permute(1, 2, 0), self.pad).permute(2, 0, 1)
        win = torch.view_as_complex(p.contiguous()).unfold(0, self.b + 2 * self.h, self.b).transpose(1, 2)
        return torch.bmm(op, win.contiguous()).reshape(-1, psi.shape[1])[:self.n]

    def ground_state(self, eguess=-1.0, cv=1e-15):
        n, dx, V = self.n, self.dx, self.V
        K = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        k = torch.arange(n, device="cuda")
        K[k, k] = 1 / dx ** 2 + 10 / 12 * V - eguess * 10 / 12
        K[k[1:], k[:-1]] = -0.5 / dx ** 2 + V[:-1] / 12 - eguess / 12
        K[k[:-1], k[1:]] = -0.5 / dx ** 2 + V[1:] / 12 - eguess / 12
        lu = torch.linalg.lu_factor(K)

        def m2(v):
            p = torch.nn.functional.pad(v, (1, 1))
            return (10 * p[1:-1] + p[2:] + p[:-2]) / 12

        psi, e = torch.ones(n, dtype=torch.float64, device="cuda"), eguess
        for _ in range(200):
            psi = torch.linalg.lu_solve(*lu, m2(psi)[:, None])[:, 0]
            psi = psi / psi.norm()
            p, v = torch.nn.functional.pad(psi, (1, 1)), torch.nn.functional.pad(V * psi, (1, 1))
            kp = (psi - 0.5 * (p[2:] + p[:-2])) / dx ** 2 + (10 * v[1:-1] + v[2:] + v[:-2]) / 12
            mp = m2(psi)
            new = float((kp * mp).sum() / (mp * mp).sum())
            if abs(new - e) <= cv:
                break
            e = new
        return psi / psi.norm(), new

    def propagate(self, psi0, F, x_int=2.0, keep=False):
        """Series [n_inst, 4, S + 1] (sourceterm, PopTot, PopInt, expval) for the applied fields F [n_inst, S]."""
        n_inst, S = F.shape
        psi = psi0.to(torch.complex128)[:, None].expand(-1, n_inst).contiguous()
        win = torch.zeros_like(self.x)
        lo = max(0, int(torch.searchsorted(self.x, -x_int)) - 1)
        win[lo:min(self.n - 1, int(torch.searchsorted(self.x, x_int))) + 1] = 1.0
        obs = torch.stack([self.dV, self.x, win])  # [3, n]
        out = torch.zeros(n_inst, 4, S + 1, dtype=torch.float64, device="cuda")
        out[:, 1, 0] = 1.0
        out[:, 2, 0] = (win * psi0 ** 2).sum()
        kept = [psi] if keep else None
        p0 = psi0.to(torch.complex128)[None]
        for k in range(S):
            ph = self.x[:, None] * (F[:, k] * self.dt)[None, :]
            psi = torch.polar(torch.ones_like(ph), ph) * self.apply(self.U, psi)
            o = obs @ (psi.real ** 2 + psi.imag ** 2)
            pr = (p0 @ psi)[0]
            out[:, 0, k + 1] = F[:, k] - o[0]
            out[:, 1, k + 1] = pr.real ** 2 + pr.imag ** 2
            out[:, 2, k + 1] = o[2]
            out[:, 3, k + 1] = o[1]
            if keep:
                kept.append(psi)
        return (out, kept) if keep else out


def _applied(f, S, floor=None):
    """The field of each step: 0 up to the first k with f[k] f[k+1] <= 0, and beyond its samples."""
    n_inst, nf = f.shape
    F = torch.zeros(n_inst, S, dtype=torch.float64, device=f.device)
    F[:, :nf] = f
    g = torch.zeros(n_inst, S + 1, dtype=torch.float64, device=f.device)
    g[:, :nf] = f if floor is None else torch.where(f.abs() <= floor, torch.zeros_like(f), f)
    gate = ((g[:, :-1] * g[:, 1:]) <= 0).to(torch.int8).argmax(dim=1)
    return torch.where(torch.arange(S, device=f.device)[None] <= gate[:, None], torch.zeros_like(F), F), gate


def _spectrum(series, dt):
    return dt / math.sqrt(2 * math.pi) * torch.fft.rfft(series).conj()


def _packed(tmin, dt, F, out):
    """The six series [n_inst, 6, S + 1] as the framework orders them."""
    n_inst, S = F.shape
    t = tmin + dt * torch.arange(S + 1, dtype=torch.float64, device="cuda")
    E = torch.nn.functional.pad(F, (1, 0))
    return torch.stack([t.expand(n_inst, -1), E, out[:, 0], out[:, 1], out[:, 2], out[:, 3]], dim=1)


def _exact_call(c, seed):
    t, E = _call_inputs(c, seed)
    dtf = t[1] - t[0]
    k1 = int(math.floor(dtf / DT))
    k1 += k1 != 1
    dt = dtf / k1
    f = torch.tensor(E, device="cuda")[None]
    floor = None
    if k1 > 1:
        floor = 1e-13 * float(f.abs().max())
        f = k1 * torch.fft.irfft(torch.fft.rfft(f), n=k1 * f.shape[1])
    S = f.shape[1] + 2
    F, _ = _applied(f, S, floor)
    g = _Tdse(c["num_r"], c["dx"], A_CONFIG, dt)
    psi0, e = g.ground_state()
    s = _packed(0.0, dt, F, g.propagate(psi0, F))[0, :, :S]
    return {"x": g.x, "psi0": psi0.to(torch.complex128), "Einit": e, "tgrid": s[0], "Efield": s[1], "sourceterm": s[2],
            "PopTot": s[3], "PopInt": s[4], "expval": s[5], "Fsourceterm": _spectrum(s[2], dt),
            "FEfield": _spectrum(s[1], dt),
            "omegagrid": torch.arange(S // 2 + 1, dtype=torch.float64) * (2 * math.pi / (t[-1] - t[0]))}


def _exact_batch(c, seed):
    n_inst, n = c["n_r"] * c["n_z"], c["num_r"] + 1
    t, f = _map_fields(c["n_r"], c["n_z"], c["cycles"], seed)
    S = f.shape[1] + 2
    if float(n_inst) * n * S > 2.5e9:
        return None
    dt = float(t[1] - t[0])
    F, _ = _applied(torch.tensor(f, device="cuda"), S)
    g = _Tdse(c["num_r"], c["dx"], A_CONFIG, dt)
    psi0, _ = g.ground_state()
    s = _packed(0.0, dt, F, g.propagate(psi0, F))
    return {"series": s.reshape(-1), "F": [_spectrum(s[:, 2, :S], dt)]}


def _exact_adjoint(c, seed):
    t, f = _map_fields(c["n_inst"], 1, c["cycles"], seed)
    nf, n_inst, n = f.shape[1], c["n_inst"], c["num_r"] + 1
    S, dt = nf + 2, float(t[1] - t[0])
    if float(n_inst) * n * S > 8e8:
        return None
    F, gate = _applied(torch.tensor(f, device="cuda"), S)
    g = _Tdse(c["num_r"], c["dx"], A_CONFIG, dt, adjoint=True)
    psi0, _ = g.ground_state()
    out, psi = g.propagate(psi0, F, keep=True)
    s = out[:, 0, :S].clone().requires_grad_(True)
    om = torch.arange(S // 2 + 1, device="cuda", dtype=torch.float64) * (2 * math.pi / ((nf - 1) * dt))
    sel = (om >= BAND[0]) & (om <= BAND[1])
    L = (dt ** 2 / (2 * math.pi) * torch.fft.rfft(s)[:, sel].abs() ** 2).sum(dim=1)
    L.sum().backward()
    a = torch.nn.functional.pad(s.grad, (0, 1))  # the last state's sample is not in the series
    grad = torch.zeros(n_inst, S, dtype=torch.float64, device="cuda")
    lam = torch.zeros(n, n_inst, dtype=torch.complex128, device="cuda")
    for k in range(S - 1, -1, -1):
        lam = lam - 2 * a[None, :, k + 1] * g.dV[:, None] * psi[k + 1]
        grad[:, k] = a[:, k + 1] - dt * (g.x[:, None] * (lam.conj() * psi[k + 1]).imag).sum(dim=0)
        ph = -g.x[:, None] * (F[:, k] * dt)[None, :]
        lam = g.apply(g.UH, torch.polar(torch.ones_like(ph), ph) * lam)
    grad = torch.where(torch.arange(S, device="cuda")[None] <= gate[:, None], torch.zeros_like(grad), grad)
    return [L.detach(), grad[:, :nf]]


class _J0:
    """J0 in 64 bits on [0, top]: Taylor sums of 12 terms about nodes 1/4 apart, whose coefficients
    follow from J0 and J1 there (trapezoid of Bessel's integral, exact to rounding) by Bessel's equation."""

    def __init__(self, top):
        x0 = (np.arange(int(4 * top) + 2) + 0.5) / 4
        th = (np.arange(2048) + 0.5) * (np.pi / 2048)
        j0, j1 = np.empty_like(x0), np.empty_like(x0)
        for i, x in enumerate(x0):
            j0[i] = math.fsum(np.cos(x * np.sin(th))) / 2048
            j1[i] = math.fsum(np.cos(th - x * np.sin(th))) / 2048
        c = [np.zeros_like(x0), j0, -j1]  # c[n + 1] multiplies d^n
        for n in range(10):
            c.append(-((n + 1) ** 2 * c[n + 2] + x0 * c[n + 1] + c[n]) / ((n + 2) * (n + 1) * x0))
        self.c = torch.tensor(np.stack(c[1:]), device="cuda")

    def __call__(self, x):
        i = (4 * x).to(torch.int32)
        d = x - (i + 0.5) / 4
        y = self.c[-1][i]
        for n in range(len(self.c) - 2, -1, -1):
            y.mul_(d).add_(self.c[n][i])
        return y


def _exact_far(c, seed):
    long_ = c["kind"] == "long"
    z, r, om, rho, S = _source(c, c["n_z"], seed, torch.complex128 if c.get("form") == "plain" else torch.complex64)
    if long_:
        z, S = z[:-1], S[:-1]
    nz, no = len(z), len(om)
    if float(nz) * no * len(r) * len(rho) > 7e10:
        return None
    pre, renorm = _medium(z, om)
    wr = np.zeros_like(r)
    wr[:-1] += 0.5 * np.diff(r)
    wr[1:] += 0.5 * np.diff(r)
    dev = "cuda"
    rt, rhot, kt = torch.tensor(r, device=dev), torch.tensor(rho, device=dev), torch.tensor(om / C_LIGHT, device=dev)
    w = torch.tensor(wr * r, device=dev)
    pt = torch.tensor(pre, device=dev)
    j0 = _J0(float(om[-1] / C_LIGHT * rho[-1] * r[-1] / (1.0 - z[-1])) + 1.0)
    P = torch.empty(nz, len(rho), no, dtype=torch.complex128, device=dev)
    step = max(1, int(6e7 // (len(r) * len(rho))))
    for k in range(nz):
        D = 1.0 - z[k]
        ph = -kt[:, None] * rt[None, :] ** 2 / (2 * D)
        A = S[k].to(torch.complex128) * w[None] * torch.polar(torch.ones_like(ph), ph) * pt[k][:, None]
        for a in range(0, no, step):
            J = j0(kt[a:a + step, None, None] * rhot[None, :, None] * rt[None, None, :] / D)
            o = torch.bmm(J, torch.view_as_real(A[a:a + step]))
            P[k, :, a:a + step] = torch.view_as_complex(o).T
    dz = torch.tensor(np.diff(z), device=dev)
    run_ = torch.cumsum(0.5 * dz[:, None, None] * (P[:-1] + P[1:]), dim=0) if nz > 1 else None
    ff = run_[-1].clone() if nz > 1 else torch.zeros_like(P[0])
    if not long_:
        return {"ff": ff, "planes": [P[0], P[-1]] if nz > 1 else [P[0]]}
    out = {"ff": ff, "entry": P[0], "exit": P[-1]}
    if c["cumulative"]:
        out["cumulative"] = torch.tensor(renorm[:nz - 1], device=dev)[:, None, :] * run_
    return out


def _exact_pes(c, seed):
    x, psi = _psi(c, seed)
    n, dx, dE = len(x), c["dx"], 5e-4
    V = (-1.0 / np.sqrt(1.68 + x ** 2)).tolist()
    E = torch.tensor(-0.6 + c["Estep"] * np.arange(c["num_E"]), device="cuda")

    def solve(rhs, e):
        """(M2 (e - V) - K) u = rhs[j], rows as lists of [num_E] (or scalar) values."""
        up, low, cp = [None] * n, [None] * n, [None] * n
        for j in range(n):
            up[j] = (e - V[j]) / 12 + 0.5 / dx ** 2
            d = (e - V[j]) * (10 / 12) - 1 / dx ** 2
            low[j] = rhs[j] / d if j == 0 else (rhs[j] - up[j - 1] * low[j - 1])
            if j > 0:
                beta = d - up[j - 1] * cp[j]
                low[j] = low[j] / beta
            else:
                beta = d
            if j + 1 < n:
                cp[j + 1] = ((e - V[j + 1]) / 12 + 0.5 / dx ** 2) / beta
            up[j - 1] = None
        for j in range(n - 2, -1, -1):
            low[j] = low[j] - cp[j + 1] * low[j + 1]
        return low

    def m2(v):
        zero = torch.zeros((), dtype=torch.complex128, device="cuda")
        return [(10 * v[j] + (v[j - 1] if j else zero) + (v[j + 1] if j + 1 < n else zero)) / 12 for j in range(n)]

    p = np.pad(psi, 1)
    rhs = ((10 * p[1:-1] + p[2:] + p[:-2]) / 12).tolist()
    u1 = solve(rhs, torch.complex(E - dE, torch.full_like(E, -dE)))
    u2 = solve(m2(u1), torch.complex(E + dE, torch.full_like(E, dE)))
    acc = torch.zeros_like(E)
    for u in u2:
        acc += u.real ** 2 + u.imag ** 2
    return acc * dx * dE ** 4


def _exact_gabor(c, seed):
    t, sig = _signals(c, seed)
    N, dt, T = len(t), float(t[1] - t[0]), float(t[-1])
    n_freq = int(np.count_nonzero(2 * np.pi * np.fft.fftfreq(N, dt)[:N // 2] <= c["omega_max"]))
    j = torch.arange(N, dtype=torch.float64, device="cuda") * dt
    tw = torch.arange(c["n_windows"], dtype=torch.float64, device="cuda") * (T / c["n_windows"])
    win = torch.exp(-((j[None] - tw[:, None]) / 8.0) ** 2)
    out = torch.empty(c["n_sig"], c["n_windows"], n_freq, dtype=torch.float64, device="cuda")
    for s in range(c["n_sig"]):
        out[s] = dt / math.sqrt(2 * math.pi) * torch.fft.rfft(win * sig[s][None])[:, :n_freq].abs()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "uneven":  # one grid per instance: too many operators
        return None
    fn = {"call": _exact_call, "batch": _exact_batch, "adjoint": _exact_adjoint, "long": _exact_far,
          "far_field": _exact_far, "pes": _exact_pes, "gabor": _exact_gabor}[kind]
    return fn(case, seed)
