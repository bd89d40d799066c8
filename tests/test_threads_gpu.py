"""Calls of different sizes from several host threads, each on its own stream.  A kernel's limit of dynamic
shared memory belongs to the whole context: a call that sets it to its own size can lower it between
another thread's set and launch, and that launch fails (cudaErrorInvalidValue, on the host).  Every pair
below runs one kernel with two sizes of shared memory."""
import threading

import numpy as np
import pytest
import torch

from tests.tdse_cases import A_CONFIG

pytestmark = pytest.mark.gpu


def _propagate(num_r, precision, ctas):
    from mma_gb300.tdse_batch import TDSEBatchPlan, TDSEGrids

    grids = TDSEGrids([dict(num_r=num_r, dx=0.2, trg_a=A_CONFIG, CV=1e-10)], dt=0.25, df64=precision == "df64")
    plan = TDSEBatchPlan(grids, [2] * 2, 0.25, precision=precision, spectra=False, grid_ctas=ctas)
    plan.load_fields(torch.zeros(2, 2, dtype=torch.float64, device="cuda"))
    return plan.launch


def _ground(num_r):
    from mma_gb300.tdse_batch import TDSEGrids

    return lambda s: TDSEGrids([dict(num_r=num_r, dx=0.4, trg_a=A_CONFIG, CV=1e-3)], dt=0.25)


def _adjoint(num_r):
    from mma_gb300.tdse_adjoint import yield_and_grad
    from mma_gb300.tdse_batch import TDSEGrids

    grids = TDSEGrids([dict(num_r=num_r, dx=0.2, trg_a=A_CONFIG, CV=1e-10)], dt=0.25, adjoint=True)
    f = torch.full((1, 4), 1e-3, dtype=torch.float64, device="cuda")
    return lambda s: yield_and_grad(grids, f, 0.25, (0.2, 20.0), ckpt_every=2)


def _far_field(nr, form, planes):
    from mma_gb300 import hankel as H

    om, r, z = np.linspace(11, 41, 2) * 2.36e15, np.linspace(0, 2e-4, nr), np.linspace(-5e-3, 5e-3, 4)
    S = torch.ones(4, 2, nr, dtype=torch.complex64, device="cuda")
    return lambda s: H.far_field(om, r, z, np.linspace(0, 5e-3, 4), S, 1.0, planes=planes, form=form, stream=s)


@pytest.mark.parametrize("make, args, n", [
    (_propagate, [(8000, "fp64", 0), (600, "fp64", 0)], 1500), (_propagate, [(8000, "df64", 0), (600, "df64", 0)], 1500),
    (_propagate, [(8000, "fp64", 1), (1500, "fp64", 1)], 3000), (_ground, [(6000,), (300,)], 300),
    (_adjoint, [(8000,), (600,)], 200), (_far_field, [(4000, "plain", (0, 1, 2)), (64, "plain", (0, 1, 2))], 400),
    (_far_field, [(512, "fast", (0,)), (64, "fast", (0,))], 400)],
    ids=["fp64", "df64", "fp64-one-cta", "ground", "adjoint", "plain", "fast"])
def test_two_threads_two_sizes(gpu_lib, make, args, n):
    calls, errors = [make(*a) for a in args], []
    streams = [torch.cuda.Stream() for _ in calls]
    for call, s in zip(calls, streams):
        with torch.cuda.stream(s):
            call(s)
    torch.cuda.synchronize()
    gate = threading.Barrier(len(calls))

    def work(call, s):
        try:
            gate.wait()
            with torch.cuda.stream(s):
                for k in range(n):
                    call(s)
                    if k % 16 == 15:
                        s.synchronize()
        except Exception as e:  # reported by the test
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
