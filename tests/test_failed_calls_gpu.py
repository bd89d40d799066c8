"""A CUDA call that fails on the host: the entry points fall back where they can, and leave no error behind
for the next call.  A preloaded library hands the runtime a launch or an allocation that it refuses (a block
of 4096 threads, 2^60 bytes), so nothing reaches the device."""
import ctypes
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stdlib.h>
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a)
{
    cudaError_t (*real)(const cudaLaunchConfig_t *, const void *, void **) = dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
    cudaLaunchConfig_t bad = *c;
    if (getenv("FAIL_CLUSTERS") && c->numAttrs == 1 && c->attrs[0].id == cudaLaunchAttributeClusterDimension)
        bad.blockDim.x = 4096;
    return real(&bad, f, a);
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s)
{
    cudaError_t (*real)(void **, size_t, cudaStream_t) = dlsym(RTLD_NEXT, "cudaMallocAsync");
    return real(p, getenv("FAIL_MALLOC") ? (size_t)1 << 60 : n, s);
}
"""

PRELUDE = r"""
import ctypes, os
import numpy as np, torch
from mma_gb300 import analysis, hankel as H
from mma_gb300.tdse_adjoint import yield_and_grad
from mma_gb300.tdse_batch import MMAStatusError, TDSEGrids, run_batch
setenv = ctypes.CDLL(None).setenv
unsetenv = ctypes.CDLL(None).unsetenv
P = dict(num_r=600, dx=0.2, trg_a=1.3)
f = torch.full((1, 8), 1e-3, dtype=torch.float64, device="cuda")
def raises(call):
    try:
        call()
    except MMAStatusError as e:
        assert "CUDA error" in str(e), e
        return True
def next_call():
    assert TDSEGrids([P] * 60, dt=0.25).iterations.min() > 1
next_call()
"""

CASES = {
    "ground": """
ref = TDSEGrids([P], dt=0.25)
setenv(b"FAIL_CLUSTERS", b"1", 1)
got = TDSEGrids([P], dt=0.25)
assert torch.equal(got.buf[:ref.buf.numel()], ref.buf)
""",
    "propagate": """
g = TDSEGrids([P], dt=0.25)
run_batch(g, f, 0.25, spectra=False)
setenv(b"FAIL_CLUSTERS", b"1", 1)
assert raises(lambda: run_batch(g, f, 0.25, spectra=False))
next_call()
""",
    "adjoint": """
import mma_gb300.tdse_adjoint as ta
g = TDSEGrids([P], dt=0.25, adjoint=True)
lib = ta._adj_sig()
class Lib:  # the propagation before the sweep succeeds
    def __getattr__(self, name):
        if name != "mma_tdse_adjoint":
            return getattr(lib, name)
        setenv(b"FAIL_CLUSTERS", b"1", 1)
        return lib.mma_tdse_adjoint
ta._adj_sig = Lib
assert raises(lambda: yield_and_grad(g, f, 0.25, (0.2, 20.0), ckpt_every=4))
next_call()
""",
    "pes": """
lib = analysis._sig()
psi = torch.ones(201, dtype=torch.complex128, device="cuda")
out = torch.empty(64, dtype=torch.float64, device="cuda")
least = (8 * 202 + 255) // 256 * 256 + (16 * 201 + 255) // 256 * 256 + 32 * 201
ws = torch.empty(least, dtype=torch.uint8, device="cuda")
setenv(b"FAIL_MALLOC", b"1", 1)
st = torch.cuda.current_stream().cuda_stream
assert lib.mma_tdse_pes(psi.data_ptr(), 200, 0.3, 1.1, 64, 4e-3, 2e-4, -0.5, out.data_ptr(), ws.data_ptr(), least, st) == 3
next_call()
""",
    "plain": """
lib = H._sig()
g = torch.linspace(1e-5, 2e-4, 8, dtype=torch.float64, device="cuda")
S = torch.ones(8, 8, 8, dtype=torch.complex128, device="cuda")
ff = torch.empty(8, 8, dtype=torch.complex128, device="cuda")
p = H.HankelProblem(8, 8, 8, 8, 1.0, 1, 1, 64, 8, 0)
setenv(b"FAIL_MALLOC", b"1", 1)
st = torch.cuda.current_stream().cuda_stream
d = g.data_ptr()
assert lib.mma_hankel_plain(ctypes.byref(p), d, d, d, d, S.data_ptr(), None, ff.data_ptr(), None, 0, None, st) == 3
next_call()
""",
}


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    src, so = d / "shim.c", d / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-I/usr/local/cuda/include", str(src), "-o", str(so), "-ldl"], check=True)
    return str(so)


@pytest.mark.parametrize("case", sorted(CASES))
def test_failed_call_is_left_behind(gpu_lib, shim, case):
    r = subprocess.run([sys.executable, "-c", PRELUDE + CASES[case] + "\nprint('done')"], cwd=ROOT, text=True,
                       capture_output=True, timeout=120, env=dict(os.environ, LD_PRELOAD=shim))
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), r.stderr[-2000:]


@pytest.mark.parametrize("num_r, launches", [(8000, 3), (24831, 3), (24832, 1)])
def test_ground_state_route_is_settled_before_the_first_launch(gpu_lib, num_r, launches):
    """Launches of one grid's build (captured, not run): tables, ground state by a cluster and step tables;
    or, where a cluster's shared memory cannot hold the vectors, the one-CTA kernel alone."""
    import torch
    from mma_gb300.tdse_batch import TDSEGrids

    # the records of a grid, from a build that one iteration ends
    g = TDSEGrids([dict(num_r=num_r, dx=0.1, trg_a=1.3, CV=1e3)], dt=0.25)
    rt = ctypes.CDLL("libcudart.so.13")
    graph, count, s = ctypes.c_void_p(), ctypes.c_size_t(), torch.cuda.Stream()
    st = ctypes.c_void_p(s.cuda_stream)
    assert rt.cudaStreamBeginCapture(st, 2) == 0
    rc = gpu_lib.mma_tdse_build_grids(ctypes.c_void_p(g.dev_recs.data_ptr()), ctypes.addressof(g.host_recs), 1, 0, st)
    assert rt.cudaStreamEndCapture(st, ctypes.byref(graph)) == 0 and rc == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    rt.cudaGraphDestroy(graph)
    assert count.value == launches
