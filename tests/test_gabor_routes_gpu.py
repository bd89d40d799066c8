"""Which way a Gabor transform goes (dft.cu, windowed): fused rows of 256 or 384 threads, or, with most bins
of a long even row wanted, passes of their own.  Read from a captured call; the values against the oracle
on both sides of each line, 1e-9 of the largest value (the analysis functions' stated bound)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Dim3(ctypes.Structure):
    _fields_ = [("x", ctypes.c_uint), ("y", ctypes.c_uint), ("z", ctypes.c_uint)]


class _KernelParams(ctypes.Structure):
    _fields_ = [("func", ctypes.c_void_p), ("grid", _Dim3), ("block", _Dim3), ("smem", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p)]


def _captured_blocks(call):
    """Threads per block of the kernels that call(stream) launches, in order of their nodes."""
    rt, s = ctypes.CDLL("libcudart.so.13"), torch.cuda.Stream()
    st, graph, n = ctypes.c_void_p(s.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    assert rt.cudaStreamBeginCapture(st, 2) == 0
    rc = call(st)
    assert rt.cudaStreamEndCapture(st, ctypes.byref(graph)) == 0 and rc == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    out = []
    for node in nodes:
        p = _KernelParams()
        assert rt.cudaGraphKernelNodeGetParams(ctypes.c_void_p(node), ctypes.byref(p)) == 0
        out.append(p.block.x)
    rt.cudaGraphDestroy(graph)
    return out


@pytest.mark.parametrize("N, n_g, n_freq, launches, threads", [
    (64, 5, 33, 2, 256), (2048, 5, 1025, 2, 256), (2050, 5, 513, 2, 384), (2050, 5, 514, 4, 0), (2050, 5, 1026, 4, 0),
    (2050, 152, 514, 4, 0), (2050, 153, 769, 2, 384), (2050, 153, 770, 4, 0), (2205, 5, 1103, 2, 384),
    (4410, 5, 352, 2, 384), (4410, 5, 2206, 4, 0)])
def test_routes(gpu_lib, N, n_g, n_freq, launches, threads):
    import oracle.analysis as oa
    from mma_gb300 import analysis

    lib = analysis._sig()
    rng = np.random.default_rng(N)
    sig = rng.standard_normal((2, N))
    s = torch.tensor(sig, device="cuda")
    dt, t_max, a = 0.25, 0.25 * N, 8.0
    out = torch.full((2, n_g, n_freq), float("nan"), dtype=torch.float64, device="cuda")
    nb = int(lib.mma_gabor_scratch_bytes(2, N, n_g))
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")

    def call(st):
        return lib.mma_gabor(s.data_ptr(), N, 2, dt, N, n_freq, n_g, 0.0, t_max, a, out.data_ptr(), ws.data_ptr(), nb, st)

    assert call(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0  # makes the length's plan
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    for i in range(2):
        ref = oa.gabor(sig[i], dt, N, n_freq, n_g, 0.0, t_max, a)
        assert np.abs(got[i] - ref).max() <= 1e-9 * np.abs(ref).max()
    blocks = _captured_blocks(call)
    assert len(blocks) == launches
    assert threads == 0 or threads in blocks
