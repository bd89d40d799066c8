"""The ground state by a cluster against one CTA per grid, to the bit, at every number of sites per thread
that splits otherwise over the cluster's four warps (tdse_ground.cu: sites i = sub, sub + 4, ...) and over
the quotient's pairs (tdse_step.cuh): full and partly filled last rows."""
import pytest
import torch

from tests.tdse_cases import A_CONFIG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_r", [2, 254, 255, 256, 511, 512, 600, 767, 768, 1023, 1024, 1279, 1280, 1535, 1536, 1791, 1792,
                                   2047, 2048, 2303])
def test_rows(gpu_lib, num_r):
    from mma_gb300.tdse_batch import TDSEGrids

    p = dict(num_r=num_r, dx=0.2, trg_a=A_CONFIG)
    one = TDSEGrids([p], dt=0.25)
    many = TDSEGrids([p] * (torch.cuda.get_device_properties(0).multi_processor_count // 4 + 1), dt=0.25)
    for name in ("x", "psi0", "cn_tab", "gs_tab", "result"):
        (o, cnt), (q, _) = one.views[0][name], many.views[-1][name]
        assert torch.equal(one.buf[o:o + cnt].view(torch.int64), many.buf[q:q + cnt].view(torch.int64)), name
