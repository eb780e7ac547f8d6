"""Device memory of an FP64 WDM plan: two work buffers and the staging series (16 bytes
per complex point each) and the passes' factors (32 bytes per point), with 2% for the
small tables and the allocation's rounding.
"""
import pytest

import glass_gb300 as gg

pytestmark = pytest.mark.gpu


def test_fp64_plan():
    import torch

    from glass_gb300 import build

    build.build()
    NF, NT = 1536, 4096
    x = torch.zeros(NF * NT, dtype=torch.float64, device="cuda")
    eng = gg.Engine(0)

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    try:
        # the kernels' modules loaded, and the plan small
        for call in (eng.wdm_forward_device, eng.wdm_inverse_device):
            call(64, 64, x[:4096], x[:4096])
        before = used()
        for call in (eng.wdm_forward_device, eng.wdm_inverse_device):
            call(NF, NT, x, x)
        grown = used() - before
    finally:
        eng.close()
    assert grown <= 1.02 * (3 * 16 + 32) * NF * NT / 2
