"""moe_finalize_routing where a CTA takes several rows, and a row several blocks of staged terms: the terms of the next
row or block are looked up while the present one is summed."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,h,dtype", [(1, 1, 8, torch.bfloat16), (1184, 2, 16, torch.float16), (1185, 2, 16, torch.bfloat16),
                                            (2500, 8, 40, torch.bfloat16), (2500, 128, 8, torch.float16),
                                            (1300, 129, 12, torch.float32), (3, 300, 4, torch.float32)])
@pytest.mark.parametrize("mode", [0, 2])
def test_matches_oracle(ops, oracle, rows, k, h, dtype, mode):
    from helpers import bits
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    src = torch.randn((rows * 2, h), generator=g, device="cuda").to(dtype)
    pos = torch.randint(-1, rows * 2 + 1, (rows * k,), generator=g, device="cuda", dtype=torch.int32)  # some out of range
    skip = torch.randn((rows, h), generator=g, device="cuda").to(dtype)
    scales = torch.rand((rows, k), generator=g, device="cuda")
    got = ops.moe_finalize_routing(src, pos, skip, None, None, scales, None, mode)
    code = {torch.bfloat16: oracle.DT_BF16, torch.float16: oracle.DT_F16, torch.float32: oracle.DT_F32}[dtype]
    host = (lambda t: t.cpu().numpy()) if dtype == torch.float32 else bits
    want = oracle.moe_finalize_routing(host(src), pos.cpu().numpy(), code, skip1=host(skip), scales=scales.cpu().numpy(),
                                       drop_pad_mode=mode)
    assert np.array_equal(host(got), want)
