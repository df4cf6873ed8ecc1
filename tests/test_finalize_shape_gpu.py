"""moe_finalize_routing over the shapes of its launch: CTAs of 96, 128 and 160 threads, one or several per row, a row in one
pass or many, more rows than CTAs.  The operator rounds each step to fp32 in a fixed order, so PyTorch's fp32 steps in that
order give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,h,dtype", [
    (1, 8, 6256, torch.float16), (3, 2, 8, torch.bfloat16), (37, 4, 768, torch.bfloat16), (37, 4, 776, torch.float16),
    (148, 2, 1024, torch.bfloat16), (149, 3, 1032, torch.float16), (700, 2, 7168, torch.bfloat16), (5000, 2, 1120, torch.float16),
    (4737, 1, 1288, torch.bfloat16), (2, 100, 776, torch.bfloat16), (40, 97, 1032, torch.float16), (5, 130, 1540, torch.float32),
    (4800, 3, 388, torch.float32), (1, 1, 40000, torch.bfloat16),
])
@pytest.mark.parametrize("bias", [False, True])
def test_bits(ops, rows, k, h, dtype, bias):
    g = torch.Generator(device="cuda").manual_seed(rows + h)
    src = torch.randn((rows * k + 1, h), generator=g, device="cuda").to(dtype)
    pos = torch.randint(-1, rows * k + 2, (rows, k), generator=g, device="cuda", dtype=torch.int32)  # some out of range
    skip = torch.randn((rows, h), generator=g, device="cuda").to(dtype)
    scales = torch.rand((rows, k), generator=g, device="cuda")
    table = torch.randn((5, h), generator=g, device="cuda").to(dtype) if bias else None
    expert = torch.randint(0, 5, (rows, k), generator=g, device="cuda", dtype=torch.int32) if bias else None
    got = ops.moe_finalize_routing(src, pos.flatten(), skip, None, table, scales, expert, 2)
    acc = skip.float()
    for j in range(k):
        p = pos[:, j].long()
        there = ((p >= 0) & (p < src.shape[0])).unsqueeze(1)
        term = src[p.clamp(0, src.shape[0] - 1)].float()
        if bias:
            term = term + table[expert[:, j].long()].float()
        acc = torch.where(there, acc + term * scales[:, j : j + 1], acc)
    assert torch.equal(got, acc.to(dtype))
