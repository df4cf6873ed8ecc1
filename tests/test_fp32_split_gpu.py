"""grouped_matmul on fp32 operands (three bf16 pieces of each, split eight values at a time) at its smallest sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", [(8, 16), (24, 48), (72, 16)])
@pytest.mark.parametrize("transpose", [False, True])
def test_fp32_split_at_its_smallest(ops, k, n, transpose):
    g = torch.Generator(device="cuda").manual_seed(k + n)
    x = torch.randn((21, k), generator=g, device="cuda")
    w = torch.randn((3, n, k) if transpose else (3, k, n), generator=g, device="cuda")
    (y,) = ops.grouped_matmul(x, w, [5, 5, 21], None, 3, transpose)
    wd = w.double().transpose(1, 2) if transpose else w.double()
    want = torch.cat([x[:5].double() @ wd[0], x[5:].double() @ wd[2]])
    # what the six piece products drop is below 2^-24 of sum |x||w|, and the fp32 sums of at most 432 terms round by
    # at most 2^-24 of it each in the worst order: 2^-15 bounds both with room
    bound = torch.cat([x[:5].abs().double() @ wd[0].abs(), x[5:].abs().double() @ wd[2].abs()]) * 2.0 ** -15
    assert ((y.double() - want).abs() <= bound).all()
