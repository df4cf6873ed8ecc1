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


@pytest.mark.parametrize("k", [8, 64, 136])  # one K block per piece, one whole, and a third with a tail
@pytest.mark.parametrize("rows", [37, 2100])  # single CTAs; pairs and leftovers
@pytest.mark.parametrize("transpose", [False, True])
def test_fp32_pieces_are_paired_as_the_split_says(ops, k, rows, transpose):
    """Each of the six piece products, K blocks in either direction: with one product of 23-bit integers per result, a
    wrong piece or K block shows at once."""
    g = torch.Generator(device="cuda").manual_seed(k + rows)
    n, ends = 272, [rows // 3, rows // 3, rows]
    # one value of x per row and one of w per column are not zero: the result is their exact product, cut to fp32
    x = torch.zeros((rows, k), device="cuda")
    w = torch.zeros((3, k, n), device="cuda")
    at = torch.randint(0, k, (rows,), generator=g, device="cuda")
    x[torch.arange(rows, device="cuda"), at] = torch.randint(1 << 22, 1 << 23, (rows,), generator=g, device="cuda").float()
    w[:] = torch.randint(1 << 22, 1 << 23, (3, k, n), generator=g, device="cuda").float()
    (y,) = ops.grouped_matmul(x, w.transpose(1, 2).contiguous() if transpose else w, ends, None, 3, transpose)
    want = torch.cat([x[: ends[0]].double() @ w[0].double(), x[ends[0] :].double() @ w[2].double()])
    # six products added in fp32, each sum cut by at most 2^-23 of the result, and three dropped ones below 2^-24 each
    assert ((y.double() - want).abs() <= want.abs() * 2.0 ** -20).all()
