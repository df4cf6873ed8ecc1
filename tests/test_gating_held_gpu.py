"""moe_gating_top_k_softmax on many rows of 129 to 256 16-bit columns, where four lanes hold a row and sort only what can be
selected, against the same rows a thousand at a time, which a warp per row selects: the same bits for ordinary rows and for
rows of ties, few values, masked and infinite logits, NaN, ascending and descending order."""
import pytest
import torch

pytestmark = pytest.mark.gpu
ROWS = 12288 + 5


def _logits(inner, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((ROWS, inner), generator=g, device="cuda")
    kind = torch.arange(ROWS, device="cuda") % 12
    rank = torch.arange(inner, device="cuda", dtype=torch.float32)
    x[kind == 1] = 0.0
    x[kind == 2] = torch.randint(-2, 3, (int((kind == 2).sum()), inner), generator=g, device="cuda").float()
    x[kind == 3] = x[kind == 3].masked_fill(torch.rand((int((kind == 3).sum()), inner), generator=g, device="cuda") < 0.9, float("-inf"))
    x[kind == 4] = rank / 16
    x[kind == 5] = -rank / 16
    x[kind == 6] *= 60.0  # most exponentials vanish
    x[kind == 7] *= 1e-6  # zeros of both signs beside tiny numbers
    x[kind == 8, 7] = float("inf")
    x[kind == 9, inner - 1] = float("nan")
    x[kind == 10] = torch.where(rank % 8 == 3, x[kind == 10] + 4.0, x[kind == 10])  # the largest all in one place of their piece
    x[kind == 11, :72] += 6.0  # and in few pieces
    return x.to(dtype)


@pytest.mark.parametrize("inner", [136, 160, 200, 256])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("k", [1, 5, 8])
def test_matches_a_warp_per_row(ops, inner, dtype, k):
    x = _logits(inner, dtype, inner + k)
    finished = torch.zeros((ROWS,), dtype=torch.bool, device="cuda")
    finished[::97] = True
    y, expert, row = ops.moe_gating_top_k_softmax(x, finished, k)
    parts = [ops.moe_gating_top_k_softmax(x[i : i + 1000], finished[i : i + 1000], k) for i in range(0, ROWS, 1000)]
    want_y, want_e = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    assert torch.equal(expert, want_e)
    assert torch.equal(y.view(torch.int16), want_y.view(torch.int16))
    want_row = torch.arange(k, device="cuda")[None, :] * ROWS + torch.arange(ROWS, device="cuda")[:, None]
    assert torch.equal(row, want_row.int())
