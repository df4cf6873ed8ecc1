"""moe_gating_top_k_softmax, k <= 8 on many rows, where different logits share an exponential in every row: selected a second
time with those logits as one key, and by a whole warp what that leaves.  Bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from helpers import best_time, bits

pytestmark = pytest.mark.gpu

ROWS = 4100


def _one_hot(inner, g):
    x = torch.full((ROWS, inner), -1e9, device="cuda")
    x[torch.arange(ROWS, device="cuda"), torch.randint(0, inner, (ROWS,), generator=g, device="cuda")] = 1.0
    return x


def _normal(inner, g):
    return torch.randn((ROWS, inner), generator=g, device="cuda")


KINDS = {
    "zeros": lambda n, g: torch.zeros((ROWS, n), device="cuda"),
    "signed_zeros": lambda n, g: _normal(n, g).sign() * 0.0,
    "one_hot": _one_hot,
    "saturated": lambda n, g: _normal(n, g) * 60,
    "one_left": lambda n, g: _normal(n, g).masked_fill(torch.arange(n, device="cuda") != n // 2, float("-inf")),
    "around_zero": lambda n, g: _normal(n, g) * 10.0 ** -(6 + 8 * torch.rand((ROWS, 1), generator=g, device="cuda")),
    "below_zero": lambda n, g: -_normal(n, g).abs() * 1e-9,
    "beside_a_peak": lambda n, g: (_normal(n, g) * 1e-6).index_fill(1, torch.tensor([n - 1], device="cuda"), 3.0),
    "under_a_far_peak": lambda n, g: (_normal(n, g) * 4).index_fill(1, torch.tensor([0], device="cuda"), 100.0),
}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("inner", [8, 31, 64, 100, 256, 1024])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_matches_oracle(ops, oracle, dtype, inner, kind):
    g = torch.Generator(device="cuda").manual_seed(inner)
    x = KINDS[kind](inner, g)
    x[1::7] = _normal(inner, g)[1::7]  # rows without ties in the same warps
    x = x.to(dtype)
    code = {torch.bfloat16: oracle.DT_BF16, torch.float16: oracle.DT_F16}[dtype]
    for k in (1, 3, 8):
        y, ei, ri = ops.moe_gating_top_k_softmax(x, None, k)
        with np.errstate(all="ignore"):
            wy, wei, wri = oracle.moe_gating_top_k_softmax(bits(x), code, k, None)
        assert np.array_equal(ei.cpu().numpy(), wei), k
        assert np.array_equal(ri.cpu().numpy(), wri), k
        assert np.array_equal(y.float().cpu().numpy(), oracle.bits_to_f32(wy, code), equal_nan=True), k


@pytest.mark.parametrize("kind", ["zeros", "one_hot"])
def test_cost_of_a_second_selection(ops, kind):
    """About twice the time of rows without ties; eight times when every such row went to a whole warp."""
    g = torch.Generator(device="cuda").manual_seed(1)
    tied = KINDS[kind](256, g).repeat(4, 1).to(torch.bfloat16)
    plain = _normal(256, g).repeat(4, 1).to(torch.bfloat16)
    t_tied = best_time(lambda: ops.moe_gating_top_k_softmax(tied, None, 8))
    t_plain = best_time(lambda: ops.moe_gating_top_k_softmax(plain, None, 8))
    assert t_tied < 4 * t_plain
