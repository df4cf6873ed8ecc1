"""moe_gating_top_k_softmax, k <= 8: the choice between four lanes and a warp per row, on both sides of it."""
import numpy as np
import pytest
import torch

from helpers import best_time, bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,inner,k", [(4096, 64, 1), (4096, 256, 2), (4096, 500, 8), (8192, 100, 1), (20000, 60, 2),
                                          (16384, 128, 4), (16384, 160, 8), (9000, 264, 1), (50000, 256, 8),
                                          (60000, 500, 8), (5000, 1000, 3)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_matches_oracle(ops, oracle, dtype, rows, inner, k):
    g = torch.Generator(device="cuda").manual_seed(rows + inner)
    x = (torch.randn((rows, inner), generator=g, device="cuda") * 3).to(dtype)
    code = {torch.bfloat16: oracle.DT_BF16, torch.float16: oracle.DT_F16, torch.float32: oracle.DT_F32}[dtype]
    y, ei, ri = ops.moe_gating_top_k_softmax(x, None, k)
    wy, wei, wri = oracle.moe_gating_top_k_softmax(x.cpu().numpy() if dtype == torch.float32 else bits(x), code, k, None)
    assert np.array_equal(ei.cpu().numpy(), wei) and np.array_equal(ri.cpu().numpy(), wri)
    assert np.array_equal(y.float().cpu().numpy(), wy if dtype == torch.float32 else oracle.bits_to_f32(wy, code))


def test_no_step_in_the_cost_where_four_lanes_become_possible(ops):
    """fp32 rows of 256, k = 1, on either side of 4096 rows: the same kernel and time; four lanes take 1.6 times as long."""
    few, many = (torch.randn(n, 256, device="cuda") for n in (4090, 4100))
    t_few = best_time(lambda: ops.moe_gating_top_k_softmax(few, None, 1), calls=20)
    t_many = best_time(lambda: ops.moe_gating_top_k_softmax(many, None, 1), calls=20)
    assert t_many < 1.3 * t_few


def test_calls_that_fill_most_of_the_chip_do_not_crowd_each_other(ops):
    """32768 rows of 256 fill two thirds of the SMs' places: 1.5 times the time of 16384 rows in a row of calls, 1.9 when
    each call starts beside the one before."""
    half, whole = (torch.randn(n, 256, device="cuda").bfloat16() for n in (16384, 32768))
    t_half = best_time(lambda: ops.moe_gating_top_k_softmax(half, None, 8), calls=20)
    t_whole = best_time(lambda: ops.moe_gating_top_k_softmax(whole, None, 8), calls=20)
    assert t_whole < 1.7 * t_half
