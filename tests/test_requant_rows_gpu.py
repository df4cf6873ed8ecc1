"""Requantisation of SwiGLU activations with a row held by one CTA: row lengths around a warp's and a CTA's worth, one too long
to be held, one and several rows per CTA, rows that hold infinities and NaN, against the definition."""
import array

import pytest
import torch

from cannbench_operator_solutions_b200 import _lib as L

pytestmark = pytest.mark.gpu


LENGTHS = [16, 496, 512, 528, 2048, 2064, 16384, 16400]
# more rows than CTAs (at most 32 per SM of one warp, 12 of four, one of 32): each takes several in turn
SEVERAL_PER_CTA = [(64, 12000), (512, 9000), (2048, 5000), (2064, 4000), (16384, 1000), (16400, 500)]


@pytest.mark.parametrize("h,rows", [(h, 1) for h in LENGTHS] + [(h, 2500 if h <= 528 else 37) for h in LENGTHS] + SEVERAL_PER_CTA)
def test_matches_the_definition(h, rows):
    lib, st = L.load(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(h + rows)
    k, n = 16, 2 * h
    need = lib.w8a8_grouped_matmul_swiglu_quant_workspace_size(rows, k, n, 1)
    ws = torch.zeros((need,), dtype=torch.uint8, device="cuda")
    y = torch.empty((rows, h), dtype=torch.int8, device="cuda")
    scale = torch.empty((rows,), device="cuda")
    x, w = torch.zeros((rows, k), dtype=torch.int8, device="cuda"), torch.zeros((1, k, n), dtype=torch.int8, device="cuda")
    w_scale, x_scale = torch.ones((1, n), device="cuda"), torch.ones((rows,), device="cuda")
    ends = array.array("q", [rows])

    def run(flags):
        return lib.w8a8_grouped_matmul_swiglu_quant(
            x.data_ptr(), w.data_ptr(), w_scale.data_ptr(), x_scale.data_ptr(), y.data_ptr(), scale.data_ptr(), rows, k, n, 1,
            ends.buffer_info()[0], 0, L.W_KN, flags, ws.data_ptr(), need, st)

    assert run(L.F_STAGE_MATMUL) == L.OK  # the header
    # the activations are the last M x H floats before the second table (256 bytes of header, 16-byte tiles of E + 1 groups)
    tail = 256 + 256
    first = need - tail - (rows * h * 4 + 255) // 256 * 256
    act = ws[first : first + rows * h * 4].view(torch.float32).view(rows, h)
    assert (act == 0).all()
    # in no order: a row whose maximum came from another row of its CTA could not pass
    size_of_row = torch.logspace(-3, 3, rows, device="cuda")[torch.randperm(rows, generator=g, device="cuda")]
    act.copy_(torch.randn((rows, h), generator=g, device="cuda") * size_of_row.unsqueeze(1))
    if rows > 1:
        act[0, 3], act[1, h - 1], act[2] = float("nan"), float("inf"), 0.0
    assert run(L.F_STAGE_REQUANT) == L.OK
    a = act.nan_to_num(nan=0.0, posinf=float("inf"), neginf=float("-inf"))
    amax = a.abs().amax(1).clamp_min(1.1754944e-38)
    assert torch.equal(scale, amax * torch.tensor(1.0 / 127.0, device="cuda"))
    inv = torch.full_like(amax, 127.0) / amax  # (127.0 / amax would multiply by a reciprocal)
    want = (act * inv.unsqueeze(1)).half().float().round().clamp(-128, 127).nan_to_num(nan=0.0)
    assert torch.equal(y.float(), want)
