"""The kernel shape that is chosen by an estimate of its time gives the bits of the shapes that the caller can force, on
both sides of the lines between them (dense: narrow and wide single CTAs, pairs, K split over two and four; grouped: singles,
pairs, both)."""
import pytest
import torch

from cannbench_operator_solutions_b200 import _lib

pytestmark = pytest.mark.gpu


def _under(shape, call):
    lib = _lib.load()
    before = lib.w8a8_set_gemm_shape(shape)
    try:
        return call()
    finally:
        lib.w8a8_set_gemm_shape(before)


@pytest.mark.parametrize("m,k,n", [
    (1, 256, 512), (3, 1776, 1584), (8, 1504, 7168), (17, 1296, 736), (33, 1568, 832), (76, 4608, 512), (85, 5776, 816),
    (129, 2064, 400), (178, 1200, 11920), (223, 528, 14784), (721, 848, 8384), (1112, 1760, 4032), (2702, 2048, 1632),
    (1309, 560, 6880), (3000, 1024, 2064),
])
def test_dense(ops, m, k, n):
    g = torch.Generator(device="cuda").manual_seed(m + k)
    x = torch.randint(-127, 128, (m, k), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-127, 128, (k, n), generator=g, device="cuda", dtype=torch.int8)
    scale, pt = torch.rand((n,), generator=g, device="cuda") * 1e-3, torch.rand((m,), generator=g, device="cuda")
    bias = torch.randn((n,), generator=g, device="cuda").to(torch.bfloat16)

    def call():
        return ops.quant_matmul(x, w, scale, pertoken_scale=pt, bias=bias, output_dtype="bfloat16")

    own = call()
    assert torch.equal(own, _under(1, call)) and torch.equal(own, _under(2, call))
    assert _lib.load().w8a8_pipeline_error(torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("rows,experts,k,n", [(300, 8, 512, 608), (2500, 16, 1024, 1024), (3000, 8, 528, 2048), (9000, 4, 256, 768),
                                              (6000, 128, 256, 512)])
@pytest.mark.parametrize("skew", [0.0, 1.0])
def test_grouped(ops, rows, experts, k, n, skew):
    g = torch.Generator(device="cuda").manual_seed(rows)
    odds = torch.arange(1, experts + 1, device="cuda", dtype=torch.float32).pow(-skew)
    pick = torch.multinomial(odds, rows, replacement=True, generator=g)
    ends = torch.bincount(pick, minlength=experts).cumsum(0)
    x = torch.randint(-127, 128, (rows, k), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-127, 128, (experts, k, n), generator=g, device="cuda", dtype=torch.int8)
    ws, xs = torch.rand((experts, n), generator=g, device="cuda") * 1e-3, torch.rand((rows,), generator=g, device="cuda")
    for lst in (ends.tolist(), ends):  # the tiles are known, and assumed
        def down():
            return ops.grouped_matmul(x, w, lst, None, 3, x_scale=xs, weight_scale=ws)[0]

        def up():
            return torch.cat([t.view(torch.uint8).flatten() for t in ops.grouped_matmul_swiglu_quant(x, w, ws, xs, lst)])

        for call in (down, up):
            own = call()
            assert all(torch.equal(own, _under(shape, call)) for shape in (1, 2, 3))
