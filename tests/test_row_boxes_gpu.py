"""Grouped matmuls with enough weights that single-CTA tiles load their own rows only (boxes of 16 or 32 rows; what the
stages hold below is multiplied and not stored): group sizes around the boxes and the tile, against the CTA-pair form of the same operator, which loads whole
tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

E, K, N = 64, 2048, 2048  # 256 MB of int8


def ends(sizes):
    return torch.tensor(sizes + [0] * (E - len(sizes))).cumsum(0).tolist()


SIZES = {
    "box16": [0, 1, 15, 16, 17, 32, 33, 128, 129, 0, 257, 2],                       # 630 rows: boxes of 16
    "box32": [31, 32, 33, 64, 65, 96, 97, 127, 128, 129, 200, 0, 256, 300, 1],      # 1655 rows: boxes of 32
    "leftovers": [1, 127, 128, 129, 256, 257, 287, 288, 289, 384, 385, 513, 31, 32, 33],  # pairs, then boxes of 32
}


@pytest.fixture(scope="module")
def weights():
    g = torch.Generator(device="cuda").manual_seed(1)
    return torch.randint(-127, 128, (E, K, N), generator=g, device="cuda", dtype=torch.int8)


@pytest.mark.parametrize("case", sorted(SIZES))
def test_same_bits_as_pairs(ops, weights, case):
    from cannbench_operator_solutions_b200 import _lib as L
    lib = L.load()
    gl = ends(SIZES[case])
    m = gl[-1]
    assert m < 2048 or case == "leftovers"
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randint(-127, 128, (m, K), generator=g, device="cuda", dtype=torch.int8)
    xs = torch.rand((m,), generator=g, device="cuda") * 1e-2 + 1e-3
    ws = torch.rand((E, N), generator=g, device="cuda") * 1e-3 + 1e-4

    def both():
        y, s = ops.grouped_matmul_swiglu_quant(x, weights, ws, xs, gl)
        (d,) = ops.grouped_matmul(x, weights, gl, None, 3, x_scale=xs, weight_scale=ws)
        return y, s, d
    got = both()
    lib.w8a8_set_gemm_shape(2)
    try:
        want = both()
    finally:
        lib.w8a8_set_gemm_shape(0)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_bf16_rows_and_a_device_list_that_ends_early(ops, weights):
    g = torch.Generator(device="cuda").manual_seed(9)
    gl = ends([1, 40, 16, 0, 129])
    m = gl[-1]
    x = torch.randn((m, K), generator=g, device="cuda").to(torch.bfloat16)
    w = (weights[:, :, :1024].to(torch.float32) / 73.0 / K ** 0.5).to(torch.bfloat16)  # 256 MB
    (y,) = ops.grouped_matmul(x, w, torch.tensor(gl, device="cuda"), None, 3)
    first = 0
    for e, end in enumerate(gl):
        if end > first:
            want = x[first:end].double() @ w[e].double()
            # bf16 rounding of the result (2^-8 relative) beside fp32 sums
            assert ((y[first:end].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16 * want.abs().max()).all()
        first = end
