"""dequant_swiglu_quant where its register-resident rows change shape (chunks per thread, threads per row, dividing
or multiplying form) and where its pair arithmetic leaves its range, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# half-row lengths: one chunk per thread / two, the dividing form's last length and the next, 576 threads and the
# next, the longest register-resident row and the first of the any-length kernel
@pytest.mark.parametrize("h", [8, 256, 264, 1984, 1992, 9208, 9216, 9224, 16384, 16392])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_16_bit_rows_with_gates_out_of_range(ops, oracle, dtype, h):
    from helpers import assert_same_f32, bits
    g = torch.Generator(device="cuda").manual_seed(h)
    x = (torch.randn((5, 2 * h), generator=g, device="cuda") * 4).to(dtype)
    edge = torch.tensor([80.0, -80.0, 80.5, -80.5, 88.0, -88.0, 104.0, 0.0, -0.0, 6.1e-5], device="cuda").to(dtype)
    x[1, :8] = edge[:8]
    x[1, -8:] = edge[2:]
    x[2, h // 2] = float("inf")
    x[3, h + 1] = float("nan")
    for left in (False, True):
        y, sc = ops.dequant_swiglu_quant(x, activate_left=left)
        wy, wsc = oracle.dequant_swiglu_quant(bits(x), oracle.DT_BF16 if dtype == torch.bfloat16 else oracle.DT_F16,
                                              activate_left=left)
        assert_same_f32(sc, wsc, "scale")
        assert np.array_equal(y.cpu().numpy(), wy)


@pytest.mark.parametrize("h", [4, 128, 132, 1984, 1988, 4096, 8192, 8196])
def test_int32_rows_with_exact_ties_of_the_exponent(ops, oracle, h):
    from helpers import assert_same_f32
    g = torch.Generator(device="cuda").manual_seed(h)
    x = torch.randint(-200000, 200000, (4, 2 * h), generator=g, device="cuda", dtype=torch.int32)
    ws = torch.empty((2 * h,), device="cuda").uniform_(1e-6, 1e-4, generator=g)
    # gate * log2(e) rounds to n + 1/2 exactly: the multiplication and the rounding to an integer are two roundings
    x[0, :] = 1
    ws[:4] = torch.tensor([float.fromhex("0x1.92068p+5"), float.fromhex("0x1.a56ef8p+2"), 80.0, 81.0], device="cuda")
    x[1, :] = 0
    a_s = torch.ones((4,), device="cuda")
    for sign in (1, -1):
        for left in (False, True):
            y, sc = ops.dequant_swiglu_quant(x * sign, ws, a_s, None, left)
            wy, wsc = oracle.dequant_swiglu_quant((x * sign).cpu().numpy(), oracle.DT_I32, weight_scale=ws.cpu().numpy(),
                                                  activation_scale=a_s.cpu().numpy(), activate_left=left)
            assert_same_f32(sc, wsc, "scale")
            assert np.array_equal(y.cpu().numpy(), wy)
