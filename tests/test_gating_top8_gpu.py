"""moe_gating_top_k_softmax with k <= 8 on many rows (four lanes per row) at the edges of its rows, pieces and warps, and on rows
whose selection has to be redone on the exponentials, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def special_rows(inner, dtype, g):
    """Rows in which different x share an exponential, equal x sit far apart, or the maximum is not finite."""
    n = torch.randn((14, inner), generator=g, device="cuda") * 2
    n[0] = 0.0
    n[1] = torch.where(torch.arange(inner, device="cuda") % 2 == 0, 0.0, -0.0)
    n[2] = float("-inf")
    n[2, inner // 2] = 1.0
    n[3] = n[3].abs() * 1e-7                       # differences below the resolution of x - max
    n[3, 0] = 3.0
    n[4] = n[4].round()                            # many equal values
    n[5, inner - 1] = float("nan")
    n[6, inner // 3] = float("inf")
    n[7] = float("-inf")
    n[8] = -100.0 - n[8].abs()                     # exponentials down to subnormals and zero
    n[8, inner // 2] = 0.0
    n[9] = torch.arange(inner, device="cuda").float()
    n[10] = -torch.arange(inner, device="cuda").float() / 64
    n[11] = n[11] * 30
    n[12] = n[12] * 6e-8
    n[13, : inner // 2] = float("-inf")
    return n.to(dtype)


@pytest.mark.parametrize("inner", [1, 7, 8, 31, 32, 33, 60, 64, 160, 256, 264, 1000, 1024])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_matches_oracle(ops, oracle, dtype, inner):
    from helpers import bits
    g = torch.Generator(device="cuda").manual_seed(inner)
    code = {torch.bfloat16: oracle.DT_BF16, torch.float16: oracle.DT_F16, torch.float32: oracle.DT_F32}[dtype]
    for rows in (4096, 4097, 4103):
        x = (torch.randn((rows, inner), generator=g, device="cuda") * 2).to(dtype)
        x[:14] = special_rows(inner, dtype, g)
        x[-14:] = special_rows(inner, dtype, g)
        fin = torch.rand((rows,), generator=g, device="cuda") < 0.2
        host = x.cpu().numpy() if dtype == torch.float32 else bits(x)
        for k in sorted({1, 2, 3, 5, 8, min(8, inner)}):
            if k > inner:
                continue
            y, ei, ri = ops.moe_gating_top_k_softmax(x, fin, k)
            with np.errstate(all="ignore"):
                wy, wei, wri = oracle.moe_gating_top_k_softmax(host, code, k, fin.cpu().numpy())
            # with nothing selectable left (NaN exponentials) the oracle has no index, the operator index 0
            wei = np.where(wei == -1, 0, wei)
            got = y.cpu().numpy() if dtype == torch.float32 else y.float().cpu().numpy()
            want = wy if dtype == torch.float32 else oracle.bits_to_f32(wy, code)
            assert np.array_equal(ei.cpu().numpy(), wei), (rows, k)
            assert np.array_equal(ri.cpu().numpy(), wri), (rows, k)
            assert np.array_equal(got, want, equal_nan=True), (rows, k)


def test_unaligned_rows(ops):
    g = torch.Generator(device="cuda").manual_seed(5)
    flat = torch.randn((4099 * 64 + 1,), generator=g, device="cuda").to(torch.bfloat16)
    x = flat[1:].view(4099, 64)
    for a, b in zip(ops.moe_gating_top_k_softmax(x, None, 6), ops.moe_gating_top_k_softmax(x.clone(), None, 6)):
        assert torch.equal(a, b)
