"""The pair forms of the exponential and the quotient, and the order that the router selects by, on every input that can
tell."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CHECKS = ["negated exponential", "exponential of x <= 0", "exponential of neighbours", "quotient near midpoints"]


def test_pair_arithmetic_equals_the_scalar_forms():
    from cannbench_operator_solutions_b200 import _lib as L

    lib = L.load()
    res = torch.empty(9, dtype=torch.int64, device="cuda")
    rc = lib.w8a8_selftest_pairs(res.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, L.status_string(rc)
    torch.cuda.synchronize()
    got = res.tolist()
    for c, name in enumerate(CHECKS):
        assert got[2 * c] == 0, f"{name}: {got[2 * c]} differ, the smallest pattern is {got[2 * c + 1] & 0xffffffff:#010x}"
    assert got[8] > 50_000_000  # divisions tested
    assert lib.w8a8_selftest_pairs(None, None) == L.ERR_INVALID
