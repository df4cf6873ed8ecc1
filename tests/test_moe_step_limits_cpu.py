"""What the C++ expert step refuses does not depend on whether it can do without the address tables, and is refused before
anything is launched."""
import ctypes

import pytest

from cannbench_operator_solutions_b200 import _lib as L


@pytest.mark.parametrize("cap_rows", [32, 4096], ids=["tables", "one chain"])
@pytest.mark.parametrize("experts", [1025, 4096])
def test_more_experts_than_the_tables_hold(experts, cap_rows):
    from cannbench_operator_solutions_b200 import build

    build.build_library()
    lib = L.load()
    buf = (ctypes.c_char * 1024)()
    p = (ctypes.addressof(buf) + 255) & ~255
    step = L.MoeFfnStep()
    step.world, step.rank, step.num_experts, step.topk, step.dtype = 1, 0, experts, 4, L.DT_BF16
    step.tokens, step.hidden, step.inter, step.cap_rows, step.home_rows = 16, 64, 32, cap_rows, 4096
    for name in ("peer_base", "local_base", "w_up", "s_up", "w_down", "s_down", "workspace"):
        setattr(step, name, p)
    step.workspace_bytes = lib.w8a8_moe_ffn_step_workspace_size(ctypes.byref(step))
    launches = lib.w8a8_kernel_launch_count()
    assert lib.w8a8_moe_ffn_step(ctypes.byref(step), p, p, p, 1e-6, p, p, p, p, None) == L.ERR_LIMIT
    assert lib.w8a8_kernel_launch_count() == launches
