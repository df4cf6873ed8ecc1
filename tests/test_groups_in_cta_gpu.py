"""Grouped matmuls around the number of groups up to which every CTA plans its tiles itself (256; beyond it a kernel builds
a table): host and device lists, empty groups at either end, lists that end before the rows do, and lists out of order."""
import ctypes

import pytest
import torch

from cannbench_operator_solutions_b200 import _lib

pytestmark = pytest.mark.gpu
K, N = 32, 48


def _ends(experts, rows, seed):
    g = torch.Generator().manual_seed(seed)
    cuts = torch.randint(0, rows + 1, (experts - 1,), generator=g).sort().values if experts > 1 else torch.zeros(0).long()
    cuts[: experts // 8] = 0  # empty groups first
    cuts[experts - experts // 8 :] = rows  # and last
    return [*cuts.tolist(), rows]


def _operands(experts, rows, seed):
    """bf16 integers whose products and sums fp32 holds exactly, with results that bf16 holds exactly: -1, 0 and 1."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-1, 2, (rows, K), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randint(-1, 2, (experts, K, N), generator=g, device="cuda").to(torch.bfloat16)
    return x, w


def _want(x, w, ends):
    out, first = torch.zeros((x.size(0), N), device="cuda"), 0
    for e, end in enumerate(ends):
        out[first:end] = x[first:end].float() @ w[e].float()
        first = end
    return out.to(torch.bfloat16)


@pytest.mark.parametrize("experts", [1, 7, 8, 9, 255, 256, 257, 600])
@pytest.mark.parametrize("rows", [300, 4100])  # one launch; pairs and leftovers
@pytest.mark.parametrize("on_device", [False, True])
def test_tiles_of_the_groups(ops, experts, rows, on_device):
    ends = _ends(experts, rows, experts + rows)
    x, w = _operands(experts, rows, experts)
    lst = torch.tensor(ends, device="cuda") if on_device else ends
    (y,) = ops.grouped_matmul(x, w, lst, None, 3)
    assert torch.equal(y, _want(x, w, ends))


@pytest.mark.parametrize("experts", [256, 257])
@pytest.mark.parametrize("rows", [300, 4100])
def test_prefix_and_invalid_device_lists(ops, experts, rows):
    lib = _lib.load()
    ends = _ends(experts, rows - 37, experts)
    x, w = _operands(experts, rows, experts)
    need = lib.w8a8_grouped_matmul_workspace_size(rows, N, K, experts)
    ws = torch.empty((need,), dtype=torch.uint8, device="cuda")

    def run(values, mode):
        y = torch.full((rows, N), 7.0, dtype=torch.bfloat16, device="cuda")
        lst = torch.tensor(values, device="cuda")
        rc = lib.w8a8_grouped_matmul(x.data_ptr(), w.data_ptr(), None, y.data_ptr(), None, None, rows, N, K, experts,
                                     lst.data_ptr(), mode, 1, 1, 1, 0, ws.data_ptr(), need,
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        return y, lib.w8a8_workspace_error(ws.data_ptr(), None)

    y, error = run(ends, 2)  # ends 37 rows early: those rows stay as they are
    assert error == 0 and torch.equal(y[: rows - 37], _want(x, w, ends)[: rows - 37]) and (y[rows - 37 :] == 7.0).all()
    for values, mode in ((ends, 1), ([*ends[:5], ends[-1] + 50, *ends[6:]], 2), ([-1, *ends[1:]], 2)):
        y, error = run(values, mode)
        assert error == 1 and (y == 7.0).all()
