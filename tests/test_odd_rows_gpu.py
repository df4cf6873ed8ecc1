"""Regrouping of token rows whose length is no multiple of 16 bytes, or that start off a 16-byte boundary: copied byte by
byte, with the loads of a step ahead of its stores."""
import pytest
import torch

from helpers import best_time

pytestmark = pytest.mark.gpu


def _problem(rows, row_bytes, ranks, experts, offset=0):
    g = torch.Generator(device="cuda").manual_seed(rows * 31 + row_bytes)
    store = torch.randint(-128, 128, (rows * row_bytes + offset,), generator=g, device="cuda", dtype=torch.int8)
    tokens = store[offset:].view(rows, row_bytes)
    cell = torch.randint(0, ranks * experts, (rows,), generator=g, device="cuda")
    counts = torch.bincount(cell, minlength=ranks * experts).view(ranks, experts)
    return tokens, counts


@pytest.mark.parametrize("offset", [0, 1, 8])
@pytest.mark.parametrize("row_bytes", [1, 31, 33, 255, 257, 512, 1000])  # a step of a warp is 256 bytes
def test_rows_are_copied_whole(ops, row_bytes, offset):
    tokens, counts = _problem(300, row_bytes, 3, 5, offset)
    got, _, index, _ = ops.moe_re_routing(tokens, counts)
    cell = torch.repeat_interleave(torch.arange(counts.numel(), device="cuda"), counts.flatten())
    order = torch.argsort(cell % 5, stable=True)
    assert torch.equal(index.long(), order)
    assert torch.equal(got, tokens[order])


def test_odd_rows_cost_at_most_twice_the_vectorised_copy(ops):
    """1.8 times; 2.5 with every load waiting for the store before it."""
    odd, counts = _problem(65536, 1000, 1, 8)
    even, counts2 = _problem(65536, 1024, 1, 8)
    t_odd = best_time(lambda: ops.moe_re_routing(odd, counts))
    t_even = best_time(lambda: ops.moe_re_routing(even, counts2))
    assert t_odd < 2.15 * t_even
