"""The C++ expert step on one GPU in both of its forms - one chain of kernels where the buffers hold every pair, and the
general one (address tables, a second stream, output addresses, capacity-sized matmuls) that several ranks run - against
the oracle, eager and from a captured graph.  A buffer of fewer rows than there are pairs takes the general form; its
results mean something where enough pairs have no valid expert for the rest to fit."""
import numpy as np
import pytest
import torch

from helpers import bits

pytestmark = pytest.mark.gpu


def _reference(problem, experts):
    """The chain by the oracle; pairs without a valid expert are routed to one more expert, behind all others, and dropped."""
    from test_ep_cpu import OracleBackend

    from cannbench_operator_solutions_b200.ep import ExpertShard, MoeFfnChain

    class Backend(OracleBackend):
        def route_plan(self, expert_idx, num_experts):
            idx = torch.where((expert_idx < 0) | (expert_idx >= num_experts), num_experts, expert_idx)
            count, cumsum, pos = super().route_plan(idx, num_experts + 1)
            self.rows = int(cumsum[num_experts - 1])
            return count[:num_experts], cumsum[:num_experts], torch.where(pos < self.rows, pos, -1)

        def scatter_rows(self, src, src_scale, pos, total_rows):
            spare = torch.where(pos < 0, self.rows, pos)
            dst, scale = super().scatter_rows(src, src_scale, spare, self.rows + 1)
            return dst[: self.rows], scale[: self.rows]

    x, res, gamma, idx, probs, *weights = problem
    return MoeFfnChain(experts, ExpertShard(*weights), backend=Backend()).forward(x, res, gamma, 1e-6, idx, probs)


def _problem(seed, tokens, hidden, inter, experts, topk):
    """Every third pair or so, and the first, without a valid expert, on both sides of the valid ones."""
    from test_ep_cpu import _problem as valid

    problem = list(valid(seed=seed, tokens=tokens, hidden=hidden, inter=inter, experts=experts, topk=topk))
    lost = torch.from_numpy(np.random.default_rng(seed + 1).integers(0, 6, problem[3].shape))
    problem[3] = torch.where(lost == 0, -1, torch.where(lost == 1, experts, problem[3])).to(torch.int32)
    problem[3][0, 0] = -1
    return problem


def _chain(problem, experts, general):
    from cannbench_operator_solutions_b200.ep import ExpertShard, MoeFfnChain

    idx = problem[3]
    valid = int(((idx >= 0) & (idx < experts)).sum())
    # room for other inputs' valid pairs too, but not for all pairs
    capacity = min(idx.numel() - 1, valid + idx.numel() // 8) if general else None
    return MoeFfnChain(experts, ExpertShard(*(t.cuda() for t in problem[5:])), transport="p2p", device_tables=True,
                       capacity_rows=capacity)


def _args(problem, off=0):
    def at(t):
        held = torch.empty((t.numel() + off,), dtype=t.dtype, device="cuda")
        held[off:].copy_(t.reshape(-1))
        return held[off:].view(t.shape)

    x, res, gamma, idx, probs = problem[:5]
    return [at(x), at(res), at(gamma), idx.cuda(), probs.cuda()]


# one and several CTAs of the route plan; up to 256 groups planned in the matmuls and more by their own kernel; the most
# experts; rows that the normalisation reads an element at a time (their addresses miss 16 bytes); more tokens than SMs
@pytest.mark.parametrize("tokens,hidden,inter,experts,topk,off", [
    (200, 512, 256, 8, 4, 0), (5, 64, 32, 5, 2, 0), (700, 256, 128, 16, 8, 0), (150, 256, 64, 300, 4, 0), (60, 64, 32, 1024, 8, 0),
    (90, 512, 64, 8, 2, 3), (2600, 128, 64, 4, 2, 0)])
@pytest.mark.parametrize("general", [False, True], ids=["one chain", "general"])
def test_eager(ops, tokens, hidden, inter, experts, topk, off, general):
    problem = _problem(tokens, tokens, hidden, inter, experts, topk)
    want, want_x = _reference(problem, experts)
    chain = _chain(problem, experts, general)
    x, res, gamma, idx, probs = _args(problem, off)
    for _ in range(2):  # the second pass reuses the buffers of the first
        out, x_out = chain.forward(x, res, gamma, 1e-6, idx, probs)
        assert np.array_equal(bits(x_out), bits(want_x))
        assert np.array_equal(bits(out), bits(want))
    assert chain._native is not None
    chain.check()


@pytest.mark.parametrize("general", [False, True], ids=["one chain", "general"])
def test_captured(ops, general):
    """Nothing is read back or allocated and all streams join the caller's, so a capture holds the whole step: replayed after
    the inputs have been overwritten in place it gives the result on the new ones."""
    experts = 16
    problems = [_problem(seed, 256, 512, 256, experts, 4) for seed in (7, 8)]
    problems[1][5:] = problems[0][5:]
    want = [_reference(problem, experts) for problem in problems]
    chain = _chain(problems[0], experts, general)
    static = _args(problems[0])
    chain.forward(static[0], static[1], static[2], 1e-6, static[3], static[4])  # first-use set-up outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, x_out = chain.forward(static[0], static[1], static[2], 1e-6, static[3], static[4])
    for i in (0, 1, 0):
        for dst, src in zip(static, _args(problems[i])):
            dst.copy_(src)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(bits(out), bits(want[i][0])) and np.array_equal(bits(x_out), bits(want[i][1]))
    chain.check()


def test_requantisation_inside_the_matmuls(ops):
    """The optional in-kernel requantisation under both forms: a device list that ends below the matmul's row count."""
    from cannbench_operator_solutions_b200 import _lib as L

    experts, lib = 8, L.load()
    problem = _problem(11, 700, 512, 384, experts, 4)
    want, want_x = _reference(problem, experts)
    x, res, gamma, idx, probs = _args(problem)
    try:
        lib.w8a8_set_gmsq_fused_requant(1)
        for general in (False, True):
            chain = _chain(problem, experts, general)
            out, x_out = chain.forward(x, res, gamma, 1e-6, idx, probs)
            chain.check()
            assert np.array_equal(bits(out), bits(want)) and np.array_equal(bits(x_out), bits(want_x))
    finally:
        lib.w8a8_set_gmsq_fused_requant(0)
    assert lib.w8a8_pipeline_error(None) == 0
