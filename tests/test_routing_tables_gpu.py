"""Route plan and expert-parallel address tables where their launches change: around one CTA's worth of pairs, around
the shared-memory expert limit, with ids out of range, and with more than one rank's counts."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference_plan(idx, e):
    flat = idx.reshape(-1)
    ok = (flat >= 0) & (flat < e)
    count = np.bincount(flat[ok], minlength=e).astype(np.int64)
    base = np.concatenate([[0], np.cumsum(count)[:-1]])
    pos = np.full(flat.size, -1, np.int64)
    for x in np.unique(flat[ok]):
        at = np.flatnonzero(flat == x)
        pos[at] = base[x] + np.arange(at.size)
    return count, np.cumsum(count), pos.reshape(idx.shape)


@pytest.mark.parametrize("e", [1, 3, 256, 1000, 1024, 1025])
@pytest.mark.parametrize("t,topk", [(1, 1), (255, 4), (256, 4), (257, 4), (1025, 1), (5000, 8), (33 * 1024 + 5, 2)])
def test_route_plan(e, t, topk):
    from cannbench_operator_solutions_b200 import ep
    rng = np.random.default_rng(e * 1000 + t)
    idx = (rng.zipf(1.3, size=(t, topk)) % e).astype(np.int32)
    idx[rng.random((t, topk)) < 0.01] = e
    idx[rng.random((t, topk)) < 0.01] = -1
    count, cumsum, pos = ep.CudaBackend().route_plan(torch.from_numpy(idx).cuda(), e)
    want = reference_plan(idx, e)
    for got, w in zip((count, cumsum, pos), want):
        assert np.array_equal(got.cpu().numpy(), w)


@pytest.mark.parametrize("p,e,cap", [(1, 1, 100), (1, 1024, 4000), (2, 1024, 9000), (8, 256, 30000), (32, 64, 40000),
                                     (8, 256, 500)])
def test_ep_tables(p, e, cap):
    from cannbench_operator_solutions_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(p * 7 + e)
    counts = rng.integers(0, 7, size=(p, e)).astype(np.int64)
    base = (1 << 40) + (np.arange(p, dtype=np.int64) << 32)
    e_local = e // p
    off_x, off_s, off_back, row_bytes, back_bytes = 4096, 1 << 20, 1 << 21, 112, 224
    for rank in {0, p - 1}:
        dev = dict(device="cuda", dtype=torch.int64)
        row_dst, scale_dst, my_base = (torch.full((e,), -7, **dev) for _ in range(3))
        group_list, seg_first, seg_ptr = torch.full((e_local,), -7, **dev), torch.full((e + 1,), -7, **dev), torch.full((e,), -7, **dev)
        status = torch.zeros((4,), device="cuda", dtype=torch.int32)
        c, b = torch.from_numpy(counts).cuda(), torch.from_numpy(base).cuda()
        rc = lib.w8a8_ep_tables(c.data_ptr(), p, e, rank, b.data_ptr(), off_x, off_s, off_back, row_bytes, back_bytes, cap,
                                row_dst.data_ptr(), scale_dst.data_ptr(), my_base.data_ptr(), group_list.data_ptr(),
                                seg_first.data_ptr(), seg_ptr.data_ptr(), status.data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        per_rank = np.concatenate([np.zeros((p, 1), np.int64), counts.cumsum(1)], 1)  # exclusive prefix of each rank
        col = counts.sum(0)
        bad = bool((col.reshape(p, e_local).sum(1) > cap).any())
        assert int(status[0]) == int(bad)
        owner = np.arange(e) // e_local
        ex = np.concatenate([[0], col.cumsum()])
        first = ex[:-1] - ex[owner * e_local] + counts[:rank].sum(0)
        assert np.array_equal(my_base.cpu().numpy(), per_rank[rank, :-1])
        mine = np.arange(rank * e_local, (rank + 1) * e_local)
        seg = counts[:, mine].T.reshape(-1)
        want = dict(row_dst=base[owner] + off_x + first * row_bytes, scale_dst=base[owner] + off_s + first * 4,
                    group_list=col[mine].cumsum(), seg_first=np.concatenate([[0], seg.cumsum()]),
                    seg_ptr=(base[None, :] + off_back + per_rank[:, mine].T * back_bytes).reshape(-1))
        got = dict(row_dst=row_dst, scale_dst=scale_dst, group_list=group_list, seg_first=seg_first[: e_local * p + 1],
                   seg_ptr=seg_ptr[: e_local * p])
        for k, w in want.items():
            assert np.array_equal(got[k].cpu().numpy(), w * (0 if bad else 1)), k
