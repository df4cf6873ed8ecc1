"""quant_matmul where its K is split over a cluster (few 128 x 128 tiles): every split, ragged rows, columns and K
blocks, several row tiles and batches, against the oracle bit for bit, and the tile counts on both sides of each line."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (1, 16, 2048),           # one tile, a cluster of four
    (8, 144, 1536),          # a cluster of two, six K blocks each; the second column tile holds one 16-column piece
    (17, 1024, 2048 + 16),   # seventeen K blocks over four CTAs, the last one partial
    (65, 528, 3072 + 16), (129, 528, 3072 + 16), (300, 640, 7168), (16, 7168, 9216), (64, 4096, 2048),
    (512, 2032, 3200),       # 64 tiles, split in two
    (16, 9472, 1536),        # 74 tiles: the last count that splits
    (16, 9488, 1536),        # 75 tiles: none
    (64, 1024, 1408), (65, 1024, 2944),  # one K block too few to split
    (600, 3680, 256),        # 145 tiles: single CTAs
    (600, 3856, 256),        # 155 tiles: CTA pairs
])
@pytest.mark.parametrize("layout", ["kn", "nk"])
def test_matches_oracle(ops, oracle, m, n, k, layout):
    from helpers import bits
    from cannbench_operator_solutions_b200 import _lib as L
    rng = np.random.default_rng(m + n + k)
    x = rng.integers(-128, 128, (m, k)).astype(np.int8)
    w = rng.integers(-128, 128, (n, k) if layout == "nk" else (k, n)).astype(np.int8)
    scale = rng.uniform(1e-4, 1e-3, n).astype(np.float32)
    pt = rng.uniform(0.5, 2.0, m).astype(np.float32)
    off = rng.uniform(-1, 1, n).astype(np.float32)
    fbias = rng.normal(size=n).astype(np.float32)
    ibias = rng.integers(-1000, 1000, n).astype(np.int32)
    d = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    for bias, kind in ((None, 0), (fbias, L.QM_BIAS_F32), (ibias, L.QM_BIAS_I32)):
        flags = L.QM_SCALE_PERCHAN | L.QM_HAS_OFFSET | L.QM_OFFSET_PERCHAN | L.QM_HAS_PT
        if bias is not None:
            flags |= (kind << L.QM_BIAS_SHIFT) | L.QM_BIAS_PERCHAN
        got = ops.quant_matmul(d(x), d(w), d(scale), offset=d(off), pertoken_scale=d(pt), bias=None if bias is None else d(bias),
                               output_dtype="bfloat16", transpose_x2=layout == "nk")
        want = oracle.quant_matmul(x, w, scale, offset=off, pertoken=pt, bias=bias, flags=flags, out_dtype=oracle.DT_BF16,
                                   x2_transposed=layout == "nk")
        assert np.array_equal(bits(got), want)
    got = ops.quant_matmul(d(x), d(w), d(scale[:1]), output_dtype="float16", transpose_x2=layout == "nk")
    want = oracle.quant_matmul(x, w, scale[:1], flags=0, out_dtype=oracle.DT_F16, x2_transposed=layout == "nk")
    assert np.array_equal(bits(got), want)
    c = torch.empty((m, n), device="cuda", dtype=torch.int32)
    dx, dw = d(x), d(w)
    rc = L.load().w8a8_matmul_i8_i32(dx.data_ptr(), dw.data_ptr(), c.data_ptr(), 1, m, n, k,
                                     L.W_NK if layout == "nk" else L.W_KN, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    acc = x.astype(np.int64) @ (w.T if layout == "nk" else w).astype(np.int64)
    assert np.array_equal(c.cpu().numpy(), acc)
    assert L.load().w8a8_pipeline_error(torch.cuda.current_stream().cuda_stream) == 0


def test_batches_and_repeats(ops):
    """Several matrices in one launch, and the same launch again and again on one stream."""
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randint(-128, 128, (3, 130, 3200), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-128, 128, (3, 3200, 400), generator=g, device="cuda", dtype=torch.int8)
    scale = torch.rand((400,), generator=g, device="cuda") * 1e-3
    want = ((x.double() @ w.double()).float() * scale).to(torch.bfloat16)
    for _ in range(20):
        assert torch.equal(ops.quant_matmul(x, w, scale, output_dtype="bfloat16"), want)
