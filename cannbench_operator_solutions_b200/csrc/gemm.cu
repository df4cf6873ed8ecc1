// Host side of the tensor-core operators: argument validation (mirroring the
// reference plugins' checks), TMA tensor maps, the device-side group planner,
// kernel selection, and the C-ABI entry points for quant_matmul,
// grouped_matmul_swiglu_quant and grouped_matmul.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <atomic>
#include <mutex>

#include "gemm_kernel.cuh"

namespace w8a8 {

// ---------------------------------------------------------------------------
// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (the
// library does not link libcuda directly).
// ---------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(sym);
        }
    });
    return fn;
}

static CUtensorMapDataType tm_dtype(int kind)
{
    switch (kind) {
    case KIND_F16:
        return CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    case KIND_BF16:
        return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    default:
        return CU_TENSOR_MAP_DATA_TYPE_UINT8;
    }
}

// A: [rows, K] row-major.  Box = 128 bytes of K x 128 rows.
static bool make_map_a(CUtensorMap* m, const void* base, int64_t rows, int64_t K, int kind, int box_rows = 128)
{
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) {
        return false;
    }
    const int elem = (kind == KIND_I8) ? 1 : 2;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * elem};
    cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem), static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, tm_dtype(kind), 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// B: [G, K, N] (mn_major) or [G, N, K].  Box = 128 bytes of the contiguous
// dimension x 128 bytes-worth of K rows (mn_major: BLOCK_K rows) or 128 N rows.  L2 promotion to 128 bytes: to 256, the
// neighbouring column tile's half of each line pair came along, to be fetched again where that tile runs at another time
// or on the other die (SwiGLU form, 512 rows of 256 experts of 7168 x 4096 927 us, 953 so; 7724 of 64 of 1712 x 3808 159,
// 171).
static bool make_map_b(CUtensorMap* m, const void* base, int64_t G, int64_t N, int64_t K, int kind, bool mn_major)
{
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) {
        return false;
    }
    const int elem = (kind == KIND_I8) ? 1 : 2;
    const int64_t inner = mn_major ? N : K;
    const int64_t outer = mn_major ? K : N;
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer), static_cast<cuuint64_t>(G)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(inner) * elem, static_cast<cuuint64_t>(inner) * outer * elem};
    cuuint32_t box[3] = {static_cast<cuuint32_t>(128 / elem), static_cast<cuuint32_t>(mn_major ? 128 / elem : 128), 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, tm_dtype(kind), 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CG, int BLOCK_N>
constexpr size_t gemm_smem_bytes()
{
    return static_cast<size_t>(gemm_stages(CG, BLOCK_N)) * (GEMM_A_BYTES + (BLOCK_N / CG) * GEMM_KBYTES) +
           1024 /*alignment slack*/ + 512 /*barriers, tmem slot, abort flag*/ + GEMM_EPI_PATCH_BYTES /*store patches*/ +
           (GROUPS_IN_CTA + 1) * sizeof(int32_t) /*first tiles of the groups*/;
}

// number of workers (CTAs, or CTA pairs) a persistent launch uses
template <int CG>
static int64_t worker_count(int64_t max_tiles)
{
    int64_t workers = sm_count() / CG;
    if (max_tiles < workers) {
        workers = max_tiles;
    }
    return workers < 1 ? 1 : workers;
}

template <int CG, int BLOCK_N, int KIND, int EPI, bool B_MN, int EPI_WARPS = 8, bool SPLITK = false, bool ROW_BOXES = false>
static cudaError_t launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int64_t max_tiles,
                               cudaStream_t st, const GroupListOf<EPI>& groups = {})
{
    auto kern = gemm_tc_kernel<CG, BLOCK_N, KIND, EPI, B_MN, EPI_WARPS, SPLITK, ROW_BOXES>;
    constexpr size_t smem = gemm_smem_bytes<CG, BLOCK_N>();
    static KernelFacts facts;
    const cudaError_t e = allow_dynamic_smem(facts, kern, smem);
    if (e != cudaSuccess) {
        return e;
    }
    const unsigned cluster = SPLITK ? static_cast<unsigned>(p.split) : CG;
    const int64_t workers = SPLITK ? max_tiles : worker_count<CG>(max_tiles);  // split K: one tile per cluster
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(workers * cluster), 1, 1);
    cfg.blockDim = dim3(gemm_threads(EPI_WARPS), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = p.order == ORDER_PLAIN ? 0 : 1;
    if (cluster > 1) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = cluster;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    note_launch();
    return cudaLaunchKernelEx(&cfg, kern, ta, tb, p, groups);
}

static std::atomic<int> g_gmsq_epilogue_warps{16};

template <int KIND, int EPI>
static cudaError_t dispatch_gemm(int cta_group, int block_n, bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb,
                                 const GemmParams& p, int64_t max_tiles, cudaStream_t st,
                                 const GroupListOf<EPI>& groups = {})
{
    if constexpr (EPI == EPI_GMSQ) {
        // the SwiGLU epilogue with sixteen epilogue warps (see w8a8_set_gmsq_epilogue_warps)
        if (g_gmsq_epilogue_warps.load(std::memory_order_relaxed) == 16) {
            if (cta_group == 2) {
                return b_mn ? launch_gemm<2, 256, KIND, EPI, true, 16>(ta, tb, p, max_tiles, st, groups)
                            : launch_gemm<2, 256, KIND, EPI, false, 16>(ta, tb, p, max_tiles, st, groups);
            }
            return b_mn ? launch_gemm<1, 256, KIND, EPI, true, 16>(ta, tb, p, max_tiles, st, groups)
                        : launch_gemm<1, 256, KIND, EPI, false, 16>(ta, tb, p, max_tiles, st, groups);
        }
    }
    // Sixteen warps for the int8 operators' 16-bit results: eight, at two per scheduler, take 6 us for a 128 x 256 tile, as
    // long as the main loop of K = 2048 (8192 x 512 x 4096 with bias 43 us, 60 with eight; 4096 x 1024 x 8192 48.8, 50.4;
    // 1000 x 2048 x 4096 16.1, 17.2; expert layer of 2000 x 8 rows over 64 experts of 2688 x 1008 295, 303).  16-bit operands,
    // with nothing to convert or scale, are no faster (16000 rows of 8 experts of 512 x 4096 89.4, 88.3), and rows stored
    // at addresses of their own, which may be another GPU's, leave eight warps in whole lines.
    if constexpr (EPI == EPI_QMM || (EPI == EPI_GMM && KIND == KIND_I8)) {
        if (EPI == EPI_QMM || p.out_row_ptrs == nullptr) {
            if (cta_group == 2) {
                return b_mn ? launch_gemm<2, 256, KIND, EPI, true, 16>(ta, tb, p, max_tiles, st, groups)
                            : launch_gemm<2, 256, KIND, EPI, false, 16>(ta, tb, p, max_tiles, st, groups);
            }
            if (block_n == 128) {
                return b_mn ? launch_gemm<1, 128, KIND, EPI, true, 16>(ta, tb, p, max_tiles, st, groups)
                            : launch_gemm<1, 128, KIND, EPI, false, 16>(ta, tb, p, max_tiles, st, groups);
            }
            return b_mn ? launch_gemm<1, 256, KIND, EPI, true, 16>(ta, tb, p, max_tiles, st, groups)
                        : launch_gemm<1, 256, KIND, EPI, false, 16>(ta, tb, p, max_tiles, st, groups);
        }
    }
    if constexpr (EPI != EPI_QMM) {
        if (cta_group == 2) {
            return b_mn ? launch_gemm<2, 256, KIND, EPI, true>(ta, tb, p, max_tiles, st, groups)
                        : launch_gemm<2, 256, KIND, EPI, false>(ta, tb, p, max_tiles, st, groups);
        }
        if constexpr (EPI == EPI_RAW || (EPI == EPI_GMM && KIND != KIND_I8)) {
            if (block_n == 128) {
                return b_mn ? launch_gemm<1, 128, KIND, EPI, true>(ta, tb, p, max_tiles, st, groups)
                            : launch_gemm<1, 128, KIND, EPI, false>(ta, tb, p, max_tiles, st, groups);
            }
        }
        return b_mn ? launch_gemm<1, 256, KIND, EPI, true>(ta, tb, p, max_tiles, st, groups)
                    : launch_gemm<1, 256, KIND, EPI, false>(ta, tb, p, max_tiles, st, groups);
    }
}

// Single-CTA tiles of a grouped problem that load their own rows only (see run_grouped).
template <int KIND, int EPI>
static cudaError_t dispatch_row_boxes(bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                                      int64_t max_tiles, cudaStream_t st, const GroupListOf<EPI>& groups)
{
    if constexpr (EPI == EPI_GMSQ) {
        if (g_gmsq_epilogue_warps.load(std::memory_order_relaxed) == 16) {
            return b_mn ? launch_gemm<1, 256, KIND, EPI, true, 16, false, true>(ta, tb, p, max_tiles, st, groups)
                        : launch_gemm<1, 256, KIND, EPI, false, 16, false, true>(ta, tb, p, max_tiles, st, groups);
        }
    }
    if constexpr (EPI == EPI_GMM && KIND == KIND_I8) {
        if (p.out_row_ptrs == nullptr) {
            return b_mn ? launch_gemm<1, 256, KIND, EPI, true, 16, false, true>(ta, tb, p, max_tiles, st, groups)
                        : launch_gemm<1, 256, KIND, EPI, false, 16, false, true>(ta, tb, p, max_tiles, st, groups);
        }
    }
    return b_mn ? launch_gemm<1, 256, KIND, EPI, true, 8, false, true>(ta, tb, p, max_tiles, st, groups)
                : launch_gemm<1, 256, KIND, EPI, false, 8, false, true>(ta, tb, p, max_tiles, st, groups);
}

// w8a8_set_gemm_shape() (1, 2, or 3 = pairs plus singles for grouped problems; 0 = the library's choice) overrides the
// kernel shape process-wide; the tests use it to run every case on every shape.
constexpr int GEMM_SHAPE_HYBRID = 3;
constexpr int GEMM_SHAPE_NARROW = 4;  // single CTAs on 128 x 128 tiles: never forced
static std::atomic<int> g_shape_override{0};
static std::atomic<int> g_fuse_requant{0};  // see w8a8_set_gmsq_fused_requant

struct DenseShape {
    int cta_group, block_n, split;
};

// Dense problems: single CTAs on 128 x 128 or 128 x 256 tiles, CTA pairs on 256 x 256, or, where most SMs would have no
// tile, clusters of two or four CTAs that share a 128 x 128 tile's K (clusters of eight do not find a place for every tile,
// clusters of four count on 128 SMs).  The shape is the one with the smallest estimate, in us: waves of tiles over the SMs,
// a tile taking its K blocks (0.244, 0.356, 0.245) or its epilogue (1.8, 3.1, 3.3) if that is longer; no less than the
// weights at 5.5 TB/s; and what the shape costs besides - wide tiles 0.5, a pair's cluster 3, a split 0.8 and the exchange of
// the accumulators, by the 32-row quarters of a tile that hold rows (0.55 for two CTAs, 0.83 for four).  Fitted to 220
// problems of 1 - 8192 rows, 512 - 9216 x 512 - 18432, each timed in all shapes: 0.2 % from the best of each on average and
// 8 % at worst, where the rule before it - singles up to one tile per SM, pairs from 256 rows on, splits by thresholds - is
// 2.3 % and 41 % from it (1112 x 1760 x 4032 15.8 us, 11.2 on wide singles; 178 x 4384 x 11920 26.2, 20.5 on pairs; 85 x 5776 x
// 816 14.9, 11.3 split over four).
static DenseShape choose_dense_shape(int64_t batch, int64_t M, int64_t N, int64_t k_blocks, double weight_bytes)
{
    const int v = g_shape_override.load(std::memory_order_relaxed);
    const int64_t sms = sm_count();
    const auto tiles = [&](int64_t rows, int64_t cols) { return batch * ((M + rows - 1) / rows) * ((N + cols - 1) / cols); };
    if (v == 1 || v == 2) {
        return {v, v == 1 && tiles(128, 256) < sms ? 128 : 256, 1};
    }
    const double kb = static_cast<double>(k_blocks), weights = weight_bytes * 1e-6 / 5.5;
    const auto estimate = [&](int64_t count, int64_t workers, double tile, double besides) {
        return std::max(static_cast<double>((count + workers - 1) / workers) * tile, weights) + besides;
    };
    const int64_t narrow = tiles(128, 128);
    const double quarters = static_cast<double>(std::min<int64_t>(4, (M + 31) / 32));
    DenseShape best{1, 128, 1};
    double least = estimate(narrow, sms, std::max(0.244 * kb, 1.8), 0.0);
    const auto offer = [&](const DenseShape& shape, double us) {
        if (us < least) {
            least = us;
            best = shape;
        }
    };
    offer({1, 256, 1}, estimate(tiles(128, 256), sms, std::max(0.356 * kb, 3.1), 0.5));
    offer({2, 256, 1}, estimate(tiles(256, 256), sms / 2, std::max(0.245 * kb, 3.3), 3.0));
    for (int split : {2, 4}) {
        // no share of a tile's K blocks may be empty
        if (narrow * split <= std::min<int64_t>(sms, split == 4 ? 128 : sms) && k_blocks >= split) {
            const double share = static_cast<double>((k_blocks + split - 1) / split);
            offer({1, 128, split}, std::max(share * 0.244, weights) + 0.8 + quarters * (split == 2 ? 0.55 : 0.83));
        }
    }
    return best;
}

// Grouped problems: single CTAs on 128-row tiles, CTA pairs on 256-row tiles, or both in two launches - pairs on every
// group's 256-row blocks (the last one partial when it holds more than 128 rows) and singles on leftovers of at most 128
// rows, which pads the least and takes the least energy, but starts and ends twice.  The shape is the one with the
// smallest of three estimates, in us: waves of tiles over the SMs, a tile taking its K blocks (0.405 on a single CTA,
// 0.326 on a pair) or its epilogue (2.7, 3.15) if that is longer; no less than the touched groups' weights at 7.7 TB/s; and
// what the shape costs besides (2.5 for pairs, 20 for two launches, whose leftovers partly overlap the pairs: 0.55 of
// their time counts).  Fitted to 290 problems of 200 - 65000 rows, 4 - 128 groups, int8 and 16-bit, both epilogues, each
// timed under load in all three shapes: 0.2 % from the best shape of each on average and 6 % at worst.  Two launches from
// 2048 rows on, as the rule was, are 6.4 % from it on average and 52 % at worst (3000 rows of 8 groups of 2048 x 4096 bf16
// 74 us, 59 on single CTAs; SwiGLU form, 6000 of 8 of 4096 x 2048 69, 58).  Of a device list only the rows and the number of
// groups are known here: even groups with remainders of all sizes are assumed (0.8 % and 31 % on the same problems).
// Where one wave of narrow tiles holds the whole problem (`n_narrow` > 0 of them side by side: not for the SwiGLU epilogue,
// whose tile is 128 gate and 128 up columns), they are one more candidate, 0.244 a K block and 1.8 an epilogue as in the
// dense estimate: 64 rows of 4 groups of 512 x 512 bf16 5.2 us (6.6 on wide tiles), 200 of 8 of 1024 x 2048 10.3 (12.4), 500 of
// 8 of 2048 x 1024 12.8 (17.1), 200 of 8 of 4000 x 2048 29.4 (35.9).
static int choose_grouped_shape(const int64_t* host_ends, int64_t E, int64_t M, int64_t n_tiles, int64_t n_narrow,
                                int64_t k_blocks, double group_weight_bytes)
{
    const int v = g_shape_override.load(std::memory_order_relaxed);
    if (v != 0) {
        return v;
    }
    double singles = 0, pairs = 0, whole = 0, leftover = 0, touched = 0;  // row tiles of the three shapes
    if (host_ends != nullptr) {
        int64_t prev = 0;
        for (int64_t g = 0; g < E; ++g) {
            const int64_t rows = host_ends[g] - prev, rest = rows % 256;
            prev = host_ends[g];
            singles += static_cast<double>((rows + 127) / 128);
            pairs += static_cast<double>((rows + 255) / 256);
            whole += static_cast<double>(rows / 256 + (rest > 128 ? 1 : 0));
            leftover += (rest > 0 && rest <= 128) ? 1 : 0;
            touched += rows > 0 ? 1 : 0;
        }
    } else {
        const double e = static_cast<double>(E), m = static_cast<double>(M);
        touched = std::min(e, m);
        if (M >= 256 * E) {
            singles = m / 128 + e / 2;
            pairs = m / 256 + e / 2;
            whole = m / 256;
            leftover = e / 2;
        } else {
            singles = M > 128 * E ? 2 * e : touched;
            pairs = touched;
            whole = M > 128 * E ? e : 0;
            leftover = touched - whole;
        }
    }
    const double sms = sm_count(), nt = static_cast<double>(n_tiles), kb = static_cast<double>(k_blocks);
    const double single_tile = std::max(0.405 * kb, 2.7), pair_tile = std::max(0.326 * kb, 3.15);
    const double weights = touched * group_weight_bytes * 1e-6 / 7.7;
    const double t1 = std::max(std::ceil(singles * nt / sms) * single_tile, weights);
    const double t2 = std::max(std::ceil(pairs * nt / (sms / 2)) * pair_tile, weights) + 2.5;
    const double t3 =
        std::max(std::ceil(whole * nt / (sms / 2)) * pair_tile + leftover * nt / sms * single_tile * 0.55, weights) + 20.0;
    const double t4 = std::max(std::max(0.244 * kb, 1.8), weights);
    if (n_narrow > 0 && singles * static_cast<double>(n_narrow) <= sms && t4 < std::min({t1, t2, t3})) {
        return GEMM_SHAPE_NARROW;
    }
    return t1 <= t2 && t1 <= t3 ? 1 : (t2 <= t3 ? 2 : GEMM_SHAPE_HYBRID);
}

// ---------------------------------------------------------------------------
// Group planner: cumulative group list -> table of row tiles (128 rows for single CTAs, 256 for CTA pairs).
// The list arrives by value (host lists, validated by the caller) or from
// device memory (validated here; an invalid list yields zero tiles and
// error = 1).
// ---------------------------------------------------------------------------
constexpr int PLAN_MAX_BY_VALUE = 1024;
struct GroupEndsByValue {
    int32_t ends[PLAN_MAX_BY_VALUE];
};

__device__ __forceinline__ void plan_groups_body(int64_t zero, const int64_t* dev_list,
                                                 const GroupEndsByValue& by_value, int use_by_value, int64_t E,
                                                 int64_t M, GroupedHeader* header, TileEntry* tiles,
                                                 int64_t max_tiles, int tile_m, int mode, int allow_prefix)
{
    extern __shared__ int32_t s_first[];  // first tile index of each group, E + 1 entries
    __shared__ int32_t s_warp_sum[8];
    __shared__ int s_bad;
    __shared__ int32_t s_carry;
    auto end_of = [&](int64_t g) -> int64_t {
        return use_by_value ? static_cast<int64_t>(by_value.ends[g]) : dev_list[g];
    };
    const int tid = static_cast<int>(threadIdx.x + zero);
    const int lane = tid & 31;
    const int wid = tid >> 5;
    if (tid == 0) {
        s_bad = 0;
        s_carry = 0;
    }
    __syncthreads();
    // groups in chunks of 256: validate, count tiles, block-wide exclusive scan
    for (int64_t base = 0; base < E; base += 256) {
        const int64_t g = base + tid;
        int32_t cnt = 0;
        if (g < E) {
            const int64_t prev = (g == 0) ? 0 : end_of(g - 1);
            const int64_t e = end_of(g);
            if (e < prev || e > M || (g == E - 1 && e != M && !allow_prefix)) {
                s_bad = 1;
            } else {
                cnt = group_tiles(static_cast<uint32_t>(e - prev), static_cast<uint32_t>(tile_m), mode);
            }
        }
        int32_t incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int32_t v = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) {
                incl += v;
            }
        }
        if (lane == 31) {
            s_warp_sum[wid] = incl;
        }
        __syncthreads();
        int32_t warp_off = 0;
        for (int w = 0; w < wid; ++w) {
            warp_off += s_warp_sum[w];
        }
        const int32_t carry = s_carry;
        if (g < E) {
            s_first[g] = carry + warp_off + incl - cnt;
        }
        __syncthreads();
        if (tid == 255) {
            s_carry = carry + warp_off + incl;
        }
        __syncthreads();
    }
    const int32_t total = s_carry;
    const int bad = (s_bad != 0 || total > max_tiles) ? 1 : 0;
    if (tid == 0) {
        s_first[E] = total;
        header->num_m_tiles = bad ? 0 : total;
        header->error = bad;
        header->rows_total = bad ? 0 : static_cast<int32_t>(end_of(E - 1));
    }
    __syncthreads();
    if (bad) {
        return;
    }
    // a thread per tile looks up its group (the last one whose first tile is at or before it; groups without tiles
    // share their first tile with the next one, and s_first[E] = total ends the search): 3.5 us for 512 rows of 256
    // experts, 10 with a warp per group in turn, whose loads of the list waited for one another
    for (int32_t i = tid; i < total; i += 256) {
        int lo = 0, hi = static_cast<int>(E);
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_first[mid] <= i) {
                lo = mid;
            } else {
                hi = mid;
            }
        }
        tiles[i] = group_tile(lo, lo == 0 ? 0 : end_of(lo - 1), end_of(lo), i - s_first[lo], tile_m, mode);
    }
}

__global__ void __launch_bounds__(256) plan_groups_kernel(const int64_t* dev_list,
                                                          const GroupEndsByValue by_value, int use_by_value,
                                                          int64_t E, int64_t M, GroupedHeader* header,
                                                          TileEntry* tiles, int64_t max_tiles, int tile_m,
                                                          int allow_prefix)
{
    const int64_t zero = after_previous();
    plan_groups_body(zero, dev_list, by_value, use_by_value, E, M, header, tiles, max_tiles, tile_m, PLAN_ALL, allow_prefix);
}

__global__ void __launch_bounds__(256) zero_words_kernel(uint4* __restrict__ words, int64_t count)
{
    const int64_t zero = after_previous();
    const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = zero + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += step) {
        words[i] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// Both tile tables of the two-launch form in one launch: CTA 0 plans the 256-row blocks, CTA 1 the leftovers of at
// most 128 rows (each validates the list itself; the leftover table cannot overflow, every group adds at most one
// tile to it), and the remaining CTAs zero `clear16` 16-byte words at `clear` (row maxima and tile counters of the
// SwiGLU form), which saves a second planner launch and a memset per call.
constexpr int PLAN_CLEAR_CTAS = 30;

__global__ void __launch_bounds__(256) plan_groups_both_kernel(const int64_t* dev_list,
                                                               const GroupEndsByValue by_value, int use_by_value,
                                                               int64_t E, int64_t M, GroupedHeader* header,
                                                               TileEntry* tiles, int64_t max_tiles,
                                                               GroupedHeader* tail_header, TileEntry* tail_tiles,
                                                               int64_t tail_max_tiles, int allow_prefix,
                                                               uint4* __restrict__ clear, int64_t clear16)
{
    const int64_t zero = after_previous();
    if (blockIdx.x == 0) {
        plan_groups_body(zero, dev_list, by_value, use_by_value, E, M, header, tiles, max_tiles, 256, PLAN_WHOLE,
                         allow_prefix);
    } else if (blockIdx.x == 1) {
        plan_groups_body(zero, dev_list, by_value, use_by_value, E, M, tail_header, tail_tiles, tail_max_tiles, 128,
                         PLAN_LEFTOVER, allow_prefix);
    } else {
        const int64_t stride = static_cast<int64_t>(gridDim.x - 2) * blockDim.x;
        for (int64_t i = static_cast<int64_t>(blockIdx.x - 2) * blockDim.x + threadIdx.x; i < clear16; i += stride) {
            clear[i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
}

// ---------------------------------------------------------------------------
// Requantisation of the SwiGLU activations (second, bandwidth-bound half of grouped_matmul_swiglu_quant): a CTA holds a row
// in registers between its maximum and its quantisation, so the matmul keeps no maxima and nothing has to be zeroed for them.
// Bound: HBM (5 H bytes per row).  131072 x 2048 198 us, 40000 x 1792 56, 8000 x 512 5.5, 64 x 2048 1.8; with two pieces per
// thread 248, 71, 7.9, 1.8, with eight 209, 56, 6.5, 2.0.  The operator: 64 rows of 8 experts of 1024 x 1024 10.7 us (12.1 with a
// zeroing kernel ahead, a maximum per row and column tile kept by the matmul, and warps that read it), 100 of 8 of 4096 x 2048
// 22.4 (24.2), 40000 of 32 of 1280 x 3584 312 (320).
// CPT: 16-byte pieces of the row per thread; 0: rows of any length, read twice (the second time from L2).
// ---------------------------------------------------------------------------
template <bool DIRECT, int CPT>
__global__ void __launch_bounds__(1024) gmsq_requant_kernel(const float* act, int8_t* __restrict__ y,
                                                            float* __restrict__ y_scale, int64_t M, int64_t H,
                                                            const GroupedHeader* header)
{
    __shared__ int s_max[2][32];
    const int64_t zero = after_previous();
    if (header->error != 0) {
        return;
    }
    const int64_t rows = min(M, static_cast<int64_t>(header->rows_total));  // a device list may end before M
    const int tid = threadIdx.x, threads = blockDim.x, lane = tid & 31, warps = threads >> 5;
    const int64_t n4 = H / 4;
    int parity = 0;
    for (int64_t row = blockIdx.x + zero; row < rows; row += gridDim.x, parity ^= 1) {
        const float4* src = reinterpret_cast<const float4*>(act + row * H);
        uint32_t* dst = reinterpret_cast<uint32_t*>(y + row * H);
        constexpr int HELD = CPT > 0 ? CPT : 1;
        float4 a[HELD];
        float m = 0.0f;
        if constexpr (CPT > 0) {
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
                const int c = tid + i * threads;
                a[i] = c < n4 ? __ldcs(src + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
                m = requant_max4(m, a[i]);
            }
        } else {
            for (int64_t c = tid; c < n4; c += threads) {
                m = requant_max4(m, src[c]);
            }
        }
        // magnitudes order like their bit patterns
        const int own = __reduce_max_sync(FULL_MASK, __float_as_int(m));
        if (lane == 0) {
            s_max[parity][tid >> 5] = own;
        }
        __syncthreads();
        const int top = __reduce_max_sync(FULL_MASK, lane < warps ? s_max[parity][lane] : 0);
        const float amax = requant_amax(__int_as_float(top));
        if (tid == 0) {
            y_scale[row] = __fmul_rn(amax, INV127);
        }
        const float inv = __fdiv_rn(127.0f, amax);
        if constexpr (CPT > 0) {
#pragma unroll
            for (int i = 0; i < CPT; ++i) {
                const int c = tid + i * threads;
                if (c < n4) {
                    __stcs(dst + c, requant4<DIRECT>(a[i], inv));
                }
            }
        } else {
            for (int64_t c = tid; c < n4; c += threads) {
                __stcs(dst + c, requant4<DIRECT>(src[c], inv));
            }
        }
    }
}

template <bool DIRECT>
static cudaError_t requant(const float* act, int8_t* y, float* y_scale, int64_t M, int64_t H, const GroupedHeader* header,
                           cudaStream_t st)
{
    constexpr int CPT = 4;
    const int64_t n4 = H / 4;
    const bool held = n4 <= 1024 * CPT;
    const int threads = held ? static_cast<int>((n4 + 32 * CPT - 1) / (32 * CPT)) * 32 : 1024;
    auto kern = held ? gmsq_requant_kernel<DIRECT, CPT> : gmsq_requant_kernel<DIRECT, 0>;
    const int64_t cap = static_cast<int64_t>(sm_count()) * std::min(32, std::max(1, 65536 / (40 * threads)));  // 37 registers
    return launch_chained(kern, static_cast<unsigned>(std::min(M, cap)), static_cast<unsigned>(threads), 0, st, act, y, y_scale,
                          M, H, header);
}

static inline size_t align_up_sz(size_t v, size_t a) { return (v + a - 1) / a * a; }

// ---------------------------------------------------------------------------
// fp32 operands on the bf16 tensor path (gemm_kernel.cuh): each operand is split once into SPLIT_PIECES arrays of bf16
// pieces.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void split3(float v, __nv_bfloat16 (&piece)[3])
{
    piece[0] = __float2bfloat16_rn(v);
    const float r1 = __fsub_rn(v, __bfloat162float(piece[0]));
    piece[1] = __float2bfloat16_rn(r1);
    const float r2 = __fsub_rn(r1, __bfloat162float(piece[1]));
    piece[2] = __float2bfloat16_rn(r2);
}

// The pieces of eight consecutive values as three 16-byte words (hi, mid, lo)
__device__ __forceinline__ void split8(const float* src, uint4 (&word)[3])
{
    const float4 a = __ldcs(reinterpret_cast<const float4*>(src)), b = __ldcs(reinterpret_cast<const float4*>(src) + 1);
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    __nv_bfloat16 piece[3][8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        __nv_bfloat16 p[3];
        split3(v[j], p);
        piece[0][j] = p[0], piece[1][j] = p[1], piece[2][j] = p[2];
    }
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            w[j] = static_cast<uint32_t>(__bfloat16_as_ushort(piece[t][2 * j])) |
                   (static_cast<uint32_t>(__bfloat16_as_ushort(piece[t][2 * j + 1])) << 16);
        }
        word[t] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// src: `blocks` blocks of `len` fp32 values (a row of x, or an expert's weight) -> dst: per block, its hi, its mid
// and its lo pieces, `len` bf16 values each.  `len` is a multiple of 8 and both ends are 16-byte aligned (K of the
// operator is a multiple of 8).
// Bound: HBM (10 bytes per value).  With every piece stored once and found by the matmul's producer through its map,
// instead of six copies laid out along K (16 bytes per value, twice the workspace): 8 experts of 4096 x 4096 with 1000
// rows, matmul included, 629 us (769 before); 32 of 1024 x 2048 with 333 rows 241 (324); 32 of 4096 x 7168 with 2000
// rows 3.47 ms (4.45); 16000 rows, bound by the six products, 2.62 (2.90).
__global__ void __launch_bounds__(256) split_blocks_kernel(const float* src, __nv_bfloat16* __restrict__ dst,
                                                           int64_t blocks, int64_t len)
{
    const int64_t zero = after_previous();
    const int64_t n8 = len / 8, total = blocks * n8;
    const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = zero + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
        const int64_t r = i / n8, c = i - r * n8;
        uint4 w[SPLIT_PIECES];
        split8(src + i * 8, w);
        uint4* out = reinterpret_cast<uint4*>(dst + r * (SPLIT_PIECES * len)) + c;
#pragma unroll
        for (int t = 0; t < SPLIT_PIECES; ++t) {
            out[t * n8] = w[t];
        }
    }
}

struct GroupedWorkspace {
    GroupedHeader* header;
    TileEntry* tiles;
    int64_t max_tiles;
    uint32_t* amax;
    float* act;
    // second tile table: what a group leaves over after its 256-row blocks when that is at most 128 rows (one tile
    // per group), used when the blocks run on CTA pairs and these leftovers on single CTAs
    GroupedHeader* tail_header;
    TileEntry* tail_tiles;
    int64_t tail_max_tiles;
    // finished-column-tile counters of the fused requantisation, one per (row tile, CTA of the tile): for the first
    // table, then for the tail table; they follow the row maxima so that one memset clears both
    int32_t* tile_done;
    int32_t* tail_tile_done;
    size_t clear_bytes;  // from `amax`: row maxima + counters
    size_t total;
};

static GroupedWorkspace carve_workspace(void* ws, int64_t M, int64_t E, int64_t act_cols)
{
    GroupedWorkspace g;
    uint8_t* p = static_cast<uint8_t*>(ws);
    size_t off = 0;
    g.header = reinterpret_cast<GroupedHeader*>(p + off);
    off += align_up_sz(sizeof(GroupedHeader), 256);
    g.max_tiles = M / GEMM_BLOCK_M + E + 1;
    g.tiles = reinterpret_cast<TileEntry*>(p + off);
    off += align_up_sz(static_cast<size_t>(g.max_tiles) * sizeof(TileEntry), 256);
    g.amax = reinterpret_cast<uint32_t*>(p + off);
    const size_t clear_from = off;
    off += (act_cols > 0) ? align_up_sz(static_cast<size_t>(M) * sizeof(uint32_t), 256) : 0;
    g.tile_done = reinterpret_cast<int32_t*>(p + off);
    off += (act_cols > 0) ? align_up_sz(static_cast<size_t>(g.max_tiles) * 2 * sizeof(int32_t), 256) : 0;
    g.tail_tile_done = reinterpret_cast<int32_t*>(p + off);
    off += (act_cols > 0) ? align_up_sz(static_cast<size_t>(E + 1) * 2 * sizeof(int32_t), 256) : 0;
    g.clear_bytes = off - clear_from;
    g.act = reinterpret_cast<float*>(p + off);
    off += (act_cols > 0) ? align_up_sz(static_cast<size_t>(M) * act_cols * sizeof(float), 256) : 0;
    g.tail_header = reinterpret_cast<GroupedHeader*>(p + off);
    off += align_up_sz(sizeof(GroupedHeader), 256);
    g.tail_max_tiles = E + 1;
    g.tail_tiles = reinterpret_cast<TileEntry*>(p + off);
    off += align_up_sz(static_cast<size_t>(g.tail_max_tiles) * sizeof(TileEntry), 256);
    g.total = off;
    return g;
}

// A host group list is checked before any CUDA call is made for the operator.
static int check_host_group_list(const int64_t* group_list, int list_on_device, int64_t E, int64_t M)
{
    if (list_on_device < 0 || list_on_device > 2) {
        return W8A8_ERR_INVALID;
    }
    if (list_on_device) {
        return W8A8_OK;
    }
    if (E > PLAN_MAX_BY_VALUE) {
        return W8A8_ERR_UNSUPPORTED;
    }
    int64_t prev = 0;
    for (int64_t i = 0; i < E; ++i) {
        const int64_t v = group_list[i];
        if (v < prev || v > M) {
            return W8A8_ERR_GROUP_LIST;
        }
        prev = v;
    }
    return (prev == M) ? W8A8_OK : W8A8_ERR_GROUP_LIST;
}

// returns W8A8_OK or an error; launches the planner on `st`: of one table with tiles of tile_m rows, or of `both` tables of
// the two-launch form, which zeroes `clear` too
static int plan_groups(const int64_t* group_list, int list_on_device, int64_t E, int64_t M, const GroupedWorkspace& g,
                       cudaStream_t st, int tile_m, bool both = false, void* clear = nullptr, size_t clear_bytes = 0)
{
    GroupEndsByValue bv;
    int use_bv = 0;
    const int64_t* dev_list = group_list;
    if (!list_on_device) {
        if (E > PLAN_MAX_BY_VALUE) {
            return W8A8_ERR_UNSUPPORTED;
        }
        int64_t prev = 0;
        for (int64_t i = 0; i < E; ++i) {
            const int64_t v = group_list[i];
            if (v < prev || v > M) {
                return W8A8_ERR_GROUP_LIST;
            }
            bv.ends[i] = static_cast<int32_t>(v);
            prev = v;
        }
        if (prev != M) {
            return W8A8_ERR_GROUP_LIST;
        }
        for (int64_t i = E; i < PLAN_MAX_BY_VALUE; ++i) {
            bv.ends[i] = 0;
        }
        use_bv = 1;
        dev_list = nullptr;
    }
    const size_t smem = static_cast<size_t>(E + 1) * sizeof(int32_t);
    if (smem > 48 * 1024) {
        return W8A8_ERR_UNSUPPORTED;
    }
    cudaError_t e;
    if (both) {
        const int64_t clear16 = static_cast<int64_t>(clear_bytes / 16);
        const unsigned grid = 2 + (clear16 > 0 ? PLAN_CLEAR_CTAS : 0);
        e = launch_chained(plan_groups_both_kernel, grid, 256, smem, st, dev_list, bv, use_bv, E, M, g.header, g.tiles,
                           g.max_tiles, g.tail_header, g.tail_tiles, g.tail_max_tiles, list_on_device == 2 ? 1 : 0,
                           static_cast<uint4*>(clear), clear16);
    } else {
        e = launch_chained(plan_groups_kernel, 1, 256, smem, st, dev_list, bv, use_bv, E, M, g.header, g.tiles, g.max_tiles,
                           tile_m, list_on_device == 2 ? 1 : 0);
    }
    return launch_status(e);
}

// Runs a grouped problem whose GemmParams are filled in except for the tile table: plans the groups and launches
// the kernel shape(s) choose_grouped_shape picked.
template <int KIND, int EPI>
static int run_grouped(const int64_t* group_list, int list_on_device, int64_t E, int64_t M, const GroupedWorkspace& g,
                       bool b_mn, const void* a, const CUtensorMap& tb, GemmParams p, cudaStream_t st,
                       void* clear = nullptr, size_t clear_bytes = 0)
{
    constexpr int64_t ELEM = (KIND == KIND_I8) ? 1 : 2;
    const bool split = p.k_blocks_per_term != 0;
    const int64_t a_cols = split ? SPLIT_PIECES * p.K : p.K;
    const int64_t group_bytes = p.N * p.K * ELEM * (split ? SPLIT_TERMS : 1);  // of weights, as the kernel streams them
    const int64_t n_narrow = (EPI == EPI_GMM && p.out_row_ptrs == nullptr) ? (p.N + 127) / 128 : 0;
    const int chosen = choose_grouped_shape(list_on_device ? nullptr : group_list, E, M, p.n_tiles, n_narrow, p.num_k_blocks,
                                            static_cast<double>(group_bytes));
    const bool narrow = chosen == GEMM_SHAPE_NARROW;
    const int shape = narrow ? 1 : chosen;
    if (narrow) {
        p.n_tiles = static_cast<int32_t>(n_narrow);
    }
    p.error = &g.header->error;
    // Rows per A load.  Pairs take whole tiles.  A single CTA's tile holds at most 128 rows of one group and often far
    // fewer - what a group leaves over, or a whole group of a small batch.  Where there are 256 MB of weights to stream
    // it loads its own rows in boxes of 32 or 16 instead of 128 rows that are mostly another group's, and multiplies
    // what the stages hold below them - zeros, as long as no taller tile of the CTA has used them: 512 rows of 256
    // experts (7168 x 4096 and 2048 x 7168) 1.55 ms back to back, 1.80 before (the SM clock held near 0.8 GHz by the
    // power cap), 1.44 and 1.53 from rest; 1500 rows of 32 experts of 2048 x 7168 bf16 161 us, 165.  Smaller problems do
    // not pay for clearing the stages and the longer loop (512 rows of 32 experts of 2048 x 2048: 38.7 us, 37.6).
    // Calls that the cap does not bound gain little - 64 experts of 4096 x 4096, 4 - 64 rows each: 152.8 - 182.8 us,
    // 153.7 - 184 with whole tiles - the same with boxes of 16 and of 32, and nothing from 96 rows per expert on, which
    // is where the rule ends; at 12 rows per expert most tiles still fit into one box of 16.
    int box_rows = (shape == GEMM_SHAPE_HYBRID) ? 32 : (M <= 12 * E ? 16 : (M <= 96 * E ? 32 : GEMM_BLOCK_M));
    if (shape == 2 || narrow || E * group_bytes < (int64_t(256) << 20)) {
        box_rows = GEMM_BLOCK_M;
    }
    const bool row_boxes = box_rows < GEMM_BLOCK_M;
    CUtensorMap ta;
    p.a_box_rows = (shape == 1) ? box_rows : GEMM_BLOCK_M;
    if (!make_map_a(&ta, a, M, a_cols, KIND, p.a_box_rows)) {
        return W8A8_ERR_CUDA;
    }
    // Up to GROUPS_IN_CTA groups every CTA of the matmul plans its tiles itself; more take a table, planned by a kernel of
    // its own.  `clear` (the SwiGLU form's row maxima and tile counters) must be zero before the first matmul launch: a
    // kernel zeroes it, the planner's own launch where that builds two tables.
    const bool hybrid = shape == GEMM_SHAPE_HYBRID;
    GroupList groups{};
    if (E <= GROUPS_IN_CTA) {
        groups.E = static_cast<int32_t>(E);
        groups.allow_prefix = list_on_device == 2 ? 1 : 0;
        groups.mode = hybrid ? PLAN_WHOLE : PLAN_ALL;
        groups.tile_m = hybrid ? 256 : 128 * shape;
        if (list_on_device) {
            groups.dev = group_list;
        } else {
            std::copy(group_list, group_list + E, groups.ends);  // checked by the caller
        }
    }
    if (clear_bytes != 0 && (E <= GROUPS_IN_CTA || !hybrid)) {
        const int64_t words = static_cast<int64_t>(clear_bytes / 16);
        const unsigned ctas = static_cast<unsigned>(std::min<int64_t>((words + 255) / 256, sm_count()));
        const cudaError_t e = launch_chained(zero_words_kernel, ctas, 256, 0, st, static_cast<uint4*>(clear), words);
        if (e != cudaSuccess) {
            return launch_status(e);
        }
    }
    if (E > GROUPS_IN_CTA) {
        const int rc = hybrid ? plan_groups(group_list, list_on_device, E, M, g, st, 256, true, clear, clear_bytes)
                              : plan_groups(group_list, list_on_device, E, M, g, st, 128 * shape);
        if (rc != W8A8_OK) {
            return rc;
        }
    }
    p.tiles = g.tiles;
    p.header = g.header;
    p.tile_done = g.tile_done;
    // (with a table of its own the second launch would read what the planner wrote: it waits)
    const bool overlap = hybrid && E <= GROUPS_IN_CTA;
    // The SwiGLU form on single CTAs, with enough weights to be long, starts on an idle chip: launched beside the kernel
    // before, its CTAs come to lie on the SMs as those fall free, and neighbouring column tiles no longer on the two SMs of a
    // TPC, which share what they fetch.  9328 rows of 128 experts of 4784 x 2752 326 us (413 overlapped), 2296 of 128 of
    // 2464 x 3360 196 (231), 20000 of 64 of 4096 x 2048 237 (244), 3000 of 32 of 7168 x 4096 201 (199); shorter calls lose
    // the 2 us of the overlap (600 rows of 32 experts of 4096 x 2912, 381 MB: 80.7, 79.0).  The other epilogue, whose tiles
    // are 256 contiguous columns, shows no difference.
    const bool plain = EPI == EPI_GMSQ && shape == 1 && E * group_bytes >= int64_t(400000000);
    p.order = overlap ? ORDER_FIRST_OF_TWO : (plain ? ORDER_PLAIN : ORDER_ALONE);
    const int64_t most = (hybrid ? M / 256 + E + 1 : g.max_tiles) * p.n_tiles;
    cudaError_t e = (!hybrid && row_boxes) ? dispatch_row_boxes<KIND, EPI>(b_mn, ta, tb, p, most, st, groups)
                                           : dispatch_gemm<KIND, EPI>(hybrid ? 2 : shape, narrow ? 128 : 256, b_mn, ta, tb, p, most, st, groups);
    if (e != cudaSuccess || !hybrid) {
        return launch_status(e);
    }
    p.tiles = g.tail_tiles;
    p.header = g.tail_header;
    p.tile_done = g.tail_tile_done;
    p.order = overlap ? ORDER_SECOND_OF_TWO : ORDER_ALONE;
    groups.mode = PLAN_LEFTOVER;
    groups.tile_m = 128;
    const int64_t tail_most = g.tail_max_tiles * p.n_tiles;
    if (row_boxes) {
        p.a_box_rows = box_rows;
        if (!make_map_a(&ta, a, M, a_cols, KIND, box_rows)) {
            return W8A8_ERR_CUDA;
        }
        e = dispatch_row_boxes<KIND, EPI>(b_mn, ta, tb, p, tail_most, st, groups);
    } else {
        e = dispatch_gemm<KIND, EPI>(1, 256, b_mn, ta, tb, p, tail_most, st, groups);
    }
    return launch_status(e);
}

// ---------------------------------------------------------------------------
// Error word of launches that have no workspace to carry one (the dense matmuls): one int32 in the library's
// device image per GPU.  A kernel whose bounded wait ran out stores 2 there; w8a8_pipeline_error() reads and
// clears it.  The address is looked up once per device, with that device current.
// ---------------------------------------------------------------------------
static __device__ int32_t g_pipeline_error_word;

static int32_t* pipeline_error_word()
{
    constexpr int MAX_DEVICES = 64;
    static std::atomic<int32_t*> cache[MAX_DEVICES];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) {
        return nullptr;
    }
    int32_t* p = cache[dev].load(std::memory_order_relaxed);
    if (p == nullptr) {
        void* sym = nullptr;
        if (cudaGetSymbolAddress(&sym, g_pipeline_error_word) != cudaSuccess) {
            return nullptr;
        }
        p = static_cast<int32_t*>(sym);
        cache[dev].store(p, std::memory_order_relaxed);
    }
    return p;
}

}  // namespace w8a8

using namespace w8a8;

// ===========================================================================
// quant_matmul
// ===========================================================================
// The epilogues read per-channel vectors in 16-byte pieces from their first element on (see load_vec), each batch's bias
// from its own; a single value and the rows' factors are read as what they are.
static bool qmm_vectors_aligned(const void* scale, const float* offset, const float* pertoken, const void* bias,
                                int64_t flags, int64_t batch, int64_t bias_batch_stride)
{
    const size_t scale_size = (flags & W8A8_QM_SCALE_BF16) ? 2 : 4;
    if (!is_aligned(scale, (flags & W8A8_QM_SCALE_PERCHAN) ? 16 : scale_size)) {
        return false;
    }
    if ((flags & W8A8_QM_HAS_OFFSET) && !is_aligned(offset, (flags & W8A8_QM_OFFSET_PERCHAN) ? 16 : 4)) {
        return false;
    }
    if ((flags & W8A8_QM_HAS_PT) && !is_aligned(pertoken, 4)) {
        return false;
    }
    const int64_t bias_kind = (flags & W8A8_QM_BIAS_MASK) >> W8A8_QM_BIAS_SHIFT;
    if (bias_kind == W8A8_QM_BIAS_NONE) {
        return true;
    }
    const int64_t bias_size = (bias_kind == W8A8_QM_BIAS_F16 || bias_kind == W8A8_QM_BIAS_BF16) ? 2 : 4;
    if (!(flags & W8A8_QM_BIAS_PERCHAN)) {
        return is_aligned(bias, static_cast<size_t>(bias_size));
    }
    return is_aligned(bias, 16) && (batch == 1 || (bias_batch_stride * bias_size) % 16 == 0);
}

static int quant_matmul_impl(const int8_t* x1, const int8_t* x2, const void* scale, const float* offset,
                             const float* pertoken, const void* bias, void* out, int64_t batch, int64_t M, int64_t N,
                             int64_t K, int64_t flags, int out_dtype, int x2_layout, int64_t bias_batch_stride,
                             bool raw_i32, void* stream)
{
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) {
        return W8A8_ERR_INVALID;  // quant_matmul_plugin.cpp:100 "requires non-empty shapes"
    }
    if (x1 == nullptr || x2 == nullptr || out == nullptr) {
        return W8A8_ERR_INVALID;
    }
    if (x2_layout != W8A8_W_KN && x2_layout != W8A8_W_NK) {
        return W8A8_ERR_INVALID;
    }
    if (!raw_i32) {
        if (scale == nullptr || (out_dtype != W8A8_DT_F16 && out_dtype != W8A8_DT_BF16)) {
            return W8A8_ERR_INVALID;
        }
        const int64_t bias_kind = (flags & W8A8_QM_BIAS_MASK) >> W8A8_QM_BIAS_SHIFT;
        if (bias_kind > W8A8_QM_BIAS_F32 || (bias_kind != W8A8_QM_BIAS_NONE && bias == nullptr)) {
            return W8A8_ERR_INVALID;
        }
        if (((flags & W8A8_QM_HAS_OFFSET) && offset == nullptr) || ((flags & W8A8_QM_HAS_PT) && pertoken == nullptr)) {
            return W8A8_ERR_INVALID;
        }
    }
    if ((K % 16) != 0 || (N % 16) != 0) {
        return W8A8_ERR_UNSUPPORTED;
    }
    if (!is_aligned(x1, 16) || !is_aligned(x2, 16) || !is_aligned(out, 16)) {
        return W8A8_ERR_ALIGN;
    }
    if (!raw_i32 && !qmm_vectors_aligned(scale, offset, pertoken, bias, flags, batch, bias_batch_stride)) {
        return W8A8_ERR_ALIGN;
    }
    if (batch * M >= (int64_t(1) << 31) || N >= (int64_t(1) << 31) || K >= (int64_t(1) << 31)) {
        return W8A8_ERR_UNSUPPORTED;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool b_mn = (x2_layout == W8A8_W_KN);
    // With fewer than 128 rows in all, the A load only brings the rows that exist (rounded up to 8): the rest of the
    // 128-row shared-memory tile keeps whatever it held, which only reaches accumulator rows the epilogue never stores.
    const int a_box_rows = (batch * M < 128) ? static_cast<int>((batch * M + 7) / 8 * 8) : 128;
    CUtensorMap ta, tb;
    if (!make_map_a(&ta, x1, batch * M, K, KIND_I8, a_box_rows) || !make_map_b(&tb, x2, batch, N, K, KIND_I8, b_mn)) {
        return W8A8_ERR_CUDA;
    }
    GemmParams p{};
    p.a_box_rows = a_box_rows;
    p.M = M;
    p.N = N;
    p.K = K;
    p.num_k_blocks = static_cast<int32_t>((K + GEMM_KBYTES - 1) / GEMM_KBYTES);
    p.m_tiles_per_batch = static_cast<int32_t>((M + GEMM_BLOCK_M - 1) / GEMM_BLOCK_M);
    p.batch = static_cast<int32_t>(batch);
    p.scale = scale;
    p.offset = offset;
    p.row_scale = pertoken;
    p.bias = bias;
    p.out = out;
    p.flags = flags;
    p.out_dtype = out_dtype;
    p.bias_batch_stride = bias_batch_stride;
    p.prefetch_k_blocks = GEMM_PREFETCH_K_BLOCKS;
    p.error = pipeline_error_word();  // null (no report) only if the symbol lookup failed
    const DenseShape shape = choose_dense_shape(batch, M, N, p.num_k_blocks, static_cast<double>(batch * N * K));
    if (shape.split > 1) {
        p.split = shape.split;
        p.n_tiles = static_cast<int32_t>((N + 127) / 128);
        const int64_t tiles = batch * p.m_tiles_per_batch * p.n_tiles;
        cudaError_t e;
        if (raw_i32) {
            e = b_mn ? launch_gemm<1, 128, KIND_I8, EPI_RAW, true, 8, true>(ta, tb, p, tiles, st)
                     : launch_gemm<1, 128, KIND_I8, EPI_RAW, false, 8, true>(ta, tb, p, tiles, st);
        } else {
            e = b_mn ? launch_gemm<1, 128, KIND_I8, EPI_QMM, true, 8, true>(ta, tb, p, tiles, st)
                     : launch_gemm<1, 128, KIND_I8, EPI_QMM, false, 8, true>(ta, tb, p, tiles, st);
        }
        return launch_status(e);
    }
    const int cg = shape.cta_group, block_n = shape.block_n;
    const int tile_m = 128 * cg;
    p.m_tiles_per_batch = static_cast<int32_t>((M + tile_m - 1) / tile_m);
    const int64_t m_tiles = batch * p.m_tiles_per_batch;
    p.n_tiles = static_cast<int32_t>((N + block_n - 1) / block_n);
    const int64_t total = m_tiles * p.n_tiles;
    cudaError_t e;
    if (raw_i32) {
        e = dispatch_gemm<KIND_I8, EPI_RAW>(cg, block_n, b_mn, ta, tb, p, total, st);
    } else {
        e = dispatch_gemm<KIND_I8, EPI_QMM>(cg, block_n, b_mn, ta, tb, p, total, st);
    }
    return launch_status(e);
}

extern "C" int w8a8_quant_matmul(const int8_t* x1, const int8_t* x2, const void* scale, const float* offset,
                                 const float* pertoken, const void* bias, void* out, int64_t batch, int64_t M,
                                 int64_t N, int64_t K, int64_t flags, int out_dtype, int x2_layout,
                                 int64_t bias_batch_stride, void* stream)
{
    return quant_matmul_impl(x1, x2, scale, offset, pertoken, bias, out, batch, M, N, K, flags, out_dtype, x2_layout,
                             bias_batch_stride, false, stream);
}

extern "C" int w8a8_matmul_i8_i32(const int8_t* x1, const int8_t* x2, int32_t* c, int64_t batch, int64_t M, int64_t N,
                                  int64_t K, int x2_layout, void* stream)
{
    return quant_matmul_impl(x1, x2, nullptr, nullptr, nullptr, nullptr, c, batch, M, N, K, 0, 0, x2_layout, 0, true,
                             stream);
}

// ===========================================================================
// grouped_matmul_swiglu_quant
// ===========================================================================
extern "C" size_t w8a8_grouped_matmul_swiglu_quant_workspace_size(int64_t M, int64_t K, int64_t N, int64_t E)
{
    (void)K;
    if (M < 0 || N <= 0 || E <= 0) {
        return 0;
    }
    return carve_workspace(nullptr, M, E, N / 2).total;
}

extern "C" int w8a8_grouped_matmul_swiglu_quant(const int8_t* x, const int8_t* w, const float* w_scale,
                                                const float* x_scale, int8_t* y, float* y_scale, int64_t M, int64_t K,
                                                int64_t N, int64_t E, const int64_t* group_list, int list_on_device,
                                                int w_layout, int flags, void* workspace, size_t workspace_bytes,
                                                void* stream)
{
    if (M < 0 || K <= 0 || N <= 0 || E <= 0 || (N & 1) != 0) {
        return W8A8_ERR_INVALID;  // gmsq_plugin.cpp:52 "N must be even"
    }
    if ((flags & ~(W8A8_F_ROUND_DIRECT | W8A8_F_STAGE_MATMUL | W8A8_F_STAGE_REQUANT)) != 0 ||
        (w_layout != W8A8_W_KN && w_layout != W8A8_W_NK)) {
        return W8A8_ERR_INVALID;
    }
    const int stages = flags & (W8A8_F_STAGE_MATMUL | W8A8_F_STAGE_REQUANT);
    const bool run_matmul = (stages == 0) || (stages & W8A8_F_STAGE_MATMUL);
    const bool run_requant = (stages == 0) || (stages & W8A8_F_STAGE_REQUANT);
    if (M == 0) {
        return W8A8_OK;  // gmsq_plugin.cpp:93-95
    }
    if (x == nullptr || w == nullptr || w_scale == nullptr || x_scale == nullptr || y == nullptr ||
        y_scale == nullptr || group_list == nullptr) {
        return W8A8_ERR_INVALID;
    }
    if ((K % 16) != 0 || (N % 32) != 0) {
        return W8A8_ERR_UNSUPPORTED;
    }
    if (!is_aligned(x, 16) || !is_aligned(w, 16) || !is_aligned(w_scale, 16) || !is_aligned(x_scale, 4) || !is_aligned(y, 4) ||
        !is_aligned(y_scale, 4)) {
        return W8A8_ERR_ALIGN;
    }
    if (M >= (int64_t(1) << 31) - 256 || N >= (int64_t(1) << 31) || K >= (int64_t(1) << 31)) {
        return W8A8_ERR_UNSUPPORTED;
    }
    const int64_t H = N / 2;
    const size_t need = w8a8_grouped_matmul_swiglu_quant_workspace_size(M, K, N, E);
    if (workspace == nullptr || workspace_bytes < need) {
        return W8A8_ERR_WORKSPACE;
    }
    if (!is_aligned(workspace, 256)) {
        return W8A8_ERR_ALIGN;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const GroupedWorkspace g = carve_workspace(workspace, M, E, H);
    bool fused = false;
    if (run_matmul) {
        const int list_rc = check_host_group_list(group_list, list_on_device, E, M);
        if (list_rc != W8A8_OK) {
            return list_rc;
        }
        const bool b_mn = (w_layout == W8A8_W_KN);
        CUtensorMap tb;
        if (!make_map_b(&tb, w, E, N, K, KIND_I8, b_mn)) {
            return W8A8_ERR_CUDA;
        }
        GemmParams p{};
        p.M = M;
        p.N = N;
        p.K = K;
        p.num_k_blocks = static_cast<int32_t>((K + GEMM_KBYTES - 1) / GEMM_KBYTES);
        p.n_tiles = static_cast<int32_t>((H + 127) / 128);
        p.scale = w_scale;
        p.row_scale = x_scale;
        p.act = g.act;
        p.amax = g.amax;
        // Optional (off by default, it measures slower): the matmul kernels quantise each row block themselves as
        // soon as its last column tile is done, and no second kernel runs.
        // (a CTA waits for the other column tiles of its rows, which must then be running on other CTAs: only with
        // at least as many workers as column tiles)
        p.fuse_requant =
            (run_requant && g_fuse_requant.load(std::memory_order_relaxed) && p.n_tiles <= sm_count() / 2) ? 1 : 0;
        p.y = y;
        p.y_scale = y_scale;
        p.round_direct = (flags & W8A8_F_ROUND_DIRECT) ? 1 : 0;
        fused = p.fuse_requant != 0;
        // row maxima and finished-tile counters, where the matmul kernels requantise, start at zero
        const int rc = run_grouped<KIND_I8, EPI_GMSQ>(group_list, list_on_device, E, M, g, b_mn, x, tb, p, st,
                                                      fused ? g.amax : nullptr, fused ? g.clear_bytes : 0);
        if (rc != W8A8_OK) {
            return rc;
        }
    }
    if (!run_requant || fused) {
        return W8A8_OK;
    }
    const cudaError_t e = (flags & W8A8_F_ROUND_DIRECT) ? requant<true>(g.act, y, y_scale, M, H, g.header, st)
                                                        : requant<false>(g.act, y, y_scale, M, H, g.header, st);
    return launch_status(e);
}

// ===========================================================================
// grouped_matmul
// ===========================================================================
extern "C" size_t w8a8_grouped_matmul_workspace_size(int64_t M, int64_t N, int64_t K, int64_t E)
{
    (void)N;
    (void)K;
    if (M < 0 || E <= 0) {
        return 0;
    }
    return carve_workspace(nullptr, M, E, 0).total;
}

extern "C" size_t w8a8_grouped_matmul_f32_workspace_size(int64_t M, int64_t N, int64_t K, int64_t E)
{
    if (M < 0 || N <= 0 || K <= 0 || E <= 0) {
        return 0;
    }
    const size_t base = carve_workspace(nullptr, M, E, 0).total;
    const size_t xs = align_up_sz(static_cast<size_t>(M) * SPLIT_PIECES * K * 2, 256);
    const size_t ws = align_up_sz(static_cast<size_t>(E) * SPLIT_PIECES * K * N * 2, 256);
    return base + xs + ws;
}

static int grouped_matmul_impl(const void* x, const void* w, const void* bias, void* y, const uint64_t* out_row_ptrs,
                               const float* x_scale, const float* w_scale, int64_t M, int64_t N, int64_t K, int64_t E,
                               const int64_t* group_list, int list_on_device, int dtype, int bias_dtype,
                               int out_dtype, int w_layout, void* workspace, size_t workspace_bytes, void* stream)
{
    if (M < 0 || K <= 0 || N <= 0 || E <= 0) {
        return W8A8_ERR_INVALID;
    }
    if (w_layout != W8A8_W_KN && w_layout != W8A8_W_NK) {
        return W8A8_ERR_INVALID;
    }
    int kind;
    if (dtype == W8A8_DT_I8) {
        kind = KIND_I8;
        if (x_scale == nullptr || w_scale == nullptr) {
            return W8A8_ERR_INVALID;
        }
        if (out_dtype != W8A8_DT_F16 && out_dtype != W8A8_DT_BF16) {
            return W8A8_ERR_INVALID;
        }
    } else if (dtype == W8A8_DT_F16 || dtype == W8A8_DT_BF16) {
        kind = (dtype == W8A8_DT_F16) ? KIND_F16 : KIND_BF16;
        if (out_dtype != dtype) {
            return W8A8_ERR_INVALID;  // the reference's output takes x's dtype
        }
    } else if (dtype == W8A8_DT_F32) {
        kind = KIND_BF16;  // three-piece bf16 split of both operands, fp32 accumulation (see split3)
        if (out_dtype != W8A8_DT_F32 || out_row_ptrs != nullptr) {
            return W8A8_ERR_INVALID;
        }
    } else {
        return W8A8_ERR_INVALID;
    }
    if (bias != nullptr && bias_dtype != W8A8_DT_F16 && bias_dtype != W8A8_DT_BF16 && bias_dtype != W8A8_DT_F32) {
        return W8A8_ERR_INVALID;
    }
    if (M == 0) {
        return W8A8_OK;
    }
    if (x == nullptr || w == nullptr || (y == nullptr && out_row_ptrs == nullptr) || group_list == nullptr) {
        return W8A8_ERR_INVALID;
    }
    const int elem = (kind == KIND_I8) ? 1 : 2;
    const bool f32 = (dtype == W8A8_DT_F32);
    // the epilogue fetches per-channel operands and stores outputs in 16-column pieces
    if ((K * elem) % 16 != 0 || (N % 16) != 0) {
        return W8A8_ERR_UNSUPPORTED;
    }
    if (!is_aligned(x, 16) || !is_aligned(w, 16) || (y != nullptr && !is_aligned(y, 16))) {
        return W8A8_ERR_ALIGN;
    }
    // the epilogue reads both vectors in 16-byte pieces; scales belong to int8 operands only
    if (!is_aligned(bias, 16) || (kind == KIND_I8 && (!is_aligned(w_scale, 16) || !is_aligned(x_scale, 4)))) {
        return W8A8_ERR_ALIGN;
    }
    if (M >= (int64_t(1) << 31) - 256 || N >= (int64_t(1) << 31) || K >= (int64_t(1) << 31)) {
        return W8A8_ERR_UNSUPPORTED;
    }
    const size_t need = f32 ? w8a8_grouped_matmul_f32_workspace_size(M, N, K, E)
                            : w8a8_grouped_matmul_workspace_size(M, N, K, E);
    if (workspace == nullptr || workspace_bytes < need) {
        return W8A8_ERR_WORKSPACE;
    }
    if (!is_aligned(workspace, 256)) {
        return W8A8_ERR_ALIGN;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const GroupedWorkspace g = carve_workspace(workspace, M, E, 0);
    const int list_rc = check_host_group_list(group_list, list_on_device, E, M);
    if (list_rc != W8A8_OK) {
        return list_rc;
    }
    const bool b_mn = (w_layout == W8A8_W_KN);
    if (f32) {
        if (SPLIT_TERMS * K >= (int64_t(1) << 31)) {
            return W8A8_ERR_UNSUPPORTED;
        }
        uint8_t* base = static_cast<uint8_t*>(workspace) + g.total;
        __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(base);
        __nv_bfloat16* wsplit =
            reinterpret_cast<__nv_bfloat16*>(base + align_up_sz(static_cast<size_t>(M) * SPLIT_PIECES * K * 2, 256));
        const unsigned grid = static_cast<unsigned>(sm_count()) * 8;
        cudaError_t e = launch_chained(split_blocks_kernel, grid, 256, 0, st, static_cast<const float*>(x), xs, M, K);
        if (e == cudaSuccess) {
            e = launch_chained(split_blocks_kernel, grid, 256, 0, st, static_cast<const float*>(w), wsplit, E, K * N);
        }
        if (e != cudaSuccess) {
            return launch_status(e);
        }
        x = xs;
        w = wsplit;
    }
    CUtensorMap tb;
    if (!make_map_b(&tb, w, f32 ? E * SPLIT_PIECES : E, N, K, kind, b_mn)) {
        return W8A8_ERR_CUDA;
    }
    GemmParams p{};
    p.M = M;
    p.N = N;
    p.K = K;
    const int block_k = GEMM_KBYTES / elem;
    p.num_k_blocks = static_cast<int32_t>((K + block_k - 1) / block_k);
    if (f32) {
        p.k_blocks_per_term = p.num_k_blocks;
        p.num_k_blocks *= SPLIT_TERMS;
    }
    p.scale = w_scale;
    p.row_scale = x_scale;
    p.bias = bias;
    p.out = y;
    p.out_row_ptrs = out_row_ptrs;
    p.flags = (bias != nullptr ? 4 : 0) | (bias_dtype & 3);
    p.out_dtype = out_dtype;
    p.n_tiles = static_cast<int32_t>((N + 255) / 256);
    if (kind == KIND_I8) {
        return run_grouped<KIND_I8, EPI_GMM>(group_list, list_on_device, E, M, g, b_mn, x, tb, p, st);
    }
    if (kind == KIND_F16) {
        return run_grouped<KIND_F16, EPI_GMM>(group_list, list_on_device, E, M, g, b_mn, x, tb, p, st);
    }
    return run_grouped<KIND_BF16, EPI_GMM>(group_list, list_on_device, E, M, g, b_mn, x, tb, p, st);
}

extern "C" int w8a8_grouped_matmul(const void* x, const void* w, const void* bias, void* y, const float* x_scale,
                                   const float* w_scale, int64_t M, int64_t N, int64_t K, int64_t E,
                                   const int64_t* group_list, int list_on_device, int dtype, int bias_dtype,
                                   int out_dtype, int w_layout, void* workspace, size_t workspace_bytes, void* stream)
{
    return grouped_matmul_impl(x, w, bias, y, nullptr, x_scale, w_scale, M, N, K, E, group_list, list_on_device, dtype,
                               bias_dtype, out_dtype, w_layout, workspace, workspace_bytes, stream);
}

extern "C" int w8a8_grouped_matmul_to_rows(const void* x, const void* w, const void* bias,
                                           const uint64_t* out_row_ptrs, const float* x_scale, const float* w_scale,
                                           int64_t M, int64_t N, int64_t K, int64_t E, const int64_t* group_list,
                                           int list_on_device, int dtype, int bias_dtype, int out_dtype, int w_layout,
                                           void* workspace, size_t workspace_bytes, void* stream)
{
    if (out_row_ptrs == nullptr) {
        return W8A8_ERR_INVALID;
    }
    return grouped_matmul_impl(x, w, bias, nullptr, out_row_ptrs, x_scale, w_scale, M, N, K, E, group_list,
                               list_on_device, dtype, bias_dtype, out_dtype, w_layout, workspace, workspace_bytes,
                               stream);
}

extern "C" int w8a8_pipeline_error(void* stream)
{
    int32_t* word = pipeline_error_word();
    if (word == nullptr) {
        return W8A8_ERR_CUDA;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int32_t v = 0;
    if (cudaMemcpyAsync(&v, word, sizeof(v), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemsetAsync(word, 0, sizeof(v), st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
        return W8A8_ERR_CUDA;
    }
    return v;
}

extern "C" int w8a8_set_gmsq_epilogue_warps(int warps)
{
    if (warps != 8 && warps != 16) {
        return W8A8_ERR_INVALID;
    }
    return g_gmsq_epilogue_warps.exchange(warps, std::memory_order_relaxed);
}

extern "C" int w8a8_set_gmsq_fused_requant(int on)
{
    return g_fuse_requant.exchange(on ? 1 : 0, std::memory_order_relaxed);
}

extern "C" int w8a8_set_gemm_shape(int shape)
{
    if (shape < 0 || shape > GEMM_SHAPE_HYBRID) {
        return W8A8_ERR_INVALID;
    }
    return g_shape_override.exchange(shape, std::memory_order_relaxed);
}

extern "C" int w8a8_workspace_error(const void* workspace, void* stream)
{
    if (workspace == nullptr) {
        return W8A8_ERR_INVALID;
    }
    GroupedHeader h;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(&h, workspace, sizeof(int32_t) * 2, cudaMemcpyDeviceToHost, st) != cudaSuccess) {
        return W8A8_ERR_CUDA;
    }
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        return W8A8_ERR_CUDA;
    }
    return h.error;
}

// ===========================================================================
// grouped_matmul_swiglu_quant without a caller workspace
// ===========================================================================
// Scratch for w8a8_grouped_matmul_swiglu_quant_static: lives in the library's
// device image, so every GPU that loads the library sets these bytes aside
// until the process exits.  In host code this name is only a handle for
// cudaGetSymbolAddress; it is never a device address by itself.
static __device__ __align__(256) unsigned char g_gmsq_static_scratch[W8A8_STATIC_SCRATCH_BYTES];

// One address lookup per device, made with that device current.  Racing first calls store the same value.
static int static_scratch_address(void** out)
{
    constexpr int MAX_DEVICES = 64;
    static std::atomic<void*> scratch_of_device[MAX_DEVICES];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) {
        return W8A8_ERR_CUDA;
    }
    if (dev >= MAX_DEVICES) {
        return W8A8_ERR_LIMIT;  // the address cache is fixed-size; nothing in CUDA failed
    }
    void* scratch = scratch_of_device[dev].load(std::memory_order_relaxed);
    if (scratch == nullptr) {
        if (cudaGetSymbolAddress(&scratch, g_gmsq_static_scratch) != cudaSuccess || scratch == nullptr) {
            return W8A8_ERR_CUDA;
        }
        scratch_of_device[dev].store(scratch, std::memory_order_relaxed);
    }
    *out = scratch;
    return W8A8_OK;
}

// The error word of the last *_static call on the current device (it lives in the built-in scratch, which the
// caller never sees): 0 = none, 1 = invalid device group list (y was left untouched), 2 = a pipeline wait ran out.
extern "C" int w8a8_static_scratch_error(void* stream)
{
    void* scratch = nullptr;
    const int rc = static_scratch_address(&scratch);
    if (rc != W8A8_OK) {
        return rc;
    }
    return w8a8_workspace_error(scratch, stream);
}

extern "C" int w8a8_grouped_matmul_swiglu_quant_static(const int8_t* x, const int8_t* w, const float* w_scale,
                                                       const float* x_scale, int8_t* y, float* y_scale, int64_t M,
                                                       int64_t K, int64_t N, int64_t E, const int64_t* group_list,
                                                       int list_on_device, int w_layout, int flags, void* stream)
{
    if (M < 0 || K <= 0 || N <= 0 || E <= 0) {
        return W8A8_ERR_INVALID;
    }
    // the built-in scratch is fixed: refuse anything whose workspace would not fit
    const size_t need = w8a8_grouped_matmul_swiglu_quant_workspace_size(M, K, N, E);
    if (need == 0 || need > static_cast<size_t>(W8A8_STATIC_SCRATCH_BYTES)) {
        return W8A8_ERR_LIMIT;
    }
    void* scratch = nullptr;
    const int rc = static_scratch_address(&scratch);
    if (rc != W8A8_OK) {
        return rc;
    }
    // From here on this is the ordinary operator with the built-in bytes as its workspace.  Whatever the call before left
    // there is never read: the first matmul launch rewrites the header (the planner does, and the tile tables with it, for
    // more than GROUPS_IN_CTA groups) once that call is complete, the matmuls write every activation that the
    // requantisation reads, and row maxima and counters, where they are used, are zeroed first.
    return w8a8_grouped_matmul_swiglu_quant(x, w, w_scale, x_scale, y, y_scale, M, K, N, E, group_list, list_on_device,
                                            w_layout, flags, scratch, static_cast<size_t>(W8A8_STATIC_SCRATCH_BYTES),
                                            stream);
}
