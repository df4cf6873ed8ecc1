// Persistent, warp-specialised tcgen05 GEMM for sm_100a with fused epilogues.
//
// One CTA per SM, 320 threads (576 with sixteen epilogue warps):
//   warp 0      TMA producer: fills a ring of shared-memory stages (128-byte
//               swizzle) with A and B tiles, one mbarrier per stage.
//   warp 1      MMA issuer: the warp walks the loop and waits together, an elected
//               lane issues tcgen05.mma into one of two TMEM accumulator stages;
//               tcgen05.commit releases the shared-memory stage and finally
//               publishes the accumulator.
//   warps 2-9   epilogue: tcgen05.ld the accumulator (a warp may read the 32 TMEM
//               lanes its index modulo 4 selects; two warps share each lane
//               quarter and split the columns), apply the operator's dequant
//               chain, store.  Double-buffered TMEM lets the epilogue of tile i
//               overlap the main loop of tile i+1.  The epilogues that work on
//               every element - SwiGLU with its exponential and correctly
//               rounded quotient, the dequantisation of int8 products - run on
//               warps 2-17, four per lane quarter: eight take as long per tile
//               as the main loop, all of it where K is short.
//
// Two shapes of the same kernel (template parameter CG):
//   CG = 1  one CTA per tile of 128 rows x BLOCK_N columns, 4 stages of
//           {A 128x128 B, B BLOCK_N x128 B}.  Used for small row counts.
//   CG = 2  a pair of CTAs (cluster of 2, tcgen05 cta_group::2) per tile of 256
//           rows x 256 columns.  Each CTA loads its 128 rows of A and its 128
//           columns of B (6 stages of 32 KB), the even CTA issues the MMAs for
//           both, each CTA's tensor memory receives its 128 rows of the
//           accumulator and each CTA runs its own epilogue.  Halving the B bytes
//           per CTA takes shared-memory and L2->SM traffic per MMA from 96 to 64
//           bytes per clock, which is what lets the tensor pipe stay busy.  No
//           load is multicast: each CTA fetches exactly what it stores.
//
// A is always K-major ([rows, K], K contiguous).  B is either K-major
// ([.., N, K]) or MN-major ([.., K, N], the reference catalog's weight layout);
// both are consumed directly by the tensor core through the descriptor's
// major bit, no transposition pass.
//
// Dense problems enumerate (row tile, column tile) with the row index fastest
// so that concurrently running CTAs share a B column block in L2.  Grouped
// problems cut the cumulative group list into tiles - every CTA for itself, or
// a kernel ahead of this one where there are many groups - that never straddle
// groups (rows past a group's end inside a tile are computed and discarded),
// with the column index fastest, so the A tile and the expert's weights stay
// L2-resident.
#pragma once

#include <type_traits>

#include "beside.cuh"
#include "common.cuh"
#include "tc_ptx.cuh"

namespace w8a8 {

// producer warp, MMA warp and the epilogue warps (8 or 16)
__host__ __device__ constexpr int gemm_threads(int epi_warps) { return 64 + 32 * epi_warps; }
constexpr int GEMM_EPI_PATCH_BYTES = 8 * 4096;  // shared by the epilogue warps: 4 KB each for 8, 2 KB each for 16
constexpr int GEMM_BLOCK_M = 128;
constexpr int GEMM_KBYTES = 128;  // bytes of K per stage row (one swizzle atom)
constexpr int GEMM_PREFETCH_K_BLOCKS = 4;  // of a dense problem's weights, asked into L2 ahead of the kernel's start
constexpr int GEMM_A_BYTES = GEMM_BLOCK_M * GEMM_KBYTES;

// pipeline depth: as many 1 KB-aligned stages as fit beside the barriers
__host__ __device__ constexpr int gemm_stages(int cg, int block_n)
{
    return (GEMM_A_BYTES + (block_n / cg) * GEMM_KBYTES) <= 32768 ? 6 : 4;
}

// K blocks (128 bytes of K each) per pipeline stage.  The thread that issues the MMAs pays a fixed price for every
// barrier wait, satisfied or not (measured with the issue probe: about 0.3 us per wait-and-commit against 45 ns
// per instruction, so 4 instructions per wait sustain 2.5 - 3.0 POPS at full clock, 8 per wait 3.5 - 4.3): a stage
// therefore carries two K blocks wherever that still leaves three stages.
__host__ __device__ constexpr int gemm_kblocks_per_stage(int cg, int block_n)
{
#ifdef W8A8_ONE_KBLOCK_PER_STAGE  // comparison builds only
    return 1;
#else
    return (GEMM_A_BYTES + (block_n / cg) * GEMM_KBYTES) <= 32768 ? 2 : 1;
#endif
}

// fp32 operands on the bf16 tensor path: v = hi + mid + lo with three bf16 pieces (8 + 8 + 8 significand bits, each
// remainder exact in fp32), and x.w is the sum of the six piece products whose orders add up to at most two (hi.hi,
// hi.mid, mid.hi, hi.lo, mid.mid, lo.hi; what is dropped is below 2^-24 of |x||w|).  The products are accumulated one
// after the other, hi.hi last, as one matmul of SPLIT_TERMS times the K blocks; two bits per term name the piece (0 hi,
// 1 mid, 2 lo).  Neighbouring terms share a piece and every other one runs through K backwards, so that a term starts
// on the K blocks that the one before it has left in L2.
constexpr int SPLIT_PIECES = 3;
constexpr int SPLIT_TERMS = 6;
constexpr uint32_t SPLIT_PICK_A = 0x016;  // lo mid mid hi  hi  hi
constexpr uint32_t SPLIT_PICK_B = 0x250;  // hi hi  mid mid lo  hi

enum GemmKind { KIND_I8 = 0, KIND_F16 = 1, KIND_BF16 = 2 };
enum GemmEpi { EPI_RAW = 0, EPI_QMM = 1, EPI_GMSQ = 2, EPI_GMM = 3 };

struct TileEntry {
    int32_t group;
    int32_t m_start;
    int32_t m_rows;
    int32_t pad;
};

struct GroupedHeader {
    int32_t num_m_tiles;
    int32_t error;  // 0 ok, 1 invalid group list, 2 pipeline wait ran out
    int32_t rows_total;  // the list's last entry: rows the groups cover (may be below M for a device prefix list)
    int32_t pad[61];
};

// How groups become row tiles:
// PLAN_ALL: every row of a group, in tiles of tile_m (the last one partial).
// PLAN_WHOLE: the whole tile_m-row tiles of a group, plus its last partial tile when that holds more than
//             tile_m / 2 rows (as a pair tile it pads no more rows than two single tiles would).
// PLAN_LEFTOVER: what a group leaves over after its (2 * tile_m)-row blocks when that is at most tile_m rows:
//             one tile of tile_m.
// PLAN_WHOLE at 256 rows and PLAN_LEFTOVER at 128 rows together cover every row exactly once.
constexpr int PLAN_ALL = 0;
constexpr int PLAN_WHOLE = 1;
constexpr int PLAN_LEFTOVER = 2;

// (tile_m is a power of two)
__device__ __forceinline__ int32_t group_tiles(uint32_t rows, uint32_t tile_m, int mode)
{
    if (mode == PLAN_LEFTOVER) {
        const uint32_t rest = rows & (2 * tile_m - 1);
        return (rest >= 1 && rest <= tile_m) ? 1 : 0;
    }
    const uint32_t whole = rows >> (31 - __clz(tile_m)), rest = rows & (tile_m - 1);
    return static_cast<int32_t>(whole + (rest > (mode == PLAN_WHOLE ? tile_m / 2 : 0) ? 1 : 0));
}

// tile `t` of group `group`, whose rows are [start, end)
__device__ __forceinline__ TileEntry group_tile(int group, int64_t start, int64_t end, int32_t t, int tile_m, int mode)
{
    if (mode == PLAN_LEFTOVER) {
        start += (end - start) & ~static_cast<int64_t>(2 * tile_m - 1);
    }
    TileEntry te;
    te.group = group;
    te.m_start = static_cast<int32_t>(start + static_cast<int64_t>(t) * tile_m);
    const int64_t left = end - te.m_start;
    te.m_rows = static_cast<int32_t>(left < tile_m ? left : tile_m);
    te.pad = 0;
    return te;
}

// The group list of a grouped problem with at most GROUPS_IN_CTA groups: every CTA plans the tiles for itself - one warp,
// 0.5 us, and for a host list before the wait for the kernel before.  A planner kernel that wrote a table took 2 - 3 us of
// every call (and, for the SwiGLU form of few rows, a memset that no launch overlaps): 64 rows of 4 experts of 512 x 512
// bf16 6.7 us (8.7 with it), 200 of 8 of 1024 x 2048 14.1 (16.0); SwiGLU form, 64 rows of 32 experts of 1024 x 1024 16.1
// (22.4), 100 of 8 of 4096 x 2048 23.5 (28.8).  The bound is the shared memory that is left beside the stages.
constexpr int GROUPS_IN_CTA = 256;
struct GroupList {
    const int64_t* dev;  // device list, or null: `ends`
    int32_t E;           // 0: the tiles come from the table of plan_groups_kernel
    int32_t mode;
    int32_t tile_m;
    int32_t allow_prefix;
    int32_t ends[GROUPS_IN_CTA];

    __device__ __forceinline__ int64_t end_of(int g) const { return dev != nullptr ? dev[g] : ends[g]; }
};
struct NoGroupList {
};
// how many groups a CTA has planned for itself (0: none)
__device__ __forceinline__ int32_t groups_planned(const GroupList& list) { return list.E; }
__device__ __forceinline__ int32_t groups_planned(const NoGroupList&) { return 0; }
template <int EPI>
using GroupListOf = std::conditional_t<EPI == EPI_GMSQ || EPI == EPI_GMM, GroupList, NoGroupList>;

// One warp: first[g] = the first tile of group g, first[E] = the number of tiles, and whether the list is in order.  An
// invalid one has no tiles.  Behind first[E] come numbers that no tile has.
__device__ __forceinline__ bool plan_in_cta(const GroupList& list, int64_t M, int32_t* first)
{
    constexpr int PER_LANE = GROUPS_IN_CTA / 32;
    const int lane = threadIdx.x & 31;
    int32_t count[PER_LANE], sum = 0;
    bool bad = false;
    int64_t prev = 0;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int g = lane * PER_LANE + i;
        count[i] = 0;
        if (g < list.E) {
            if (i == 0 && g > 0) {
                prev = list.end_of(g - 1);
            }
            const int64_t end = list.end_of(g);
            const bool ok = end >= prev && prev >= 0 && end <= M && (g != list.E - 1 || end == M || list.allow_prefix != 0);
            bad |= !ok;
            count[i] = ok ? group_tiles(static_cast<uint32_t>(end - prev), static_cast<uint32_t>(list.tile_m), list.mode) : 0;
            prev = end;
        }
        sum += count[i];
    }
    bad = __any_sync(FULL_MASK, bad);
    int32_t incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int32_t v = __shfl_up_sync(FULL_MASK, incl, off);
        incl += lane >= off ? v : 0;
    }
    int32_t at = incl - sum;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int g = lane * PER_LANE + i;
        if (g != list.E) {
            first[g] = g < list.E ? (bad ? 0 : at) : INT32_MAX;
        }
        at += count[i];
        if (g == list.E - 1) {
            first[list.E] = bad ? 0 : at;
        }
    }
    return !bad;
}

// Tile `mt` by the first tiles: its group is the last one whose first tile is at or before it (groups without tiles
// share their first tile with the next one), found by a whole warp at once.  (Between two tiles an epilogue warp has
// nothing else to do: with a search by halves and the tile number divided, SwiGLU tiles of K = 1280 took 4 % longer.)
__device__ __forceinline__ TileEntry tile_in_cta(const GroupList& list, const int32_t* first, int32_t mt)
{
    const int4* mine = reinterpret_cast<const int4*>(first) + (threadIdx.x & 31) * (GROUPS_IN_CTA / 32 / 4);
    int at_or_before = 0;
#pragma unroll
    for (int i = 0; i < GROUPS_IN_CTA / 32 / 4; ++i) {
        const int4 f = mine[i];
        at_or_before += (f.x <= mt) + (f.y <= mt) + (f.z <= mt) + (f.w <= mt);
    }
    const int g = __reduce_add_sync(FULL_MASK, at_or_before) - 1;
    return group_tile(g, g == 0 ? 0 : list.end_of(g - 1), list.end_of(g), mt - first[g], list.tile_m, list.mode);
}

// A grouped problem's two launches (pairs, then leftovers) share no output row and read nothing of one another, so the
// second one's CTAs start as the first one's leave their SMs, whose last wave of tiles is rarely full.  What orders them:
// the first one lets the second in only after its own wait, when all that came before is complete; the second one waits
// for the first only before it ends, so that whoever waits for the second has waited for both.  2500 rows of 16 experts of
// 1024 x 1024 bf16 21.1 us (28.1 one after the other), 4000 of 32 of 2048 x 7168 205 (214), 16000 of 4 of 4096 x 2048 223
// (236); SwiGLU form, 2500 of 8 of 2048 x 2048 35.8 (39.3), 3000 of 32 of 7168 x 4096 206 (218); what the power cap bounds
// (8000 of 32 of 2048 x 7168 317, the 131072-row Zipf load 4060) stays.
constexpr int ORDER_ALONE = 0;
constexpr int ORDER_FIRST_OF_TWO = 1;
constexpr int ORDER_SECOND_OF_TWO = 2;
constexpr int ORDER_PLAIN = 3;  // not launched beside the kernel before (see run_grouped)

struct GemmParams {
    int64_t M;  // rows per batch (dense) or total rows (grouped)
    int64_t N;  // logical output columns of the matmul
    int64_t K;
    int32_t num_k_blocks;
    int32_t n_tiles;
    int32_t m_tiles_per_batch;
    int32_t batch;
    const TileEntry* tiles;
    GroupedHeader* header;  // grouped: tile count + error word; dense: may be null
    int32_t* error;         // device error word (may be null)
    // epilogue operands
    const void* scale;       // QMM: scale; GMSQ/GMM: w_scale [E, N]
    const float* offset;     // QMM
    const float* row_scale;  // QMM: pertoken; GMSQ/GMM: x_scale
    const void* bias;
    void* out;
    int64_t flags;  // QMM flag word; GMM: bias dtype in bits 0-1, bit 2 = has bias
    int32_t out_dtype;
    int64_t bias_batch_stride;
    const uint64_t* out_row_ptrs;  // GMM: when set, row r is stored at this address instead of out + r*N
    int32_t a_box_rows;  // rows of one A load: 128, or fewer (a multiple of 8) on single CTAs
    // fp32 operands split into bf16 pieces (SPLIT_PIECES of each): K blocks of one piece product, num_k_blocks being
    // SPLIT_TERMS times that; 0: operands as they are
    int32_t k_blocks_per_term;
    // dense: K blocks of a CTA's first tile of B that it asks L2 for while the kernel before it may still be running
    int32_t prefetch_k_blocks;
    int32_t order;  // ORDER_*
    float* act;       // GMSQ: fp32 activations [M, N/2]
    uint32_t* amax;   // GMSQ with fuse_requant: per-row max|act| bit patterns
    // GMSQ with the requantisation fused in: the CTA that finishes the last column tile of its rows quantises them
    int32_t* tile_done;   // per (row tile, CTA of the tile): epilogue warps done with a column tile (zeroed by the caller)
    int8_t* y;            // [M, N/2]
    float* y_scale;       // [M]
    int32_t split;  // SPLITK kernels: CTAs of a cluster that share a tile's K
    int32_t fuse_requant;
    int32_t round_direct;
};

__device__ __forceinline__ float vec_elem_as_float(const void* p, int64_t i, int kind)
{
    switch (kind) {
    case W8A8_QM_BIAS_I32:
        return static_cast<float>(static_cast<const int32_t*>(p)[i]);
    case W8A8_QM_BIAS_F16:
        return __half2float(static_cast<const __half*>(p)[i]);
    case W8A8_QM_BIAS_BF16:
        return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
    default:
        return static_cast<const float*>(p)[i];
    }
}

// NV (32 or 16) consecutive per-channel values starting at element `idx0` (16-byte aligned
// for every kind because idx0 is a multiple of 16), widened to fp32; a vector
// that is not per-channel broadcasts element 0.  `valid` is 32, 16 or 0.
template <int NV>
__device__ __forceinline__ void load_vec(const void* base, int64_t idx0, int kind, bool perchan, int valid,
                                         float (&out)[NV])
{
    if (!perchan) {
        const float s = vec_elem_as_float(base, 0, kind);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            out[j] = s;
        }
        return;
    }
    if (kind == W8A8_QM_BIAS_F32 || kind == W8A8_QM_BIAS_I32) {
        const uint4* p4 = reinterpret_cast<const uint4*>(static_cast<const uint32_t*>(base) + idx0);
#pragma unroll
        for (int q = 0; q < NV / 4; ++q) {
            uint4 t = make_uint4(0, 0, 0, 0);
            if (q * 4 < valid) {
                t = __ldca(p4 + q);
            }
            if (kind == W8A8_QM_BIAS_I32) {
                out[q * 4 + 0] = static_cast<float>(static_cast<int32_t>(t.x));
                out[q * 4 + 1] = static_cast<float>(static_cast<int32_t>(t.y));
                out[q * 4 + 2] = static_cast<float>(static_cast<int32_t>(t.z));
                out[q * 4 + 3] = static_cast<float>(static_cast<int32_t>(t.w));
            } else {
                out[q * 4 + 0] = __uint_as_float(t.x);
                out[q * 4 + 1] = __uint_as_float(t.y);
                out[q * 4 + 2] = __uint_as_float(t.z);
                out[q * 4 + 3] = __uint_as_float(t.w);
            }
        }
    } else {
        const uint4* p4 = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + idx0);
#pragma unroll
        for (int q = 0; q < NV / 8; ++q) {
            uint4 t = make_uint4(0, 0, 0, 0);
            if (q * 8 < valid) {
                t = __ldca(p4 + q);
            }
            const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (kind == W8A8_QM_BIAS_BF16) {
                    unpack2<W8A8_DT_BF16>(w[i], out[q * 8 + 2 * i], out[q * 8 + 2 * i + 1]);
                } else {
                    unpack2<W8A8_DT_F16>(w[i], out[q * 8 + 2 * i], out[q * 8 + 2 * i + 1]);
                }
            }
        }
    }
}


// What the dequant chain of quant_matmul needs besides the accumulator, the same for all columns of a row.
struct QmmTerms {
    float row_mul;
    const void* bias;
    int bias_kind;
    bool has_pt, bias_perchan, scale_perchan, scale_bf16, has_offset, offset_perchan;
};

__device__ __forceinline__ QmmTerms qmm_terms(const GemmParams& p, int32_t group, int64_t row, bool row_ok)
{
    const int64_t f = p.flags;
    QmmTerms t;
    t.has_pt = (f & W8A8_QM_HAS_PT) != 0;
    t.row_mul = 1.0f;
    if (t.has_pt && row_ok) {
        // the plugin's layouts make (row mod M) the token index in every case
        t.row_mul = p.row_scale[(group == 0) ? row : (row - static_cast<int64_t>(group) * p.M)];
    }
    t.bias = p.bias;
    t.bias_kind = static_cast<int>((f & W8A8_QM_BIAS_MASK) >> W8A8_QM_BIAS_SHIFT);
    t.bias_perchan = (f & W8A8_QM_BIAS_PERCHAN) != 0;
    t.scale_perchan = (f & W8A8_QM_SCALE_PERCHAN) != 0;
    t.scale_bf16 = (f & W8A8_QM_SCALE_BF16) != 0;
    t.has_offset = (f & W8A8_QM_HAS_OFFSET) != 0;
    t.offset_perchan = (f & W8A8_QM_OFFSET_PERCHAN) != 0;
    if (t.bias != nullptr && p.bias_batch_stride != 0) {
        const int64_t esz = (t.bias_kind == W8A8_QM_BIAS_F16 || t.bias_kind == W8A8_QM_BIAS_BF16) ? 2 : 4;
        t.bias = static_cast<const uint8_t*>(t.bias) + group * p.bias_batch_stride * esz;
    }
    return t;
}

// ((acc + i32 bias) * scale + offset) * pertoken + float bias of NV columns, each operation rounded
template <int NV>
__device__ __forceinline__ void qmm_dequant(const GemmParams& p, const QmmTerms& t, int64_t col0, int valid,
                                            float (&v)[NV])
{
    float w[NV];
    if (t.bias_kind == W8A8_QM_BIAS_I32) {
        load_vec<NV>(t.bias, col0, t.bias_kind, t.bias_perchan, valid, w);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            v[j] = __fadd_rn(v[j], w[j]);
        }
    }
    load_vec<NV>(p.scale, col0, t.scale_bf16 ? W8A8_QM_BIAS_BF16 : W8A8_QM_BIAS_F32, t.scale_perchan, valid, w);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        v[j] = __fmul_rn(v[j], w[j]);
    }
    if (t.has_offset) {
        load_vec<NV>(p.offset, col0, W8A8_QM_BIAS_F32, t.offset_perchan, valid, w);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            v[j] = __fadd_rn(v[j], w[j]);
        }
    }
    if (t.has_pt) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            v[j] = __fmul_rn(v[j], t.row_mul);
        }
    }
    if (t.bias_kind >= W8A8_QM_BIAS_F16) {
        load_vec<NV>(t.bias, col0, t.bias_kind, t.bias_perchan, valid, w);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            v[j] = __fadd_rn(v[j], w[j]);
        }
    }
}

// Requantisation of a row of SwiGLU activations by its largest magnitude: amax clamp at FLT_MIN, y_scale = amax * (1/127),
// inv = 127 / amax, clamp to [-128, 127], narrowing (gmsq_vec_kernel.cpp:233-257).
__device__ __forceinline__ float requant_amax(float amax) { return amax > 1.1754944e-38f ? amax : 1.1754944e-38f; }

// largest magnitude of four activations and `m`, NaN left out
__device__ __forceinline__ float requant_max4(float m, const float4& a)
{
    return fmaxf(fmaxf(fmaxf(m, fabsf(a.x)), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w)));
}

template <bool DIRECT>
__device__ __forceinline__ uint32_t requant4(const float4& a, float inv)
{
    const float w[4] = {__fmul_rn(a.x, inv), __fmul_rn(a.y, inv), __fmul_rn(a.z, inv), __fmul_rn(a.w, inv)};
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[q] = fminf(fmaxf(w[q], -128.0f), 127.0f);
    }
    uint32_t packed = narrow4_fast<DIRECT>(v[0], v[1], v[2], v[3]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (w[q] != w[q]) {  // a NaN activation narrows to 0 (fmaxf / fminf turned it into a bound)
            packed &= ~(0xffu << (8 * q));
        }
    }
    return packed;
}

// 16-byte pieces [c_lo, c_hi) of one finished row by one warp, inside the matmul kernel.  The activations and row maxima
// were written by other SMs: they are read through L2 (ld.global.cg), never through this SM's L1.
template <bool DIRECT>
__device__ __forceinline__ void requant_row_part(const float* act, const uint32_t* amax_bits, int8_t* y, float* y_scale,
                                                 int64_t row, int64_t H, int64_t c_lo, int64_t c_hi, bool write_scale,
                                                 int lane)
{
    const float amax = requant_amax(__uint_as_float(__ldcg(amax_bits + row)));
    if (write_scale && lane == 0) {
        y_scale[row] = __fmul_rn(amax, INV127);
    }
    const float inv = __fdiv_rn(127.0f, amax);
    const float4* src = reinterpret_cast<const float4*>(act + row * H);
    uint32_t* dst = reinterpret_cast<uint32_t*>(y + row * H);
    // eight independent 16-byte loads in flight per lane: few warps work here, and a load at a time would leave
    // them waiting on L2 latency
    constexpr int DEPTH = 8;
    for (int64_t c0 = c_lo; c0 < c_hi; c0 += 32 * DEPTH) {
        float4 a[DEPTH];
#pragma unroll
        for (int j = 0; j < DEPTH; ++j) {
            const int64_t c = c0 + lane + 32 * j;
            a[j] = (c < c_hi) ? __ldcg(src + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int j = 0; j < DEPTH; ++j) {
            const int64_t c = c0 + lane + 32 * j;
            if (c < c_hi) {
                __stcs(dst + c, requant4<DIRECT>(a[j], inv));
            }
        }
    }
}

struct TileInfo {
    int32_t a_row0;  // first row this CTA loads and owns (global row index)
    int32_t m_rows;  // valid rows among this CTA's 128
    int32_t group;   // expert / batch (B's outermost coordinate)
    int32_t nt;      // column tile
    int32_t mt;      // row tile (grouped: index into the tile table)
};

// Eight SwiGLU activations silu(g * xs * wg) * (u * xs * wu) on pairs, with the bits of canonical_silu.  The range
// that needs the scalar form is gates beyond +-80; below 2^-25 the denominator is exactly 2, so small gates need no
// lower bound (a zero gate may give a zero of the other sign, which quantises to 0 all the same).  With the faster
// requantisation: 4096 rows over 8 experts of 2048 x 4096 72.6 us, 81 with scalar arithmetic; 65536 rows of 1024 x 1024
// 149, 156; the 131072-row Zipf load, bound by the power cap, the same 4.5 ms.
__device__ __forceinline__ void swiglu8(const uint32_t* g, const uint32_t* u, float xs, const float* wg, const float* wu,
                                        float (&a)[8])
{
    f32x2 l[4], r[4], den[4], q[4];
    float l_max = 0.0f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float4 p = __ldca(reinterpret_cast<const float4*>(wg) + i), o = __ldca(reinterpret_cast<const float4*>(wu) + i);
        const f32x2 ws[4] = {pair(p.x, p.y), pair(p.z, p.w), pair(o.x, o.y), pair(o.z, o.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = 2 * i + h;
            auto f = [](uint32_t v) { return static_cast<float>(static_cast<int32_t>(v)); };
            l[j] = mul2(mul2(pair(f(g[2 * j]), f(g[2 * j + 1])), pair(xs)), ws[h]);
            r[j] = mul2(mul2(pair(f(u[2 * j]), f(u[2 * j + 1])), pair(xs)), ws[2 + h]);
            float l0, l1;
            unpair(l[j], l0, l1);
            l_max = fmaxf(l_max, fmaxf(fabsf(l0), fabsf(l1)));
        }
    }
    neg_exp_neg2<4>(l, den);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        den[j] = add2(den[j], pair(-1.0f));
    }
    quotient2<4>(l, den, q);
    if (!(l_max <= EXP2_MAX_ABS)) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float l0, l1;
            unpair(l[j], l0, l1);
            q[j] = pair(canonical_silu(l0), canonical_silu(l1));
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        unpair(mul2(q[j], r[j]), a[2 * j], a[2 * j + 1]);
    }
}

// Brings what the epilogue of a tile reads besides the accumulator into L1 while the accumulator is being computed (with
// the loads behind the wait for it, 128 x 1024 x 1024 with its quantisation takes 7.27 us, 7.13 so; 300 x 4096 x 4096
// 15.49, 15.36).
__device__ __forceinline__ void touch(const void* base, int64_t byte)
{
    uint32_t v;
    asm volatile("ld.global.ca.b32 %0, [%1];" : "=r"(v) : "l"(static_cast<const uint8_t*>(base) + byte));
}

template <int BLOCK_N, int KIND, int EPI>
__device__ __forceinline__ void touch_epilogue_operands(const GemmParams& p, const TileInfo& tl, int row_in_tile)
{
    const int lane = row_in_tile & 31;
    const bool row_ok = row_in_tile < tl.m_rows;
    const int64_t row = static_cast<int64_t>(tl.a_row0) + row_in_tile;
    if constexpr (EPI == EPI_GMSQ) {
        // lanes 0-15: 128 gate scales, 16-31: 128 up scales, a 32-byte sector each
        const int64_t H = p.N / 2, col = static_cast<int64_t>(tl.nt) * 128 + (lane & 15) * 8;
        if (col < H) {
            touch(p.scale, ((static_cast<int64_t>(tl.group) * p.N) + (lane < 16 ? col : H + col)) * 4);
        }
        if (row_ok) {
            touch(p.row_scale, row * 4);
        }
    } else if constexpr (EPI == EPI_QMM || EPI == EPI_GMM) {
        const int64_t col = static_cast<int64_t>(tl.nt) * BLOCK_N + lane * (BLOCK_N / 32);
        const int64_t at = (EPI == EPI_GMM ? static_cast<int64_t>(tl.group) * p.N : 0) + col;
        const bool col_ok = col < p.N;
        if constexpr (EPI == EPI_QMM) {
            const int64_t f = p.flags;
            if (col_ok && (f & W8A8_QM_SCALE_PERCHAN)) {
                touch(p.scale, at * ((f & W8A8_QM_SCALE_BF16) ? 2 : 4) & ~int64_t(3));
            }
            if (row_ok && (f & W8A8_QM_HAS_PT)) {
                touch(p.row_scale, (tl.group == 0 ? row : row - static_cast<int64_t>(tl.group) * p.M) * 4);
            }
            const int kind = static_cast<int>((f & W8A8_QM_BIAS_MASK) >> W8A8_QM_BIAS_SHIFT);
            if (col_ok && kind != W8A8_QM_BIAS_NONE && (f & W8A8_QM_BIAS_PERCHAN)) {
                const int size = (kind == W8A8_QM_BIAS_F16 || kind == W8A8_QM_BIAS_BF16) ? 2 : 4;
                touch(p.bias, (tl.group * p.bias_batch_stride + col) * size & ~int64_t(3));
            }
        } else {
            if constexpr (KIND == KIND_I8) {
                if (col_ok) {
                    touch(p.scale, at * 4);
                }
                if (row_ok) {
                    touch(p.row_scale, row * 4);
                }
            }
            if (col_ok && (p.flags & 4)) {
                touch(p.bias, at * ((p.flags & 3) == W8A8_DT_F32 ? 4 : 2) & ~int64_t(3));
            }
        }
    }
}

// Eight columns of a row in the form that most calls have - per-channel fp32 scales `w` (int8 operands), one factor per
// row, a per-channel float bias or none - as four words of two 16-bit results.  The order and rounding of qmm_dequant; the
// factors are multiplied two at a time, the bias is added one by one (see mul2).  `b16`: eight values of a 16-bit bias;
// `b32`: where an fp32 one is.
template <int KIND>
__device__ __forceinline__ uint4 dequant8(const uint32_t* r, const f32x2* w, float row_mul, int bias_kind, uint4 b16,
                                          const void* b32, bool bf16_out)
{
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if constexpr (KIND == KIND_I8) {
            const f32x2 a = pair(static_cast<float>(static_cast<int32_t>(r[2 * j])),
                                 static_cast<float>(static_cast<int32_t>(r[2 * j + 1])));
            unpair(mul2(mul2(a, w[j]), pair(row_mul)), v[2 * j], v[2 * j + 1]);
        } else {
            v[2 * j] = __uint_as_float(r[2 * j]);
            v[2 * j + 1] = __uint_as_float(r[2 * j + 1]);
        }
    }
    if (bias_kind != W8A8_QM_BIAS_NONE) {
        float b[8];
        if (bias_kind == W8A8_QM_BIAS_F32) {
            load_vec<8>(b32, 0, W8A8_QM_BIAS_F32, true, 8, b);
        } else {
            const uint32_t word[4] = {b16.x, b16.y, b16.z, b16.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (bias_kind == W8A8_QM_BIAS_BF16) {
                    unpack2<W8A8_DT_BF16>(word[j], b[2 * j], b[2 * j + 1]);
                } else {
                    unpack2<W8A8_DT_F16>(word[j], b[2 * j], b[2 * j + 1]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = __fadd_rn(v[j], b[j]);
        }
    }
    return bf16_out ? make_uint4(pack2<W8A8_DT_BF16>(v[0], v[1]), pack2<W8A8_DT_BF16>(v[2], v[3]),
                                 pack2<W8A8_DT_BF16>(v[4], v[5]), pack2<W8A8_DT_BF16>(v[6], v[7]))
                    : make_uint4(pack2<W8A8_DT_F16>(v[0], v[1]), pack2<W8A8_DT_F16>(v[2], v[3]),
                                 pack2<W8A8_DT_F16>(v[4], v[5]), pack2<W8A8_DT_F16>(v[6], v[7]));
}

// The 16-bit epilogue of one thread on one tile: row `row_in_tile` of this CTA's accumulator, the `share`-th of
// EPI_WARPS / 4 equal shares of its columns.
// A chunk of results is 32 or 64 bytes of this thread's row.  They are not stored from here (every lane would write
// 16-byte pieces of a different row): the warp parks two chunks, 64 or 128 bytes per row, in its private shared-memory
// patch and then writes them as whole row segments, 4 or 8 lanes per row.  (Rows whose home is another GPU take eight
// warps: NVLink carries full 128-byte lines, not fragments.)
// Bound: its warps' latency, where K is short.  What a chunk is multiplied with is requested ahead of the wait for it, and
// all that does not need the accumulator is done before the wait for that: 128 x 1024 x 1024 with its quantisation 6.8 us
// (7.2 with eight warps and everything behind the waits; 5.1 without any epilogue), 8192 x 512 x 4096 40.8 (46.5; 18.5).
template <int BLOCK_N, int KIND, int EPI, int EPI_WARPS, typename Wait>
__device__ __forceinline__ bool epilogue_16bit(const GemmParams& p, const TileInfo& tl, uint32_t t_addr, int row_in_tile,
                                               int share, uint4* stage, Wait accumulator_ready)
{
    constexpr int COLS = BLOCK_N / (EPI_WARPS / 4);  // of this warp
    constexpr int CH = (EPI_WARPS == 16) ? 16 : 32;  // columns of a chunk
    constexpr int PIECES = CH / 4;                   // 16-byte pieces of a row in the patch (two chunks)
    constexpr int COPY_ROWS = 32 / PIECES;           // rows per instruction of the copy out
    static_assert(COLS % (2 * CH) == 0, "whole patches");
    const int lane = row_in_tile & 31, first_row = row_in_tile & ~31;
    const bool row_ok = row_in_tile < tl.m_rows;
    const int64_t row = static_cast<int64_t>(tl.a_row0) + row_in_tile;
    const int64_t col_first = static_cast<int64_t>(tl.nt) * BLOCK_N + share * COLS;
    if (first_row >= tl.m_rows || col_first >= p.N) {
        return accumulator_ready();  // a whole warp without results
    }
    [[maybe_unused]] QmmTerms terms;
    const float* scale = static_cast<const float*>(p.scale);
    const uint8_t* bias = static_cast<const uint8_t*>(p.bias);
    float row_mul = 1.0f;
    int bias_kind = W8A8_QM_BIAS_NONE;
    bool plain = true;
    if constexpr (EPI == EPI_QMM) {
        terms = qmm_terms(p, tl.group, row, row_ok);
        row_mul = terms.row_mul;
        bias = static_cast<const uint8_t*>(terms.bias);
        bias_kind = terms.bias_kind;
        plain = terms.scale_perchan && !terms.scale_bf16 && !terms.has_offset && bias_kind != W8A8_QM_BIAS_I32 &&
                (bias_kind == W8A8_QM_BIAS_NONE || terms.bias_perchan);
    } else {
        scale += static_cast<int64_t>(tl.group) * p.N;
        if constexpr (KIND == KIND_I8) {
            row_mul = row_ok ? p.row_scale[row] : 0.0f;
        }
        if (p.flags & 4) {
            const int bdt = static_cast<int>(p.flags & 3);
            bias_kind = (bdt == W8A8_DT_F16) ? W8A8_QM_BIAS_F16 : (bdt == W8A8_DT_BF16 ? W8A8_QM_BIAS_BF16 : W8A8_QM_BIAS_F32);
            bias += static_cast<int64_t>(tl.group) * p.N * (bias_kind == W8A8_QM_BIAS_F32 ? 4 : 2);
        }
    }
    const bool bias16 = bias_kind == W8A8_QM_BIAS_F16 || bias_kind == W8A8_QM_BIAS_BF16;
    const bool bf16_out = p.out_dtype == W8A8_DT_BF16;
    // where this lane's pieces of the copy out go: row first_row + COPY_ROWS * it + lane / PIECES, piece lane % PIECES
    const int piece = lane % PIECES, copy_row = lane / PIECES;
    const bool addressed = EPI == EPI_GMM && EPI_WARPS == 8 && p.out_row_ptrs != nullptr;
    uint64_t row_ptr = 0;  // addressed: of this thread's own row, else of the first row that it copies
    if (addressed) {
        // the row's home may be another GPU's memory: plain peer stores over NVLink
        row_ptr = row_ok ? p.out_row_ptrs[row] : 0;
    } else {
        row_ptr = reinterpret_cast<uint64_t>(p.out) +
                  static_cast<uint64_t>(static_cast<int64_t>(tl.a_row0) + first_row + copy_row) * p.N * 2;
    }
    // the place of row `r`'s piece `q` in the patch: permuted by the row so that the eight lanes of a store or load phase
    // hit eight different bank groups
    auto patch = [&](int r, int q) -> uint4& { return stage[r * PIECES + (PIECES == 8 ? q ^ (r & 7) : q ^ ((r >> 1) & 3))]; };
    f32x2 w[CH / 2];
    uint4 b16[CH / 8];
    // (N is a multiple of 16: a chunk has 32, 16 or no valid columns)
    auto request = [&](int cc) {
#pragma unroll
        for (int q = 0; q < CH / 8; ++q) {
            const int64_t col = col_first + cc + 8 * q;
            if (col < p.N) {
                if (KIND == KIND_I8 && plain) {
                    const ulonglong2* s2 = reinterpret_cast<const ulonglong2*>(scale + col);
                    const ulonglong2 lo = __ldca(s2), hi = __ldca(s2 + 1);
                    w[4 * q] = lo.x, w[4 * q + 1] = lo.y, w[4 * q + 2] = hi.x, w[4 * q + 3] = hi.y;
                }
                if (bias16 && plain) {
                    b16[q] = __ldca(reinterpret_cast<const uint4*>(bias + col * 2));
                }
            }
        }
    };
    auto chunk = [&](const uint32_t (&r)[CH], int cc, int sub) {
#pragma unroll
        for (int h = 0; h < CH / 16; ++h) {
            const int64_t col = col_first + cc + 16 * h;
            if (col >= p.N) {
                break;  // what the patch holds there is not copied out
            }
            uint4 o[2];
            if (EPI != EPI_QMM || plain) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    o[q] = dequant8<KIND>(r + 16 * h + 8 * q, w + 8 * h + 4 * q, row_mul, bias_kind, b16[2 * h + q],
                                          bias + (col + 8 * q) * 4, bf16_out);
                }
            } else {
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    v[j] = static_cast<float>(static_cast<int32_t>(r[16 * h + j]));
                }
                qmm_dequant<16>(p, terms, col, 16, v);
                uint32_t x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    x[j] = bf16_out ? pack2<W8A8_DT_BF16>(v[2 * j], v[2 * j + 1]) : pack2<W8A8_DT_F16>(v[2 * j], v[2 * j + 1]);
                }
                o[0] = make_uint4(x[0], x[1], x[2], x[3]);
                o[1] = make_uint4(x[4], x[5], x[6], x[7]);
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                patch(lane, sub * (PIECES / 2) + 2 * h + q) = o[q];
            }
        }
    };
    auto load = [&](int cc, uint32_t (&r)[CH]) {
        if constexpr (CH == 16) {
            tc::tmem_ld_32x16(t_addr + share * COLS + cc, r);
        } else {
            tc::tmem_ld_32x32(t_addr + share * COLS + cc, r);
        }
    };
    // all of the above, and what the first chunk is multiplied with, while the accumulator is being computed
    request(0);
    if (!accumulator_ready()) {
        return false;
    }
#pragma unroll 1
    for (int cc = 0; cc < COLS; cc += 2 * CH) {
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
            uint32_t r[CH];
            load(cc + sub * CH, r);
            if (cc + sub * CH != 0) {
                request(cc + sub * CH);
            }
            tc::tmem_ld_wait(r);
            chunk(r, cc + sub * CH, sub);
        }
        __syncwarp();
        const int64_t pc = col_first + cc + piece * 8;
#pragma unroll
        for (int it = 0; it < PIECES; ++it) {
            const int rr = it * COPY_ROWS + copy_row;  // row within the warp's 32
            uint64_t rp = row_ptr + static_cast<uint64_t>(it) * (COPY_ROWS * 2) * p.N;
            if (addressed) {
                rp = __shfl_sync(FULL_MASK, row_ptr, rr);
            }
            const uint4 val = patch(rr, piece);
            if (first_row + rr < tl.m_rows && pc < p.N) {
                *reinterpret_cast<uint4*>(rp + static_cast<uint64_t>(pc) * 2) = val;
            }
        }
        __syncwarp();
    }
    return true;
}

// The work of one epilogue thread on one tile: row `row_in_tile` of this CTA's accumulator, the `col_half`-th of
// EPI_WARPS / 4 equal shares of its columns.  accumulator_ready() waits for the accumulator; false: it never came.
template <int BLOCK_N, int KIND, int EPI, int EPI_WARPS, typename Wait>
__device__ __forceinline__ bool epilogue_tile(const GemmParams& p, const TileInfo& tl, uint32_t t_addr,
                                              int row_in_tile, int col_half, int64_t H, uint4* stage, Wait accumulator_ready)
{
    const bool row_ok = row_in_tile < tl.m_rows;
    const int64_t row = static_cast<int64_t>(tl.a_row0) + row_in_tile;  // global row (A and output)
    if constexpr (EPI == EPI_GMSQ) {
        const float xs = row_ok ? p.row_scale[row] : 0.0f;
        if (!accumulator_ready()) {
            return false;
        }
        if ((row_in_tile & ~31) >= tl.m_rows) {
            return true;  // a whole warp without rows
        }
        const float* wsg = static_cast<const float*>(p.scale) + static_cast<int64_t>(tl.group) * p.N;
        float local_max = 0.0f;
        // `col_half` counts this warp among the EPI_WARPS / 4 warps that share a TMEM lane quarter: each takes
        // 128 / (EPI_WARPS / 4) activation columns, 16 at a time
        constexpr int WARP_COLS = 128 / (EPI_WARPS / 4);
#pragma unroll 1
        for (int cc = 0; cc < WARP_COLS; cc += 16) {
            const int c = col_half * WARP_COLS + cc;
            uint32_t g[16], u[16];
            tc::tmem_ld_32x16(t_addr + c, g);
            tc::tmem_ld_32x16(t_addr + 128 + c, u);
            tc::tmem_ld_wait();
            const int64_t col0 = static_cast<int64_t>(tl.nt) * 128 + c;  // column in [0, H)
            const int lane = row_in_tile & 31;
            if (row_ok && col0 < H) {  // H is a multiple of 16: a chunk is valid as a whole
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float a[8];
                    swiglu8(g + 8 * h, u + 8 * h, xs, wsg + col0 + 8 * h, wsg + H + col0 + 8 * h, a);
#pragma unroll
                    for (int j = 0; j < 8 && p.fuse_requant; ++j) {
                        local_max = fmaxf(local_max, fabsf(a[j]));
                    }
#pragma unroll
                    for (int q = 2 * h; q < 2 * h + 2; ++q) {
                        // parked in the warp's shared-memory patch: piece q of row `lane`, the pieces permuted by
                        // the row so that the eight lanes of a store phase hit eight different bank groups
                        const float* v = a + 4 * (q - 2 * h);
                        stage[lane * 4 + (q ^ ((lane ^ (lane >> 2)) & 3))] =
                            make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]),
                                       __float_as_uint(v[3]));
                    }
                }
            }
            // the 16 activations of each row are a 64-byte piece of a line: written by 4 lanes per row, 8 rows per
            // instruction, instead of 16-byte pieces of 32 different rows
            __syncwarp();
            {
                const int piece = lane & 3;
                const int64_t col = col0 + piece * 4;
                const int first_row = row_in_tile & ~31;
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    const int rr = it * 8 + (lane >> 2);
                    if (first_row + rr < tl.m_rows && col < H) {
                        const uint4 val = stage[rr * 4 + (piece ^ ((rr ^ (rr >> 2)) & 3))];
                        *reinterpret_cast<uint4*>(p.act + (static_cast<int64_t>(tl.a_row0) + first_row + rr) * H + col) =
                            val;
                    }
                }
            }
            __syncwarp();
        }
        if (p.fuse_requant && row_ok) {  // (the kernel that requantises otherwise has whole rows in hand)
            atomicMax(reinterpret_cast<int*>(p.amax + row), __float_as_int(local_max));
        }
    } else if (EPI == EPI_RAW || (KIND == KIND_BF16 && p.out_dtype == W8A8_DT_F32)) {
        // 32-bit results - accumulators, or fp32 of the split operands: 32 of them are one whole 128-byte line of the row
        if (!accumulator_ready()) {
            return false;
        }
        constexpr int COLS = BLOCK_N / (EPI_WARPS / 4);
#pragma unroll 1
        for (int cc = 0; cc < COLS; cc += 32) {
            const int c = col_half * COLS + cc;
            uint32_t r[32];
            tc::tmem_ld_32x32(t_addr + c, r);
            tc::tmem_ld_wait();
            const int64_t col0 = static_cast<int64_t>(tl.nt) * BLOCK_N + c;
            if (!row_ok || col0 >= p.N) {
                continue;
            }
            const int valid = (col0 + 32 <= p.N) ? 32 : 16;  // N is a multiple of 16
            if constexpr (EPI == EPI_GMM) {
                if (p.flags & 4) {
                    const int bdt = static_cast<int>(p.flags & 3);
                    float b[32];
                    load_vec<32>(p.bias, static_cast<int64_t>(tl.group) * p.N + col0,
                                 bdt == W8A8_DT_F16 ? W8A8_QM_BIAS_F16 : (bdt == W8A8_DT_BF16 ? W8A8_QM_BIAS_BF16 : W8A8_QM_BIAS_F32),
                                 true, valid, b);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        r[j] = __float_as_uint(__fadd_rn(__uint_as_float(r[j]), b[j]));
                    }
                }
            }
            uint4* dst = reinterpret_cast<uint4*>(static_cast<uint32_t*>(p.out) + row * p.N + col0);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (q * 4 < valid) {
                    dst[q] = make_uint4(r[q * 4], r[q * 4 + 1], r[q * 4 + 2], r[q * 4 + 3]);
                }
            }
        }
    } else if constexpr (EPI == EPI_QMM || EPI == EPI_GMM) {
        return epilogue_16bit<BLOCK_N, KIND, EPI, EPI_WARPS>(p, tl, t_addr, row_in_tile, col_half, stage, accumulator_ready);
    }
    return true;
}

// Split K (SPLITK): the CTAs of a cluster each run the main loop over their share of a tile's K blocks, then deal the
// tile's columns out in slices: every CTA sends the other CTAs their slices of its accumulator through distributed
// shared memory (the stage memory, which nothing reads any more), adds what it received to its own slice - int32,
// so the order does not matter - and runs the dequant chain on it.
struct SplitSlices {
    static constexpr int COLS = 16;            // columns exchanged as one piece, 64 bytes per row
    static constexpr int PIECES = 128 / COLS;  // of a 128-column tile
    // byte offset of row `row`'s 16-byte word `word` of piece `piece` from source slot `slot`; the words are permuted
    // by the row so that eight lanes of a store hit eight different bank groups
    static __device__ __forceinline__ uint32_t offset(int slot, int pieces_per_slice, int piece, int row, int word)
    {
        return static_cast<uint32_t>(((slot * pieces_per_slice + piece) * 128 + row) * 64 + ((word ^ ((row >> 1) & 3)) << 4));
    }
};

__device__ __forceinline__ void split_send(const GemmParams& p, int m_rows, uint32_t t_addr, int row, int half, int rank,
                                           uint32_t smem_base)
{
    if ((row & ~31) >= m_rows) {
        return;  // a whole warp
    }
    const int per = SplitSlices::PIECES / p.split;
#pragma unroll 1
    for (int piece = half; piece < SplitSlices::PIECES; piece += 2) {
        const int owner = piece / per;
        if (owner == rank) {
            continue;
        }
        uint32_t r[16];
        tc::tmem_ld_32x16(t_addr + piece * 16, r);
        tc::tmem_ld_wait();
        if (row < m_rows) {
            const uint32_t to = tc::map_to_cta(smem_base, static_cast<uint32_t>(owner));
            const int slot = rank < owner ? rank : rank - 1;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                tc::st_cluster_v4(to + SplitSlices::offset(slot, per, piece - owner * per, row, w), r[4 * w], r[4 * w + 1],
                                  r[4 * w + 2], r[4 * w + 3]);
            }
        }
    }
}

template <int EPI>
__device__ __forceinline__ void split_finish(const GemmParams& p, const TileInfo& tl, uint32_t t_addr, int row_in_tile,
                                             int half, int rank, const uint8_t* smem)
{
    if ((row_in_tile & ~31) >= tl.m_rows) {
        return;  // a whole warp
    }
    const int per = SplitSlices::PIECES / p.split;
    const bool row_ok = row_in_tile < tl.m_rows;
    const int64_t row = static_cast<int64_t>(tl.a_row0) + row_in_tile;
    [[maybe_unused]] QmmTerms terms;
    if constexpr (EPI == EPI_QMM) {
        terms = qmm_terms(p, tl.group, row, row_ok);
    }
#pragma unroll 1
    for (int piece = rank * per; piece < (rank + 1) * per; ++piece) {
        if (per > 1 && (piece & 1) != half) {
            continue;
        }
        if (per == 1 && half != 0) {
            continue;
        }
        uint32_t r[16];
        tc::tmem_ld_32x16(t_addr + piece * 16, r);
        tc::tmem_ld_wait();
        const int64_t col0 = static_cast<int64_t>(tl.nt) * 128 + piece * 16;
        if (!row_ok || col0 >= p.N) {
            continue;
        }
        for (int slot = 0; slot < p.split - 1; ++slot) {
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const uint4 o = *reinterpret_cast<const uint4*>(
                    smem + SplitSlices::offset(slot, per, piece - rank * per, row_in_tile, w));
                r[4 * w] += o.x, r[4 * w + 1] += o.y, r[4 * w + 2] += o.z, r[4 * w + 3] += o.w;
            }
        }
        if constexpr (EPI == EPI_RAW) {
            uint4* dst = reinterpret_cast<uint4*>(static_cast<int32_t*>(p.out) + row * p.N + col0);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                dst[w] = make_uint4(r[4 * w], r[4 * w + 1], r[4 * w + 2], r[4 * w + 3]);
            }
        } else {
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                v[j] = static_cast<float>(static_cast<int32_t>(r[j]));
            }
            qmm_dequant<16>(p, terms, col0, 16, v);
            uint32_t o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                o[j] = (p.out_dtype == W8A8_DT_BF16) ? pack2<W8A8_DT_BF16>(v[2 * j], v[2 * j + 1])
                                                     : pack2<W8A8_DT_F16>(v[2 * j], v[2 * j + 1]);
            }
            uint4* dst = reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.out) + row * p.N + col0);
            dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
            dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
    }
}

template <int CG, int BLOCK_N, int KIND, int EPI, bool B_MN, int EPI_WARPS, bool SPLITK, bool ROW_BOXES>
__global__ void __launch_bounds__(gemm_threads(EPI_WARPS), 1)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                   const GemmParams p, const __grid_constant__ GroupListOf<EPI> groups)
{
    constexpr int ELEM = (KIND == KIND_I8) ? 1 : 2;
    constexpr int BLOCK_K = GEMM_KBYTES / ELEM;    // elements of K per stage
    constexpr int UMMA_K = 32 / ELEM;              // elements of K per instruction
    constexpr bool SPLIT_OPERANDS = (KIND == KIND_BF16 && EPI == EPI_GMM);  // may run on pieces of fp32 operands
    constexpr int CTA_N = BLOCK_N / CG;            // B columns this CTA loads
    constexpr int NBOX = CTA_N * ELEM / 128;       // MN-major: 128-byte-wide column blocks this CTA loads
    constexpr int B_BYTES = CTA_N * GEMM_KBYTES;
    constexpr int KB_BYTES = GEMM_A_BYTES + B_BYTES;           // one K block: 128 bytes of K of A and of B
    constexpr int KPS = gemm_kblocks_per_stage(CG, BLOCK_N);   // K blocks per stage
    constexpr int STAGE_BYTES = KPS * KB_BYTES;
    constexpr int STAGES = gemm_stages(CG, BLOCK_N) / KPS;
    constexpr uint32_t TMEM_COLS = 2 * BLOCK_N;    // 256 or 512: power of two
    constexpr uint32_t UMMA_M = 128 * CG;
    constexpr uint32_t IDESC =
        (KIND == KIND_I8) ? tc::instr_desc(2u, 1u, B_MN ? 1u : 0u, UMMA_M, BLOCK_N)
                          : tc::instr_desc(1u, (KIND == KIND_BF16) ? 1u : 0u, B_MN ? 1u : 0u, UMMA_M, BLOCK_N);
    static_assert(BLOCK_N == 128 || BLOCK_N == 256, "BLOCK_N");
    static_assert(CG == 1 || BLOCK_N == 256, "CTA pairs use 256-column tiles");
    static_assert(EPI != EPI_GMSQ || BLOCK_N == 256, "the SwiGLU epilogue pairs 128 gate with 128 up columns");
    static_assert(!ROW_BOXES || (CG == 1 && BLOCK_N == 256), "row boxes: single CTAs of grouped problems");
    static_assert(!SPLITK || (CG == 1 && BLOCK_N == 128 && KIND == KIND_I8 && (EPI == EPI_QMM || EPI == EPI_RAW)),
                  "split K: dense int8 matmuls on single-CTA tiles of 128 columns");
    static_assert(EPI_WARPS == 8 || EPI_WARPS == 16, "epilogue warps");

    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment: required by the 128-byte swizzle atoms.  The dynamic shared memory window starts at
    // the same offset in both CTAs of a pair, so the layout below is identical in both.
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    // bars[0..S) full, [S..2S) empty, [2S..2S+2) tmem_full, [2S+2..2S+4) tmem_empty
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 6);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    // first tiles of the groups, behind the store patches
    [[maybe_unused]] int32_t* first_tiles = reinterpret_cast<int32_t*>(smem + STAGES * STAGE_BYTES + 512 + GEMM_EPI_PATCH_BYTES);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t cta_rank = (CG == 2) ? tc::cluster_ctarank() : 0u;
    const bool leader = (cta_rank == 0);
    // this CTA's share of the K blocks
    int kb_first = 0, kb_last = p.num_k_blocks;
    [[maybe_unused]] int split_rank = 0;
    if constexpr (SPLITK) {
        split_rank = static_cast<int>(tc::cluster_ctarank());
        // the host splits no finer than one K block each: no share is empty
        kb_first = static_cast<int>(static_cast<int64_t>(split_rank) * p.num_k_blocks / p.split);
        kb_last = static_cast<int>(static_cast<int64_t>(split_rank + 1) * p.num_k_blocks / p.split);
    }
    const uint32_t smem_base = tc::smem_u32(smem);
    const uint32_t bar_base = tc::smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tfull_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };
    auto tempty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + 2 + s); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(full_bar(s), 1);   // the (leader's) producer's arrive.expect_tx; bytes from every CTA of the tile
            tc::mbar_init(empty_bar(s), 1);  // one commit (multicast to both CTAs of a pair)
        }
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(tfull_bar(s), 1);
            tc::mbar_init(tempty_bar(s), EPI_WARPS * CG);  // one arrival per epilogue warp of every CTA on the tile
        }
        *abort_flag = 0;
        tc::fence_mbar_init();
        tc::prefetch_tensormap(&tm_a);
        tc::prefetch_tensormap(&tm_b);
    }
    // Dense problems: the first K blocks of this CTA's first column tile are asked into L2 already here, beside the kernel
    // before (usually a short one that leaves HBM idle).  Nothing is read: what that kernel still writes is what the loads
    // behind the wait see.  An epilogue warp does it, the producer has its own start to prepare (with the producer, calls
    // whose weights are in L2 anyway lose 0.15 us).  Dense layer of 100 rows of 4096 x 3008 30.0 us (30.7 without), of 40
    // rows of 4096 x 8192 36.5 (37.7), of 16 rows of 7168 x 9216 49.2 (50.5); 30 rows x 4096 x 12288 15.2 (15.9); 2 rows x
    // 4096 x 4096 out of L2 7.9 (7.8).  Two K blocks gain half of it, eight or more less than four.
    if (warp == 2 && p.prefetch_k_blocks != 0 && tc::elect_one()) {
        const int64_t first = blockIdx.x / (SPLITK ? p.split : CG);
        const int32_t m_tiles = p.batch * p.m_tiles_per_batch;
        const int32_t nt = static_cast<int32_t>(first / m_tiles);
        const int32_t group = static_cast<int32_t>(first % m_tiles) / p.m_tiles_per_batch;
        // (one CTA per column tile of a batch asks for it)
        const bool mine = (first % m_tiles) % p.m_tiles_per_batch == 0;
        const int last = mine ? min(kb_last, kb_first + p.prefetch_k_blocks) : kb_first;
        for (int kb = kb_first; kb < last; ++kb) {
            if constexpr (B_MN) {
#pragma unroll
                for (int i = 0; i < NBOX; ++i) {
                    tc::tma_prefetch_l2_3d(&tm_b, nt * BLOCK_N + (static_cast<int>(cta_rank) * NBOX + i) * (128 / ELEM),
                                           kb * BLOCK_K, group);
                }
            } else {
#pragma unroll
                for (int i = 0; i < CTA_N / 128; ++i) {
                    tc::tma_prefetch_l2_3d(&tm_b, kb * BLOCK_K,
                                           nt * BLOCK_N + (static_cast<int>(cta_rank) * (CTA_N / 128) + i) * 128, group);
                }
            }
        }
    }
    if (warp == 1) {
        // each CTA allocates its own tensor memory; a pair asks for all 512 columns in both CTAs, so the
        // accumulator has the same column address in both, as the paired MMA requires
        tc::tmem_alloc(tc::smem_u32(tmem_slot), TMEM_COLS);
        tc::tmem_relinquish();
    }
    if constexpr (ROW_BOXES) {
        // Rows that no load has brought yet are zeros: their products are never stored, but multiplying what the shared
        // memory happens to hold costs as much energy as multiplying operands, and the chip runs at its power limit.
        // They stay zeros while a CTA's tiles do not shrink, which is so where every group has a few rows; a tile with
        // fewer boxes than one before it multiplies what that one left in its stages.
        for (int i = threadIdx.x; i < STAGES * KPS * (GEMM_A_BYTES / 16); i += gemm_threads(EPI_WARPS)) {
            const int block = i / (GEMM_A_BYTES / 16), word = i % (GEMM_A_BYTES / 16);
            reinterpret_cast<uint4*>(smem + (block / KPS) * STAGE_BYTES + (block % KPS) * KB_BYTES)[word] =
                make_uint4(0u, 0u, 0u, 0u);
        }
        tc::fence_async_smem();
    }
    constexpr bool GROUPED = (EPI == EPI_GMSQ || EPI == EPI_GMM);
    if constexpr (GROUPED) {
        if (warp == 3 && groups.E != 0 && groups.dev == nullptr) {
            plan_in_cta(groups, p.M, first_tiles);
        }
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if constexpr (CG == 2) {
        // both CTAs' barriers must be initialised before either signals the other
        tc::cluster_arrive();
        tc::cluster_wait();
    }
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // everything above touches shared and tensor memory only and may run beside the kernel before
    if (p.order == ORDER_FIRST_OF_TWO) {
        after_previous<false>();  // the second one starts only when everything before this kernel is complete
    } else if (p.order == ORDER_SECOND_OF_TWO) {
        // reads nothing that the first one writes, and writes other rows: it waits for it only before it ends
        beside_previous();
    } else {
        after_previous();
    }
    if constexpr (GROUPED) {
        if (groups.E != 0) {
            bool valid = true;
            if (groups.dev != nullptr) {
                if (warp == 3) {
                    valid = plan_in_cta(groups, p.M, first_tiles);
                }
                __syncthreads();
            }
            if (blockIdx.x == 0 && threadIdx.x == 96) {  // warp 3: for the requantisation, and whoever asks for the error
                p.header->num_m_tiles = first_tiles[groups.E];
                p.header->error = valid ? 0 : 1;
                p.header->rows_total = valid ? static_cast<int32_t>(groups.end_of(groups.E - 1)) : 0;
            }
        }
    }

    // ---- tile enumeration (identical in every role and in both CTAs of a pair) ----
    constexpr int TILE_M = 128 * CG;
    // Tiles are numbered with the column tile (grouped) or the row tile (dense) fastest; a worker's are num_workers apart.
    const int32_t fast_count = GROUPED ? p.n_tiles : p.batch * p.m_tiles_per_batch;
    const int32_t slow_count =
        GROUPED ? (groups_planned(groups) ? first_tiles[groups_planned(groups)] : p.header->num_m_tiles) : p.n_tiles;
    const int64_t total_tiles = static_cast<int64_t>(slow_count) * fast_count;
    const int64_t H = p.N / 2;  // GMSQ half width
    const int32_t ctas_per_tile = SPLITK ? p.split : CG;
    const int32_t worker = static_cast<int32_t>(blockIdx.x) / ctas_per_tile;
    const int32_t num_workers = static_cast<int32_t>(gridDim.x) / ctas_per_tile;
    struct Walk {
        int32_t fast, slow;
    };
    auto first_step = [&] { return Walk{worker % fast_count, worker / fast_count}; };
    const Walk stride{num_workers % fast_count, num_workers / fast_count};
    auto next_step = [&](Walk& w) {
        w.fast += stride.fast;
        w.slow += stride.slow;
        if (w.fast >= fast_count) {
            w.fast -= fast_count;
            ++w.slow;
        }
    };

    // by a whole warp
    auto decode = [&](const Walk& w) {
        TileInfo tl;
        int64_t tile_row0;
        int32_t tile_rows;
        if constexpr (GROUPED) {
            tl.nt = w.fast;
            tl.mt = w.slow;
            const TileEntry e = groups.E != 0 ? tile_in_cta(groups, first_tiles, w.slow) : p.tiles[w.slow];
            tile_row0 = e.m_start;
            tile_rows = e.m_rows;
            tl.group = e.group;
        } else {
            tl.nt = w.slow;
            tl.mt = w.fast;
            const int32_t b = p.batch == 1 ? 0 : w.fast / p.m_tiles_per_batch;
            const int64_t m0 = static_cast<int64_t>(w.fast - b * p.m_tiles_per_batch) * TILE_M;
            tile_row0 = b * p.M + m0;
            const int64_t left = p.M - m0;
            tile_rows = static_cast<int32_t>(left < TILE_M ? left : TILE_M);
            tl.group = b;
        }
        tl.a_row0 = static_cast<int32_t>(tile_row0 + 128 * static_cast<int64_t>(cta_rank));
        int32_t mine = tile_rows - 128 * static_cast<int32_t>(cta_rank);
        tl.m_rows = mine < 0 ? 0 : (mine > 128 ? 128 : mine);
        return tl;
    };
    // first column (MN-major) / first N row (K-major) of block `i` among the blocks THIS CTA loads for column
    // tile nt.  With the SwiGLU epilogue the first half of the tile's columns are gate columns and the second
    // half the matching up columns, H apart in the weight.
    auto b_block_origin = [&](int32_t nt, int i, int block_width) -> int32_t {
        const int g = static_cast<int>(cta_rank) * (CTA_N / block_width) + i;  // block index within the full tile
        const int per_half = (BLOCK_N / 2) / block_width;
        if constexpr (EPI == EPI_GMSQ) {
            const int64_t base = (g < per_half ? 0 : H) + static_cast<int64_t>(nt) * (BLOCK_N / 2);
            return static_cast<int32_t>(base + (g % per_half) * block_width);
        } else {
            return nt * BLOCK_N + g * block_width;
        }
    };

    if (warp == 0) {
        // ===================== TMA producer =====================
        {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            // a pair credits both CTAs' bytes to the leader's barrier
            const uint32_t full0 = (CG == 2) ? tc::map_to_cta(full_bar(0), 0) : full_bar(0);
            Walk at = first_step();
            for (int64_t t = worker; ok && t < total_tiles; t += num_workers, next_step(at)) {
                const TileInfo tl = decode(at);
                // ROW_BOXES: the tile's rows only, in boxes of a_box_rows
                const int a_loads = ROW_BOXES ? (tl.m_rows + p.a_box_rows - 1) / p.a_box_rows : 1;
                const uint32_t a_box_bytes = static_cast<uint32_t>(p.a_box_rows) * GEMM_KBYTES;
                const uint32_t stage_bytes = a_loads * a_box_bytes + B_BYTES;  // of one K block, per CTA
                [[maybe_unused]] int term = 0, term_kb = 0;  // SPLIT_OPERANDS: the next K block's product, and place in it
                for (int kb0 = kb_first; kb0 < kb_last; kb0 += KPS) {
                    [[maybe_unused]] int piece_kb[KPS], a_piece[KPS], b_piece[KPS];
                    if constexpr (SPLIT_OPERANDS) {
                        // (counted along, and A on a 2D map: a division, or a third coordinate, per K block held the
                        // producer up by 0.05 - 0.1 us)
#pragma unroll
                        for (int sub = 0; sub < KPS; ++sub) {
                            piece_kb[sub] = (term & 1) ? p.k_blocks_per_term - 1 - term_kb : term_kb;
                            a_piece[sub] = static_cast<int>((SPLIT_PICK_A >> (2 * term)) & 3u);
                            b_piece[sub] = static_cast<int>((SPLIT_PICK_B >> (2 * term)) & 3u);
                            if (++term_kb == p.k_blocks_per_term) {
                                term_kb = 0;
                                ++term;
                            }
                        }
                    }
                    if (!__all_sync(FULL_MASK, tc::mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag))) {
                        ok = false;
                        break;
                    }
                    const int left = kb_last - kb0;
                    const int n_sub = left < KPS ? left : KPS;  // K blocks this stage carries (the tile's last may be short)
                    const uint32_t fb = full0 + 8u * stage;
                    if (tc::elect_one()) {
                        // Only the leader announces the bytes (its own and its partner's).  The partner's copies may
                        // complete first: the barrier's phase cannot end before the leader's arrival, and a
                        // transaction count may run ahead of its announcement.
                        if (leader) {
                            tc::mbar_arrive_expect_tx(full_bar(stage),
                                                      CG * n_sub * stage_bytes);
                        }
#pragma unroll
                        for (int sub = 0; sub < KPS; ++sub) {
                            if (sub >= n_sub) {
                                break;
                            }
                            int kb = kb0 + sub;
                            int b_group = tl.group;
                            const uint32_t a_dst = smem_base + stage * STAGE_BYTES + sub * KB_BYTES;
                            const uint32_t b_dst = a_dst + GEMM_A_BYTES;
                            int a_x = kb * BLOCK_K;
                            if (SPLIT_OPERANDS && p.k_blocks_per_term != 0) {
                                kb = piece_kb[sub];
                                // a piece's last K block may run into the next piece of the row: those columns meet
                                // zeros, which is what B's map gives past K
                                a_x = a_piece[sub] * static_cast<int>(p.K) + kb * BLOCK_K;
                                b_group = b_group * SPLIT_PIECES + b_piece[sub];
                            }
                            if constexpr (CG == 2) {
                                tc::tma_load_2d_pair(a_dst, &tm_a, fb, a_x, tl.a_row0);
                            } else {
                                tc::tma_load_2d(a_dst, &tm_a, fb, a_x, tl.a_row0);
                                if constexpr (ROW_BOXES) {
#pragma unroll 1
                                    for (int i = 1; i < a_loads; ++i) {
                                        tc::tma_load_2d(a_dst + i * a_box_bytes, &tm_a, fb, a_x,
                                                        tl.a_row0 + i * p.a_box_rows);
                                    }
                                }
                            }
                            if constexpr (B_MN) {
                                // boxes of {128 bytes of N, BLOCK_K rows of K}
                                constexpr int BOX_BYTES = BLOCK_K * 128;
                                constexpr int BOX_COLS = 128 / ELEM;
#pragma unroll
                                for (int i = 0; i < NBOX; ++i) {
                                    const int32_t col = b_block_origin(tl.nt, i, BOX_COLS);
                                    if constexpr (CG == 2) {
                                        tc::tma_load_3d_pair(b_dst + i * BOX_BYTES, &tm_b, fb, col, kb * BLOCK_K, b_group);
                                    } else {
                                        tc::tma_load_3d(b_dst + i * BOX_BYTES, &tm_b, fb, col, kb * BLOCK_K, b_group);
                                    }
                                }
                            } else {
                                // boxes of {128 bytes of K, 128 rows of N}
                                constexpr int BOXES = CTA_N / 128;
#pragma unroll
                                for (int i = 0; i < BOXES; ++i) {
                                    const int32_t n_row = b_block_origin(tl.nt, i, 128);
                                    if constexpr (CG == 2) {
                                        tc::tma_load_3d_pair(b_dst + i * 128 * GEMM_KBYTES, &tm_b, fb, kb * BLOCK_K, n_row,
                                                             b_group);
                                    } else {
                                        tc::tma_load_3d(b_dst + i * 128 * GEMM_KBYTES, &tm_b, fb, kb * BLOCK_K, n_row,
                                                        b_group);
                                    }
                                }
                            }
                        }
                    }
                    __syncwarp();
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ===================== MMA issuer (leader CTA only) =====================
        // The whole warp walks the loop and waits; one elected lane issues.  (A loop run by lane 0 alone had every
        // descriptor moved to a uniform register on its way into each instruction: 8192 x 7168 x 18432 with all-zero
        // operands, which the power cap does not bound, 574 us, 590 then; 2048 x 7168 x 4096 47.2, 51.9.)
        if (leader) {
            // Descriptors as {lo, hi}: hi is loop invariant; a byte offset adds (offset >> 4) to lo.
            const uint64_t a_desc0 = tc::smem_desc_sw128(smem_base, 16, 1024);
            const uint64_t b_desc0 = B_MN ? tc::smem_desc_sw128(smem_base + GEMM_A_BYTES, BLOCK_K * 128, 1024)
                                          : tc::smem_desc_sw128(smem_base + GEMM_A_BYTES, 16, 1024);
            const uint32_t a_hi = static_cast<uint32_t>(a_desc0 >> 32);
            const uint32_t b_hi = static_cast<uint32_t>(b_desc0 >> 32);
            const uint32_t a_lo0 = static_cast<uint32_t>(a_desc0);
            const uint32_t b_lo0 = static_cast<uint32_t>(b_desc0);
            constexpr uint32_t STAGE_STEP = STAGE_BYTES >> 4;
            constexpr uint32_t KB_STEP = KB_BYTES >> 4;
            constexpr uint32_t A_KSTEP = 32 >> 4;                                   // 32 bytes of K
            constexpr uint32_t B_KSTEP = B_MN ? ((UMMA_K * 128) >> 4) : (32 >> 4);  // UMMA_K rows of 128 bytes, or 32 bytes
            constexpr int KSTEPS = BLOCK_K / UMMA_K;
            int stage = 0;
            uint32_t phase = 0;
            int64_t it = 0;
            bool ok = true;
            for (int64_t t = worker; ok && t < total_tiles; t += num_workers, ++it) {
                const int acc = static_cast<int>(it & 1);
                const uint32_t acc_phase = static_cast<uint32_t>((it >> 1) & 1);
                if (!__all_sync(FULL_MASK, tc::mbar_wait_cluster(tempty_bar(acc), acc_phase ^ 1u, abort_flag))) {
                    ok = false;
                    break;
                }
                tc::tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BLOCK_N);
                uint32_t accumulate = 0;
                for (int kb0 = kb_first; kb0 < kb_last; kb0 += KPS) {
                    // The copies are consumed by the tensor core (async proxy), not by this thread: the barrier's
                    // default acquire plus the tcgen05 fence is what orders them, also for the partner CTA's
                    // copies that complete on this barrier.
                    if (!__all_sync(FULL_MASK, tc::mbar_wait(full_bar(stage), phase, abort_flag))) {
                        ok = false;
                        break;
                    }
                    tc::tc_fence_after_sync();
                    const int left = kb_last - kb0;
                    const int n_sub = left < KPS ? left : KPS;
                    if (tc::elect_one()) {
#pragma unroll
                        for (int sub = 0; sub < KPS; ++sub) {
                            if (sub >= n_sub) {
                                break;
                            }
                            const uint32_t a_lo = a_lo0 + stage * STAGE_STEP + sub * KB_STEP;
                            const uint32_t b_lo = b_lo0 + stage * STAGE_STEP + sub * KB_STEP;
#pragma unroll
                            for (int k = 0; k < KSTEPS; ++k) {
                                tc::mma_lohi<CG, KIND == KIND_I8>(d_tmem, a_lo + k * A_KSTEP, a_hi, b_lo + k * B_KSTEP, b_hi,
                                                                 IDESC, accumulate | static_cast<uint32_t>(sub | k));
                            }
                        }
                        // one commit hands the whole stage back to the producer
                        if constexpr (CG == 2) {
                            tc::tc_commit_pair(empty_bar(stage));
                        } else {
                            tc::tc_commit(empty_bar(stage));
                        }
                    }
                    __syncwarp();
                    accumulate = 1;
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (ok && tc::elect_one()) {
                    if constexpr (CG == 2) {
                        tc::tc_commit_pair(tfull_bar(acc));
                    } else {
                        tc::tc_commit(tfull_bar(acc));
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();
    } else {
        // ===================== epilogue (warps 2 .. 2 + EPI_WARPS) =====================
        // EPI_WARPS / 4 warps per TMEM lane quarter; they split the tile's columns evenly.
        const int quarter = warp & 3;          // TMEM lanes [32*quarter, 32*quarter+32)
        const int col_half = (warp - 2) >> 2;  // which share of the columns
        const int row_in_tile = quarter * 32 + lane;
        // this warp's patch (4 KB, or 2 KB with 16 warps) for turning per-thread rows into whole-segment stores
        uint4* stage = reinterpret_cast<uint4*>(smem + STAGES * STAGE_BYTES + 512) +
                       (warp - 2) * (GEMM_EPI_PATCH_BYTES / 16 / EPI_WARPS);
        const uint32_t tempty0 = (CG == 2) ? tc::map_to_cta(tempty_bar(0), 0) : tempty_bar(0);
        int64_t it = 0;
        bool ok = true;
        // Requantisation inside this kernel (SwiGLU epilogue, optional).  The rows of a row tile are shared out
        // among the CTAs that compute its column tiles: the CTA of column tile nt quantises rows nt, nt + n_tiles,
        // ... of its 128, one row per warp at a time, once every column tile of the rows has been counted in
        // tile_done.  Column tiles of one row tile are consecutive tile numbers, so they run on different CTAs at
        // the same time (the host switches this on only when there are at least n_tiles workers): a wait here
        // only ever depends on tiles with smaller numbers than the waiter's current one, and it is bounded like
        // every other wait of the kernel.
        TileInfo late{};
        bool have_late = false;
        auto requant_share = [&](const TileInfo& d) -> bool {
            // work units of this CTA for the tile: (row d.nt + n_tiles * k, half h of the row), unit = 2 k + h
            const int units = 2 * ((d.m_rows - d.nt + p.n_tiles - 1) / p.n_tiles);
            if (warp - 2 >= units) {
                return true;
            }
            const int want = p.n_tiles * EPI_WARPS;
            int seen = 0;
            if (lane == 0) {
                const int* counter = p.tile_done + static_cast<int64_t>(d.mt) * CG + cta_rank;
                const long long t0 = clock64();
                while ((seen = tc::ld_acquire_gpu(counter)) < want) {
                    if (*abort_flag != 0 || clock64() - t0 > tc::WAIT_LIMIT_CYCLES) {
                        *abort_flag = 1;
                        break;
                    }
                    __nanosleep(100);
                }
            }
            seen = __shfl_sync(0xffffffffu, seen, 0);
            if (seen < want) {
                return false;
            }
            const int64_t n4 = H / 4, mid = n4 / 2;
            for (int u = warp - 2; u < units; u += EPI_WARPS) {
                const int64_t row = static_cast<int64_t>(d.a_row0) + d.nt + p.n_tiles * (u >> 1);
                const bool second = (u & 1) != 0;
                if (p.round_direct) {
                    requant_row_part<true>(p.act, p.amax, p.y, p.y_scale, row, H, second ? mid : 0, second ? n4 : mid,
                                           !second, lane);
                } else {
                    requant_row_part<false>(p.act, p.amax, p.y, p.y_scale, row, H, second ? mid : 0, second ? n4 : mid,
                                            !second, lane);
                }
            }
            return true;
        };
        Walk at = first_step();
        for (int64_t t = worker; ok && t < total_tiles; t += num_workers, ++it, next_step(at)) {
            const TileInfo tl = decode(at);
            touch_epilogue_operands<BLOCK_N, KIND, EPI>(p, tl, row_in_tile);
            const int acc = static_cast<int>(it & 1);
            const uint32_t acc_phase = static_cast<uint32_t>((it >> 1) & 1);
            auto accumulator_ready = [&]() {
                const bool ready = tc::mbar_wait(tfull_bar(acc), acc_phase, abort_flag);
                tc::tc_fence_after_sync();
                return ready;
            };
            if constexpr (SPLITK) {
                ok = accumulator_ready();
                break;  // one tile per cluster: its accumulators are exchanged below, by all warps together
            }
            const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                    static_cast<uint32_t>(acc * BLOCK_N);
            if (!epilogue_tile<BLOCK_N, KIND, EPI, EPI_WARPS>(p, tl, t_addr, row_in_tile, col_half, H, stage,
                                                              accumulator_ready)) {
                ok = false;
                break;
            }
            // accumulator stage drained: hand it back to the MMA issuer (one arrival per warp)
            tc::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if constexpr (CG == 2) {
                    tc::mbar_arrive_cluster(tempty0 + 8u * acc);
                } else {
                    tc::mbar_arrive(tempty0 + 8u * acc);
                }
            }
            if constexpr (EPI == EPI_GMSQ) {
                if (p.fuse_requant) {
                    // Publish this warp's activation stores and row maxima, then count the warp on its row tile:
                    // the rows are complete when n_tiles * EPI_WARPS warps have been counted.
                    __threadfence();
                    __syncwarp();
                    if (lane == 0) {
                        atomicAdd(p.tile_done + static_cast<int64_t>(tl.mt) * CG + cta_rank, 1);
                    }
                    // This tile's share of the requantisation is taken one tile late: by then the other column
                    // tiles of the same rows (on other CTAs, at about the same time) have been counted, so the wait
                    // inside costs one load.  (Two tiles late measured slower: the second pending tile goes to
                    // local memory.)
                    if (have_late && !requant_share(late)) {
                        ok = false;
                        break;
                    }
                    late = tl;
                    have_late = true;
                }
            }
        }
        if constexpr (EPI == EPI_GMSQ) {
            if (p.fuse_requant && ok && have_late) {
                requant_share(late);
            }
        }
    }

    if constexpr (SPLITK) {
        // Every CTA of the cluster has its accumulator: nothing reads the stage memory any more.
        __syncwarp();
        tc::tc_fence_before_sync();
        tc::cluster_arrive();
        tc::cluster_wait();
        tc::tc_fence_after_sync();
        const bool mine = warp >= 2 && worker < total_tiles && *abort_flag == 0;
        const int row_in_tile = (warp & 3) * 32 + lane;
        const uint32_t t_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        TileInfo tl{};
        if (mine) {
            tl = decode(first_step());
            split_send(p, tl.m_rows, t_addr, row_in_tile, (warp - 2) >> 2, split_rank, smem_base);
        }
        __syncwarp();
        tc::cluster_arrive();
        tc::cluster_wait();
        if (mine) {
            split_finish<EPI>(p, tl, t_addr, row_in_tile, (warp - 2) >> 2, split_rank, smem);
        }
        __syncwarp();
    }

    // ---- teardown ----
    if (p.order == ORDER_SECOND_OF_TWO) {
        previous_complete();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag != 0) {
        // a wait ran out: record it, then give copies still in flight time to land
        if (threadIdx.x == 0 && p.error != nullptr) {
            atomicExch(p.error, 2);
        }
        const long long t0 = clock64();
        while (clock64() - t0 < 400000ll) {
            __nanosleep(1000);
        }
        __syncthreads();
    }
    if constexpr (CG == 2) {
        // neither CTA may release tensor memory or exit while its partner can still signal it
        tc::cluster_arrive();
        tc::cluster_wait();
    }
    if (warp == 1) {
        tc::tc_fence_after_sync();
        tc::tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace w8a8
