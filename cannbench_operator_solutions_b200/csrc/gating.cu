// MoeGatingTopKSoftmax for sm_100a: per-row softmax over the experts, the k largest probabilities with their
// expert indices, and the flattened row index j * rows + r.
//
// Arithmetic follows operators/moegatingtopksoftmax/csrc/ops/moe_gating_top_k_softmax/op_kernel/
// moe_gating_kernel.cpp of the reference catalog: everything in fp32 (:28), row maximum (:305-312), x - max
// (:327), exp (:329), row sum (:333-339), descending sort of the exponentials with their indices (:344-368),
// division of the selected values by the row sum (:390), round-to-nearest-even cast to the input type (:392);
// a finished row reports `inner` as every expert index and keeps y and row_idx (:21, :285-300).
//
// Two choices the reference leaves to its hardware are fixed here and shared bit for bit with the CPU oracle:
// exp is the canonical fp32 sequence of common.cuh, and the row sum is taken in a 32-lane order (lane t adds
// elements t, t+32, ... in ascending order, then a butterfly over lane distances 16, 8, 4, 2, 1).  Equal
// exponentials are ordered by ascending expert index.
//
// Two kernels.  gating_top8_kernel (k <= 8, many rows, see four_lanes_pay) gives a row to four lanes, which is where the
// summation order puts whole 8-element pieces of a row into one lane; see there.  gating_kernel (the rest) gives a row
// to a warp: lane t owns elements t + 32 v, ranks its own once (larger exponential first, equal ones by ascending index) and parks them in
// that order in shared memory; the k selections are then k rounds of "largest head of the 32 lists" - two
// `redux.sync`, one 8-byte shared-memory load and a counter per round.  The operator moves rows * inner input
// elements and 10 k bytes of output per row; at router sizes (inner <= 1024) it is bound by issue slots, not by HBM.
#include <type_traits>

#include "common.cuh"

namespace w8a8 {

template <int DT>
__device__ __forceinline__ float gating_load(const void* x, int64_t i)
{
    if constexpr (DT == W8A8_DT_F32) {
        return static_cast<const float*>(x)[i];
    } else {
        return bits16_to_float<DT>(static_cast<const uint16_t*>(x)[i]);
    }
}

template <int DT>
__device__ __forceinline__ void gating_store(void* y, int64_t i, float v)
{
    if constexpr (DT == W8A8_DT_F32) {
        static_cast<float*>(y)[i] = v;
    } else {
        static_cast<uint16_t*>(y)[i] = float_to_bits16<DT>(v);
    }
}

constexpr int GATING_WARPS = 4;

// FULL: inner == 32 * VPT, so no element needs a bounds check.
template <int DT, int VPT, bool FULL>
__global__ void __launch_bounds__(GATING_WARPS * 32) gating_kernel(const void* x,
                                                                   const uint8_t* finished,
                                                                   void* __restrict__ y,
                                                                   int32_t* __restrict__ expert_idx,
                                                                   int32_t* __restrict__ row_idx, int64_t rows,
                                                                   int inner, int k)
{
    __shared__ int2 lists[GATING_WARPS][(VPT + 1) * 32];
    const int64_t zero = after_previous();
    const int lane = threadIdx.x & 31;
    int2* list = lists[threadIdx.x >> 5];
    const int64_t warps = static_cast<int64_t>(gridDim.x) * GATING_WARPS;
    for (int64_t r = zero + static_cast<int64_t>(blockIdx.x) * GATING_WARPS + (threadIdx.x >> 5); r < rows; r += warps) {
        float v[VPT];
        float m = -INFINITY;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int c = lane + 32 * i;
            v[i] = (FULL || c < inner) ? gating_load<DT>(x, r * inner + c) : -INFINITY;
            m = fmaxf(m, v[i]);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            m = fmaxf(m, __shfl_xor_sync(FULL_MASK, m, off));
        }
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int c = lane + 32 * i;
            if (FULL || c < inner) {
                v[i] = canonical_expf(__fsub_rn(v[i], m));
                s = __fadd_rn(s, v[i]);
            } else {
                v[i] = -1.0f;  // below every exponential: never selected
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            s = __fadd_rn(s, __shfl_xor_sync(FULL_MASK, s, off));
        }
        const bool fin = (finished != nullptr) && (finished[r] != 0);
        // Selection keys: exponentials are >= 0, so their bit patterns order like integers; what can never be
        // selected (a NaN, which fmaxf drops, and the padding past `inner`) gets the bits of -1, a negative integer.
        int key[VPT];
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            key[i] = __float_as_int(fmaxf(v[i], -1.0f));
        }
        // position of each element in the lane's own order: larger key first, equal keys by ascending i
        int pos[VPT];
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            pos[i] = 0;
        }
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
#pragma unroll
            for (int j = i + 1; j < VPT; ++j) {
                const bool first = key[i] >= key[j];  // i stays in front of j
                pos[j] += first ? 1 : 0;
                pos[i] += first ? 0 : 1;
            }
        }
        // list[p * 32 + lane] = the lane's p-th element as (key, expert index); one more entry that ends the list
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            list[pos[i] * 32 + lane] = make_int2(key[i], lane + 32 * i);
        }
        list[VPT * 32 + lane] = make_int2(-1, 0);
        // Lane j keeps the j-th selection and the lanes store together after every 32 rounds: one division and one
        // store instruction per 32 results instead of one per result.
        int keep_top = -1;
        int keep_win = 0;
        int taken = 0;  // how many of this lane's elements have been selected
        for (int j = 0; j < k; ++j) {
            const int2 head = list[taken * 32 + lane];
            const int top = __reduce_max_sync(FULL_MASK, head.x);
            // the largest exponential, and among equal ones the smallest expert index; with nothing selectable left
            // (only after NaNs) the result is a NaN with index 0
            const unsigned cand = (head.x == top && top >= 0) ? static_cast<unsigned>(head.y) : 0xffffffffu;
            const unsigned win = __reduce_min_sync(FULL_MASK, cand);
            taken += (cand == win && top >= 0) ? 1 : 0;
            if (lane == (j & 31)) {
                keep_top = top;
                keep_win = (top >= 0) ? static_cast<int>(win) : 0;
            }
            if ((j & 31) == 31 || j == k - 1) {
                const int jj = (j & ~31) + lane;  // the round this lane holds
                if (jj <= j) {
                    const float e = (keep_top >= 0) ? __int_as_float(keep_top) : NAN;
                    const int64_t o = r * k + jj;
                    gating_store<DT>(y, o, __fdiv_rn(e, s));
                    expert_idx[o] = fin ? inner : keep_win;
                    row_idx[o] = static_cast<int32_t>(static_cast<int64_t>(jj) * rows + r);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// k <= 8.  Eight rows per warp, four lanes per row: lane q of a row owns the elements 32 i + 8 q + j (j < 8), one
// 16-byte load of a 16-bit row per i, and with them the terms of the partial sums t = 8 q + j of the 32-lane order,
// so that order costs three in-lane additions and two exchanges.  Each 8 elements are sorted by a 19-comparator
// network and merged into the lane's eight best by a bitonic half-cleaner; two exchanges merge the four lanes.
//
// 16-bit rows are selected on one integer per element, the ordered bits of x above 8191 - column (the low 13 bits
// of a bf16 or fp16 value widened to fp32 are zero).  That is the order of the exponentials too - the exponential
// does not decrease (w8a8_selftest_pairs, over all floats) - except where two different x have the same exponential: such a row
// (seen from the selected exponentials, and for the last one from the exponential of the next smaller x) is selected
// once more by gating_settle, which knows the two ways in which that happens to real rows.  What is left, and a
// row whose maximum is not finite, goes to the whole warp.  fp32 rows are selected on the exponential above the column
// in 64 bits, where the question does not arise.
//
// Bound: issue slots.  65536 x 256 bf16, k = 8: 24 us (18 where rows are held, see below), was 55 with a warp per row (869
// warp instructions per row); fp32: 45 us.
// ---------------------------------------------------------------------------
constexpr int GATING_TOP = 8;
constexpr int GATING_TOP_THREADS = 64;
constexpr int GATING_COL_MASK = 0x1fff;

template <typename Key>
__device__ __forceinline__ void order_desc(Key& a, Key& b)
{
    const Key hi = a > b ? a : b;
    b = a > b ? b : a;
    a = hi;
}

template <typename Key>
__device__ __forceinline__ void sort8_desc(Key (&v)[8])
{
    order_desc(v[0], v[1]), order_desc(v[2], v[3]), order_desc(v[4], v[5]), order_desc(v[6], v[7]);
    order_desc(v[0], v[2]), order_desc(v[1], v[3]), order_desc(v[4], v[6]), order_desc(v[5], v[7]);
    order_desc(v[1], v[2]), order_desc(v[5], v[6]), order_desc(v[0], v[4]), order_desc(v[3], v[7]);
    order_desc(v[1], v[5]), order_desc(v[2], v[6]);
    order_desc(v[1], v[4]), order_desc(v[3], v[6]);
    order_desc(v[2], v[4]), order_desc(v[3], v[5]);
    order_desc(v[3], v[4]);
}

// best = the eight largest of two descending lists, descending
template <typename Key>
__device__ __forceinline__ void merge8_desc(Key (&best)[8], const Key (&other)[8])
{
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        best[i] = best[i] > other[7 - i] ? best[i] : other[7 - i];
    }
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if ((i & d) == 0) {
                order_desc(best[i], best[i + d]);
            }
        }
    }
}

// elements 8 c .. 8 c + 7 of a row, -inf past its end
template <int DT, bool VEC>
__device__ __forceinline__ void gating_load8(const void* x, int64_t row, int inner, int c, float (&v)[8])
{
    if constexpr (VEC) {
        if (8 * c >= inner) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = -INFINITY;
            }
        } else if constexpr (DT == W8A8_DT_F32) {
            const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(x) + row * inner) + 2 * c;
            const float4 a = __ldca(p), b = __ldca(p + 1);
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
            const uint4 w = __ldca(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + row * inner) + c);
            unpack2<DT>(w.x, v[0], v[1]);
            unpack2<DT>(w.y, v[2], v[3]);
            unpack2<DT>(w.z, v[4], v[5]);
            unpack2<DT>(w.w, v[6], v[7]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = (8 * c + j < inner) ? gating_load<DT>(x, row * inner + 8 * c + j) : -INFINITY;
        }
    }
}

__device__ __forceinline__ float max_nan(float a, float b)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// One row by a whole warp, straight from the definition: every round looks for the largest exponential behind the
// last selection.  For rows the fast selection cannot vouch for.
template <int DT>
__device__ __noinline__ void gating_row_by_warp(const void* x, int64_t row, int64_t rows, int inner, int k, bool fin,
                                                void* y, int32_t* expert_idx, int32_t* row_idx)
{
    const int lane = threadIdx.x & 31;
    float m = -INFINITY;
    for (int c = lane; c < inner; c += 32) {
        m = fmaxf(m, gating_load<DT>(x, row * inner + c));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        m = fmaxf(m, __shfl_xor_sync(FULL_MASK, m, off));
    }
    float s = 0.0f;
    for (int c = lane; c < inner; c += 32) {
        s = __fadd_rn(s, canonical_expf(__fsub_rn(gating_load<DT>(x, row * inner + c), m)));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        s = __fadd_rn(s, __shfl_xor_sync(FULL_MASK, s, off));
    }
    int last_key = INT32_MAX, last_col = -1;
    for (int j = 0; j < k; ++j) {
        int best = -1, best_col = 0;  // what can never be selected (a NaN) has a negative key
        for (int c = lane; c < inner; c += 32) {
            const int key = __float_as_int(fmaxf(canonical_expf(__fsub_rn(gating_load<DT>(x, row * inner + c), m)), -1.0f));
            const bool behind = key < last_key || (key == last_key && c > last_col);
            if (behind && key > best) {
                best = key;
                best_col = c;
            }
        }
        const int top = __reduce_max_sync(FULL_MASK, best);
        const unsigned col = __reduce_min_sync(FULL_MASK, best == top && top >= 0 ? static_cast<unsigned>(best_col) : ~0u);
        if (lane == 0) {
            const int64_t o = row * k + j;
            gating_store<DT>(y, o, __fdiv_rn(top >= 0 ? __int_as_float(top) : NAN, s));
            expert_idx[o] = fin ? inner : (top >= 0 ? static_cast<int>(col) : 0);
            row_idx[o] = static_cast<int32_t>(static_cast<int64_t>(j) * rows + row);
        }
        last_key = top;
        last_col = static_cast<int>(col);
    }
}

// x in the order of its value as an integer with the low 13 bits clear, and back
__device__ __forceinline__ int gating_ordered(float v)
{
    const int bits = __float_as_int(v);
    return bits ^ ((bits >> 31) & (0x7fffffff & ~GATING_COL_MASK));
}

__device__ __forceinline__ float gating_value(int ordered)
{
    return __int_as_float(ordered ^ ((ordered >> 31) & (0x7fffffff & ~GATING_COL_MASK)));
}

// A lower bound of the 16-bit x next below one that is not zero, in the same order.  (Below +0 comes -0, 0x2000 away
// for bf16 too: what is reached from +0 is a smaller x with the same exponential, which is what the caller asks for.)
template <int DT>
__device__ __forceinline__ int gating_next_below(int ordered)
{
    return ordered - ((DT == W8A8_DT_BF16) ? 0x10000 : 0x2000);
}

// lane q of a row stores the selections 2 q and 2 q + 1
template <int DT>
__device__ __forceinline__ void gating_store_two(int64_t row, int64_t rows, int inner, int k, const float (&e)[2],
                                                 const int (&col)[2], float s, const uint8_t* finished, void* y,
                                                 int32_t* expert_idx, int32_t* row_idx)
{
    const bool fin = (finished != nullptr) && (finished[row] != 0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j = 2 * (threadIdx.x & 3) + h;
        if (j < k) {
            const int64_t o = row * k + j;
            gating_store<DT>(y, o, __fdiv_rn(e[h], s));
            expert_idx[o] = fin ? inner : col[h];
            row_idx[o] = static_cast<int32_t>(static_cast<int64_t>(j) * rows + row);
        }
    }
}

// entries 2 q and 2 q + 1 of a list that the lanes of a row hold alike
template <typename Key>
__device__ __forceinline__ void gating_own_two(const Key (&best)[8], Key (&own)[2])
{
    own[0] = best[0], own[1] = best[1];
#pragma unroll
    for (int h = 1; h < 4; ++h) {
        if (static_cast<int>(threadIdx.x & 3) == h) {
            own[0] = best[2 * h];
            own[1] = best[2 * h + 1];
        }
    }
}

// Rows in which different x share an exponential, four lanes per row as in gating_top8_kernel (m: the maximum, s: the
// sum of exponentials, which that kernel has).  Two sets of x share one in real rows: those so far below the maximum
// that it is zero or nearly so (saturated or masked logits), and those around zero, whose difference from the maximum
// rounds alike (all of a row of zeros: signed zeros and the smallest numbers).  The key of the first is the exponential
// itself, below every ordered x, that of the second zero, so that the column decides among equal ones.
// Returns whether the row is settled, and stored if `wanted`; an x shared otherwise leaves it unsettled.
// 16384 rows of 256 zeros: 16.5 us, 78 by the whole warp (14.4 by the kernel with a warp per row).
template <int DT, bool VEC>
__device__ __forceinline__ bool gating_tied_rows(const void* x, int64_t row, int64_t rows, int inner, int k, float m,
                                                 float s, bool wanted, const uint8_t* finished, void* y,
                                                 int32_t* expert_idx, int32_t* row_idx)
{
    // exponentials with a bit pattern below 1024 fit between the smallest integer and the ordered bits of -inf
    constexpr int LOW = INT32_MIN, LOW_END = LOW + (1023 << 13);
    const int q = threadIdx.x & 3;
    const int pieces = (inner + 31) / 32;
    const float e_zero = m > 0.0f ? canonical_expf(-m) : 1.0f;  // of x = 0, or of the maximum where every x is negative
    int best[8];
    for (int i = 0; i < pieces; ++i) {
        float v[8];
        gating_load8<DT, VEC>(x, row, inner, 4 * i + q, v);
        f32x2 d[4], e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            d[j] = add2(pair(v[2 * j], v[2 * j + 1]), pair(-m));
        }
        exp_nonpositive2<4>(d, e);
        int key[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float e0, e1;
            unpair(e[j / 2], e0, e1);
            const float ej = (j & 1) ? e1 : e0;
            const int bits = __float_as_int(ej);
            const int value = bits < 1024 ? LOW + (bits << 13) : (ej == e_zero ? 0 : gating_ordered(v[j]));
            key[j] = value + (GATING_COL_MASK - 32 * i - 8 * q - j);
        }
        sort8_desc(key);
        if (i == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                best[j] = key[j];
            }
        } else {
            merge8_desc(best, key);
        }
    }
#pragma unroll
    for (int off = 2; off > 0; off >>= 1) {
        int other[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            other[j] = __shfl_xor_sync(FULL_MASK, best[j], off);
        }
        merge8_desc(best, other);
    }
    int own[2], xo[2], col[2];
    float e[2];
    gating_own_two(best, own);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        col[h] = GATING_COL_MASK - (own[h] & GATING_COL_MASK);
        xo[h] = own[h] & ~GATING_COL_MASK;
        e[h] = xo[h] <= LOW_END ? __int_as_float((xo[h] - LOW) >> 13)
                                : (xo[h] == 0 ? e_zero : canonical_expf(__fsub_rn(gating_value(xo[h]), m)));
    }
    const float next_e = __shfl_down_sync(FULL_MASK, e[0], 1);
    const int next_x = __shfl_down_sync(FULL_MASK, xo[0], 1);
    const int j = 2 * q;
    bool shared = j + 1 < k && e[0] == e[1] && xo[0] != xo[1];
    shared |= j + 2 < k && e[1] == next_e && xo[1] != next_x;
    const bool last0 = j == k - 1;
    const int last_x = last0 ? xo[0] : xo[1];
    if ((last0 || j + 1 == k - 1) && last_x > LOW_END && last_x != 0) {
        shared |= canonical_expf(__fsub_rn(gating_value(gating_next_below<DT>(last_x)), m)) == (last0 ? e[0] : e[1]);
    }
    const unsigned open = __ballot_sync(FULL_MASK, shared);
    const bool settled = wanted && ((open >> (threadIdx.x & 28)) & 0xfu) == 0;
    if (settled) {
        gating_store_two<DT>(row, rows, inner, k, e, col, s, finished, y, expert_idx, row_idx);
    }
    return settled;
}

// What gating_top8_kernel leaves open: rows with `open` set in their four lanes (row0: the warp's first row)
template <int DT, bool VEC>
__device__ __noinline__ void gating_settle(const void* x, int64_t row0, int64_t row, int64_t rows, int inner, int k, float m,
                                           float s, bool open, const uint8_t* finished, void* y, int32_t* expert_idx,
                                           int32_t* row_idx)
{
    if constexpr (DT != W8A8_DT_F32) {
        const bool finite = fabsf(m) < INFINITY;
        open &= !gating_tied_rows<DT, VEC>(x, row, rows, inner, k, m, s, open && finite, finished, y, expert_idx, row_idx);
    }
    unsigned again = __ballot_sync(FULL_MASK, open);
    while (again != 0) {
        const int g = (__ffs(again) - 1) >> 2;
        again &= ~(0xfu << (4 * g));
        const bool fin = (finished != nullptr) && (finished[row0 + g] != 0);
        gating_row_by_warp<DT>(x, row0 + g, rows, inner, k, fin, y, expert_idx, row_idx);
    }
}

// ---------------------------------------------------------------------------
// Rows of 129 to 256 aligned 16-bit elements: the four lanes hold their row, up to eight pieces of eight elements each, and
// sort only what can be selected.  The eighth largest of the row's 32 piece maxima is no larger than its eighth largest
// element, so only elements at or above it count: about eleven of 256, found with packed comparisons and picked out one by
// one.  A lane that has more than eight of them (rows of ties) sends its warp back to sorting every piece.
// Bound: issue slots, the integer pipe above all, of which sorting every piece takes half.  65536 x 256 bf16, k = 8 18.3 us
// (24.3 sorting every piece), x 160 14.7 (16.1), 16384 x 256 7.3 (8.3); rows that come back - few different values, or in
// order - 25.5 (22.9).  A grid that does not fill the chip twice waits for the longer chain: 8192 x 256 5.7 (5.5).
// ---------------------------------------------------------------------------
constexpr int GATING_HELD_PIECES = 8;
constexpr int64_t GATING_HELD_ROWS = 12288;

template <int DT>
struct Half2 {
    using type = std::conditional_t<DT == W8A8_DT_BF16, __nv_bfloat162, __half2>;
    static constexpr uint32_t NEG_INF = (DT == W8A8_DT_BF16) ? 0xff80ff80u : 0xfc00fc00u;
    static __device__ __forceinline__ type of(uint32_t w) { return *reinterpret_cast<const type*>(&w); }
    static __device__ __forceinline__ uint32_t bits(type v) { return *reinterpret_cast<const uint32_t*>(&v); }
    static __device__ __forceinline__ uint32_t max_nan(uint32_t a, uint32_t b) { return bits(__hmax2_nan(of(a), of(b))); }
    // all ones in the halves in which a >= b
    static __device__ __forceinline__ uint32_t at_least(uint32_t a, uint32_t b) { return __hge2_mask(of(a), of(b)); }
};

// The row's pieces of this lane, the row's maximum, and whether the row is not a regular one
template <int DT>
__device__ __forceinline__ void gating_hold(const void* x, int64_t row, int inner, int q, uint4 (&raw)[GATING_HELD_PIECES],
                                            float (&top)[GATING_HELD_PIECES])
{
    using H = Half2<DT>;
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + row * inner) + q;
#pragma unroll
    for (int i = 0; i < GATING_HELD_PIECES; ++i) {
        raw[i] = make_uint4(H::NEG_INF, H::NEG_INF, H::NEG_INF, H::NEG_INF);
        if (8 * (4 * i + q) < inner) {
            raw[i] = __ldca(p + 4 * i);
        }
    }
#pragma unroll
    for (int i = 0; i < GATING_HELD_PIECES; ++i) {
        float lo, hi;
        unpack2<DT>(H::max_nan(H::max_nan(raw[i].x, raw[i].y), H::max_nan(raw[i].z, raw[i].w)), lo, hi);
        top[i] = max_nan(lo, hi);
    }
}

// best = the lane's eight largest keys (fewer, and INT32_MIN, where it has fewer elements that can be selected)
template <int DT>
__device__ __forceinline__ void gating_held_best(const void* x, int64_t row, int inner, int q,
                                                 const uint4 (&raw)[GATING_HELD_PIECES],
                                                 const float (&top)[GATING_HELD_PIECES], int (&best)[8])
{
    using H = Half2<DT>;
    int t[8], other[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        t[i] = gating_ordered(top[i]);
    }
    sort8_desc(t);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        other[i] = __shfl_xor_sync(FULL_MASK, t[i], 2);
    }
    merge8_desc(t, other);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        other[i] = __shfl_xor_sync(FULL_MASK, t[i], 1);
    }
    int eighth = max(t[0], other[7]);
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        eighth = min(eighth, max(t[i], other[7 - i]));
    }
    const float least = gating_value(eighth);
    const uint32_t least2 = pack2<DT>(least, least);
    // bit 4 (i % 4) + w of half h: element 2 w + h of piece i
    uint32_t found[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < GATING_HELD_PIECES; ++i) {
        const uint32_t word[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            found[i >> 2] |= H::at_least(word[w], least2) & (0x00010001u << (4 * (i & 3) + w));
        }
    }
    const int count = __popc(found[0]) + __popc(found[1]);
    const int most = __reduce_max_sync(FULL_MASK, count);
    if (most > 8) {
        const int pieces = (inner + 31) / 32;
#pragma unroll 1
        for (int i = 0; i < pieces; ++i) {
            float v[8];
            gating_load8<DT, true>(x, row, inner, 4 * i + q, v);
            int key[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                key[j] = gating_ordered(v[j]) + (GATING_COL_MASK - 32 * i - 8 * q - j);
            }
            sort8_desc(key);
            if (i == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    best[j] = key[j];
                }
            } else {
                merge8_desc(best, key);
            }
        }
        return;
    }
    const uint16_t* xr = static_cast<const uint16_t*>(x) + row * inner;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        best[n] = INT32_MIN;
    }
#pragma unroll
    for (int n0 = 0; n0 < 8; n0 += 4) {
        if (n0 < most) {
#pragma unroll
            for (int n = n0; n < n0 + 4; ++n) {
                const bool low = found[0] != 0u;
                const uint32_t from = low ? found[0] : found[1];
                const int bit = __ffs(from) - 1;
                found[0] &= found[0] - 1u;
                found[1] = low ? found[1] : (found[1] & (found[1] - 1u));
                const int at = bit & 15;
                const int col = 32 * ((at >> 2) + (low ? 0 : 4)) + 8 * q + 2 * (at & 3) + (bit >> 4);
                if (n < count) {
                    best[n] = gating_ordered(bits16_to_float<DT>(xr[col])) + (GATING_COL_MASK - col);
                }
            }
        }
    }
    sort8_desc(best);
}

// HELD: rows of 129 to 256 aligned 16-bit elements
template <int DT, bool VEC, bool HELD>
__global__ void __launch_bounds__(GATING_TOP_THREADS) gating_top8_kernel(const void* x,
                                                                         const uint8_t* finished,
                                                                         void* __restrict__ y,
                                                                         int32_t* __restrict__ expert_idx,
                                                                         int32_t* __restrict__ row_idx, int64_t rows,
                                                                         int inner, int k)
{
    constexpr bool WIDE = (DT == W8A8_DT_F32);
    using Key = std::conditional_t<WIDE, unsigned long long, int>;
    const int64_t zero = after_previous();
    const int lane = threadIdx.x & 31;
    const int q = lane & 3;
    const int64_t row0 = zero + (static_cast<int64_t>(blockIdx.x) * GATING_TOP_THREADS + (threadIdx.x & ~31)) / 4;
    if (row0 >= rows) {
        return;  // a whole warp
    }
    const int64_t mine = row0 + (lane >> 2);
    const int64_t row = mine < rows ? mine : rows - 1;  // lanes past the last row work on it and store nothing
    const int pieces = (inner + 31) / 32;

    Key best[8];
    f32x2 sum[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        sum[i] = pair(0.0f);
    }
    float m = -INFINITY;
    bool redo;
    if constexpr (HELD) {
        uint4 raw[GATING_HELD_PIECES];
        float top[GATING_HELD_PIECES];
        gating_hold<DT>(x, row, inner, q, raw, top);
#pragma unroll
        for (int i = 0; i < GATING_HELD_PIECES; ++i) {
            m = max_nan(m, top[i]);
        }
        m = max_nan(m, __shfl_xor_sync(FULL_MASK, m, 1));
        m = max_nan(m, __shfl_xor_sync(FULL_MASK, m, 2));
        redo = !(fabsf(m) < INFINITY);
        gating_held_best<DT>(x, row, inner, q, raw, top, best);
#pragma unroll
        for (int i = 0; i < GATING_HELD_PIECES; ++i) {
            if (i < pieces) {
                const uint32_t word[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
                f32x2 d[4], e[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float lo, hi;
                    unpack2<DT>(word[j], lo, hi);
                    d[j] = add2(pair(lo, hi), pair(-m));
                }
                exp_nonpositive2<4>(d, e);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sum[j] = add2(sum[j], e[j]);
                }
            }
        }
    } else {
#pragma unroll 4
        for (int i = 0; i < pieces; ++i) {
            float v[8];
            gating_load8<DT, VEC>(x, row, inner, 4 * i + q, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                m = max_nan(m, v[j]);
            }
        }
        m = max_nan(m, __shfl_xor_sync(FULL_MASK, m, 1));
        m = max_nan(m, __shfl_xor_sync(FULL_MASK, m, 2));
        redo = !(fabsf(m) < INFINITY);
        // two pieces per step: 4096 x 256 bf16 4.5 us, 4.9 one at a time; 4096 x 1024 12.4, 13.2; 65536 x 256 22.8, 23.8
#pragma unroll 2
        for (int i = 0; i < pieces; ++i) {
            float v[8];
            gating_load8<DT, VEC>(x, row, inner, 4 * i + q, v);
            const int col = 32 * i + 8 * q;
            f32x2 d[4], e[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                d[j] = add2(pair(v[2 * j], v[2 * j + 1]), pair(-m));
            }
            exp_nonpositive2<4>(d, e);
            Key key[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                sum[j] = add2(sum[j], e[j]);
                if constexpr (WIDE) {
                    float e0, e1;
                    unpair(e[j], e0, e1);
                    key[2 * j] = (static_cast<Key>(__float_as_uint(e0)) << 32) | static_cast<uint32_t>(~(col + 2 * j));
                    key[2 * j + 1] = (static_cast<Key>(__float_as_uint(e1)) << 32) | static_cast<uint32_t>(~(col + 2 * j + 1));
                }
            }
            if constexpr (!WIDE) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    key[j] = gating_ordered(v[j]) + (GATING_COL_MASK - col - j);
                }
            }
            sort8_desc(key);
            if (i == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    best[j] = key[j];
                }
            } else {
                merge8_desc(best, key);
            }
        }
    }
    float part[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        unpair(sum[j], part[2 * j], part[2 * j + 1]);
    }
    // distances 16 and 8 of the 32-lane order are the lane's neighbours, 4, 2 and 1 its own eight sums
#pragma unroll
    for (int off = 2; off > 0; off >>= 1) {
        Key other[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            part[j] = __fadd_rn(part[j], __shfl_xor_sync(FULL_MASK, part[j], off));
            other[j] = __shfl_xor_sync(FULL_MASK, best[j], off);
        }
        merge8_desc(best, other);
    }
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {
#pragma unroll
        for (int j = 0; j < d; ++j) {
            part[j] = __fadd_rn(part[j], part[j + d]);
        }
    }
    const float s = part[0];

    Key own[2];
    gating_own_two(best, own);
    float e[2];
    int col[2];
    if constexpr (WIDE) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            e[h] = __uint_as_float(static_cast<uint32_t>(own[h] >> 32));
            col[h] = static_cast<int>(~static_cast<uint32_t>(own[h]));
        }
    } else {
        int xo[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            col[h] = GATING_COL_MASK - (own[h] & GATING_COL_MASK);
            xo[h] = own[h] & ~GATING_COL_MASK;
            e[h] = canonical_expf(__fsub_rn(gating_value(xo[h]), m));
        }
        const float next_e = __shfl_down_sync(FULL_MASK, e[0], 1);
        const int next_x = __shfl_down_sync(FULL_MASK, xo[0], 1);
        const int j = 2 * q;
        redo |= j + 1 < k && e[0] == e[1] && xo[0] != xo[1];
        redo |= j + 2 < k && e[1] == next_e && xo[1] != next_x;
        const bool last0 = j == k - 1;
        if (last0 || j + 1 == k - 1) {
            redo |= canonical_expf(__fsub_rn(gating_value(gating_next_below<DT>(last0 ? xo[0] : xo[1])), m)) ==
                    (last0 ? e[0] : e[1]);
        }
    }
    const unsigned flagged = __ballot_sync(FULL_MASK, redo && mine < rows);
    const bool open = ((flagged >> (lane & ~3)) & 0xfu) != 0;
    if (mine < rows && !open) {
        gating_store_two<DT>(row, rows, inner, k, e, col, s, finished, y, expert_idx, row_idx);
    }
    if (flagged != 0) {
        gating_settle<DT, VEC>(x, row0, row, rows, inner, k, m, s, open, finished, y, expert_idx, row_idx);
    }
}

// A grid that fills more than half of the SMs but not all of them starts when the kernel before it has completed: of two
// such grids at once only part of the second finds a place beside the first, and the rest piles onto the SMs that the
// first leaves early.  Back to back, 32768 x 256 bf16 17.1 us, 13.8 in turn; 2048 x 1024 with a warp per row 18.5, 14.3.
template <auto KERN, typename... Args>
static cudaError_t launch_router(unsigned grid, unsigned threads, cudaStream_t st, Args... args)
{
    static KernelFacts facts;
    int ctas = 1;
    const cudaError_t e = resident_ctas(facts, KERN, static_cast<int>(threads), &ctas);
    if (e != cudaSuccess) {
        return e;
    }
    const int64_t places = static_cast<int64_t>(sm_count()) * ctas;
    return launch_chained_if(2 * static_cast<int64_t>(grid) <= places || grid >= places, KERN, grid, threads, 0, st, args...);
}

template <int DT>
static cudaError_t launch_gating_top8(const void* x, const uint8_t* finished, void* y, int32_t* expert_idx,
                                      int32_t* row_idx, int64_t rows, int inner, int k, cudaStream_t st)
{
    constexpr int64_t ROWS = GATING_TOP_THREADS / 4;
    const unsigned grid = static_cast<unsigned>((rows + ROWS - 1) / ROWS);
    if (inner % 8 == 0 && is_aligned(x, 16)) {
        if constexpr (DT != W8A8_DT_F32) {
            if (inner > 128 && inner <= 32 * GATING_HELD_PIECES && rows >= GATING_HELD_ROWS) {
                return launch_router<gating_top8_kernel<DT, true, true>>(grid, GATING_TOP_THREADS, st, x, finished, y,
                                                                         expert_idx, row_idx, rows, inner, k);
            }
        }
        return launch_router<gating_top8_kernel<DT, true, false>>(grid, GATING_TOP_THREADS, st, x, finished, y, expert_idx, row_idx,
                                                           rows, inner, k);
    }
    return launch_router<gating_top8_kernel<DT, false, false>>(grid, GATING_TOP_THREADS, st, x, finished, y, expert_idx, row_idx,
                                                        rows, inner, k);
}

template <int DT, int VPT>
static cudaError_t launch_gating(const void* x, const uint8_t* finished, void* y, int32_t* expert_idx,
                                 int32_t* row_idx, int64_t rows, int inner, int k, cudaStream_t st)
{
    const int64_t want = (rows + GATING_WARPS - 1) / GATING_WARPS;
    const int64_t cap = static_cast<int64_t>(sm_count()) * 16;
    const unsigned grid = static_cast<unsigned>(want < cap ? want : cap);
    if (inner == 32 * VPT) {
        return launch_router<gating_kernel<DT, VPT, true>>(grid, GATING_WARPS * 32, st, x, finished, y, expert_idx, row_idx,
                                                           rows, inner, k);
    }
    return launch_router<gating_kernel<DT, VPT, false>>(grid, GATING_WARPS * 32, st, x, finished, y, expert_idx, row_idx,
                                                        rows, inner, k);
}

// Four lanes per row or a warp?  Both kernels' times in us are close to lines in the rows (r thousand of them), fitted to
// 896 calls of 4096 - 65536 rows, 8 - 1024 columns, k = 1 - 8, bf16 and fp32, and the shorter one is taken.  A warp pays
// for the columns rounded up to 32, 64, ... 1024 and for every selection; four lanes pay for the columns themselves, not
// for k, more for fp32 (64-bit keys) and for rows that are read an element at a time, and start later.  Measured, warp
// and four lanes: 65536 x 256 bf16, k = 8 53 and 24; 16384 x 256 fp32, k = 1 10.5 and 15.4; 4096 x 500 bf16, k = 1 8.0 and
// 10.5; 4096 x 264 bf16, k = 1 7.3 and 5.4.  The choice lost 0.2 % on the average and 20 % at most (8192 x 500, k = 4).
template <int DT>
static bool four_lanes_pay(int64_t rows, int inner, int k, bool vec)
{
    constexpr double WARP_ROW[6] = {0.139, 0.174, 0.268, 0.500, 1.333, 5.393};
    int v = 0;
    while ((32 << v) < inner) {
        ++v;
    }
    const double r = static_cast<double>(rows) * 1e-3;
    const double warp = 1.76 + r * (WARP_ROW[v] + 0.033 * k);
    const double four = (DT == W8A8_DT_F32) ? (vec ? 1.64 + 0.0079 * inner + r * (0.067 + 0.0026 * inner)
                                                   : 1.77 + 0.0097 * inner + r * (0.056 + 0.0034 * inner))
                                            : (vec ? 1.63 + 0.0068 * inner + r * (0.050 + 0.00118 * inner)
                                                   : 1.66 + 0.0102 * inner + r * (0.048 + 0.00162 * inner));
    return four < warp;
}

template <int DT>
static cudaError_t dispatch_gating(const void* x, const uint8_t* finished, void* y, int32_t* expert_idx,
                                   int32_t* row_idx, int64_t rows, int inner, int k, cudaStream_t st)
{
    if (k <= GATING_TOP && rows >= 4096 && four_lanes_pay<DT>(rows, inner, k, inner % 8 == 0 && is_aligned(x, 16))) {
        return launch_gating_top8<DT>(x, finished, y, expert_idx, row_idx, rows, inner, k, st);
    }
    if (inner <= 32) {
        return launch_gating<DT, 1>(x, finished, y, expert_idx, row_idx, rows, inner, k, st);
    }
    if (inner <= 64) {
        return launch_gating<DT, 2>(x, finished, y, expert_idx, row_idx, rows, inner, k, st);
    }
    if (inner <= 128) {
        return launch_gating<DT, 4>(x, finished, y, expert_idx, row_idx, rows, inner, k, st);
    }
    if (inner <= 256) {
        return launch_gating<DT, 8>(x, finished, y, expert_idx, row_idx, rows, inner, k, st);
    }
    if (inner <= 512) {
        return launch_gating<DT, 16>(x, finished, y, expert_idx, row_idx, rows, inner, k, st);
    }
    return launch_gating<DT, 32>(x, finished, y, expert_idx, row_idx, rows, inner, k, st);
}

}  // namespace w8a8

extern "C" int w8a8_moe_gating_top_k_softmax(const void* x, const uint8_t* finished, void* y, int32_t* expert_idx,
                                             int32_t* row_idx, int64_t rows, int64_t inner, int64_t k, int dtype,
                                             void* stream)
{
    if (dtype != W8A8_DT_F16 && dtype != W8A8_DT_BF16 && dtype != W8A8_DT_F32) {
        return W8A8_ERR_INVALID;
    }
    if (rows < 0 || inner <= 0 || k <= 0 || k > inner) {
        return W8A8_ERR_INVALID;
    }
    if (inner > W8A8_GATING_MAX_EXPERTS || rows * k > INT32_MAX) {
        return W8A8_ERR_LIMIT;
    }
    if (rows == 0) {
        return W8A8_OK;
    }
    if (x == nullptr || y == nullptr || expert_idx == nullptr || row_idx == nullptr) {
        return W8A8_ERR_INVALID;
    }
    const size_t elem = (dtype == W8A8_DT_F32) ? 4 : 2;
    if (!w8a8::is_aligned(x, elem) || !w8a8::is_aligned(y, elem)) {
        return W8A8_ERR_ALIGN;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int in = static_cast<int>(inner), kk = static_cast<int>(k);
    cudaError_t e;
    switch (dtype) {
    case W8A8_DT_F16:
        e = w8a8::dispatch_gating<W8A8_DT_F16>(x, finished, y, expert_idx, row_idx, rows, in, kk, st);
        break;
    case W8A8_DT_BF16:
        e = w8a8::dispatch_gating<W8A8_DT_BF16>(x, finished, y, expert_idx, row_idx, rows, in, kk, st);
        break;
    default:
        e = w8a8::dispatch_gating<W8A8_DT_F32>(x, finished, y, expert_idx, row_idx, rows, in, kk, st);
        break;
    }
    return w8a8::launch_status(e);
}
