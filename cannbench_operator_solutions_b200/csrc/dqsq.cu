// DequantSwigluQuant for sm_100a: dequantise a [M, 2H] matmul result, SwiGLU, smooth scale, per-token int8
// quantisation, one HBM pass.
//
// Arithmetic follows operators/dequantswigluquant/csrc/ops/dequant_swiglu_quant/op_kernel/dqsq_kernel.cpp of the
// reference catalog, in the order its vector instructions run:
//   int32 input:  a = float(x[:, :H]) * weight_scale[:H], b = float(x[:, H:]) * weight_scale[H:]   (:335-347)
//   16-bit input: a, b = float(x) halves                                                            (:298-329)
//   quant_scale multiplies the half that is NOT the gate input, before the gate is formed          (:349-363)
//   int32 input:  a *= activation_scale[row], b *= activation_scale[row]                            (:386-410)
//   gate = b (activate_left == 0) or a: out = (a * b) / (1 + exp(gate * -1))                        (:415-428)
//   m = max |out| (not-greater-than-zero, NaN included, counts as 0), s = max(m * (1/127), 1e-12)   (:434-499)
//   y = narrow(clamp(out / s, -128, 127)), fp32 -> fp16 -> int8 with round-to-nearest-even twice    (:509-524)
// The reference scales by out / s in its batched short-row layout (:482) and by out * (1 / s) otherwise
// (:500-504).  Its batched layout needs a padded half-row of at most 1984 elements (:97) and, per tile, fewer
// 64-column chunks than rows (:272), which depends on its on-chip buffer tiling; this build divides when the
// padded half-row is at most 1984 elements long and multiplies by the reciprocal for longer rows, so the two
// can differ by one int8 step on the rare element where the two roundings disagree.  exp is the canonical fp32
// sequence shared with the CPU oracle; a NaN activation quantises to 0.
//
// Mapping: one CTA per row at a time (grid-stride, one wave), one or two 16-byte chunks of each half per thread and
// as many threads as that takes.  The fp32 results stay in registers between the row maximum and the quantisation,
// so x is read once and y written once: 8H + H + 4 bytes per row for int32 input, 4H + H + 4 for 16-bit input; the
// next row's chunks are requested before the barrier of the present one.
#include <algorithm>

#include "common.cuh"

namespace w8a8 {

constexpr int DQSQ_X_I32 = 0;
constexpr int DQSQ_X_F16 = 1;
constexpr int DQSQ_X_BF16 = 2;
constexpr int DQSQ_THREADS = 256;       // any-length kernel
constexpr int DQSQ_MAX_THREADS = 1024;  // register-resident rows
constexpr int DQSQ_PAIR_THREADS = 576;  // up to here two CTAs share an SM's registers at 56 per thread

template <int XT>
struct DqsqChunk {
    static constexpr int EL = (XT == DQSQ_X_I32) ? 4 : 8;

    // 16 raw bytes starting at element `first` of the row
    static __device__ __forceinline__ uint4 load_raw(const void* row, int64_t first)
    {
        constexpr size_t ELEM = (XT == DQSQ_X_I32) ? 4 : 2;
        return __ldcs(reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(row) + first * ELEM));
    }

    static __device__ __forceinline__ void unpack(const uint4& v, float (&f)[EL])
    {
        if constexpr (XT == DQSQ_X_I32) {
            f[0] = static_cast<float>(static_cast<int32_t>(v.x)), f[1] = static_cast<float>(static_cast<int32_t>(v.y));
            f[2] = static_cast<float>(static_cast<int32_t>(v.z)), f[3] = static_cast<float>(static_cast<int32_t>(v.w));
        } else {
            constexpr int DT = (XT == DQSQ_X_F16) ? W8A8_DT_F16 : W8A8_DT_BF16;
            unpack2<DT>(v.x, f[0], f[1]);
            unpack2<DT>(v.y, f[2], f[3]);
            unpack2<DT>(v.z, f[4], f[5]);
            unpack2<DT>(v.w, f[6], f[7]);
        }
    }

    static __device__ __forceinline__ float load1(const void* row, int64_t i)
    {
        if constexpr (XT == DQSQ_X_I32) {
            return static_cast<float>(static_cast<const int32_t*>(row)[i]);
        } else if constexpr (XT == DQSQ_X_F16) {
            return bits16_to_float<W8A8_DT_F16>(static_cast<const uint16_t*>(row)[i]);
        } else {
            return bits16_to_float<W8A8_DT_BF16>(static_cast<const uint16_t*>(row)[i]);
        }
    }
};

// one output element, in the reference's operation order
template <int XT>
__device__ __forceinline__ float dqsq_element(float a, float b, float wa, float wb, float qs, float as, bool has_q,
                                              bool left)
{
    if constexpr (XT == DQSQ_X_I32) {
        a = __fmul_rn(a, wa);
        b = __fmul_rn(b, wb);
    }
    if (has_q) {
        if (left) {
            b = __fmul_rn(b, qs);
        } else {
            a = __fmul_rn(a, qs);
        }
    }
    if constexpr (XT == DQSQ_X_I32) {
        a = __fmul_rn(a, as);
        b = __fmul_rn(b, as);
    }
    const float gate = left ? a : b;
    const float den = __fadd_rn(canonical_expf(__fmul_rn(gate, -1.0f)), 1.0f);
    return __fdiv_rn(__fmul_rn(a, b), den);
}

// N elements with the two halves named by role (g: the half the gate is formed from, o: the other one) and the
// smooth scale always applied (1 when the caller gave none; a multiplication by 1 is exact): a * b commutes, and
// gate * -1 is a sign flip, so the bits are those of dqsq_element.  Two at a time by the pair forms where all of
// them are in range, which only gates beyond +-80 or products beyond 2^100 are not.  (Products below 2^-60 may come
// out one unit off there: at most 1e-18, they neither reach the scale, which is at least 1e-12, nor any value but 0.)
template <int XT, int N>
__device__ __forceinline__ void dqsq_elements(const float (&g)[N], const float (&o)[N], const float (&wg)[N],
                                              const float (&wo)[N], const float (&qs)[N], float as, float (&out)[N])
{
    f32x2 gate[N / 2], num[N / 2], den[N / 2], res[N / 2];
    float g_max = 0.0f, n_max = 0.0f;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        f32x2 op = pair(o[2 * i], o[2 * i + 1]);
        gate[i] = pair(g[2 * i], g[2 * i + 1]);
        if constexpr (XT == DQSQ_X_I32) {
            gate[i] = mul2(mul2(gate[i], pair(wg[2 * i], wg[2 * i + 1])), pair(as));
            op = mul2(op, pair(wo[2 * i], wo[2 * i + 1]));
        }
        op = mul2(op, pair(qs[2 * i], qs[2 * i + 1]));
        if constexpr (XT == DQSQ_X_I32) {
            op = mul2(op, pair(as));
        }
        num[i] = mul2(gate[i], op);
        float a0, a1, n0, n1;
        unpair(gate[i], a0, a1);
        unpair(num[i], n0, n1);
        g_max = fmaxf(g_max, fmaxf(fabsf(a0), fabsf(a1)));
        n_max = fmaxf(n_max, fmaxf(fabsf(n0), fabsf(n1)));
    }
    neg_exp_neg2<N / 2>(gate, den);
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        den[i] = add2(den[i], pair(-1.0f));
    }
    quotient2<N / 2>(num, den, res);
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        unpair(res[i], out[2 * i], out[2 * i + 1]);
    }
    if (!(g_max <= EXP2_MAX_ABS && n_max <= 1.2676506e30f)) {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            float a0, a1, n0, n1;
            unpair(gate[i], a0, a1);
            unpair(num[i], n0, n1);
            out[2 * i] = __fdiv_rn(n0, __fadd_rn(canonical_expf(-a0), 1.0f));
            out[2 * i + 1] = __fdiv_rn(n1, __fadd_rn(canonical_expf(-a1), 1.0f));
        }
    }
}

// `slots`: two sets of one float per warp of the CTA, used in turn
__device__ __forceinline__ float dqsq_block_max(float m, float* slots, int parity)
{
    const int warps = static_cast<int>(blockDim.x >> 5);
    const int lane = threadIdx.x & 31;
    // non-negative floats order like their bit patterns
    const int own = __reduce_max_sync(FULL_MASK, __float_as_int(m));
    float* slot = slots + parity * 32;
    if (lane == 0) {
        slot[threadIdx.x >> 5] = __int_as_float(own);
    }
    __syncthreads();
    return __int_as_float(__reduce_max_sync(FULL_MASK, lane < warps ? __float_as_int(slot[lane]) : 0));
}

// out / s, or out * (1 / s) with `s` already holding the reciprocal
__device__ __forceinline__ float dqsq_scaled(float o, float s, bool divide)
{
    return divide ? __fdiv_rn(o, s) : __fmul_rn(o, s);
}

template <bool DIVIDE>
__device__ __forceinline__ uint32_t dqsq_quant4_general(const float* o, float s, bool direct)
{
    constexpr bool divide = DIVIDE;
    float v[4];
    bool any_nan = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float q = dqsq_scaled(o[j], s, divide);
        any_nan |= (q != q);
        v[j] = fmaxf(fminf(q, 127.0f), -128.0f);
    }
    uint32_t packed = direct ? narrow4_fast<true>(v[0], v[1], v[2], v[3]) : narrow4_fast<false>(v[0], v[1], v[2], v[3]);
    if (any_nan) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float q = dqsq_scaled(o[j], s, divide);
            if (q != q) {
                packed &= ~(0xffu << (8 * j));
            }
        }
    }
    return packed;
}

// Four results quantised the way narrow4_fp16_fast does, without the clamp: no |out| exceeds the row maximum, so
// every quotient is at most 127 (1 + 2^-22) and rounds to at most 127 in fp16.  `inv` is RN(1 / s).  DIVIDE: out / s
// by one remainder correction of out * inv (Markstein, as in quotient2; s is the same for the whole row, so the
// reciprocal costs nothing here).  A NaN leaves a bit set in the fp16 sum that no value from 1408 to 1663 has.
template <bool DIVIDE>
__device__ __forceinline__ uint32_t dqsq_quant4(const float* o, float s, float inv, bool regular, bool direct)
{
    if (!regular) {
        return dqsq_quant4_general<DIVIDE>(o, DIVIDE ? s : inv, direct);
    }
    __half2 h[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const f32x2 v = pair(o[2 * j], o[2 * j + 1]);
        f32x2 q = mul2(v, pair(inv));
        if constexpr (DIVIDE) {
            q = fma2(fma2(q, pair(-s), v), pair(inv), q);
        }
        float q0, q1;
        unpair(q, q0, q1);
        h[j] = __hadd2(__floats2half2_rn(q0, q1), __floats2half2_rn(1536.0f, 1536.0f));
    }
    const uint32_t h01 = *reinterpret_cast<const uint32_t*>(&h[0]), h23 = *reinterpret_cast<const uint32_t*>(&h[1]);
    if (((h01 | h23) & 0x10001000u) != 0) {
        return dqsq_quant4_general<DIVIDE>(o, DIVIDE ? s : inv, direct);
    }
    return __byte_perm(h01, h23, 0x6420);
}

// Register-resident rows: H a multiple of the chunk length, at most blockDim.x * EL * CPT long.
//
// Bound: issue slots (44 warp instructions per 32 elements against 73 with a scalar exponential and the compiler's
// division), then HBM.  int32 [16384, 4096] (302 MB): 66 us, was 86; fp16 [1531, 18432] (70 MB): 24 us, was 58
// with a fixed 256 threads per row (eight chunks per thread, 44 % of them past the row's end).
template <int XT, int CPT, bool DIVIDE, int MAX_THREADS>
__global__ void __launch_bounds__(MAX_THREADS, MAX_THREADS <= DQSQ_PAIR_THREADS ? 2 : 1)
    dqsq_rows_kernel(const void* x, const float* weight_scale,
                     const float* activation_scale, const float* quant_scale,
                     int8_t* __restrict__ y, float* __restrict__ scale, int64_t M, int64_t H, int left, int direct, int)
{
    using C = DqsqChunk<XT>;
    constexpr int EL = C::EL;
    constexpr int N = CPT * EL;
    constexpr int GROUP = (EL == 4) ? CPT : 1;  // chunks that go through the arithmetic together: 8 elements
    constexpr int GN = GROUP * EL;
    constexpr size_t ELEM = (XT == DQSQ_X_I32) ? 4 : 2;
    __shared__ float s_red[2 * 32];
    const int64_t zero = after_previous<false>();
    const int64_t first_row = blockIdx.x + zero;
    const int tid = threadIdx.x;
    const int threads = static_cast<int>(blockDim.x);
    const int nchunks = static_cast<int>(H / EL);
    const bool has_q = (quant_scale != nullptr);
    // where the gate half and the other half start, in the row and in weight_scale
    const int64_t g_off = left ? 0 : H, o_off = left ? H : 0;
    // a chunk past the end is all zeros: its results are zeros, and it is not stored
    uint4 cg[CPT], co[CPT];
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
        cg[i] = co[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    float as = 1.0f;
    const uint8_t* xg = static_cast<const uint8_t*>(x) + (static_cast<size_t>(first_row) * 2 * H + g_off) * ELEM + tid * 16;
    const int64_t to_other = (o_off - g_off) * static_cast<int64_t>(ELEM);
    const size_t row_step = static_cast<size_t>(gridDim.x) * 2 * H * ELEM;
    auto load_row = [&](int64_t row) {
#pragma unroll
        for (int i = 0; i < CPT; ++i) {
            if (tid + i * threads < nchunks) {
                cg[i] = C::load_raw(xg + i * threads * 16, 0);
                co[i] = C::load_raw(xg + to_other + i * threads * 16, 0);
            }
        }
        if constexpr (XT == DQSQ_X_I32) {
            as = activation_scale[row];
        }
        xg += row_step;
    };
    int parity = 0;
    if (first_row < M) {
        load_row(first_row);
    }
    for (int64_t row = first_row; row < M; row += gridDim.x, parity ^= 1) {
        float out[N];
#pragma unroll
        for (int i0 = 0; i0 < CPT; i0 += GROUP) {
            float g[GN], o[GN], wg[GN], wo[GN], qs[GN];
#pragma unroll
            for (int i = 0; i < GROUP; ++i) {
                float gi[EL], oi[EL];
                C::unpack(cg[i0 + i], gi);
                C::unpack(co[i0 + i], oi);
                // per-channel vectors are re-read by every row: cached 128-bit loads (the launcher checks alignment)
                const int64_t j0 = static_cast<int64_t>(min(tid + (i0 + i) * threads, nchunks - 1)) * EL;
#pragma unroll
                for (int q = 0; q < EL / 4; ++q) {
                    float4 a = make_float4(1.0f, 1.0f, 1.0f, 1.0f), b = a, c = a;
                    if constexpr (XT == DQSQ_X_I32) {
                        a = __ldca(reinterpret_cast<const float4*>(weight_scale + g_off + j0) + q);
                        b = __ldca(reinterpret_cast<const float4*>(weight_scale + o_off + j0) + q);
                    }
                    if (has_q) {
                        c = __ldca(reinterpret_cast<const float4*>(quant_scale + j0) + q);
                    }
                    const int at = i * EL + 4 * q;
                    wg[at] = a.x, wg[at + 1] = a.y, wg[at + 2] = a.z, wg[at + 3] = a.w;
                    wo[at] = b.x, wo[at + 1] = b.y, wo[at + 2] = b.z, wo[at + 3] = b.w;
                    qs[at] = c.x, qs[at + 1] = c.y, qs[at + 2] = c.z, qs[at + 3] = c.w;
                }
#pragma unroll
                for (int j = 0; j < EL; ++j) {
                    g[i * EL + j] = gi[j];
                    o[i * EL + j] = oi[j];
                }
            }
            float r[GN];
            dqsq_elements<XT, GN>(g, o, wg, wo, qs, as, r);
#pragma unroll
            for (int j = 0; j < GN; ++j) {
                out[i0 * EL + j] = r[j];
            }
        }
        float m = 0.0f;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            m = fmaxf(m, fabsf(out[j]));
        }
        if (row + gridDim.x < M) {
            load_row(row + gridDim.x);
        }
        m = dqsq_block_max(m, s_red, parity);
        float s = __fmul_rn(m, INV127);
        if (s < 1e-12f) {
            s = 1e-12f;
        }
        if (tid == 0) {
            scale[row] = s;
        }
        const float inv = __frcp_rn(s);
        const bool regular = (direct == 0) && s < 1.0e18f;
        int8_t* yr = y + row * H;
#pragma unroll
        for (int i = 0; i < CPT; ++i) {
            const int c = tid + i * threads;
            if (c < nchunks) {
                const int64_t j0 = static_cast<int64_t>(c) * EL;
                const float* oi = out + i * EL;
                if constexpr (EL == 4) {
                    *reinterpret_cast<uint32_t*>(yr + j0) = dqsq_quant4<DIVIDE>(oi, s, inv, regular, direct != 0);
                } else {
                    const uint2 w = make_uint2(dqsq_quant4<DIVIDE>(oi, s, inv, regular, direct != 0),
                                               dqsq_quant4<DIVIDE>(oi + 4, s, inv, regular, direct != 0));
                    *reinterpret_cast<uint2*>(yr + j0) = w;
                }
            }
        }
    }
}

// Any H and any alignment: two passes over the row, the second recomputes the activations (normally from L2).
template <int XT>
__global__ void __launch_bounds__(DQSQ_THREADS) dqsq_long_rows_kernel(const void* x,
                                                                      const float* weight_scale,
                                                                      const float* activation_scale,
                                                                      const float* quant_scale,
                                                                      int8_t* __restrict__ y, float* __restrict__ scale,
                                                                      int64_t M, int64_t H, int left, int direct, int divide)
{
    using C = DqsqChunk<XT>;
    __shared__ float s_red[2 * 32];
    const int64_t zero = after_previous<false>();
    const size_t elem = (XT == DQSQ_X_I32) ? 4 : 2;
    const bool has_q = (quant_scale != nullptr);
    int parity = 0;
    for (int64_t row = blockIdx.x + zero; row < M; row += gridDim.x, parity ^= 1) {
        const uint8_t* xr = static_cast<const uint8_t*>(x) + static_cast<size_t>(row) * 2 * H * elem;
        const float as = (XT == DQSQ_X_I32) ? activation_scale[row] : 1.0f;
        auto element = [&](int64_t j) {
            const float wa = (XT == DQSQ_X_I32) ? weight_scale[j] : 1.0f;
            const float wb = (XT == DQSQ_X_I32) ? weight_scale[H + j] : 1.0f;
            const float qs = has_q ? quant_scale[j] : 1.0f;
            return dqsq_element<XT>(C::load1(xr, j), C::load1(xr, H + j), wa, wb, qs, as, has_q, left != 0);
        };
        float m = 0.0f;
        for (int64_t j = threadIdx.x; j < H; j += DQSQ_THREADS) {
            m = fmaxf(m, fabsf(element(j)));
        }
        m = dqsq_block_max(m, s_red, parity);
        float s = __fmul_rn(m, INV127);
        if (s < 1e-12f) {
            s = 1e-12f;
        }
        if (threadIdx.x == 0) {
            scale[row] = s;
        }
        const float qf = divide ? s : __fdiv_rn(1.0f, s);
        for (int64_t j = threadIdx.x; j < H; j += DQSQ_THREADS) {
            const float q = dqsq_scaled(element(j), qf, divide != 0);
            const float v = fmaxf(fminf(q, 127.0f), -128.0f);
            y[row * H + j] = (q != q) ? static_cast<int8_t>(0)
                                      : static_cast<int8_t>(direct ? narrow1_general<true>(v) : narrow1_general<false>(v));
        }
    }
}

template <int XT>
static cudaError_t dispatch_dqsq(const void* x, const float* ws, const float* as, const float* qs, int8_t* y,
                                 float* scale, int64_t M, int64_t H, int left, int direct, bool vec, cudaStream_t st)
{
    constexpr int EL = DqsqChunk<XT>::EL;
    // padded half-row length of the reference's layout choice: H rounded up to 32 bytes of the input type
    constexpr int64_t PAD = (XT == DQSQ_X_I32) ? 8 : 16;
    const int divide = ((H + PAD - 1) / PAD * PAD <= 1984) ? 1 : 0;
    const int64_t chunks = (H + EL - 1) / EL;
    using Kern = void (*)(const void*, const float*, const float*, const float*, int8_t*, float*, int64_t, int64_t, int,
                          int, int);
    Kern kern = dqsq_long_rows_kernel<XT>;
    int threads = DQSQ_THREADS;
    int64_t per_sm = 1;
    if (vec && chunks <= 2 * DQSQ_MAX_THREADS) {
        // Two chunks of each half per thread (one where a row has at most a warp's worth), rounded up to whole warps:
        // a thread count fitted to the row leaves few lanes idle on rows that are not a power of two long.  (Four
        // int32 chunks per thread spill and take 79 us where two take 64 on [16384, 4096].)  16-bit rows take the
        // 56-register form up to 576 threads: it puts two CTAs on an SM (24 against 27 us on fp16 [1531, 18432]).
        const bool two = chunks > 32;
        threads = static_cast<int>((((two ? (chunks + 1) / 2 : chunks) + 31) / 32) * 32);
        const int regs = (XT == DQSQ_X_I32 && two) || threads > DQSQ_PAIR_THREADS ? 64 : 56;
        // (chosen where compiled, so that no form is built that no call reaches)
        if (!two) {
            kern = dqsq_rows_kernel<XT, 1, true, DQSQ_PAIR_THREADS>;  // rows this short always divide
        } else if constexpr (XT == DQSQ_X_I32) {
            kern = divide ? dqsq_rows_kernel<XT, 2, true, DQSQ_MAX_THREADS> : dqsq_rows_kernel<XT, 2, false, DQSQ_MAX_THREADS>;
        } else {
            // rows that divide are at most 1984 long: 576 threads are enough
            kern = divide ? dqsq_rows_kernel<XT, 2, true, DQSQ_PAIR_THREADS>
                          : (threads <= DQSQ_PAIR_THREADS ? dqsq_rows_kernel<XT, 2, false, DQSQ_PAIR_THREADS>
                                                          : dqsq_rows_kernel<XT, 2, false, DQSQ_MAX_THREADS>);
        }
        per_sm = std::min(std::max(1, 65536 / (regs * threads)), 32);
    } else {
        static KernelFacts facts;
        int ctas = 1;
        const cudaError_t e = resident_ctas(facts, kern, threads, &ctas);
        if (e != cudaSuccess) {
            return e;
        }
        per_sm = ctas;
    }
    // one wave: as many CTAs as the registers hold at once, each walking rows with a grid stride
    const int64_t cap = static_cast<int64_t>(sm_count()) * per_sm;
    const unsigned grid = static_cast<unsigned>(M < cap ? M : cap);
    return launch_chained(kern, grid, static_cast<unsigned>(threads), 0, st, x, ws, as, qs, y, scale, M, H, left, direct,
                          divide);
}

}  // namespace w8a8

extern "C" int w8a8_dequant_swiglu_quant(const void* x, const float* weight_scale, const float* activation_scale,
                                         const float* quant_scale, int8_t* y, float* scale, int64_t M, int64_t H,
                                         int x_dtype, int activate_left, int flags, void* stream)
{
    if (x_dtype != W8A8_DT_I32 && x_dtype != W8A8_DT_F16 && x_dtype != W8A8_DT_BF16) {
        return W8A8_ERR_INVALID;
    }
    if (M < 0 || H <= 0 || (flags & ~W8A8_F_ROUND_DIRECT) != 0) {
        return W8A8_ERR_INVALID;
    }
    const bool is_i32 = (x_dtype == W8A8_DT_I32);
    if (is_i32 != (weight_scale != nullptr) || is_i32 != (activation_scale != nullptr)) {
        return W8A8_ERR_INVALID;  // both scales with int32 input, neither with 16-bit input
    }
    if (M == 0) {
        return W8A8_OK;
    }
    if (x == nullptr || y == nullptr || scale == nullptr) {
        return W8A8_ERR_INVALID;
    }
    const size_t elem = is_i32 ? 4 : 2;
    if (!w8a8::is_aligned(x, elem) || !w8a8::is_aligned(scale, 4) || !w8a8::is_aligned(weight_scale, 4) ||
        !w8a8::is_aligned(activation_scale, 4) || !w8a8::is_aligned(quant_scale, 4)) {
        return W8A8_ERR_ALIGN;
    }
    const int64_t el = is_i32 ? 4 : 8;
    const bool vec = (H % el == 0) && w8a8::is_aligned(x, 16) && w8a8::is_aligned(y, 8) && (H * elem) % 16 == 0 &&
                     w8a8::is_aligned(weight_scale, 16) && w8a8::is_aligned(quant_scale, 16);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int left = activate_left ? 1 : 0;
    const int direct = (flags & W8A8_F_ROUND_DIRECT) ? 1 : 0;
    cudaError_t e;
    if (is_i32) {
        e = w8a8::dispatch_dqsq<w8a8::DQSQ_X_I32>(x, weight_scale, activation_scale, quant_scale, y, scale, M, H, left,
                                                  direct, vec, st);
    } else if (x_dtype == W8A8_DT_F16) {
        e = w8a8::dispatch_dqsq<w8a8::DQSQ_X_F16>(x, nullptr, nullptr, quant_scale, y, scale, M, H, left, direct, vec,
                                                  st);
    } else {
        e = w8a8::dispatch_dqsq<w8a8::DQSQ_X_BF16>(x, nullptr, nullptr, quant_scale, y, scale, M, H, left, direct, vec,
                                                   st);
    }
    return w8a8::launch_status(e);
}
