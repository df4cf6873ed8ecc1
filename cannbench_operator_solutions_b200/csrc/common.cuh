// Shared device helpers for the W8A8 quantised-FFN kernels (sm_100a).
//
// The whole library is compiled with -fmad=false: the operators' results
// depend on which multiplies and adds are rounded separately, so every fused
// multiply-add in these sources is an explicit fmaf().
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/w8a8ffn.h"

namespace w8a8 {

constexpr unsigned FULL_MASK = 0xffffffffu;
constexpr float INV127 = 1.0f / 127.0f;

// ---------------------------------------------------------------------------
// 16-bit float <-> fp32
// ---------------------------------------------------------------------------
template <int DT>
__device__ __forceinline__ void unpack2(uint32_t p, float& lo, float& hi)
{
    if constexpr (DT == W8A8_DT_BF16) {
        lo = __uint_as_float(p << 16);
        hi = __uint_as_float(p & 0xffff0000u);
    } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&p));
        lo = f.x;
        hi = f.y;
    }
}

template <int DT>
__device__ __forceinline__ uint32_t pack2(float lo, float hi)
{
    if constexpr (DT == W8A8_DT_BF16) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&b);
    } else {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
}

template <int DT>
__device__ __forceinline__ float bits16_to_float(uint32_t b)
{
    if constexpr (DT == W8A8_DT_BF16) {
        return __uint_as_float(b << 16);
    } else {
        return __half2float(__ushort_as_half(static_cast<unsigned short>(b)));
    }
}

template <int DT>
__device__ __forceinline__ uint16_t float_to_bits16(float v)
{
    if constexpr (DT == W8A8_DT_BF16) {
        return __bfloat16_as_ushort(__float2bfloat16_rn(v));
    } else {
        return __half_as_ushort(__float2half_rn(v));
    }
}

// fp32 exp shared with the CPU oracle: Cody-Waite reduction by ln2 in two
// pieces, degree-5 polynomial (the classic single-precision coefficients
// published with the Cephes library), two-step power-of-two scaling.  Built
// from IEEE mul / add / fma only, so host and device agree bit for bit.
// This is the defining sequence; the kernels call canonical_expf below, which
// returns the same bits with fewer instructions.
__device__ __forceinline__ float canonical_expf_as_defined(float x)
{
    if (x != x) {
        return x;
    }
    x = (x > 89.0f) ? 89.0f : x;
    x = (x < -104.0f) ? -104.0f : x;
    const float n = rintf(__fmul_rn(x, 1.44269504088896341f));
    float r = fmaf(n, -0.693359375f, x);
    r = fmaf(n, 2.12194440e-4f, r);
    float p = 1.9875691500e-4f;
    p = fmaf(p, r, 1.3981999507e-3f);
    p = fmaf(p, r, 8.3334519073e-3f);
    p = fmaf(p, r, 4.1665795894e-2f);
    p = fmaf(p, r, 1.6666665459e-1f);
    p = fmaf(p, r, 5.0000001201e-1f);
    const float r2 = __fmul_rn(r, r);
    float e = fmaf(p, r2, r);
    e = __fadd_rn(e, 1.0f);
    const int ni = static_cast<int>(n);
    const int n1 = ni >> 1;
    const int n2 = ni - n1;
    const float s1 = __int_as_float((n1 + 127) << 23);
    const float s2 = __int_as_float((n2 + 127) << 23);
    return __fmul_rn(__fmul_rn(e, s1), s2);
}

// The same function, bit for bit on every input (w8a8_selftest_exp sweeps all 2^32), arranged for the issue
// slots it costs in the SwiGLU epilogues and the router softmax:
//  - rint and the float -> int conversion (conversion-pipe instructions, a quarter of the fp32 rate) become an
//    add and a subtract of 1.5 * 2^23, whose sum holds the integer in its low mantissa bits (|n| <= 151);
//    a product that rounds to -0 gives n = +0 instead of -0, which the two fma that use n turn into the same r;
//  - e lies in [0.70, 1.42] and n1 = n >> 1 in [-75, 64], so the first of the two multiplications by powers of
//    two is exact and lands on a normal number: it becomes an integer add to e's exponent field.  The second
//    multiplication stays, because it is the one that rounds (subnormal results) or overflows.
__device__ __forceinline__ float canonical_expf(float x)
{
    const float xc = fminf(fmaxf(x, -104.0f), 89.0f);  // a NaN comes out as -104 here and is put back at the end
    const float t = __fadd_rn(__fmul_rn(xc, 1.44269504088896341f), 12582912.0f);
    const float n = __fsub_rn(t, 12582912.0f);
    const int ni = __float_as_int(t) - 0x4B400000;
    float r = fmaf(n, -0.693359375f, xc);
    r = fmaf(n, 2.12194440e-4f, r);
    float p = 1.9875691500e-4f;
    p = fmaf(p, r, 1.3981999507e-3f);
    p = fmaf(p, r, 8.3334519073e-3f);
    p = fmaf(p, r, 4.1665795894e-2f);
    p = fmaf(p, r, 1.6666665459e-1f);
    p = fmaf(p, r, 5.0000001201e-1f);
    const float r2 = __fmul_rn(r, r);
    float e = fmaf(p, r2, r);
    e = __fadd_rn(e, 1.0f);
    const int n1 = ni >> 1;
    const int n2 = ni - n1;
    const float e1 = __int_as_float(__float_as_int(e) + (n1 << 23));
    const float s2 = __int_as_float((n2 << 23) + 0x3f800000);
    const float out = __fmul_rn(e1, s2);
    return (x != x) ? x : out;
}

// silu(l) = l / (1 + exp(-l)), the operation sequence of the reference
// (gmsq_vec_kernel.cpp:213-217).
__device__ __forceinline__ float canonical_silu(float l)
{
    const float e = __fadd_rn(canonical_expf(-l), 1.0f);
    return __fdiv_rn(l, e);
}

// ---------------------------------------------------------------------------
// Pairs of fp32 values in one 64-bit register: sm_100 runs mul / add / fma on both halves in one issue slot, each
// half rounded like the scalar instruction.  The exponential and the quotient below are issue bound wherever they
// are used, so they are written on pairs.  Never feed mul2 to add2: the assembler contracts a pair multiplication
// and the pair addition that uses it into one rounding, whatever the rounding modifiers say.
// ---------------------------------------------------------------------------
using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pair(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ f32x2 pair(float both) { return pair(both, both); }

__device__ __forceinline__ void unpair(f32x2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// e = -canonical_expf(-g) of N pairs, bit for bit (w8a8_selftest_pairs), for |g| <= EXP2_MAX_ABS (the result is then a normal number, so
// the power of two is one integer add to the exponent field).  A NaN half gives an arbitrary value: callers
// multiply something by g that carries the NaN.  Every step is canonical_expf's with the sign of the argument or of
// the result folded into the constants, which round-to-nearest does not see.  The pairs go through each step
// together: a pair instruction has no immediate operand, so a constant costs registers or moves, and N pairs share
// them.
constexpr float EXP2_MAX_ABS = 80.0f;

template <int N>
__device__ __forceinline__ void neg_exp_neg2(const f32x2 (&g)[N], f32x2 (&e)[N])
{
    f32x2 t[N], r[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float g0, g1;
        unpair(g[i], g0, g1);
        // two scalar products: see above
        t[i] = add2(pair(__fmul_rn(g0, 1.44269504088896341f), __fmul_rn(g1, 1.44269504088896341f)), pair(12582912.0f));
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        e[i] = add2(t[i], pair(-12582912.0f));
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[i] = fma2(e[i], pair(-0.693359375f), g[i]);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[i] = fma2(e[i], pair(2.12194440e-4f), r[i]);  // minus the r of canonical_expf(-g)
    }
    constexpr float C[6] = {1.9875691500e-4f, -1.3981999507e-3f, 8.3334519073e-3f,
                            -4.1665795894e-2f, 1.6666665459e-1f, -5.0000001201e-1f};
#pragma unroll
    for (int i = 0; i < N; ++i) {
        e[i] = pair(C[0]);
    }
#pragma unroll
    for (int k = 1; k < 6; ++k) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            e[i] = fma2(e[i], r[i], pair(C[k]));
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        e[i] = add2(fma2(e[i], mul2(r[i], r[i]), r[i]), pair(-1.0f));
        float e0, e1, t0, t1;
        unpair(e[i], e0, e1);
        unpair(t[i], t0, t1);
        e[i] = pair(__int_as_float(__float_as_int(e0) - (__float_as_int(t0) << 23)),
                    __int_as_float(__float_as_int(e1) - (__float_as_int(t1) << 23)));
    }
}

// e = canonical_expf(x) of N pairs, bit for bit (w8a8_selftest_pairs), for x <= 0 (-inf included, NaN not): the power of two is applied as
// an exact integer add that leaves a normal number, 2^64 too large, and one multiplication that rounds the
// subnormal results.  (A pair addition that uses e may absorb that multiplication; it is exact unless the result is
// subnormal, where a sum of at least 2^-126 does not see the difference.)
template <int N>
__device__ __forceinline__ void exp_nonpositive2(const f32x2 (&x)[N], f32x2 (&e)[N])
{
    f32x2 t[N], r[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float x0, x1;
        unpair(x[i], x0, x1);
        x0 = fmaxf(x0, -104.0f);
        x1 = fmaxf(x1, -104.0f);
        r[i] = pair(x0, x1);
        t[i] = add2(pair(__fmul_rn(x0, 1.44269504088896341f), __fmul_rn(x1, 1.44269504088896341f)), pair(12582912.0f));
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        e[i] = add2(t[i], pair(-12582912.0f));
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[i] = fma2(e[i], pair(-0.693359375f), r[i]);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[i] = fma2(e[i], pair(2.12194440e-4f), r[i]);
    }
    constexpr float C[6] = {1.9875691500e-4f, 1.3981999507e-3f, 8.3334519073e-3f,
                            4.1665795894e-2f, 1.6666665459e-1f, 5.0000001201e-1f};
#pragma unroll
    for (int i = 0; i < N; ++i) {
        e[i] = pair(C[0]);
    }
#pragma unroll
    for (int k = 1; k < 6; ++k) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            e[i] = fma2(e[i], r[i], pair(C[k]));
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        e[i] = add2(fma2(e[i], mul2(r[i], r[i]), r[i]), pair(1.0f));
        float e0, e1, t0, t1;
        unpair(e[i], e0, e1);
        unpair(t[i], t0, t1);
        // the low bits of t are n, those above shift out
        e[i] = pair(__int_as_float(__float_as_int(e0) + (__float_as_int(t0) << 23) + (64 << 23)),
                    __int_as_float(__float_as_int(e1) + (__float_as_int(t1) << 23) + (64 << 23)));
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        e[i] = mul2(e[i], pair(5.42101086242752217e-20f));  // 2^-64
    }
}

__device__ __forceinline__ float approx_reciprocal(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// q = n / -nd of N pairs, correctly rounded, for -nd in [1, 2^116] and |n| in [2^-60, 2^100] (a zero numerator
// gives a zero whose sign may differ): one Newton step on the approximate reciprocal, then one correction of the
// quotient by its exactly computed remainder (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990).  Before the last rounding the quotient is within 2^-46 of n / d; the quotients
// that lie so close to the middle of two floats are, for each d, a handful of numerators, and all of them over all
// 2^23 significands d agree with the IEEE division (w8a8_selftest_pairs).
template <int N>
__device__ __forceinline__ void quotient2(const f32x2 (&n)[N], const f32x2 (&nd)[N], f32x2 (&q)[N])
{
    f32x2 y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float d0, d1;
        unpair(nd[i], d0, d1);
        y[i] = pair(approx_reciprocal(-d0), approx_reciprocal(-d1));
        q[i] = fma2(nd[i], y[i], pair(1.0f));
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        y[i] = fma2(q[i], y[i], y[i]);
        q[i] = mul2(n[i], y[i]);
        q[i] = fma2(fma2(nd[i], q[i], n[i]), y[i], q[i]);
    }
}

// ---------------------------------------------------------------------------
// fp32 -> int8 narrowing.
//
// "As written" (the reference's two casts): fp32 -> fp16 RNE, then fp16 ->
// int8 RNE.  For |v| <= 128 the second step is done without a conversion
// instruction: adding 1536 (= 1.5 * 2^10, where fp16 has unit spacing)
// rounds to the nearest integer, ties to even, and leaves the two's
// complement byte in the low 8 bits of the sum's bit pattern.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t narrow4_fp16_fast(float a, float b, float c, float d)
{
    const __half2 magic = __floats2half2_rn(1536.0f, 1536.0f);
    __half2 h01 = __hadd2(__floats2half2_rn(a, b), magic);
    __half2 h23 = __hadd2(__floats2half2_rn(c, d), magic);
    return __byte_perm(*reinterpret_cast<uint32_t*>(&h01), *reinterpret_cast<uint32_t*>(&h23), 0x6420);
}

// Direct fp32 -> int8 RNE for |v| <= 128: 1.5 * 2^23 trick.
__device__ __forceinline__ uint32_t narrow4_direct_fast(float a, float b, float c, float d)
{
    const float magic = 12582912.0f;
    const uint32_t ua = __float_as_uint(__fadd_rn(a, magic));
    const uint32_t ub = __float_as_uint(__fadd_rn(b, magic));
    const uint32_t uc = __float_as_uint(__fadd_rn(c, magic));
    const uint32_t ud = __float_as_uint(__fadd_rn(d, magic));
    const uint32_t ab = __byte_perm(ua, ub, 0x0040);
    const uint32_t cd = __byte_perm(uc, ud, 0x0040);
    return __byte_perm(ab, cd, 0x5410);
}

// Fully general narrowing: any fp32 including NaN (-> 0), inf and values
// outside the int8 range (saturate).
template <bool DIRECT>
__device__ __forceinline__ int narrow1_general(float v)
{
    int r;
    if constexpr (DIRECT) {
        r = (v != v) ? 0 : __float2int_rn(fminf(fmaxf(v, -128.0f), 127.0f));
    } else {
        const __half h = __float2half_rn(v);
        const float hv = __half2float(h);
        r = (hv != hv) ? 0 : __float2int_rn(fminf(fmaxf(hv, -128.0f), 127.0f));
    }
    return r;
}

template <bool DIRECT>
__device__ __forceinline__ uint32_t narrow4_general(float a, float b, float c, float d)
{
    const uint32_t ua = static_cast<uint32_t>(narrow1_general<DIRECT>(a)) & 0xffu;
    const uint32_t ub = static_cast<uint32_t>(narrow1_general<DIRECT>(b)) & 0xffu;
    const uint32_t uc = static_cast<uint32_t>(narrow1_general<DIRECT>(c)) & 0xffu;
    const uint32_t ud = static_cast<uint32_t>(narrow1_general<DIRECT>(d)) & 0xffu;
    return ua | (ub << 8) | (uc << 16) | (ud << 24);
}

template <bool DIRECT>
__device__ __forceinline__ uint32_t narrow4_fast(float a, float b, float c, float d)
{
    if constexpr (DIRECT) {
        return narrow4_direct_fast(a, b, c, d);
    } else {
        return narrow4_fp16_fast(a, b, c, d);
    }
}

// ---------------------------------------------------------------------------
// One 8-element chunk of a 16-bit row: 128-bit streaming load when the row
// is 16-byte aligned and a multiple of 8 long, element-wise otherwise
// (missing elements read as +0, the identity of both row reductions).
// ---------------------------------------------------------------------------
template <bool VEC>
__device__ __forceinline__ uint4 load_chunk16(const uint16_t* row, int c, int64_t N)
{
    if constexpr (VEC) {
        return __ldcs(reinterpret_cast<const uint4*>(row) + c);
    } else {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t e = static_cast<int64_t>(c) * 8 + 2 * i;
            const uint32_t lo = (e < N) ? row[e] : 0u;
            const uint32_t hi = (e + 1 < N) ? row[e + 1] : 0u;
            w[i] = lo | (hi << 16);
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// gamma-like vectors are re-read by every row: keep them cacheable
template <bool VEC>
__device__ __forceinline__ uint4 load_chunk16_cached(const uint16_t* row, int c, int64_t N)
{
    if constexpr (VEC) {
        return __ldca(reinterpret_cast<const uint4*>(row) + c);
    } else {
        return load_chunk16<false>(row, c, N);
    }
}

template <bool VEC>
__device__ __forceinline__ void store_chunk16(uint16_t* row, int c, int64_t N, uint4 v)
{
    if constexpr (VEC) {
        __stcs(reinterpret_cast<uint4*>(row) + c, v);
    } else {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t e = static_cast<int64_t>(c) * 8 + 2 * i;
            if (e < N) {
                row[e] = static_cast<uint16_t>(w[i] & 0xffffu);
            }
            if (e + 1 < N) {
                row[e + 1] = static_cast<uint16_t>(w[i] >> 16);
            }
        }
    }
}

template <bool VEC>
__device__ __forceinline__ void store_chunk8(int8_t* row, int c, int64_t N, uint32_t lo, uint32_t hi)
{
    if constexpr (VEC) {
        __stcs(reinterpret_cast<uint2*>(row) + c, make_uint2(lo, hi));
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int64_t e = static_cast<int64_t>(c) * 8 + i;
            if (e < N) {
                const uint32_t w = (i < 4) ? lo : hi;
                row[e] = static_cast<int8_t>((w >> (8 * (i & 3))) & 0xffu);
            }
        }
    }
}

// Largest |.| bit pattern of the eight 16-bit values in a chunk, compared as
// unsigned integers: orders finite magnitudes, inf above them, NaN above inf.
__device__ __forceinline__ uint32_t chunk_absmax16(uint4 v, uint32_t m2)
{
    m2 = __vmaxu2(m2, v.x & 0x7fff7fffu);
    m2 = __vmaxu2(m2, v.y & 0x7fff7fffu);
    m2 = __vmaxu2(m2, v.z & 0x7fff7fffu);
    m2 = __vmaxu2(m2, v.w & 0x7fff7fffu);
    return m2;
}

void note_launch();  // counts one kernel launch of this library (w8a8_kernel_launch_count)

// ---------------------------------------------------------------------------
// Programmatic dependent launch.  A kernel launched with launch_chained may start while the kernel before it on the
// stream is still running: its launch, block setup and prologue then overlap that kernel's tail instead of following
// it.  Every such kernel opens with after_previous(), which waits until the kernel before it has completed and its
// writes are visible; no global memory is touched before that, neither read nor written (the dense matmuls ask for
// weights into L2, which reads nothing; kernels beside the one before them have an order of their own, see
// beside.cuh).  It also lets the next kernel start.  A grid of at most one block per SM does so before its own wait,
// which takes 0.2 - 0.3 us off a short kernel; a larger one after it: with three kernels resident at once their blocks share the SMs unevenly (back to back, the router
// on 16384 rows of 256 bf16 takes 9.0 us, 13.4 if it lets the next one in ahead of the wait; the SwiGLU quantiser on 300
// rows of 16384 int32 47 us, 67).  BY_GRID = false: after it in any case - the SwiGLU quantiser, whose registers are used
// up (16384 rows of 2816 int32 90 us, 99 with the grid asked for), and the sums of gathered rows, whose few blocks run
// long (64 sums of eight fp32 rows of 4095 with bias 11.2 us, 13.8).
// Two rules keep the accesses behind the wait in the compiled code:
//  - No load is a non-coherent one (ld.global.nc, __ldg): those are for memory that nothing writes during the life of
//    the kernel, and the kernel before may write its outputs while this one already lives.  So the pointers that such a
//    kernel only reads are not __restrict__ (the compiler makes those loads non-coherent, and free to move); the
//    ones that it writes are, which is what lets loads be issued ahead of the stores.
//  - after_previous() returns a zero that the compiler cannot see through.  It is part of the index that the kernel's
//    first accesses are made with or guarded by, so that loads which the compiler takes for pure (__ldca, __ldcs,
//    __ldcg) cannot move above the wait either.  (Passing the pointers through an asm instead did that too, but made
//    every access a generic one and cost a register pair per pointer: the int32 form of the SwiGLU quantiser spilled,
//    68.5 us on [16384, 4096] against 67.3, and 8192 sums of eight rows of 7164 took 746 us against 590.)
// Kernels that are launched plainly (and memsets, copies, event waits) order themselves against these as against any
// other.
// A dense layer of 16 rows 53.9 us (61.5 before), an expert layer of 2000 rows 160 (184) and of 64 rows 116 (129), a
// grouped SwiGLU matmul of 512 rows 38 (42), regroup and combine of 8192 rows 56 (62).
// ---------------------------------------------------------------------------
template <bool BY_GRID = true>
__device__ __forceinline__ int64_t after_previous()
{
    constexpr unsigned SMS = 148;
    int64_t zero;
    if (BY_GRID && gridDim.x <= SMS) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    asm volatile("griddepcontrol.wait;\n\tmov.u64 %0, 0;" : "=l"(zero)::"memory");
    if (!BY_GRID || gridDim.x > SMS) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    return zero;
}

// overlap = false: starts when the kernel before it has completed, like a plain launch.
template <typename... Params, typename... Args>
cudaError_t launch_chained_if(bool overlap, void (*kern)(Params...), dim3 grid, unsigned block, size_t smem,
                              cudaStream_t st, Args&&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    note_launch();
    return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kern)(Params...), dim3 grid, unsigned block, size_t smem, cudaStream_t st,
                           Args&&... args)
{
    return launch_chained_if(true, kern, grid, block, smem, st, static_cast<Args&&>(args)...);
}

// The status of an entry point's launches.  A failed one's error is also taken out of the thread's last-error slot, so
// that whoever looks there next (torch does after each of its own launches) does not take it for its own.
inline int launch_status(cudaError_t e)
{
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return W8A8_ERR_CUDA;
    }
    return W8A8_OK;
}

// w8a8_add_rms_norm_dynamic_quant beside the kernel before it (see beside.cuh); unvectorised rows wait for it as ever
int add_rms_norm_dynamic_quant_beside(const void* x1, const void* x2, const void* gamma, int8_t* y, void* x_out,
                                      float* scale_out, int64_t rows, int64_t N, float epsilon, int dtype, void* stream);
// w8a8_dispatch_rows where every pair's row goes to row `expanded_pos` of one buffer
int dispatch_rows_local(const void* src, const float* src_scale, const int64_t* expanded_pos, void* dst, float* dst_scale,
                        int64_t T, int64_t topk, int64_t row_bytes, void* stream);

// whether w8a8_ep_tables takes this many ranks and experts
bool ep_tables_hold(int64_t P, int64_t E);

inline bool is_aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

int sm_count();  // cached multiprocessor count of the current device

// Launch facts of one kernel that hold for the life of the process, asked for once per device (the queries cost 1 - 2 us
// each, a good part of a small call).  Racing first calls store the same values.
constexpr int MAX_CACHED_DEVICES = 64;
struct KernelFacts {
    std::atomic<int> value[MAX_CACHED_DEVICES];  // 0: not asked yet
};

// resident CTAs per SM, at least 1
template <typename Kernel>
cudaError_t resident_ctas(KernelFacts& facts, Kernel kern, int threads, int* ctas)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    const bool keep = dev >= 0 && dev < MAX_CACHED_DEVICES;
    int n = keep ? facts.value[dev].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, 0);
        if (e != cudaSuccess) {
            return e;
        }
        n = n < 1 ? 1 : n;
        if (keep) {
            facts.value[dev].store(n, std::memory_order_relaxed);
        }
    }
    *ctas = n;
    return cudaSuccess;
}

// lets a kernel use `bytes` of dynamic shared memory on the current device
template <typename Kernel>
cudaError_t allow_dynamic_smem(KernelFacts& facts, Kernel kern, size_t bytes)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    const bool keep = dev >= 0 && dev < MAX_CACHED_DEVICES;
    if (keep && facts.value[dev].load(std::memory_order_relaxed) != 0) {
        return cudaSuccess;
    }
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e == cudaSuccess && keep) {
        facts.value[dev].store(1, std::memory_order_relaxed);
    }
    return e;
}

}  // namespace w8a8
