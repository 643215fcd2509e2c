// Shared device helpers of the sm_100a kernels: element conversion, the 2:4 selection
// and encoding rules, the metadata placement formula, MVUE arithmetic and the Philox stream.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <type_traits>
#include <utility>

#include "../../include/sparse24_b200.h"

namespace sp24 {

// ---------------------------------------------------------------------------------------------
// element types
// ---------------------------------------------------------------------------------------------
struct e4m3_t { uint8_t b; };
struct e5m2_t { uint8_t b; };

template <typename T> struct Elem;
template <> struct Elem<float> {
    static constexpr int code = SP24_F32;
    __device__ static float to_f32(float v) { return v; }
    __device__ static float from_f32(float v) { return v; }
};
template <> struct Elem<__half> {
    static constexpr int code = SP24_F16;
    __device__ static float to_f32(__half v) { return __half2float(v); }
    __device__ static __half from_f32(float v) { return __float2half_rn(v); }
    // two values rounded and packed into one register (lo in bits 0..15): one conversion instruction
    __device__ static uint32_t pack2(float lo, float hi) {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
};
template <> struct Elem<__nv_bfloat16> {
    static constexpr int code = SP24_BF16;
    __device__ static float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
    __device__ static __nv_bfloat16 from_f32(float v) { return __float2bfloat16_rn(v); }
    __device__ static uint32_t pack2(float lo, float hi) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
};
template <> struct Elem<e4m3_t> {
    static constexpr int code = SP24_E4M3;
    __device__ static float to_f32(e4m3_t v) {
        return __half2float(__half(__nv_cvt_fp8_to_halfraw(v.b, __NV_E4M3)));
    }
    __device__ static e4m3_t from_f32(float v) {
        return e4m3_t{(uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3)};
    }
};
template <> struct Elem<e5m2_t> {
    static constexpr int code = SP24_E5M2;
    __device__ static float to_f32(e5m2_t v) {
        return __half2float(__half(__nv_cvt_fp8_to_halfraw(v.b, __NV_E5M2)));
    }
    __device__ static e5m2_t from_f32(float v) {
        return e5m2_t{(uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E5M2)};
    }
};
template <> struct Elem<int8_t> {
    static constexpr int code = SP24_I8;
    __device__ static float to_f32(int8_t v) { return (float)v; }
    __device__ static int8_t from_f32(float v) { return (int8_t)v; }
};

// value as stored in TIn -> value stored in TOut (one rounding from the source precision)
template <typename TOut, typename TIn> __device__ __forceinline__ TOut convert(TIn v) {
    return Elem<TOut>::from_f32(Elem<TIn>::to_f32(v));
}

// ---------------------------------------------------------------------------------------------
// vector access (16-byte, or narrower when the element count demands)
// ---------------------------------------------------------------------------------------------
template <int BYTES> struct VecBytes;
template <> struct VecBytes<16> { using type = uint4; };
template <> struct VecBytes<8> { using type = uint2; };
template <> struct VecBytes<4> { using type = uint32_t; };
template <> struct VecBytes<2> { using type = uint16_t; };
template <> struct VecBytes<1> { using type = uint8_t; };

template <typename T, int N> struct alignas(sizeof(T) * N) Vec {
    T v[N];
};

template <typename T, int N> __device__ __forceinline__ Vec<T, N> load_vec(const T *p) {
    using R = typename VecBytes<sizeof(T) * N>::type;
    Vec<T, N> out;
    *reinterpret_cast<R *>(&out) = *reinterpret_cast<const R *>(p);
    return out;
}
template <typename T, int N> __device__ __forceinline__ void store_vec(T *p, const Vec<T, N> &val) {
    using R = typename VecBytes<sizeof(T) * N>::type;
    *reinterpret_cast<R *>(p) = *reinterpret_cast<const R *>(&val);
}

// ---------------------------------------------------------------------------------------------
// 2:4 selection by magnitude: six strict comparisons, ties keep the higher index.
// Returns the keep mask as bits 0..3.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t magnitude_mask4(float a0, float a1, float a2, float a3) {
    a0 = fabsf(a0); a1 = fabsf(a1); a2 = fabsf(a2); a3 = fabsf(a3);
    const bool x1 = a0 > a1, x2 = a0 > a2, x3 = a0 > a3, x4 = a1 > a2, x5 = a1 > a3, x6 = a2 > a3;
    const bool m0 = (x2 && x3) || (x1 && x2) || (x1 && x3);
    const bool m1 = (!x1 && x5) || (x4 && x5) || (!x1 && x4);
    const bool m2 = (!x2 && !x4) || (!x2 && x6) || (!x4 && x6);
    const bool m3 = (!x3 && !x5) || (!x3 && !x6) || (!x5 && !x6);
    return (uint32_t)m0 | ((uint32_t)m1 << 1) | ((uint32_t)m2 << 2) | ((uint32_t)m3 << 3);
}

// Encoding of a keep mask (bits 0..3) into the 4-bit metadata code idx0 | idx1 << 2.  The same
// boolean formulas serve masks with fewer or more than two bits (fall-back encodings).
__device__ __forceinline__ uint32_t encode_nibble(uint32_t mask) {
    const uint32_t m0 = mask & 1u, m1 = (mask >> 1) & 1u, m2 = (mask >> 2) & 1u;
    const uint32_t bit0 = (m0 ^ 1u) & m1;
    const uint32_t bit1 = (m0 ^ 1u) & (m1 ^ 1u);
    const uint32_t bit2 = bit1 | (m2 ^ 1u);
    const uint32_t bit3 = bit0 | (m1 ^ 1u) | m2;
    return bit0 | (bit1 << 1) | (bit2 << 2) | (bit3 << 3);
}

template <typename T> __device__ __forceinline__ T pick4(uint32_t idx, T v0, T v1, T v2, T v3) {
    const T lo = (idx & 1u) ? v1 : v0;
    const T hi = (idx & 1u) ? v3 : v2;
    return (idx & 2u) ? hi : lo;
}

// ---------------------------------------------------------------------------------------------
// metadata placement: logical element (r, c) of the (m, ncols) metadata matrix -> flat offset in the
// reordered buffer.  GROUP/INTER = 32/4 for 16-bit metadata words, 16/2 for 32-bit words.
// ---------------------------------------------------------------------------------------------
template <int META_BYTES> __device__ __forceinline__ int64_t meta_offset(int64_t r, int64_t c, int64_t m) {
    constexpr int GROUP = META_BYTES == 2 ? 32 : 16;
    constexpr int INTER = META_BYTES == 2 ? 4 : 2;
    int64_t dr = r / GROUP * GROUP + (r % 8) * INTER + (r % GROUP) / 8;
    int64_t dc = c;
    const bool r_odd = dr & 1, c_odd = dc & 1;
    if (!r_odd && c_odd) { dr += 1; dc -= 1; }
    else if (r_odd && !c_odd) { dr -= 1; dc += 1; }
    return (dc >> 1) * (2 * m) + dr * 2 + (dc & 1);
}

// Inside one aligned group of GROUP rows and one column pair the destination is a contiguous run of
// 2*GROUP words.  Position (0 .. 2*GROUP-1) of (row-in-group rr, column parity cp) inside that run.
template <int META_BYTES> __device__ __forceinline__ int meta_run_pos(int rr, int cp) {
    constexpr int GROUP = META_BYTES == 2 ? 32 : 16;
    constexpr int INTER = META_BYTES == 2 ? 4 : 2;
    int dr = (rr % 8) * INTER + (rr % GROUP) / 8;
    int dc = cp;
    if (!(dr & 1) && dc) { dr += 1; dc = 0; }
    else if ((dr & 1) && !dc) { dr -= 1; dc = 1; }
    return dr * 2 + dc;
}

// ---------------------------------------------------------------------------------------------
// Philox4x32-10 and the uniform pair of a group
// ---------------------------------------------------------------------------------------------
// Philox4x32 with ROUNDS rounds: 10 for the exact MVUE mode; 7 (the fewest rounds Salmon et al. report as passing
// BigCrush) for the fast mode.  The reference draws with five (tl.rand4x(..., n_rounds=5)).
__device__ __forceinline__ uint4 philox_round(uint4 c, uint32_t k0, uint32_t k1) {
    // both halves of a product from one wide multiplication (written as two, they are two instructions)
    uint32_t hi0, lo0, hi1, lo1;
    asm("{\n\t.reg .b64 t;\n\tmul.wide.u32 t, %2, %3;\n\tmov.b64 {%0, %1}, t;\n\t}" : "=r"(lo0), "=r"(hi0) : "r"(c.x), "n"(0xD2511F53u));
    asm("{\n\t.reg .b64 t;\n\tmul.wide.u32 t, %2, %3;\n\tmov.b64 {%0, %1}, t;\n\t}" : "=r"(lo1), "=r"(hi1) : "r"(c.z), "n"(0xCD9E8D57u));
    return make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
}
template <int ROUNDS = 10> __device__ __forceinline__ uint4 philox4x32(uint4 c, uint2 k) {
#pragma unroll
    for (int i = 0; i < ROUNDS; ++i) {
        c = philox_round(c, k.x, k.y);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}
// The same with the round keys worked out beforehand (two words a round): kept in a kernel's parameters they are constant operands,
// where the schedule above takes two instructions of the uniform path a round.
template <int ROUNDS> struct PhiloxKeys {
    uint32_t k[2 * ROUNDS];
    __host__ __device__ explicit PhiloxKeys(uint64_t seed = 0) {
        for (int i = 0; i < ROUNDS; ++i) {
            k[2 * i] = (uint32_t)seed + (uint32_t)i * 0x9E3779B9u;
            k[2 * i + 1] = (uint32_t)(seed >> 32) + (uint32_t)i * 0xBB67AE85u;
        }
    }
};
template <int ROUNDS> __device__ __forceinline__ uint4 philox4x32(uint4 c, const PhiloxKeys<ROUNDS> &keys) {
#pragma unroll
    for (int i = 0; i < ROUNDS; ++i) c = philox_round(c, keys.k[2 * i], keys.k[2 * i + 1]);
    return c;
}

__device__ __forceinline__ float u32_to_uniform(uint32_t x) { return (float)(x >> 8) * 5.9604644775390625e-08f; }

// Uniform pairs of the two groups 2*pair and 2*pair+1 (linear group index over the logical matrix).
template <int ROUNDS = 10>
__device__ __forceinline__ void mvue_uniform_pairs(uint64_t pair, uint64_t seed, uint64_t offset, float &u0a,
                                                   float &u1a, float &u0b, float &u1b) {
    const uint4 r = philox4x32<ROUNDS>(make_uint4((uint32_t)pair, (uint32_t)(pair >> 32), (uint32_t)offset,
                                             (uint32_t)(offset >> 32)),
                                  make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
    u0a = u32_to_uniform(r.x); u1a = u32_to_uniform(r.y);
    u0b = u32_to_uniform(r.z); u1b = u32_to_uniform(r.w);
}

// ---------------------------------------------------------------------------------------------
// MVUE24 (approximate): float32, one rounding per operation, left-to-right sums, IEEE division.
// x[] is overwritten with x_i / p_i; returns the keep mask as bits 0..3.
// ---------------------------------------------------------------------------------------------
template <bool ALL_FOUR = true>
__device__ __forceinline__ uint32_t mvue24_group(float (&x)[4], float u0, float u1) {
    const float eps = 1.19209e-07f;
    float a[4], t[4], kk[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = __fadd_rn(fabsf(x[i]), eps);
    const float s = __fadd_rn(__fadd_rn(__fadd_rn(a[0], a[1]), a[2]), a[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        t[i] = __fdiv_rn(a[i], s);
        kk[i] = __fdiv_rn(t[i], __fsub_rn(s, a[i]));
    }
    const float ks = __fadd_rn(__fadd_rn(__fadd_rn(kk[0], kk[1]), kk[2]), kk[3]);
    const float t01 = __fadd_rn(t[0], t[1]);
    const float t012 = __fadd_rn(t01, t[2]);
    const bool m0 = u0 <= t[0];
    const bool m1 = (u0 <= t01) && !m0;
    const bool m2 = (u0 <= t012) && !m1 && !m0;
    const bool m3 = !m2 && !m1 && !m0;
    // (~m) * a : 0 * a when picked (NaN for an infinite a, like the reference), 1 * a otherwise
    const float d0 = __fmul_rn(m0 ? 0.f : 1.f, a[0]);
    const float d1 = __fmul_rn(m1 ? 0.f : 1.f, a[1]);
    const float d2 = __fmul_rn(m2 ? 0.f : 1.f, a[2]);
    const float d3 = __fmul_rn(m3 ? 0.f : 1.f, a[3]);
    const float d01 = __fadd_rn(d0, d1);
    const float d012 = __fadd_rn(d01, d2);
    const float ds = __fadd_rn(d012, d3);
    const float tt = __fmul_rn(u1, ds);
    const bool e0 = tt <= d0;
    const bool e1 = (tt <= d01) && !e0;
    const bool e2 = (tt <= d012) && !e1 && !e0;
    const bool e3 = !e2 && !e1 && !e0;
    const uint32_t keep = (uint32_t)(m0 || e0) | ((uint32_t)(m1 || e1) << 1) | ((uint32_t)(m2 || e2) << 2) |
                          ((uint32_t)(m3 || e3) << 3);
    if constexpr (ALL_FOUR) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float p = __fadd_rn(t[i], __fmul_rn(a[i], __fsub_rn(ks, kk[i])));
            x[i] = __fdiv_rn(x[i], p);
        }
    } else {
        // compressed output: only the two stored positions are divided (the same two quotients the full form
        // would pick); they come back in x[0], x[1]
        float p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = __fadd_rn(t[i], __fmul_rn(a[i], __fsub_rn(ks, kk[i])));
        const uint32_t nib = encode_nibble(keep);
        const float q0 = __fdiv_rn(pick4(nib & 3u, x[0], x[1], x[2], x[3]), pick4(nib & 3u, p[0], p[1], p[2], p[3]));
        const float q1 = __fdiv_rn(pick4(nib >> 2, x[0], x[1], x[2], x[3]), pick4(nib >> 2, p[0], p[1], p[2], p[3]));
        x[0] = q0;
        x[1] = q1;
    }
    return keep;
}

// ---------------------------------------------------------------------------------------------
// MVUE24, fast arithmetic (seeded mode only).  The same estimator - sample two of four without replacement with
// probability proportional to a_i = |x_i| + eps, store x_i / p_i with p_i the inclusion probability - arranged for
// the instruction mix of the SM instead of for bit-equality with the reference formulas:
//   * every division is a reciprocal approximation (MUFU) and a multiply;
//   * S - a_i and K - k_i are taken as the sum of the other three terms, not as a difference: no cancellation when one
//     magnitude dominates its group, so p_i is good to a few float32 ulps everywhere (the reference order loses up to
//     ~1e-4 relative there);
//   * a draw is the last threshold below the scaled uniform instead of a cascade of dependent predicates;
//   * all four quotients are formed (two more reciprocals) so that the two stored ones can be gathered with one
//     table-driven byte permute instead of select chains.
// Every operation is an explicit intrinsic (no compiler contraction), so all kernels that call this function produce
// the same bits for the same inputs.  As in the reference, a second uniform of exactly zero repeats a first pick of
// position 0 (one kept value in that group, probability ~2^-25).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float rcp_fast(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
constexpr int kMvueFastRounds = 7;

// 23 random bits -> v = 1 + u, u a float32 uniform on [0, 1) with 2^-23 spacing (v is a float's mantissa in [1, 2)).  A scaled
// uniform u * s is taken as fma(v, s, -s): the same real number rounded once, without the subtraction.
__device__ __forceinline__ float u32_to_one_plus_uniform(uint32_t x) { return __uint_as_float((x & 0x007FFFFFu) | 0x3F800000u); }

// Uniform pairs (as 1 + u) of groups 2*pair and 2*pair+1 for the fast mode: Philox4x32-7, 23-bit uniforms.
__device__ __forceinline__ void mvue_uniform_pairs_fast(uint64_t pair, uint64_t seed, uint64_t offset, float &v0a,
                                                        float &v1a, float &v0b, float &v1b) {
    const uint4 r = philox4x32<kMvueFastRounds>(make_uint4((uint32_t)pair, (uint32_t)(pair >> 32), (uint32_t)offset,
                                                           (uint32_t)(offset >> 32)),
                                                make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
    v0a = u32_to_one_plus_uniform(r.x); v1a = u32_to_one_plus_uniform(r.y);
    v0b = u32_to_one_plus_uniform(r.z); v1b = u32_to_one_plus_uniform(r.w);
}

// x[] is overwritten with x_i / p_i for ALL four positions; v0, v1 are one plus the two uniforms.  Returns the two picks as
// first + 4 * second.
//   r_j = a_j / (S - a_j), p_j = a_j (1 + sum of the other r) / S, so x_j / p_j = x_j * (S * rcp(a_j (1 + R_j)))
// Against 64 bits over 400 000 groups of gradient-like values the quotients are off by 5.6e-8 on average and 3.6e-7 at most
// (the arrangement with one more reciprocal per position: 5.7e-8 and 3.7e-7).  A group with an infinity or NaN gives NaN.
__device__ __forceinline__ uint32_t mvue24_group_fast(float (&x)[4], float v0, float v1) {
    const float eps = 1.19209e-07f;
    const float a0 = __fadd_rn(fabsf(x[0]), eps), a1 = __fadd_rn(fabsf(x[1]), eps);
    const float a2 = __fadd_rn(fabsf(x[2]), eps), a3 = __fadd_rn(fabsf(x[3]), eps);
    const float a01 = __fadd_rn(a0, a1), a23 = __fadd_rn(a2, a3);
    const float s = __fadd_rn(a01, a23), a012 = __fadd_rn(a01, a2);
    // sums of the other three
    const float r0 = __fmul_rn(a0, rcp_fast(__fadd_rn(a1, a23))), r1 = __fmul_rn(a1, rcp_fast(__fadd_rn(a0, a23)));
    const float r2 = __fmul_rn(a2, rcp_fast(__fadd_rn(a01, a3))), r3 = __fmul_rn(a3, rcp_fast(a012));
    const float r01 = __fadd_rn(r0, r1), r23 = __fadd_rn(r2, r3);
    // first pick: the interval of the cumulative sums (a0, a01, a012, s) that u0 * s falls into
    const float w = __fmaf_rn(v0, s, -s);
    const bool b0 = w > a0, b1 = w > a01, b2 = w > a012;
    // second pick among the other three: the same walk over the cumulative sums with the first pick's weight zeroed
    const float d0 = b0 ? a0 : 0.f, d1 = (b0 && !b1) ? 0.f : a1, d2 = (b1 && !b2) ? 0.f : a2, d3 = b2 ? 0.f : a3;
    const float d01 = __fadd_rn(d0, d1), d012 = __fadd_rn(d01, d2), ds = __fadd_rn(d012, d3);
    const float w2 = __fmaf_rn(v1, ds, -ds);
    // the thresholds of a walk do not decrease, so the last one passed decides
    uint32_t f = b0 ? 1u : 0u, g = w2 > d0 ? 4u : 0u;
    f = b1 ? 2u : f;
    g = w2 > d01 ? 8u : g;
    f = b2 ? 3u : f;
    g = w2 > d012 ? 12u : g;
    x[0] = __fmul_rn(x[0], __fmul_rn(s, rcp_fast(__fmaf_rn(a0, __fadd_rn(r1, r23), a0))));
    x[1] = __fmul_rn(x[1], __fmul_rn(s, rcp_fast(__fmaf_rn(a1, __fadd_rn(r0, r23), a1))));
    x[2] = __fmul_rn(x[2], __fmul_rn(s, rcp_fast(__fmaf_rn(a2, __fadd_rn(r01, r3), a2))));
    x[3] = __fmul_rn(x[3], __fmul_rn(s, rcp_fast(__fmaf_rn(a3, __fadd_rn(r01, r2), a3))));
    return f + g;
}
// The same arithmetic, bit for bit, for two groups at once: .x of every operand belongs to the first group, .y to the second.  Sums,
// multiply-adds and most products are the two-lane instructions of sm_100: half the issue slots, the same time on the FMA pipe.  The
// draws are counted instead of selected: a passed threshold is 1.0, the first pick's weight is taken out by products with 0 or 1 (NaN
// where an infinity is behind the first position, which makes the second uniform NaN in the form above too), and the picks are added up as denormal floats, whose bits are the
// shared-memory address of the pick's table entry.  That leaves 7 instead of 19 instructions a group to the integer pipe, the busiest
// one with the form above (64 % of its rate at 73 % of the issue slots); the whole is 47 instructions a group instead of 64.
__device__ __forceinline__ float passed(float v, float limit) {      // 1.0 or 0.0
    float r;
    asm("set.gt.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "f"(limit));
    return r;
}
// at: address of entry 0; returns the addresses of the two groups' entries (8 bytes each, entry first + 4 * second)
__device__ __forceinline__ uint2 mvue24_two_groups_fast(float2 (&x)[4], float2 v0, float2 v1, uint32_t at) {
    const float eps = 1.19209e-07f;
    auto abs_eps = [&](float2 v) { return make_float2(__fadd_rn(fabsf(v.x), eps), __fadd_rn(fabsf(v.y), eps)); };
    auto rcp2 = [](float2 v) { return make_float2(rcp_fast(v.x), rcp_fast(v.y)); };
    // scalar products: a two-lane one that feeds a two-lane sum is fused with it, which is one float32 ulp off the form above
    auto times = [](float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); };
    auto neg = [](float2 v) { return make_float2(-v.x, -v.y); };
    auto scaled = [&](float2 v, float2 s_) { return __ffma2_rn(v, s_, neg(s_)); };
    auto above = [](float2 v, float2 limit) { return make_float2(passed(v.x, limit.x), passed(v.y, limit.y)); };
    auto both = [](float v) { return make_float2(v, v); };
    const float2 a0 = abs_eps(x[0]), a1 = abs_eps(x[1]), a2 = abs_eps(x[2]), a3 = abs_eps(x[3]);
    const float2 a01 = __fadd2_rn(a0, a1), a23 = __fadd2_rn(a2, a3);
    const float2 s = __fadd2_rn(a01, a23), a012 = __fadd2_rn(a01, a2);
    const float2 r0 = times(a0, rcp2(__fadd2_rn(a1, a23))), r1 = times(a1, rcp2(__fadd2_rn(a0, a23)));
    const float2 r2 = times(a2, rcp2(__fadd2_rn(a01, a3))), r3 = times(a3, rcp2(a012));
    const float2 r01 = __fadd2_rn(r0, r1), r23 = __fadd2_rn(r2, r3);
    const float2 w = scaled(v0, s);
    const float2 t0 = above(w, a0), t1 = above(w, a01), t2 = above(w, a012);     // not increasing
    const float2 most = __fmul2_rn(t0, both(3.4028235e38f));       // an infinite or NaN a0 is never passed: minima, not products
    const float2 d0 = make_float2(fminf(a0.x, most.x), fminf(a0.y, most.y)), d1 = __ffma2_rn(__fadd2_rn(t1, neg(t0)), a1, a1);
    const float2 d2 = __ffma2_rn(__fadd2_rn(t2, neg(t1)), a2, a2), d3 = __ffma2_rn(neg(t2), a3, a3);
    const float2 d01 = __fadd2_rn(d0, d1), d012 = __fadd2_rn(d01, d2), ds = __fadd2_rn(d012, d3);
    const float2 w2 = scaled(v1, ds);
    const float2 e8 = both(__uint_as_float(8u)), e32 = both(__uint_as_float(32u));
    float2 p = __ffma2_rn(t0, e8, both(__uint_as_float(at)));
    p = __ffma2_rn(t1, e8, p);
    p = __ffma2_rn(t2, e8, p);
    p = __ffma2_rn(above(w2, d0), e32, p);
    p = __ffma2_rn(above(w2, d01), e32, p);
    p = __ffma2_rn(above(w2, d012), e32, p);
    x[0] = __fmul2_rn(x[0], __fmul2_rn(s, rcp2(__ffma2_rn(a0, __fadd2_rn(r1, r23), a0))));
    x[1] = __fmul2_rn(x[1], __fmul2_rn(s, rcp2(__ffma2_rn(a1, __fadd2_rn(r0, r23), a1))));
    x[2] = __fmul2_rn(x[2], __fmul2_rn(s, rcp2(__ffma2_rn(a2, __fadd2_rn(r01, r3), a2))));
    x[3] = __fmul2_rn(x[3], __fmul2_rn(s, rcp2(__ffma2_rn(a3, __fadd2_rn(r01, r2), a3))));
    return make_uint2(__float_as_uint(p.x), __float_as_uint(p.y));
}
__device__ __forceinline__ uint32_t picks_to_keep(uint32_t picks) { return (1u << (picks & 3u)) | (1u << (picks >> 2)); }

// ---------------------------------------------------------------------------------------------
// float8 scales from a tensor's absolute maximum on the device: the dequantisation scale is amax / 448 in double (1 for
// an all-zero or NaN tensor), as a host that reads amax back works it out
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ double f8_scale(float amax) { return amax > 0.f ? (double)amax / 448.0 : 1.0; }
// The factor every quantising kernel multiplies by: the reciprocal in double, rounded once.  Two roundings (the scale, then
// its reciprocal) move products that are exact ties of e4m3 to the other side: 0.6 % of 16-bit values at some maxima.
__device__ __forceinline__ float f8_store_scale(float amax) { return (float)(1.0 / f8_scale(amax)); }

// Rows first, first + 8, ... of one column of parts (rows of `pitch` values) added up in that order: an eighth of a fixed-order sum.
__device__ __forceinline__ float sum_every_eighth(const float *column, int64_t n_parts, int64_t pitch, int first) {
    float s = 0.f;
#pragma unroll 8
    for (int64_t p = first; p < n_parts; p += 8) s += column[p * pitch];
    return s;
}

// ---------------------------------------------------------------------------------------------
// host-side helpers
// ---------------------------------------------------------------------------------------------
inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline int dtype_size(int dt) {
    switch (dt) {
        case SP24_F32: return 4;
        case SP24_F16: case SP24_BF16: return 2;
        case SP24_E4M3: case SP24_E5M2: case SP24_I8: return 1;
        case SP24_I32: return 4;
        default: return 0;
    }
}
int check_device();            // SP24_OK when the current device is compute capability 10.x
int launch_status();           // maps cudaGetLastError() to SP24_OK / SP24_ERR_CUDA
int runtime_error();           // for a failed runtime call: takes its error out of the runtime (and with SP24_DEBUG prints it), so
                               // that no later call reports it; always SP24_ERR_CUDA
int sm_count();                // SMs of the current device
int clear_words(void *dst, int64_t words, cudaStream_t st);      // zeros at dst, 4-byte aligned memory of the current device

// Programmatic dependent launch.  A kernel launched by launch_chained may start while the kernel before it on the
// stream is still finishing (as soon as all blocks of that one have called chain_enter or left), so its launch latency and set-up are
// hidden behind the other's last wave.  chain_enter first waits until everything before on the stream is complete and visible: no kernel
// reads or writes global memory before it, and every thread calls it, so a kernel's completion implies that of all kernels before it.  Its memory
// clobber holds plain loads back.  It does not bind loads that promise read-only data (__ldg, ld.global.nc, __restrict__): the kernel
// before may still be writing during this one's life, so there are none.
__device__ __forceinline__ void chain_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Asks L2 for `bytes` at p (both multiples of 16, more than none).  No value is read: the one access that may come before chain_enter, since what
// the kernel before still writes arrives in L2 as well.
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// Errors are left for launch_status, as with a <<<>>> launch.
template <typename... P, typename... A>
inline void launch_chained(cudaStream_t st, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, A &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Blocks of a kernel that an SM holds at once (kept per thread; the runtime's answer is the same for every device this library runs on).
int resident_blocks(const void *kern, unsigned threads, size_t smem);
// For kernels whose blocks compute for long: plain stream order where the grid has more blocks than the GPU SMs and an SM has room for more
// than its even share.  Placed while the kernel before it still holds some SMs, its blocks fill the others up to their resident limit, three
// on some and one on others where two each take two thirds of the time.  us, replayed back to back, chained -> here: exact MVUE
// 2048 x 2048 17.7 -> 13.4, dense MVUE fp16 2048 x 1024 5.5 -> 4.6, selection fp16 2048 x 1024 7.2 -> 6.1; layer steps of 4096 tokens,
// float8 1024 -> 1024 71.5 -> 68.7, fst 3072 -> 768 60.0 -> 57.3.  Kernels that stream keep their 0.4 us from the chain at most sizes (layer norm 2048 x 512 2.4,
// here 2.8) and lose more than that at a few (4096 x 512 3.1 -> 3.6).  Letting the next kernel in at the end of each kernel only (no
// launch_dependents) mends all of these, but takes 2 - 10 % from layer steps: fst 256 tokens, 256 -> 512, 22.7 -> 25.4.
template <typename... P, typename... A>
inline void launch_balanced(cudaStream_t st, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, A &&...args) {
    const int64_t blocks = (int64_t)grid.x * grid.y * grid.z, sms = sm_count();
    if (blocks > sms && (blocks + sms - 1) / sms < resident_blocks(reinterpret_cast<const void *>(kern), threads, smem))
        kern<<<grid, threads, smem, st>>>(std::forward<A>(args)...);
    else
        launch_chained(st, kern, grid, threads, smem, std::forward<A>(args)...);
}

}  // namespace sp24
