// Dense -> 2:4 compressed conversion: fused prune (magnitude / supplied mask / MVUE) + value
// compaction + metadata packing, for row-major and column-major storage of the logical matrix.
//
// Both kernels are HBM-bound streaming kernels.  Values leave through 16-byte coalesced stores;
// metadata words are first placed in shared memory at their position inside the destination run
// (the reordered layout keeps every aligned group of 32 rows x 2 metadata columns contiguous) and
// then written with 16-byte stores, so no partial sector is ever written.
#include "sp24_common.cuh"

namespace sp24 {
namespace {

struct PcParams {
    const void *dense;
    void *packed;
    void *meta;
    const uint8_t *mask;
    const float *uniforms;
    int64_t m, k, ld_dense, ld_packed, ld_mask, ld_u;
    uint64_t seed, offset;
    const unsigned long long *offset_dev;   // optional device word added to offset at run time
    int16_t *tc;                            // optional metadata copy in tensor-core atom order (16-bit outputs)
    int64_t k_atoms;                        // 128-column atoms per 128-row block
    float *row_sums;                        // optional (column-major only): row_sums[r] += sum over k of dense[r, k] ...
    int64_t ld_sums;                        // ... or, non-zero: block row y stores its share to row_sums[y * ld_sums + r]
    int packed_rm;                          // column-major input, 8-bit output: packed is written row-major (m, k/2)
    float out_scale;                        // 8-bit outputs: stored value = value * out_scale (1 = none)
    float soft_scale;                       // soft-threshold mode: kept values are also multiplied by this ...
    int soft_use_scale;                     // ... when this is set (one more rounding in the input type)
    const float *amax;                      // optional: 8-bit outputs take their scale from this device word (f8_store_scale)
    void *q_dense;                          // optional (column-major input, 8-bit output): dense * f8_store_scale in the output
    int64_t ld_q;                           // type, same storage order, pitch ld_q
    uint4 *zero;                            // optional (fast MVUE, column-major input): a buffer of n_zero 16-byte pieces that is
    int64_t n_zero;                         // cleared on the way
};

// internal mode code of the fused soft-threshold + compress entry point (not part of the public enum)
constexpr int PRUNE_SOFT = 4;

template <typename T, int N> __device__ __forceinline__ void load_elems(const T *p, T (&out)[N]) {
    constexpr int PER = (sizeof(T) * N >= 16) ? 16 / sizeof(T) : N;
#pragma unroll
    for (int i = 0; i < N / PER; ++i) {
        Vec<T, PER> v = load_vec<T, PER>(p + i * PER);
#pragma unroll
        for (int j = 0; j < PER; ++j) out[i * PER + j] = v.v[j];
    }
}
template <typename T, int N> __device__ __forceinline__ void store_elems(T *p, const T (&in)[N]) {
    constexpr int PER = (sizeof(T) * N >= 16) ? 16 / sizeof(T) : N;
#pragma unroll
    for (int i = 0; i < N / PER; ++i) {
        Vec<T, PER> v;
#pragma unroll
        for (int j = 0; j < PER; ++j) v.v[j] = in[i * PER + j];
        store_vec<T, PER>(p + i * PER, v);
    }
}

// V float32 values -> V consecutive float8 values, two per conversion instruction
template <typename TOut, int V> __device__ __forceinline__ void store_f8(TOut *p, const float (&f)[V]) {
    constexpr __nv_fp8_interpretation_t KIND = std::is_same<TOut, e5m2_t>::value ? __NV_E5M2 : __NV_E4M3;
    using R = typename VecBytes<V>::type;
    Vec<uint16_t, (V + 1) / 2> o;
#pragma unroll
    for (int v = 0; v < V; v += 2)
        o.v[v / 2] = (uint16_t)__nv_cvt_float2_to_fp8x2(make_float2(f[v], v + 1 < V ? f[v + 1] : 0.f), __NV_SATFINITE, KIND);
    *reinterpret_cast<R *>(p) = *reinterpret_cast<const R *>(&o);
}

constexpr bool is_mvue(int mode) { return mode == SP24_PRUNE_MVUE || mode == SP24_PRUNE_MVUE_FAST; }
// uniform pairs of the two groups of one Philox block, in the stream of the pruning mode
template <int MODE>
__device__ __forceinline__ void mode_uniform_pairs(uint64_t pair, uint64_t seed, uint64_t offset, float &u0a, float &u1a,
                                                   float &u0b, float &u1b) {
    if constexpr (MODE == SP24_PRUNE_MVUE_FAST) mvue_uniform_pairs_fast(pair, seed, offset, u0a, u1a, u0b, u1b);
    else mvue_uniform_pairs(pair, seed, offset, u0a, u1a, u0b, u1b);
}

// Entry of the pick table (16 entries in shared memory): byte-permute selector that gathers the two stored values from the four
// rounded quotients, and the metadata code.
struct PickEntry { uint32_t sel, code; };
__device__ __forceinline__ uint2 pick_entry(uint32_t addr) {      // written once, before a barrier
    uint2 e;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(e.x), "=r"(e.y) : "r"(addr));
    return e;
}
// Two groups of the fast MVUE mode.  x[] as mvue24_two_groups_fast takes it.  The quotients are rounded (8-bit outputs: times the
// caller's quantisation scale first, one more float32 rounding), then one table lookup and one byte permute a group gather the two
// stored values into oa, ob (low 16 / 8 bits: the lower position).  Returns the two 4-bit codes, the second group's in bits 4..7.
template <typename TOut>
__device__ __forceinline__ uint32_t two_groups_fast(float2 (&x)[4], float2 v0, float2 v1, uint32_t picks, float scale, uint32_t &oa, uint32_t &ob) {
    const uint2 at = mvue24_two_groups_fast(x, v0, v1, picks);
    const uint2 ea = pick_entry(at.x), eb = pick_entry(at.y);
    if constexpr (sizeof(TOut) == 2) {
        oa = __byte_perm(Elem<TOut>::pack2(x[0].x, x[1].x), Elem<TOut>::pack2(x[2].x, x[3].x), ea.x);
        ob = __byte_perm(Elem<TOut>::pack2(x[0].y, x[1].y), Elem<TOut>::pack2(x[2].y, x[3].y), eb.x);
    } else {
        static_assert(!std::is_same<TOut, int8_t>::value, "no integer form");
        constexpr __nv_fp8_interpretation_t KIND = std::is_same<TOut, e5m2_t>::value ? __NV_E5M2 : __NV_E4M3;
        const float2 sc = make_float2(scale, scale);
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = __fmul2_rn(x[j], sc);
        auto two = [](float lo, float hi) { return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, KIND); };
        oa = __byte_perm(two(x[0].x, x[1].x) | (two(x[2].x, x[3].x) << 16), 0u, ea.x);
        ob = __byte_perm(two(x[0].y, x[1].y) | (two(x[2].y, x[3].y) << 16), 0u, eb.x);
    }
    return ea.y + eb.y * 16u;
}

// One group of the fast MVUE mode, after the arithmetic: q[] holds all four quotients, picks the two picks (first + 4 * second).  16-bit
// results: round all four, then one table lookup (pick_lut, in shared memory) and one byte permute gather the two stored ones.
template <typename TOut>
__device__ __forceinline__ uint32_t emit_fast(const float (&q)[4], uint32_t picks, TOut &o0, TOut &o1, const uint32_t *pick_lut, float scale) {
    if constexpr (sizeof(TOut) == 2) {
        const uint32_t e = pick_lut[picks];
        const uint32_t o = __byte_perm(Elem<TOut>::pack2(q[0], q[1]), Elem<TOut>::pack2(q[2], q[3]), e >> 8);
        const uint16_t lo = (uint16_t)(o & 0xFFFFu), hi = (uint16_t)(o >> 16);
        o0 = *reinterpret_cast<const TOut *>(&lo);
        o1 = *reinterpret_cast<const TOut *>(&hi);
        return e & 0xFu;
    } else {
        // the caller's quantisation scale is applied before the cast (one more float32 rounding)
        const uint32_t nib = encode_nibble(picks_to_keep(picks));
        o0 = Elem<TOut>::from_f32(__fmul_rn(pick4(nib & 3u, q[0], q[1], q[2], q[3]), scale));
        o1 = Elem<TOut>::from_f32(__fmul_rn(pick4(nib >> 2, q[0], q[1], q[2], q[3]), scale));
        return nib;
    }
}

// One group of four: decide the keep mask, emit the two stored values and the 4-bit code.
// pick_lut: words 80..95 of the group table (indexed by the two picks of a draw) in shared memory; only the fast MVUE mode with 16-bit
// results reads it.
template <typename TIn, typename TOut, int MODE>
__device__ __forceinline__ uint32_t do_group(const TIn (&in)[4], uint32_t given_mask, float u0, float u1, TOut &o0,
                                             TOut &o1, const uint32_t *pick_lut = nullptr, float scale = 1.f) {
    // `scale` only acts on 8-bit outputs (float8 quantisation); 16-bit outputs ignore it
    constexpr bool SCALED = sizeof(TOut) == 1 && !std::is_same<TOut, int8_t>::value;
    uint32_t keep;
    if constexpr (MODE == SP24_PRUNE_MVUE_FAST) {
        float x[4] = {Elem<TIn>::to_f32(in[0]), Elem<TIn>::to_f32(in[1]), Elem<TIn>::to_f32(in[2]),
                      Elem<TIn>::to_f32(in[3])};
        const uint32_t picks = mvue24_group_fast(x, u0, u1);         // all four quotients in x[]
        return emit_fast<TOut>(x, picks, o0, o1, pick_lut, scale);
    } else if constexpr (MODE == SP24_PRUNE_MVUE) {
        float x[4] = {Elem<TIn>::to_f32(in[0]), Elem<TIn>::to_f32(in[1]), Elem<TIn>::to_f32(in[2]),
                      Elem<TIn>::to_f32(in[3])};
        keep = mvue24_group<false>(x, u0, u1);     // quotients of the two stored positions in x[0], x[1]
        const uint32_t nib = encode_nibble(keep);
        o0 = Elem<TOut>::from_f32(SCALED ? __fmul_rn(x[0], scale) : x[0]);
        o1 = Elem<TOut>::from_f32(SCALED ? __fmul_rn(x[1], scale) : x[1]);
        return nib;
    } else if constexpr (MODE == PRUNE_SOFT) {
        // S-STE: magnitude 2:4 mask; the two kept values move toward zero by the group's second-smallest magnitude
        // (one rounding in the input type), then optionally times the frozen scale (one more rounding in the input
        // type), then the cast to the packed type.  u0 carries the scale, u1 != 0 says whether to apply it.
        const float x0 = Elem<TIn>::to_f32(in[0]), x1 = Elem<TIn>::to_f32(in[1]), x2 = Elem<TIn>::to_f32(in[2]),
                    x3 = Elem<TIn>::to_f32(in[3]);
        keep = magnitude_mask4(x0, x1, x2, x3);
        const float a0 = fabsf(x0), a1 = fabsf(x1), a2 = fabsf(x2), a3 = fabsf(x3);
        const float thr = fminf(fmaxf(fminf(a0, a1), fminf(a2, a3)), fminf(fmaxf(a0, a1), fmaxf(a2, a3)));
        const uint32_t nib = encode_nibble(keep);
        float kv[2] = {pick4(nib & 3u, x0, x1, x2, x3), pick4(nib >> 2, x0, x1, x2, x3)};
        TIn t[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            t[i] = Elem<TIn>::from_f32(kv[i] > 0.f ? __fsub_rn(kv[i], thr) : __fadd_rn(kv[i], thr));
            if (u1 != 0.f) t[i] = Elem<TIn>::from_f32(__fmul_rn(Elem<TIn>::to_f32(t[i]), u0));
        }
        o0 = convert<TOut>(t[0]);
        o1 = convert<TOut>(t[1]);
        return nib;
    } else {
        if constexpr (MODE == SP24_PRUNE_MASK) {
            keep = given_mask;
        } else {
            keep = magnitude_mask4(Elem<TIn>::to_f32(in[0]), Elem<TIn>::to_f32(in[1]), Elem<TIn>::to_f32(in[2]),
                                   Elem<TIn>::to_f32(in[3]));
        }
        const uint32_t nib = encode_nibble(keep);
        if constexpr (SCALED) {
            o0 = Elem<TOut>::from_f32(__fmul_rn(Elem<TIn>::to_f32(pick4(nib & 3u, in[0], in[1], in[2], in[3])), scale));
            o1 = Elem<TOut>::from_f32(__fmul_rn(Elem<TIn>::to_f32(pick4(nib >> 2, in[0], in[1], in[2], in[3])), scale));
        } else {
            o0 = convert<TOut>(pick4(nib & 3u, in[0], in[1], in[2], in[3]));
            o1 = convert<TOut>(pick4(nib >> 2, in[0], in[1], in[2], in[3]));
        }
        return nib;
    }
}

// ---------------------------------------------------------------------------------------------
// Table-driven group processing for 16-bit -> same 16-bit type (magnitude and mask modes).
// Words 0..63: indexed by the six magnitude comparisons x1 | x2<<1 | x3<<2 | x4<<3 | x5<<4 | x6<<5
// (x1 = |a0|>|a1|, x2 = |a0|>|a2|, x3 = |a0|>|a3|, x4 = |a1|>|a2|, x5 = |a1|>|a3|, x6 = |a2|>|a3|);
// words 64..79: indexed by a 4-bit keep mask; words 80..95: by the two picks of a draw, first + 4 * second.  Each word: bits 0..3 the metadata code idx0 | idx1<<2,
// bits 8..23 the byte-permute selector that gathers elements idx0, idx1 from a (lo, hi) register pair.
// ---------------------------------------------------------------------------------------------
struct GroupLut { uint32_t v[96]; };
__host__ __device__ constexpr uint32_t lut_word_for_keep(uint32_t keep) {
    const uint32_t m0 = keep & 1u, m1 = (keep >> 1) & 1u, m2 = (keep >> 2) & 1u;
    const uint32_t bit0 = (m0 ^ 1u) & m1, bit1 = (m0 ^ 1u) & (m1 ^ 1u);
    const uint32_t bit2 = bit1 | (m2 ^ 1u), bit3 = bit0 | (m1 ^ 1u) | m2;
    const uint32_t i0 = bit0 | (bit1 << 1), i1 = bit2 | (bit3 << 1);
    const uint32_t sel = (2 * i0) | ((2 * i0 + 1) << 4) | ((2 * i1) << 8) | ((2 * i1 + 1) << 12);
    return (i0 | (i1 << 2)) | (sel << 8);
}
constexpr GroupLut make_group_lut() {
    GroupLut L{};
    for (uint32_t i = 0; i < 64; ++i) {
        const bool x1 = i & 1, x2 = i & 2, x3 = i & 4, x4 = i & 8, x5 = i & 16, x6 = i & 32;
        const bool m0 = (x2 && x3) || (x1 && x2) || (x1 && x3);
        const bool m1 = (!x1 && x5) || (x4 && x5) || (!x1 && x4);
        const bool m2 = (!x2 && !x4) || (!x2 && x6) || (!x4 && x6);
        const bool m3 = (!x3 && !x5) || (!x3 && !x6) || (!x5 && !x6);
        L.v[i] = lut_word_for_keep((uint32_t)m0 | ((uint32_t)m1 << 1) | ((uint32_t)m2 << 2) | ((uint32_t)m3 << 3));
    }
    for (uint32_t k = 0; k < 16; ++k) L.v[64 + k] = lut_word_for_keep(k);
    for (uint32_t k = 0; k < 16; ++k) L.v[80 + k] = lut_word_for_keep((1u << (k & 3u)) | (1u << (k >> 2)));
    return L;
}
__constant__ GroupLut kGroupLut = make_group_lut();

// Pick tables: indexed by the two picks of a draw, first + 4 * second; selectors over four 16-bit (0) or 8-bit (1) values.
struct PickLut { uint32_t v[2][16][2]; };
constexpr PickLut make_pick_lut() {
    PickLut L{};
    for (uint32_t k = 0; k < 16; ++k) {
        const uint32_t w = lut_word_for_keep((1u << (k & 3u)) | (1u << (k >> 2))), code = w & 0xFu;
        L.v[0][k][0] = w >> 8;
        L.v[1][k][0] = (code & 3u) | (code >> 2) << 4 | 0x4400u;
        L.v[0][k][1] = L.v[1][k][1] = code;
    }
    return L;
}
__constant__ PickLut kPickLut = make_pick_lut();
template <typename TOut> __device__ __forceinline__ void load_pick_lut(PickEntry *to) {
    if (threadIdx.x < 16) {
        constexpr int which = sizeof(TOut) == 2 ? 0 : 1;
        to[threadIdx.x] = PickEntry{kPickLut.v[which][threadIdx.x][0], kPickLut.v[which][threadIdx.x][1]};
    }
    __syncthreads();
}

template <typename T> struct Packed16;
template <> struct Packed16<__half> {
    __device__ static uint32_t gt_mask(uint32_t a, uint32_t b) {
        return __hgt2_mask(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
    }
};
template <> struct Packed16<__nv_bfloat16> {
    __device__ static uint32_t gt_mask(uint32_t a, uint32_t b) {
        return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162 *>(&a), *reinterpret_cast<const __nv_bfloat162 *>(&b));
    }
};

// lo = (x0, x1), hi = (x2, x3) as packed 16-bit values.  Returns the table word of the magnitude rule.
template <typename T> __device__ __forceinline__ uint32_t mse_lookup(uint32_t lo, uint32_t hi, const uint32_t *lut) {
    const uint32_t a = lo & 0x7FFF7FFFu, b = hi & 0x7FFF7FFFu;          // |x0|,|x1| and |x2|,|x3|
    const uint32_t c1 = Packed16<T>::gt_mask(a, b);                       // x2 (low half), x5 (high half)
    const uint32_t c2 = Packed16<T>::gt_mask(a, __byte_perm(b, b, 0x1032));  // x3, x4
    const uint32_t c3 = Packed16<T>::gt_mask(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));  // x1, x6
    const uint32_t t = (c3 & 0x00200001u) | (c1 & 0x00100002u) | (c2 & 0x00080004u);
    return lut[(t | (t >> 16)) & 0x3Fu];
}

// ---------------------------------------------------------------------------------------------
// row-major storage: groups of four run along the contiguous axis.
// Tile = 32 rows x 32 metadata columns; 8 warps, lane = metadata column, warp w owns rows 4w..4w+3.
// ---------------------------------------------------------------------------------------------
// Clears this block's share of the buffer that the launch was given: the weight gradient that the next kernel adds to.  The stores go
// out beside the arithmetic, where a memset of its own (9.4 MB: 3.1 us) held up the stream.
__device__ __forceinline__ void clear_share(const PcParams &P, int64_t block, int64_t blocks) {
    if (!P.zero) return;
    const int64_t per = (P.n_zero + blocks - 1) / blocks, end = min(P.n_zero, (block + 1) * per);
    for (int64_t i = block * per + threadIdx.x; i < end; i += 256) P.zero[i] = make_uint4(0, 0, 0, 0);
}

// Store scale of an 8-bit output: the caller's, or the reciprocal of the tensor's quantisation scale, worked out by one
// thread from the absolute maximum that an earlier launch left on the device.  Call with all threads of the block.
template <typename TOut> __device__ __forceinline__ float out_scale_of(const PcParams &P) {
    if constexpr (sizeof(TOut) == 1 && !std::is_same<TOut, int8_t>::value) {
        if (P.amax) {
            __shared__ float sc;
            if (threadIdx.x == 0) sc = f8_store_scale(*P.amax);
            __syncthreads();
            return sc;
        }
    }
    return P.out_scale;
}

// Fast MVUE with 8-bit results of 16-bit input: two groups at a time.  Float32 input, whose operands take twice the registers, stays with
// one group.  us a replayed launch, one group -> two: bf16 64 x 1024 8.1 -> 6.9, 2048 x 4096 13.8 -> 11.5, 4128 x 8192 44.2 -> 36.6; float32
// 7.1 -> 8.1, 14.1 -> 14.5, 42.3 -> 46.2.
template <typename TIn, typename TOut, int MODE> constexpr bool row_pairs() {
    return MODE == SP24_PRUNE_MVUE_FAST && sizeof(TOut) == 1 && sizeof(TIn) == 2;
}

template <typename TIn, typename TOut, int MODE, bool HAS_U>
__global__ void __launch_bounds__(256, is_mvue(MODE) ? 3 : 1) pc_row_kernel(PcParams P) {
    chain_enter();
    const uint64_t rng_offset = P.offset + (P.offset_dev ? *P.offset_dev : 0ull);
    const float out_scale = out_scale_of<TOut>(P);
    constexpr int CH = sizeof(TOut) == 2 ? 16 : 32;  // dense elements per metadata word
    constexpr int MB = sizeof(TOut) == 2 ? 2 : 4;    // bytes per metadata word
    constexpr int GROUP = MB == 2 ? 32 : 16;
    using MetaT = typename VecBytes<MB>::type;
    // rows in flight per thread; MVUE is arithmetic-bound, so it trades memory-level parallelism for
    // fewer registers (more resident warps)
    constexpr int RPI = (is_mvue(MODE) || CH * sizeof(TIn) >= 128) ? 1 : (CH * sizeof(TIn) >= 64 ? 2 : 4);

    __shared__ __align__(16) MetaT smeta[16][64];
    constexpr bool PACKED = !is_mvue(MODE) && MODE != PRUNE_SOFT && std::is_same<TIn, TOut>::value && sizeof(TIn) == 2;
    constexpr bool PICK_LUT = MODE == SP24_PRUNE_MVUE_FAST && sizeof(TOut) == 2;   // words 80..95 only
    constexpr bool PAIRS = row_pairs<TIn, TOut, MODE>();
    __shared__ uint32_t glut[PACKED ? 80 : (PICK_LUT ? 16 : 1)];
    __shared__ __align__(8) PickEntry picks[PAIRS ? 16 : 1];
    if constexpr (PACKED) {
        if (threadIdx.x < 80) glut[threadIdx.x] = kGroupLut.v[threadIdx.x];
        __syncthreads();
    }
    if constexpr (PICK_LUT) {
        if (threadIdx.x < 16) glut[threadIdx.x] = kGroupLut.v[80 + threadIdx.x];
        __syncthreads();
    }
    if constexpr (PAIRS) load_pick_lut<TOut>(picks);
    const uint32_t picks_at = (uint32_t)__cvta_generic_to_shared(picks);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t ncols = P.k / CH;
    const int64_t c = (int64_t)blockIdx.x * 32 + lane;
    const int64_t r0 = (int64_t)blockIdx.y * 32;
    const TIn *dense = static_cast<const TIn *>(P.dense);
    TOut *packed = static_cast<TOut *>(P.packed);

    if (c < ncols) {
#pragma unroll(is_mvue(MODE) ? 1 : 4)
        for (int it = 0; it < 4 / RPI; ++it) {
            TIn in[RPI][CH];
            uint8_t mk[RPI][CH];
#pragma unroll
            for (int j = 0; j < RPI; ++j) {
                const int64_t r = r0 + warp * 4 + it * RPI + j;
                load_elems<TIn, CH>(dense + r * P.ld_dense + c * CH, in[j]);
                if constexpr (MODE == SP24_PRUNE_MASK) load_elems<uint8_t, CH>(P.mask + r * P.ld_mask + c * CH, mk[j]);
            }
#pragma unroll
            for (int j = 0; j < RPI; ++j) {
                const int rr = warp * 4 + it * RPI + j;
                const int64_t r = r0 + rr;
                alignas(16) TOut out[CH / 2];
                uint32_t word = 0;
                if constexpr (PACKED) {
                    // one table lookup and one byte permute per group of four
                    const uint32_t *raw = reinterpret_cast<const uint32_t *>(&in[j][0]);
                    uint32_t *o32 = reinterpret_cast<uint32_t *>(&out[0]);
#pragma unroll
                    for (int g = 0; g < CH / 4; ++g) {
                        uint32_t e;
                        if constexpr (MODE == SP24_PRUNE_MASK) {
                            const uint32_t mw = *reinterpret_cast<const uint32_t *>(&mk[j][4 * g]);
                            e = glut[64 + (((__vcmpne4(mw, 0u) & 0x01010101u) * 0x01020408u) >> 24)];
                        } else {
                            e = mse_lookup<TIn>(raw[2 * g], raw[2 * g + 1], glut);
                        }
                        o32[g] = __byte_perm(raw[2 * g], raw[2 * g + 1], e >> 8);
                        word |= (e & 0xFu) << (4 * g);
                    }
                } else if constexpr (PAIRS) {
#pragma unroll
                    for (int g2 = 0; g2 < CH / 8; ++g2) {
                        const uint64_t gi = (uint64_t)r * (uint64_t)(P.k / 4) + (uint64_t)(c * (CH / 4) + g2 * 2);
                        float2 v0, v1, x[4];
                        mode_uniform_pairs<MODE>(gi >> 1, P.seed, rng_offset, v0.x, v1.x, v0.y, v1.y);
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            x[e] = make_float2(Elem<TIn>::to_f32(in[j][8 * g2 + e]), Elem<TIn>::to_f32(in[j][8 * g2 + 4 + e]));
                        uint32_t oa, ob;
                        word += two_groups_fast<TOut>(x, v0, v1, picks_at, out_scale, oa, ob) << (8 * g2);
                        reinterpret_cast<uint32_t *>(&out[0])[g2] = oa | (ob << 16);
                    }
                } else
#pragma unroll
                for (int g2 = 0; g2 < CH / 8; ++g2) {
                    float u[4] = {0.f, 0.f, 0.f, 0.f};
                    if constexpr (MODE == PRUNE_SOFT) { u[0] = u[2] = P.soft_scale; u[1] = u[3] = P.soft_use_scale ? 1.f : 0.f; }
                    if constexpr (is_mvue(MODE)) {
                        if constexpr (HAS_U) {
                            const float *up = P.uniforms + r * P.ld_u + c * CH + g2 * 8;
                            const float2 ua = *reinterpret_cast<const float2 *>(up);
                            const float2 ub = *reinterpret_cast<const float2 *>(up + 4);
                            u[0] = ua.x; u[1] = ua.y; u[2] = ub.x; u[3] = ub.y;
                        } else {
                            const uint64_t gi = (uint64_t)r * (uint64_t)(P.k / 4) + (uint64_t)(c * (CH / 4) + g2 * 2);
                            mode_uniform_pairs<MODE>(gi >> 1, P.seed, rng_offset, u[0], u[1], u[2], u[3]);
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int g = g2 * 2 + h;
                        const TIn grp[4] = {in[j][4 * g], in[j][4 * g + 1], in[j][4 * g + 2], in[j][4 * g + 3]};
                        uint32_t given = 0;
                        if constexpr (MODE == SP24_PRUNE_MASK) {
                            given = (mk[j][4 * g] != 0) | ((mk[j][4 * g + 1] != 0) << 1) | ((mk[j][4 * g + 2] != 0) << 2) |
                                    ((mk[j][4 * g + 3] != 0) << 3);
                        }
                        const uint32_t nib =
                            do_group<TIn, TOut, MODE>(grp, given, u[2 * h], u[2 * h + 1], out[2 * g], out[2 * g + 1], glut, out_scale);
                        word |= nib << (4 * g);
                    }
                }
                store_elems<TOut, CH / 2>(packed + r * P.ld_packed + c * (CH / 2), out);
                smeta[lane >> 1][(rr / GROUP) * 2 * GROUP + meta_run_pos<MB>(rr % GROUP, lane & 1)] = (MetaT)word;
                // 8-bit tensor-core order: 16 bytes per row and 128 columns, i.e. four lanes write one 16-byte piece
                if constexpr (MB == 4)
                    if (P.tc) reinterpret_cast<uint32_t *>(P.tc)[(((r >> 7) * P.k_atoms + (c >> 2)) * 128 + (r & 127)) * 4 + (c & 3)] = word;
            }
        }
    }
    __syncthreads();
    // 16 column pairs x 64 words, written as 16-byte pieces
    constexpr int PIECES = 64 * MB / 16;
    for (int i = threadIdx.x; i < 16 * PIECES; i += 256) {
        const int pair = i / PIECES, piece = i % PIECES;
        const int64_t cp = (int64_t)blockIdx.x * 16 + pair;
        if (cp * 2 < ncols) {
            char *dst = static_cast<char *>(P.meta) + (cp * 2 * P.m + 2 * r0) * MB + piece * 16;
            *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(
                reinterpret_cast<const char *>(&smeta[pair][0]) + piece * 16);
        }
    }
    if constexpr (MB == 2) {
        if (P.tc && threadIdx.x < 128) {
            // Second copy in tensor-core order, gathered from the staged runs: the tile's 32 rows x 32 word columns
            // are 32 whole 16-byte lines in each of four atoms.  Line L holds rows 16*(L/16) + 8*h + L%8 (h = 0, 1) of
            // word columns 2*q + (L/8)%2 (q = 0..3) at int16 slot 2*q + h.
            const int atom = threadIdx.x >> 5, L = threadIdx.x & 31, par = (L >> 3) & 1;
            const int64_t atom_col = (int64_t)blockIdx.x * 4 + atom;
            if (atom_col < P.k_atoms) {
                uint32_t o[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int wc = atom * 8 + 2 * q + par;                  // word column inside the tile
                    uint32_t lo = 0, hi = 0;
                    if ((int64_t)blockIdx.x * 32 + wc < ncols) {
                        lo = (uint16_t)smeta[wc >> 1][meta_run_pos<MB>(16 * (L >> 4) + (L & 7), wc & 1)];
                        hi = (uint16_t)smeta[wc >> 1][meta_run_pos<MB>(16 * (L >> 4) + 8 + (L & 7), wc & 1)];
                    }
                    o[q] = lo | (hi << 16);
                }
                const int64_t off = ((r0 >> 7) * P.k_atoms + atom_col) * 2048 + ((r0 & 127) + L) * 16;
                if (off + 16 <= (P.m >> 7) * P.k_atoms * 2048)   // every store is checked against the buffer size
                    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(P.tc) + off) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// column-major storage: element (r, c) at c*ld + r, groups of four run along the strided axis.
// Everything is element-wise across r, so loads and stores are naturally coalesced along r.
// Thread = V consecutive rows x one metadata column; warp = 32*V rows; 8 warps = 8 metadata columns.
// ---------------------------------------------------------------------------------------------
template <typename TIn> struct ColVec {
    static constexpr int wide = sizeof(TIn) == 1 ? 8 : 16 / sizeof(TIn);   // streaming modes: 16-byte (8 for int8) loads
    // Exact MVUE is bound by instruction issue, not by load width: one row per thread makes blocks of 32 rows, which
    // balances the SMs better on short matrices and is never slower on long ones.
    static constexpr int narrow = 1;
    // Fast MVUE with 8-bit results of float32 input, or stored in columns: two rows, two groups at a time, three blocks per SM, where one
    // group at a time took four rows at two blocks: the quantised bytes are gathered by one permute a group.
    static constexpr int fast8 = 2;
};

// resident blocks per SM the register budget is set for
constexpr int col_min_blocks(int mode) {
    return mode == SP24_PRUNE_MVUE_FAST ? 3 : (mode == SP24_PRUNE_MVUE ? 4 : 1);
}

template <typename TIn, typename TOut, int MODE, bool HAS_U, int V>
__global__ void __launch_bounds__(256, col_min_blocks(MODE)) pc_col_kernel(PcParams P) {
    chain_enter();
    const uint64_t rng_offset = P.offset + (P.offset_dev ? *P.offset_dev : 0ull);
    const float out_scale = out_scale_of<TOut>(P);
    constexpr int CH = sizeof(TOut) == 2 ? 16 : 32;
    constexpr int MB = sizeof(TOut) == 2 ? 2 : 4;
    constexpr int GROUP = MB == 2 ? 32 : 16;
    constexpr int RT = 32 * V;  // rows per block
    using MetaT = typename VecBytes<MB>::type;

    __shared__ __align__(16) MetaT smeta[4][2 * RT];
    // tensor-core order: line L = 16*(r/16) + 8*(c%2) + r%8 of 16 bytes, int16 slot 2*((c/2)%4) + (r/8)%2; the block's
    // RT rows x 8 word columns fill RT whole lines of one atom per 128-row block
    // (8-bit outputs: RT rows x 4 32-bit words = RT lines of each of two atoms)
    __shared__ __align__(16) MetaT stc[RT * 8];
    __shared__ float ssum[8][RT];           // per-warp partial row sums (only used when row sums are asked for)
    constexpr bool PAIRS = MODE == SP24_PRUNE_MVUE_FAST;      // two groups at a time, see ColVec
    __shared__ __align__(8) PickEntry picks[PAIRS ? 16 : 1];
    if constexpr (PAIRS) load_pick_lut<TOut>(picks);
    const uint32_t picks_at = (uint32_t)__cvta_generic_to_shared(picks);
    if constexpr (PAIRS) clear_share(P, (int64_t)blockIdx.y * gridDim.x + blockIdx.x, (int64_t)gridDim.x * gridDim.y);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t ncols = P.k / CH;
    const int64_t r0 = (int64_t)blockIdx.x * RT;
    const int64_t r = r0 + lane * V;
    const int64_t c = (int64_t)blockIdx.y * 8 + warp;
    TOut *packed = static_cast<TOut *>(P.packed);

    if (r < P.m && c < ncols) {
        uint32_t word[V];
        float rsum[V];
#pragma unroll
        for (int v = 0; v < V; ++v) { word[v] = 0; rsum[v] = 0.f; }
        // one running pointer per array: the eight storage rows of a step are ld apart
        const TIn *src = static_cast<const TIn *>(P.dense) + (c * CH) * P.ld_dense + r;
        const uint8_t *msrc = MODE == SP24_PRUNE_MASK ? P.mask + (c * CH) * P.ld_mask + r : nullptr;
        TOut *dst = packed + (c * (CH / 2)) * P.ld_packed + r;
        // 8-bit outputs can also leave row-major (the K-major operand order of the 8-bit sparse GEMM): a thread's
        // 32 logical columns are 16 contiguous packed bytes of its row
        constexpr bool CAN_RM = sizeof(TOut) == 1;
        constexpr bool CAN_Q = CAN_RM && !std::is_same<TOut, int8_t>::value;
        TOut *qdst = CAN_Q && P.q_dense ? static_cast<TOut *>(P.q_dense) + (c * CH) * P.ld_q + r : nullptr;
        alignas(16) TOut orow[CAN_RM ? V : 1][CAN_RM ? CH / 2 : 1];
        // a step = 8 consecutive storage rows = two groups of four per logical row = one Philox block, counted along the row
        uint64_t pair0[V];
#pragma unroll
        for (int v = 0; v < V; ++v) pair0[v] = (uint64_t)(r + v) * (uint64_t)(P.k / 8) + (uint64_t)(c * (CH / 8));
#pragma unroll
        for (int step = 0; step < CH / 8; ++step) {
            Vec<TIn, V> in[8];
            Vec<uint8_t, V> mk[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                in[j] = load_vec<TIn, V>(src + j * P.ld_dense);
                if constexpr (MODE == SP24_PRUNE_MASK) mk[j] = load_vec<uint8_t, V>(msrc + j * P.ld_mask);
            }
            src += 8 * P.ld_dense;
            if constexpr (MODE == SP24_PRUNE_MASK) msrc += 8 * P.ld_mask;
            if constexpr (CAN_Q) {
                if (P.q_dense) {   // the whole tensor quantised on the way (the other operand of the layer's GEMMs)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float f[V];
#pragma unroll
                        for (int v = 0; v < V; ++v) f[v] = __fmul_rn(Elem<TIn>::to_f32(in[j].v[v]), out_scale);
                        store_f8<TOut, V>(qdst + j * P.ld_q, f);
                    }
                    qdst += 8 * P.ld_q;
                }
            }
            if constexpr (PAIRS) {
                uint32_t o[2][V];                // per group and row: the two stored values
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    float2 v0, v1, x[4];
                    mode_uniform_pairs<MODE>(pair0[v] | step, P.seed, rng_offset, v0.x, v1.x, v0.y, v1.y);
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[j] = make_float2(Elem<TIn>::to_f32(in[j].v[v]), Elem<TIn>::to_f32(in[4 + j].v[v]));
                    if (P.row_sums) {   // sums of the unpruned values, fp32
                        const float2 a = __fadd2_rn(__fadd2_rn(x[0], x[1]), __fadd2_rn(x[2], x[3]));
                        rsum[v] += a.x + a.y;
                    }
                    word[v] += two_groups_fast<TOut>(x, v0, v1, picks_at, out_scale, o[0][v], o[1][v]) << (8 * step);
                }
                static_assert(CAN_RM && V == 2, "8-bit results, two rows a thread");
#pragma unroll
                for (int v = 0; v < V; ++v) *reinterpret_cast<uint32_t *>(&orow[v][4 * step]) = o[0][v] | (o[1][v] << 16);
                if (!P.packed_rm) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {       // the lower and the higher stored values of two rows
                        const uint32_t both = __byte_perm(o[h][0], o[h][1], 0x5140u);
                        *reinterpret_cast<uint16_t *>(dst) = (uint16_t)both;
                        *reinterpret_cast<uint16_t *>(dst + P.ld_packed) = (uint16_t)(both >> 16);
                        dst += 2 * P.ld_packed;
                    }
                }
            } else {
                if (P.row_sums) {   // sums of the unpruned values, fp32
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float a = 0.f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) a += Elem<TIn>::to_f32(in[j].v[v]);
                        rsum[v] += a;
                    }
                }
                float u[V][4];
                if constexpr (is_mvue(MODE)) {
                    const int64_t gcol = c * (CH / 4) + step * 2;  // first of the two groups
                    if constexpr (HAS_U) {
                        float t0[V], t1[V], t2[V], t3[V];
                        load_elems<float, V>(P.uniforms + (gcol * 4 + 0) * P.ld_u + r, t0);
                        load_elems<float, V>(P.uniforms + (gcol * 4 + 1) * P.ld_u + r, t1);
                        load_elems<float, V>(P.uniforms + (gcol * 4 + 4) * P.ld_u + r, t2);
                        load_elems<float, V>(P.uniforms + (gcol * 4 + 5) * P.ld_u + r, t3);
#pragma unroll
                        for (int v = 0; v < V; ++v) { u[v][0] = t0[v]; u[v][1] = t1[v]; u[v][2] = t2[v]; u[v][3] = t3[v]; }
                    } else {
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            mode_uniform_pairs<MODE>(pair0[v] + step, P.seed, rng_offset, u[v][0], u[v][1], u[v][2], u[v][3]);
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    Vec<TOut, V> o0, o1;
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        const TIn grp[4] = {in[4 * h].v[v], in[4 * h + 1].v[v], in[4 * h + 2].v[v], in[4 * h + 3].v[v]};
                        uint32_t given = 0;
                        if constexpr (MODE == SP24_PRUNE_MASK) {
                            given = (mk[4 * h].v[v] != 0) | ((mk[4 * h + 1].v[v] != 0) << 1) | ((mk[4 * h + 2].v[v] != 0) << 2) |
                                    ((mk[4 * h + 3].v[v] != 0) << 3);
                        }
                        float ua = 0.f, ub = 0.f;
                        if constexpr (is_mvue(MODE)) { ua = u[v][2 * h]; ub = u[v][2 * h + 1]; }
                        if constexpr (MODE == PRUNE_SOFT) { ua = P.soft_scale; ub = P.soft_use_scale ? 1.f : 0.f; }
                        const uint32_t nib = do_group<TIn, TOut, MODE>(grp, given, ua, ub, o0.v[v], o1.v[v], nullptr, out_scale);
                        word[v] |= nib << (4 * (step * 2 + h));
                        if constexpr (CAN_RM) {
                            orow[v][(step * 2 + h) * 2] = o0.v[v];
                            orow[v][(step * 2 + h) * 2 + 1] = o1.v[v];
                        }
                    }
                    if (!CAN_RM || !P.packed_rm) {
                        store_vec<TOut, V>(dst, o0);
                        store_vec<TOut, V>(dst + P.ld_packed, o1);
                        dst += 2 * P.ld_packed;
                    }
                }
            }
        }
        if constexpr (CAN_RM) {
            if (P.packed_rm) {
#pragma unroll
                for (int v = 0; v < V; ++v) store_elems<TOut, CH / 2>(packed + (r + v) * P.ld_packed + c * (CH / 2), orow[v]);
            }
        }
        if (P.row_sums) {
#pragma unroll
            for (int v = 0; v < V; ++v) ssum[warp][lane * V + v] = rsum[v];
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int rr = lane * V + v;
            smeta[warp >> 1][(rr / GROUP) * 2 * GROUP + meta_run_pos<MB>(rr % GROUP, warp & 1)] = (MetaT)word[v];
            if constexpr (MB == 2) {
                if (P.tc) stc[8 * (16 * (rr >> 4) + 8 * (warp & 1) + (rr & 7)) + 2 * (warp >> 1) + ((rr >> 3) & 1)] = (uint16_t)word[v];
            } else {
                if (P.tc) stc[(warp >> 2) * RT * 4 + rr * 4 + (warp & 3)] = word[v];
            }
        }
    } else {
        if (P.row_sums) {
#pragma unroll
            for (int v = 0; v < V; ++v) ssum[warp][lane * V + v] = 0.f;
        }
        if constexpr (MB == 2) {
            // word columns past the matrix (K not a multiple of 128): zeros, the GEMM multiplies them by zero-filled operands
            if (P.tc && r < P.m) {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const int rr = lane * V + v;
                    stc[8 * (16 * (rr >> 4) + 8 * (warp & 1) + (rr & 7)) + 2 * (warp >> 1) + ((rr >> 3) & 1)] = 0;
                }
            }
        }
    }
    __syncthreads();
    if (P.row_sums) {
        // the eight warps hold eight K ranges of the same rows: one reduction per row and block
        for (int t = threadIdx.x; t < RT; t += 256) {
            if (r0 + t < P.m) {
                // parts are of 128 storage rows: the block's eight words of 16 bits are one, of 32 bits two
                constexpr int HALVES = MB == 4 ? 2 : 1;
#pragma unroll
                for (int h = 0; h < HALVES; ++h) {
                    float a = 0.f;
#pragma unroll
                    for (int w = 0; w < 8 / HALVES; ++w) a += ssum[h * 4 + w][t];
                    const int64_t part = (int64_t)blockIdx.y * HALVES + h;
                    if (!P.ld_sums) atomicAdd(P.row_sums + r0 + t, a);
                    else if (part < P.k_atoms) P.row_sums[part * P.ld_sums + r0 + t] = a;
                }
            }
        }
    }
    const int64_t rows_here = (P.m - r0 < RT) ? (P.m - r0) : RT;
    const int pieces = (int)(rows_here * 2 * MB / 16);
    for (int i = threadIdx.x; i < 4 * (2 * RT * MB / 16); i += 256) {
        const int pair = i / (2 * RT * MB / 16), piece = i % (2 * RT * MB / 16);
        const int64_t cp = (int64_t)blockIdx.y * 4 + pair;
        if (piece < pieces && cp * 2 < ncols) {
            char *dstm = static_cast<char *>(P.meta) + (cp * 2 * P.m + 2 * r0) * MB + piece * 16;
            *reinterpret_cast<uint4 *>(dstm) = *reinterpret_cast<const uint4 *>(
                reinterpret_cast<const char *>(&smeta[pair][0]) + piece * 16);
        }
    }
    if constexpr (MB == 4) {
        if (P.tc) {
            for (int i = threadIdx.x; i < 2 * RT; i += 256) {
                const int half = i / RT, pline = i % RT;
                const int64_t atom = (int64_t)blockIdx.y * 2 + half, gr = r0 + pline;
                if (pline < rows_here && atom < P.k_atoms)
                    reinterpret_cast<uint4 *>(P.tc)[((gr >> 7) * P.k_atoms + atom) * 128 + (gr & 127)] = reinterpret_cast<const uint4 *>(stc)[i];
            }
        }
    }
    if constexpr (MB == 2) {
        if (P.tc) {
            for (int pline = threadIdx.x; pline < RT; pline += 256) {
                if (pline < rows_here) {
                    const int64_t gr = r0 + pline;   // line index inside the 128-row block = row index of its first writer
                    const int64_t off = ((gr >> 7) * P.k_atoms + blockIdx.y) * 2048 + (gr & 127) * 16;
                    if (off + 16 <= (P.m >> 7) * P.k_atoms * 2048)   // every store is checked against the buffer size
                        *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(P.tc) + off) =
                            *reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(stc) + pline * 16);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Fast MVUE, column-major storage, 16-bit results, or row-major float8 ones of 16-bit input: dY^T, the sparse operand of every
// weight-gradient GEMM.
// ---------------------------------------------------------------------------------------------
// Bound by arithmetic: about 80 instructions a group of four for the draws, quotients and random numbers, which by themselves (operands
// in shared memory, no traffic) take 115 cycles a warp and group, 67 % of the time measured here; the rest are copies, addresses and
// metadata.  So: persistent blocks, whose warps fetch their 16 columns of the next two tiles by asynchronous copies (no registers hold
// loads, no warp waits at the start of a block), compressed rows written over storage rows that have been read and stored
// 16 bytes a lane, one barrier a tile (for the metadata, which eight warps assemble), and two groups at a time in two-lane arithmetic.
// Two blocks of 128 registers: with three (80) or four (64) the loop's constants no longer fit and the same work is 106 and 109
// instructions a group instead of 98.  us a replayed launch, one group at a time in a block per tile -> here: bf16 4096 x 8192 45.0 -> 38.0,
// fp16 3072 x 16384 63.9 -> 55.9, bf16 with row sums 3072 x 8192 37.0 -> 29.2, 768 x 8192 11.2 -> 9.4, fp16 512 x 256 5.1 -> 3.1, float32
// 4096 x 8192 42.7 -> 42.4, 512 x 256 5.0 -> 3.3.
// Float8 results with the quantised tensor and row sums (stored rows staged for one 16-byte store a thread, quantised rows for two a
// lane), blocks of their own tile each -> here: bf16 3072 x 8192 40.8 -> 34.8, 768 x 8192 12.3 -> 11.7, 1024 x 4096 9.8 -> 8.8, 1024 x 1024
// 6.6 -> 4.2.  Float8 results of float32 input stay with the other kernel.
// Three or four stages of copies instead of two, and tiles of two or four 16-column slices a warp, gained nothing.
template <typename TIn, typename TOut> struct MvueCol {
    static constexpr bool F8 = sizeof(TOut) == 1;
    static constexpr int RT = 64;                                // rows of a tile; each of its eight warps takes 16 logical columns
    static constexpr int ROW = RT * sizeof(TIn);                 // bytes of one storage row of a tile
    static constexpr int SLICE = 16 * ROW, STAGES = 2;           // a warp's share, and how many of them are under way
    static constexpr int RUN = 0, LINE = 4 * 2 * RT * 2, SUMS = LINE + RT * 16, PACK = SUMS + 8 * RT * 4;     // staged results
    static constexpr int OUT = PACK + (F8 ? RT * 64 : 0);
    static constexpr int QUANT = STAGES * 8 * SLICE + 2 * OUT;   // float8: a warp's 16 storage rows quantised
    static constexpr int SMEM = QUANT + (F8 ? 8 * 16 * RT : 0);
    static constexpr int BLOCKS = 2;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// Keeps a value that a loop needs in its register: worked out anew in every pass, such values cost more than the arithmetic they serve.
template <typename T> __device__ __forceinline__ void pin(T &v) {
    if constexpr (sizeof(T) == 8) asm volatile("" : "+l"(v));
    else asm volatile("" : "+r"(v));
}
__device__ __forceinline__ void st_shared16(uint32_t addr, uint32_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((uint16_t)v) : "memory"); }

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256, MvueCol<TIn, TOut>::BLOCKS)
mvue_col_kernel(const __grid_constant__ PcParams P, const __grid_constant__ PhiloxKeys<kMvueFastRounds> keys) {
    chain_enter();
    using Cfg = MvueCol<TIn, TOut>;
    constexpr bool F8 = Cfg::F8;
    constexpr int RT = Cfg::RT, ROW = Cfg::ROW, STAGES = Cfg::STAGES, V = 2;
    static_assert(!F8 || sizeof(TIn) == 2, "float8 from 16-bit values only");
    const float out_scale = out_scale_of<TOut>(P);
    // 16-bit input: a lane writes only over the four bytes of a row that it alone reads.  Float32 rows are twice as long: other lanes
    // read where it writes.
    constexpr bool OWN_BYTES = ROW == RT * sizeof(TOut) && V * sizeof(TIn) == 4;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ __align__(8) PickEntry picks[16];
    load_pick_lut<TOut>(picks);
    const uint32_t picks_at = (uint32_t)__cvta_generic_to_shared(picks);
    const uint64_t rng_offset = P.offset + (P.offset_dev ? *P.offset_dev : 0ull);

    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);
    const int m = (int)P.m, ncols = (int)(P.k / 16);
    const int n_rt = (m + RT - 1) / RT, n_ct = (ncols + 7) / 8;
    // tile -> (row tile, column tile), the row tile varying fastest; both advance by the grid without a division
    const int grid_r = (int)(gridDim.x % n_rt), grid_c = (int)(gridDim.x / n_rt);
    auto advance = [&](int &tr, int &tc) {
        tr += grid_r;
        tc += grid_c;
        if (tr >= n_rt) { tr -= n_rt; ++tc; }
    };
    // asynchronous copies of a slice's 16 storage rows, 16 bytes a lane and copy
    constexpr int PIECES = ROW / 16, AT_ONCE = 32 / PIECES;
    const uint32_t ld_in = (uint32_t)P.ld_dense * (uint32_t)sizeof(TIn), ld_out = (uint32_t)P.ld_packed * 2u;      // bytes
    uint8_t *const slices = smem + warp * (STAGES * Cfg::SLICE);
    uint32_t fetch_to = (uint32_t)__cvta_generic_to_shared(slices) + lane * 16;
    const char *fetch_from = static_cast<const char *>(P.dense) + (uint64_t)(lane / PIECES) * ld_in + lane % PIECES * 16;
    int fetch_row = lane % PIECES * (16 / (int)sizeof(TIn));
    pin(fetch_to);
    pin(fetch_from);
    pin(fetch_row);
    int ftr = blockIdx.x % n_rt, ftc = blockIdx.x / n_rt;
    auto fetch = [&](int buf) {
        const int c = ftc * 8 + warp;
        if (fetch_row + ftr * RT < m && c < ncols) {
            const char *src = fetch_from + ((uint64_t)(uint32_t)(c * 16) * ld_in + (uint32_t)(ftr * ROW));
#pragma unroll
            for (int i = 0; i < 16 / AT_ONCE; ++i, src += (uint64_t)AT_ONCE * ld_in) cp_async16(fetch_to + buf * Cfg::SLICE + i * 512, src);
        }
        cp_async_commit();
        advance(ftr, ftc);
    };
    // where a lane's two words go in the staged metadata (the second 8 words behind the first in both orders), and its 16 bytes of the
    // stored rows
    const int rr = lane * V;
    // (float8: half a 32-bit word each; the row after is 16 bytes further in either order and either type)
    const uint32_t staged = (uint32_t)__cvta_generic_to_shared(smem + STAGES * 8 * Cfg::SLICE);
    uint32_t run_at = staged + Cfg::RUN + (F8 ? 4 * ((warp >> 2) * 2 * RT + (rr / 16) * 32 + meta_run_pos<4>(rr % 16, (warp >> 1) & 1)) + 2 * (warp & 1)
                                              : 2 * ((warp >> 1) * 2 * RT + (rr / 32) * 64 + meta_run_pos<2>(rr % 32, warp & 1)));
    uint32_t line_at = staged + Cfg::LINE + (F8 ? rr * 16 + warp * 2
                                                : 2 * (8 * (16 * (rr >> 4) + 8 * (warp & 1) + (rr & 7)) + 2 * (warp >> 1) + ((rr >> 3) & 1)));
    char *store_to = static_cast<char *>(P.packed) + (uint64_t)(lane >> 3) * ld_out + (lane & 7) * 16;
    // float8: a row's 64 stored bytes of a tile are eight pieces of 8, one a warp; rows 2 l and 2 l + 1 share 128 bytes whose halves change
    // places every eight l, the pieces exchanged by l % 8: no bank is met twice
    auto pack_at = [](int row, int piece) {
        const int l = row >> 1;
        return Cfg::PACK + l * 128 + (((row & 1) ^ ((l >> 3) & 1)) << 6) + ((piece ^ (l & 7)) << 3);
    };
    uint32_t pack_to[2] = {staged + pack_at(rr, warp), staged + pack_at(rr + 1, warp)};
    uint8_t *const quant = smem + Cfg::QUANT + warp * (16 * RT);
    pin(run_at);
    pin(line_at);
    pin(store_to);

    for (int i = 0; i < STAGES; ++i) fetch(i);
    clear_share(P, blockIdx.x, gridDim.x);
    int tr = blockIdx.x % n_rt, tc = blockIdx.x / n_rt, buf = 0;
    uint32_t out_off = 0;
    const uint32_t row_pairs = (uint32_t)(P.k / 8);
#pragma unroll 1
    for (; tc < n_ct; advance(tr, tc)) {
        const int r0 = tr * RT, c = tc * 8 + warp;
        uint8_t *const sl = slices + buf * Cfg::SLICE;
        cp_async_wait<STAGES - 1>();
        __syncwarp();
        uint32_t word[V] = {0, 0};
        float rsum[V] = {0.f, 0.f};
        const bool mine = r0 + lane * V < m && c < ncols;      // all lanes, the first 16 or none
        const uint32_t together = OWN_BYTES ? 0u : __ballot_sync(0xFFFFFFFFu, mine);
        if (mine) {
            uint64_t pair[V];
            pair[0] = (uint64_t)(uint32_t)(r0 + lane * V) * row_pairs + (uint32_t)(c * 2);
            pair[1] = pair[0] + row_pairs;
            uint32_t stored[F8 ? V : 1][2];
#pragma unroll
            for (int step = 0; step < 2; ++step) {
                Vec<TIn, V> in[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) in[j] = load_vec<TIn, V>(reinterpret_cast<const TIn *>(sl + (8 * step + j) * ROW) + lane * V);
                if constexpr (F8) {
                    if (P.q_dense) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float f[V] = {__fmul_rn(Elem<TIn>::to_f32(in[j].v[0]), out_scale), __fmul_rn(Elem<TIn>::to_f32(in[j].v[1]), out_scale)};
                            store_f8<TOut, V>(reinterpret_cast<TOut *>(quant + (8 * step + j) * RT + lane * V), f);
                        }
                    }
                }
                uint32_t o[2][V];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    // the count of blocks before the slice is even: K is a multiple of 64
                    const uint4 u = philox4x32<kMvueFastRounds>(make_uint4((uint32_t)pair[v] | step, (uint32_t)(pair[v] >> 32), (uint32_t)rng_offset, (uint32_t)(rng_offset >> 32)), keys);
                    const float2 v0 = make_float2(u32_to_one_plus_uniform(u.x), u32_to_one_plus_uniform(u.z));
                    const float2 v1 = make_float2(u32_to_one_plus_uniform(u.y), u32_to_one_plus_uniform(u.w));
                    float2 x[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[j] = make_float2(Elem<TIn>::to_f32(in[j].v[v]), Elem<TIn>::to_f32(in[4 + j].v[v]));
                    if (P.row_sums) {   // sums of the unpruned values, fp32
                        const float2 a = __fadd2_rn(__fadd2_rn(x[0], x[1]), __fadd2_rn(x[2], x[3]));
                        rsum[v] += a.x + a.y;
                    }
                    word[v] += two_groups_fast<TOut>(x, v0, v1, picks_at, out_scale, o[0][v], o[1][v]) << (8 * step);
                    if constexpr (F8) stored[v][step] = o[0][v] | (o[1][v] << 16);
                }
                if constexpr (F8) continue;
                // stored rows (128 bytes) take the place of the first storage rows, which all lanes have read by now
                if constexpr (!OWN_BYTES) __syncwarp(together);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t *to = reinterpret_cast<uint32_t *>(sl + (4 * step + 2 * h) * 128) + lane;
                    to[0] = __byte_perm(o[h][0], o[h][1], 0x5410u);
                    to[32] = __byte_perm(o[h][0], o[h][1], 0x7632u);
                }
            }
            if constexpr (F8) {
#pragma unroll
                for (int v = 0; v < V; ++v)
                    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(pack_to[v] + out_off), "r"(stored[v][0]), "r"(stored[v][1]) : "memory");
            }
        }
        // word columns past the matrix (K not a multiple of 128) are zeros in the tensor-core copy: the GEMM multiplies them by
        // zero-filled operands
        st_shared16(run_at + out_off, word[0]);
        st_shared16(run_at + out_off + 16, word[1]);
        st_shared16(line_at + out_off, word[0]);
        st_shared16(line_at + out_off + 16, word[1]);
        if (P.row_sums) *reinterpret_cast<float2 *>(smem + STAGES * 8 * Cfg::SLICE + out_off + Cfg::SUMS + (warp * RT + rr) * 4) = make_float2(rsum[0], rsum[1]);
        __syncwarp();
        if constexpr (F8) {
            if (P.q_dense && r0 + (lane & 3) * 16 < m) {       // 16 rows of 64 bytes (float8: columns come in whole tiles)
                char *dst = static_cast<char *>(P.q_dense) + (c * 16 + (lane >> 2)) * P.ld_q + r0 + (lane & 3) * 16;
                *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(quant + lane * 16);
                *reinterpret_cast<uint4 *>(dst + 8 * P.ld_q) = *reinterpret_cast<const uint4 *>(quant + 512 + lane * 16);
            }
        } else if (r0 + (lane & 7) * 8 < m && c < ncols) {       // 8 rows of 128 bytes, 16 bytes a lane and store
            char *dst = store_to + ((uint64_t)(uint32_t)(c * 8) * ld_out + (uint32_t)(r0 * 2));
            *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(sl + lane * 16);
            *reinterpret_cast<uint4 *>(dst + 4ull * ld_out) = *reinterpret_cast<const uint4 *>(sl + 512 + lane * 16);
        }
        __syncwarp();
        fetch(buf);
        if (++buf == STAGES) buf = 0;
        __syncthreads();
        // metadata and row sums of the tile, one piece a thread; the next tile's are staged in the other buffer, and nobody is two
        // tiles ahead
        const uint8_t *out = smem + STAGES * 8 * Cfg::SLICE + out_off;
        const int t = threadIdx.x & 63, rows_here = m - r0;
        if constexpr (F8) {
            const int row = threadIdx.x >> 2, piece = threadIdx.x & 3;       // 16 bytes a thread
            if (row < rows_here) {
                const uint2 lo = *reinterpret_cast<const uint2 *>(out + pack_at(row, 2 * piece)), hi = *reinterpret_cast<const uint2 *>(out + pack_at(row, 2 * piece + 1));
                *reinterpret_cast<uint4 *>(static_cast<char *>(P.packed) + (int64_t)(r0 + row) * P.ld_packed + tc * 64 + piece * 16) =
                    make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
        }
        if (F8 && warp < 2) {
            // 2 column pairs x 2 RT words of 4 bytes
            const int cp = tc * 2 + (t >> 5), pc = t & 31;
            if (pc * 2 < rows_here)
                *reinterpret_cast<uint4 *>(static_cast<char *>(P.meta) + ((uint64_t)(uint32_t)cp * (uint32_t)m + (uint32_t)r0) * 8 + pc * 16) =
                    *reinterpret_cast<const uint4 *>(out + Cfg::RUN + t * 16);
        } else if (warp < 2) {
            // 4 column pairs x 2 RT words
            const int cp = tc * 4 + (t >> 4), pc = t & 15;
            if (pc * 4 < rows_here && cp * 2 < ncols)
                *reinterpret_cast<uint4 *>(static_cast<char *>(P.meta) + ((uint64_t)(uint32_t)cp * (uint32_t)m + (uint32_t)r0) * 4 + pc * 16) =
                    *reinterpret_cast<const uint4 *>(out + Cfg::RUN + t * 16);
        } else if (warp < 4) {
            const int gr = r0 + t;    // line index inside the 128-row block = row index of its first writer
            if (P.tc && t < rows_here) {
                const int64_t off = ((gr >> 7) * P.k_atoms + tc) * 2048 + (gr & 127) * 16;
                if (off + 16 <= (P.m >> 7) * P.k_atoms * 2048)   // every store is checked against the buffer size
                    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(P.tc) + off) = *reinterpret_cast<const uint4 *>(out + Cfg::LINE + t * 16);
            }
        } else if (warp < 6) {
            if (P.row_sums && t < rows_here) {
                const float *ssum = reinterpret_cast<const float *>(out + Cfg::SUMS);
                float a = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) a += ssum[w * RT + t];
                if (P.ld_sums) P.row_sums[tc * P.ld_sums + r0 + t] = a;
                else atomicAdd(P.row_sums + r0 + t, a);
            }
        }
        out_off ^= Cfg::OUT;
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------------------------------------
// W and W^T of a float8 layer under one mask, e4m3, both packed row-major (K-major), from one read of W.
// ---------------------------------------------------------------------------------------------
// A warp takes 16 rows x 128 columns, a thread four columns of them, all loads under way at once: every value is quantised once, then
// the thread's 16 row groups and 16 column groups are looked up by their four mask bits.  The row groups' codes of eight lanes are a
// metadata word: an 8 x 8 transpose of nibbles in three exchanges.  A column's 16 rows are 8 stored bytes and half a word.  Nothing is
// staged; the two launches that this one replaces read W and its mask twice.  us, replayed, both copies with the masked maximum before
// them, two launches -> one: 3072 x 768 16.0 -> 9.6, 1024 x 1024 15.9 -> 7.3, 256 x 256 13.0 -> 6.6, 4096 x 4096 60.2 -> 42.2.
struct DualF8Params {
    const void *w;
    const uint8_t *mask;
    const float *amax;
    uint8_t *packed_w, *packed_t;
    int32_t *meta_w, *tc_w;
    uint16_t *meta_t, *tc_t;            // halves of words
    int64_t m, k, ld_w, ld_mask;
};
__device__ __forceinline__ uint32_t transpose_nibbles(uint32_t x, int lane) {      // nibble j of lane l <- nibble l of lane j, in each eight lanes
#pragma unroll
    for (int s = 4; s; s >>= 1) {
        const uint32_t low = s == 4 ? 0x0000FFFFu : (s == 2 ? 0x00FF00FFu : 0x0F0F0F0Fu), y = __shfl_xor_sync(0xFFFFFFFFu, x, s);
        x = lane & s ? (x & ~low) | ((y >> (4 * s)) & low) : (x & low) | ((y & low) << (4 * s));
    }
    return x;
}

template <typename TIn> __global__ void __launch_bounds__(128) dual_f8_kernel(DualF8Params P) {
    chain_enter();
    __shared__ __align__(8) PickEntry by_keep[16];
    __shared__ float sc;
    const int lane = threadIdx.x & 31;
    const int64_t c0 = (int64_t)blockIdx.x * 128 + 4 * lane, r0 = (int64_t)blockIdx.y * 64 + (threadIdx.x >> 5) * 16;
    Vec<TIn, 4> in[16];
    uint32_t mk[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        in[i] = load_vec<TIn, 4>(static_cast<const TIn *>(P.w) + (r0 + i) * P.ld_w + c0);
        mk[i] = *reinterpret_cast<const uint32_t *>(P.mask + (r0 + i) * P.ld_mask + c0);
    }
    if (threadIdx.x < 16) {
        const uint32_t code = encode_nibble(threadIdx.x);
        by_keep[threadIdx.x] = PickEntry{(code & 3u) | (code >> 2) << 4 | 0x4400u, code};
    }
    if (threadIdx.x == 0) sc = f8_store_scale(*P.amax);
    __syncthreads();
    const float scale = sc;
    const uint32_t table = (uint32_t)__cvta_generic_to_shared(by_keep);
    auto two = [](float lo, float hi) { return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3); };

    uint32_t words[2] = {0, 0};         // codes of rows 0..7 and 8..15
    uint32_t col_word[4] = {0, 0, 0, 0}, col_packed[4][2];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        uint32_t q[4], keeps = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const Vec<TIn, 4> &x = in[4 * b + i];
            q[i] = two(__fmul_rn(Elem<TIn>::to_f32(x.v[0]), scale), __fmul_rn(Elem<TIn>::to_f32(x.v[1]), scale)) |
                   two(__fmul_rn(Elem<TIn>::to_f32(x.v[2]), scale), __fmul_rn(Elem<TIn>::to_f32(x.v[3]), scale)) << 16;
            const uint32_t keep = ((__vcmpne4(mk[4 * b + i], 0u) & 0x01010101u) * 0x01020408u) >> 24;
            keeps |= keep << (4 * i);
            const uint2 e = pick_entry(table + 8 * keep);
            const int64_t r = r0 + 4 * b + i;
            *reinterpret_cast<uint16_t *>(P.packed_w + (r * P.k + c0) / 2) = (uint16_t)__byte_perm(q[i], 0u, e.x);
            words[b >> 1] |= e.y << (4 * (4 * (b & 1) + i));
        }
        const uint32_t t0 = __byte_perm(q[0], q[1], 0x5140u), t1 = __byte_perm(q[2], q[3], 0x5140u);
        const uint32_t t2 = __byte_perm(q[0], q[1], 0x7362u), t3 = __byte_perm(q[2], q[3], 0x7362u);
        const uint32_t col[4] = {__byte_perm(t0, t1, 0x5410u), __byte_perm(t0, t1, 0x7632u), __byte_perm(t2, t3, 0x5410u), __byte_perm(t2, t3, 0x7632u)};
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const uint32_t keep = ((((keeps >> v) & 0x1111u) * 0x1248u) >> 12) & 0xFu;      // bit v of the four rows
            const uint2 e = pick_entry(table + 8 * keep);
            const uint32_t o = __byte_perm(col[v], 0u, e.x) & 0xFFFFu;
            if (b & 1) col_packed[v][b >> 1] |= o << 16;
            else col_packed[v][b >> 1] = o;
            col_word[v] |= e.y << (4 * b);
        }
    }
    // metadata of W: lane l has rows l % 8 and 8 + l % 8 of the 32 columns that its eight lanes share
    const int64_t wc = c0 / 32, atoms_w = P.k / 128, atoms_t = P.m / 128;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int32_t word = (int32_t)transpose_nibbles(words[h], lane);
        const int64_t r = r0 + 8 * h + (lane & 7);
        P.meta_w[meta_offset<4>(r, wc, P.m)] = word;
        P.tc_w[(((r >> 7) * atoms_w + (wc >> 2)) * 128 + (r & 127)) * 4 + (wc & 3)] = word;
    }
    const int64_t tw = r0 / 32, half = (r0 >> 4) & 1;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const int64_t c = c0 + v;
        *reinterpret_cast<uint2 *>(P.packed_t + (c * P.m + r0) / 2) = make_uint2(col_packed[v][0], col_packed[v][1]);
        P.meta_t[2 * meta_offset<4>(c, tw, P.k) + half] = (uint16_t)col_word[v];
        P.tc_t[2 * ((((c >> 7) * atoms_t + (tw >> 2)) * 128 + (c & 127)) * 4 + (tw & 3)) + half] = (uint16_t)col_word[v];
    }
}

// Lets a kernel take more than 48 KB of dynamic shared memory, once per kernel and device.
template <auto KERN> int allow_shared_memory(int bytes) {
    static std::atomic<bool> done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !done[dev]) {
        if (cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return runtime_error();
        if (dev >= 0 && dev < 64) done[dev] = true;
    }
    return SP24_OK;
}

template <typename TIn, typename TOut> int launch_mvue_col(const PcParams &P, cudaStream_t st) {
    using Cfg = MvueCol<TIn, TOut>;
    constexpr auto kern = mvue_col_kernel<TIn, TOut>;
    if (int rc = allow_shared_memory<mvue_col_kernel<TIn, TOut>>(Cfg::SMEM)) return rc;
    const int64_t tiles = ((P.m + Cfg::RT - 1) / Cfg::RT) * ((P.k / 16 + 7) / 8), most = (int64_t)sm_count() * Cfg::BLOCKS;
    launch_chained(st, kern, (unsigned)(tiles < most ? tiles : most), 256, Cfg::SMEM, P, PhiloxKeys<kMvueFastRounds>(P.seed));
    return launch_status();
}

template <typename TIn, typename TOut, int MODE, bool HAS_U>
int launch(const PcParams &P, int col_major, cudaStream_t st) {
    constexpr int CH = sizeof(TOut) == 2 ? 16 : 32;
    if (!col_major) {
        dim3 grid((unsigned)((P.k / CH + 31) / 32), (unsigned)(P.m / 32));
        if constexpr (is_mvue(MODE)) launch_balanced(st, pc_row_kernel<TIn, TOut, MODE, HAS_U>, grid, 256, 0, P);
        else launch_chained(st, pc_row_kernel<TIn, TOut, MODE, HAS_U>, grid, 256, 0, P);
    } else if constexpr (MODE == SP24_PRUNE_MVUE_FAST && sizeof(TOut) == 2) {
        return launch_mvue_col<TIn, TOut>(P, st);
    } else {
        if constexpr (MODE == SP24_PRUNE_MVUE_FAST && sizeof(TIn) == 2)
            if (P.packed_rm) return launch_mvue_col<TIn, TOut>(P, st);
        constexpr int V = MODE == SP24_PRUNE_MVUE_FAST ? ColVec<TIn>::fast8
                                                       : (MODE == SP24_PRUNE_MVUE ? ColVec<TIn>::narrow : ColVec<TIn>::wide);
        constexpr int RT = 32 * V;
        dim3 grid((unsigned)((P.m + RT - 1) / RT), (unsigned)((P.k / CH + 7) / 8));
        if constexpr (is_mvue(MODE)) launch_balanced(st, pc_col_kernel<TIn, TOut, MODE, HAS_U, V>, grid, 256, 0, P);
        else launch_chained(st, pc_col_kernel<TIn, TOut, MODE, HAS_U, V>, grid, 256, 0, P);
    }
    return launch_status();
}

template <typename TIn, typename TOut> int dispatch_mode(const PcParams &P, int mode, int col_major, cudaStream_t st) {
    switch (mode) {
        case SP24_PRUNE_MSE: return launch<TIn, TOut, SP24_PRUNE_MSE, false>(P, col_major, st);
        case SP24_PRUNE_MASK: return launch<TIn, TOut, SP24_PRUNE_MASK, false>(P, col_major, st);
        case SP24_PRUNE_MVUE:
            if constexpr (std::is_same<TIn, int8_t>::value) {
                return SP24_ERR_DTYPE;
            } else {
                return P.uniforms ? launch<TIn, TOut, SP24_PRUNE_MVUE, true>(P, col_major, st)
                                  : launch<TIn, TOut, SP24_PRUNE_MVUE, false>(P, col_major, st);
            }
        case SP24_PRUNE_MVUE_FAST:
            if constexpr (std::is_same<TIn, int8_t>::value) return SP24_ERR_DTYPE;
            else return launch<TIn, TOut, SP24_PRUNE_MVUE_FAST, false>(P, col_major, st);
        case PRUNE_SOFT:
            if constexpr (std::is_same<TIn, int8_t>::value || sizeof(TOut) != 2) return SP24_ERR_DTYPE;
            else return launch<TIn, TOut, PRUNE_SOFT, false>(P, col_major, st);
        default: return SP24_ERR_ARG;
    }
}

template <typename TIn> int dispatch_out(const PcParams &P, int packed_dtype, int mode, int col_major, cudaStream_t st) {
    switch (packed_dtype) {
        case SP24_F16: return dispatch_mode<TIn, __half>(P, mode, col_major, st);
        case SP24_BF16: return dispatch_mode<TIn, __nv_bfloat16>(P, mode, col_major, st);
        case SP24_E4M3: return dispatch_mode<TIn, e4m3_t>(P, mode, col_major, st);
        case SP24_E5M2: return dispatch_mode<TIn, e5m2_t>(P, mode, col_major, st);
        default: return SP24_ERR_DTYPE;
    }
}

}  // namespace
}  // namespace sp24

static int prune_compress_impl(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense,
                               int col_major, void *packed, int packed_dtype, int64_t ld_packed, void *meta,
                               int mode, const void *mask, int64_t ld_mask, const float *uniforms,
                               int64_t ld_uniforms, uint64_t seed, uint64_t offset, const uint64_t *offset_dev,
                               void *e_tc, float *row_sums, void *stream, int packed_rm = 0, float out_scale = 1.f,
                               int soft_use_scale = 0, float soft_scale = 1.f, const float *amax = nullptr, void *q_dense = nullptr,
                               int64_t ld_q = 0, bool sums_in_parts = false, void *zero = nullptr, int64_t zero_bytes = 0) {
    using namespace sp24;
    if (!dense || !packed || !meta) return SP24_ERR_ARG;
    const int so = dtype_size(packed_dtype), si = dtype_size(dense_dtype);
    if (so == 0 || si == 0 || packed_dtype == SP24_F32) return SP24_ERR_DTYPE;
    if (dense_dtype == SP24_E4M3 || dense_dtype == SP24_E5M2) return SP24_ERR_DTYPE;
    if ((dense_dtype == SP24_I8) != (packed_dtype == SP24_I8)) return SP24_ERR_DTYPE;
    const int64_t kmult = so == 2 ? 64 : 128;
    if (m <= 0 || k <= 0 || m % 32 || k % kmult) return SP24_ERR_SHAPE;
    if (mode == SP24_PRUNE_MASK && !mask) return SP24_ERR_ARG;
    if (mode != SP24_PRUNE_MASK && mask) return SP24_ERR_ARG;
    if (mode != SP24_PRUNE_MVUE && uniforms) return SP24_ERR_ARG;
    if (mode < SP24_PRUNE_MSE || mode > PRUNE_SOFT) return SP24_ERR_ARG;
    if (packed_rm && (!col_major || so != 1)) return SP24_ERR_ARG;
    if (!(out_scale > 0.f) || (out_scale != 1.f && (so != 1 || packed_dtype == SP24_I8))) return SP24_ERR_ARG;
    const int64_t inner = col_major ? m : k, inner_p = (col_major && !packed_rm) ? m : k / 2;
    if (ld_dense < inner || (ld_dense * si) % 16) return SP24_ERR_STRIDE;
    if (ld_packed < inner_p || (ld_packed * so) % 16) return SP24_ERR_STRIDE;
    if (mask && (ld_mask < inner || ld_mask % 16)) return SP24_ERR_STRIDE;
    if (uniforms && (ld_uniforms < inner || ld_uniforms % 4)) return SP24_ERR_STRIDE;
    if (!aligned16(dense) || !aligned16(packed) || !aligned16(meta) || (mask && !aligned16(mask)) ||
        (uniforms && !aligned16(uniforms)))
        return SP24_ERR_ALIGN;
    if (e_tc && (packed_dtype == SP24_I8 || m % 128 || !aligned16(e_tc))) return SP24_ERR_ARG;
    if (q_dense && (!amax || !packed_rm || ld_q < m || ld_q % 16 || !aligned16(q_dense))) return SP24_ERR_ARG;
    if (zero && (mode != SP24_PRUNE_MVUE_FAST || !col_major || zero_bytes <= 0 || zero_bytes % 16 || !aligned16(zero))) return SP24_ERR_ARG;
    if (row_sums && (!col_major || (reinterpret_cast<uintptr_t>(row_sums) & 3u))) return SP24_ERR_ARG;
    if (int rc = check_device()) return rc;
    PcParams P{dense, packed, meta, static_cast<const uint8_t *>(mask), uniforms, m, k, ld_dense, ld_packed, ld_mask,
               ld_uniforms, seed, offset, reinterpret_cast<const unsigned long long *>(offset_dev),
               static_cast<int16_t *>(e_tc), (k + 127) / 128, row_sums, sums_in_parts ? m : 0, packed_rm, out_scale, soft_scale, soft_use_scale, amax, q_dense, ld_q,
               static_cast<uint4 *>(zero), zero_bytes / 16};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (dense_dtype) {
        case SP24_F32: return dispatch_out<float>(P, packed_dtype, mode, col_major, st);
        case SP24_F16: return dispatch_out<__half>(P, packed_dtype, mode, col_major, st);
        case SP24_BF16: return dispatch_out<__nv_bfloat16>(P, packed_dtype, mode, col_major, st);
        case SP24_I8: return dispatch_mode<int8_t, int8_t>(P, mode, col_major, st);
        default: return SP24_ERR_DTYPE;
    }
}

extern "C" int sp24_prune_compress(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense,
                                   int col_major, void *packed, int packed_dtype, int64_t ld_packed, void *meta,
                                   int mode, const void *mask, int64_t ld_mask, const float *uniforms,
                                   int64_t ld_uniforms, uint64_t seed, uint64_t offset, void *stream) {
    if (mode > SP24_PRUNE_MVUE_FAST) return SP24_ERR_ARG;
    return prune_compress_impl(dense, dense_dtype, m, k, ld_dense, col_major, packed, packed_dtype, ld_packed, meta, mode,
                               mask, ld_mask, uniforms, ld_uniforms, seed, offset, nullptr, nullptr, nullptr, stream);
}

// Same conversion with three optional extras (each may be NULL).
// offset_dev: the Philox offset becomes `offset` plus the 64-bit word at `offset_dev` (device memory), read when the
//   kernel runs.  A launch recorded once (a CUDA graph) then draws fresh uniforms on every replay if the caller
//   bumps that word between replays.
// e_tc: a second copy of the metadata in the order the sparse GEMM reads (sp24_meta_tc_bytes(m, k) bytes), so that
//   no conversion launch is needed before sp24_spmm.  16-bit outputs only, m % 128 == 0.
// row_sums: m floats; row_sums[r] += sum over k of dense[r, k] (the values before pruning, fp32 partial sums added
//   with atomics: the caller zeroes the array or passes a gradient buffer).  Column-major storage only: for dY^T this
//   is the bias gradient, taken from the pass that reads dY anyway.
extern "C" int sp24_prune_compress_ex(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense,
                                      int col_major, void *packed, int packed_dtype, int64_t ld_packed, void *meta,
                                      int mode, const void *mask, int64_t ld_mask, const float *uniforms,
                                      int64_t ld_uniforms, uint64_t seed, uint64_t offset, const uint64_t *offset_dev,
                                      void *e_tc, float *row_sums, void *stream) {
    if (offset_dev && (reinterpret_cast<uintptr_t>(offset_dev) & 7u)) return SP24_ERR_ARG;
    if (mode > SP24_PRUNE_MVUE_FAST) return SP24_ERR_ARG;
    return prune_compress_impl(dense, dense_dtype, m, k, ld_dense, col_major, packed, packed_dtype, ld_packed, meta, mode,
                               mask, ld_mask, uniforms, ld_uniforms, seed, offset, offset_dev, e_tc, row_sums, stream);
}

// Float8 quantising form of the conversion: packed is ALWAYS row-major (m, k/2), the K-major operand order the 8-bit
// sparse GEMM requires, whatever the storage order of dense (col_major = 1: a transposed view such as W.T of a
// row-major weight or dY.T of a row-major gradient, converted without a transpose pass).  Stored values are
// value * out_scale rounded to the float8 type (the caller's per-tensor quantisation scale; 1 for none).  mask follows
// the storage order of dense.  Metadata: m*k/32 int32 in the reference's reordered layout, as for any 8-bit output.
extern "C" int sp24_prune_compress_q8(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense, int col_major,
                                      void *packed, int packed_dtype, int64_t ld_packed, void *meta, int mode,
                                      const void *mask, int64_t ld_mask, float out_scale, uint64_t seed, uint64_t offset,
                                      void *stream) {
    if (packed_dtype != SP24_E4M3 && packed_dtype != SP24_E5M2) return SP24_ERR_DTYPE;
    if (mode > SP24_PRUNE_MVUE_FAST) return SP24_ERR_ARG;
    return prune_compress_impl(dense, dense_dtype, m, k, ld_dense, col_major, packed, packed_dtype, ld_packed, meta, mode, mask,
                               ld_mask, nullptr, 0, seed, offset, nullptr, nullptr, nullptr, stream, col_major ? 1 : 0,
                               out_scale);
}

// The same conversion for a layer that never reads its scales back: the stored values' scale comes from the tensor's
// absolute maximum on the device (sp24_absmax), and the pass that reads dense anyway also leaves the metadata in
// tensor-core order (e_tc), the float32 row sums of the unpruned values (row_sums, column-major input, added to) and the
// whole tensor quantised in its own storage order (q_dense, column-major input).  Each of the three may be NULL.
extern "C" int sp24_prune_compress_q8_dev(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense, int col_major,
                                          void *packed, int packed_dtype, int64_t ld_packed, void *meta, int mode,
                                          const void *mask, int64_t ld_mask, const float *amax, uint64_t seed, uint64_t offset,
                                          void *e_tc, float *row_sums, void *q_dense, int64_t ld_q, void *stream) {
    if (packed_dtype != SP24_E4M3 && packed_dtype != SP24_E5M2) return SP24_ERR_DTYPE;
    if (mode > SP24_PRUNE_MVUE_FAST || !amax) return SP24_ERR_ARG;
    return prune_compress_impl(dense, dense_dtype, m, k, ld_dense, col_major, packed, packed_dtype, ld_packed, meta, mode, mask,
                               ld_mask, nullptr, 0, seed, offset, nullptr, e_tc, row_sums, stream, col_major ? 1 : 0, 1.f, 0, 1.f, amax,
                               q_dense, ld_q);
}

// One part for every 128 storage rows of a column-major matrix.
extern "C" int sp24_row_parts(int64_t k, int packed_dtype) {
    const int so = sp24::dtype_size(packed_dtype);
    return so != 1 && so != 2 ? 0 : (int)((k + 127) / 128);
}

static int prune_compress_with(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense, int col_major, void *packed,
                               int packed_dtype, int64_t ld_packed, void *meta, int mode, const void *mask, int64_t ld_mask,
                               const float *uniforms, int64_t ld_uniforms, uint64_t seed, uint64_t offset, const sp24_prune_extras *x,
                               void *zero, int64_t zero_bytes, void *stream) {
    if (!x || mode > SP24_PRUNE_MVUE_FAST) return SP24_ERR_ARG;
    if (x->offset_dev && (reinterpret_cast<uintptr_t>(x->offset_dev) & 7u)) return SP24_ERR_ARG;
    if (x->amax && packed_dtype != SP24_E4M3 && packed_dtype != SP24_E5M2) return SP24_ERR_DTYPE;
    if (x->amax && x->out_scale != 0.f) return SP24_ERR_ARG;
    return prune_compress_impl(dense, dense_dtype, m, k, ld_dense, col_major, packed, packed_dtype, ld_packed, meta, mode, mask, ld_mask,
                               uniforms, ld_uniforms, seed, offset, x->offset_dev, x->e_tc, x->row_parts, stream, x->packed_row_major && col_major ? 1 : 0,
                               x->out_scale != 0.f ? x->out_scale : 1.f, 0, 1.f, x->amax, x->q_dense, x->ld_q, true, zero, zero_bytes);
}

extern "C" int sp24_prune_compress_with(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense, int col_major,
                                        void *packed, int packed_dtype, int64_t ld_packed, void *meta, int mode, const void *mask,
                                        int64_t ld_mask, const float *uniforms, int64_t ld_uniforms, uint64_t seed, uint64_t offset,
                                        const sp24_prune_extras *x, void *stream) {
    return prune_compress_with(dense, dense_dtype, m, k, ld_dense, col_major, packed, packed_dtype, ld_packed, meta, mode, mask, ld_mask,
                               uniforms, ld_uniforms, seed, offset, x, nullptr, 0, stream);
}

extern "C" int sp24_mvue_compress_clearing(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense, void *packed,
                                           int packed_dtype, int64_t ld_packed, void *meta, uint64_t seed, uint64_t offset,
                                           const sp24_prune_extras *x, void *zero, int64_t zero_bytes, void *stream) {
    if (!zero) return SP24_ERR_ARG;
    return prune_compress_with(dense, dense_dtype, m, k, ld_dense, 1, packed, packed_dtype, ld_packed, meta, SP24_PRUNE_MVUE_FAST, nullptr, 0,
                               nullptr, 0, seed, offset, x, zero, zero_bytes, stream);
}

// Both compressed copies of a float8 layer's weight (W and W^T, e4m3, K-major) under one mask: see the header.
extern "C" int sp24_dual_compress_f8(const void *w, int dtype, int64_t m, int64_t k, int64_t ld_w, const void *mask, int64_t ld_mask, const float *amax,
                                     void *packed_w, void *meta_w, void *tc_w, void *packed_t, void *meta_t, void *tc_t, void *stream) {
    using namespace sp24;
    if (!w || !mask || !amax || !packed_w || !meta_w || !tc_w || !packed_t || !meta_t || !tc_t) return SP24_ERR_ARG;
    if (dtype != SP24_F32 && dtype != SP24_F16 && dtype != SP24_BF16) return SP24_ERR_DTYPE;
    if (m <= 0 || k <= 0 || m % 128 || k % 128 || m / 64 > 65535) return SP24_ERR_SHAPE;
    if (ld_w < k || (ld_w * dtype_size(dtype)) % 16 || ld_mask < k || ld_mask % 4) return SP24_ERR_STRIDE;
    if (!aligned16(w) || (reinterpret_cast<uintptr_t>(mask) & 3u) || !aligned16(packed_w) || !aligned16(meta_w) || !aligned16(tc_w) ||
        !aligned16(packed_t) || !aligned16(meta_t) || !aligned16(tc_t))
        return SP24_ERR_ALIGN;
    if (int rc = check_device()) return rc;
    const DualF8Params P{w, static_cast<const uint8_t *>(mask), amax, static_cast<uint8_t *>(packed_w), static_cast<uint8_t *>(packed_t),
                         static_cast<int32_t *>(meta_w), static_cast<int32_t *>(tc_w), static_cast<uint16_t *>(meta_t),
                         static_cast<uint16_t *>(tc_t), m, k, ld_w, ld_mask};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const dim3 grid((unsigned)(k / 128), (unsigned)(m / 64));
    if (dtype == SP24_F32) launch_chained(st, dual_f8_kernel<float>, grid, 128, 0, P);
    else if (dtype == SP24_F16) launch_chained(st, dual_f8_kernel<__half>, grid, 128, 0, P);
    else launch_chained(st, dual_f8_kernel<__nv_bfloat16>, grid, 128, 0, P);
    return launch_status();
}

// S-STE forward in one pass: magnitude 2:4 mask, soft threshold of the kept values (one rounding in the input type),
// optional frozen scale (one more rounding in the input type), cast to the packed 16-bit type, metadata - what
// sp24_soft_threshold24 followed by a cast and sp24_prune_compress (mask mode) produce in three passes over W.
// e_tc (optional): the metadata also in the order sp24_spmm reads (m % 128 == 0).
extern "C" int sp24_soft_threshold24_compress(const void *dense, int dense_dtype, int64_t m, int64_t k, int64_t ld_dense,
                                              int col_major, void *packed, int packed_dtype, int64_t ld_packed, void *meta,
                                              int use_scale, float scale, void *e_tc, void *stream) {
    if (packed_dtype != SP24_F16 && packed_dtype != SP24_BF16) return SP24_ERR_DTYPE;
    return prune_compress_impl(dense, dense_dtype, m, k, ld_dense, col_major, packed, packed_dtype, ld_packed, meta,
                               sp24::PRUNE_SOFT, nullptr, 0, nullptr, 0, 0, 0, nullptr, e_tc, nullptr, stream, 0, 1.f,
                               use_scale ? 1 : 0, scale);
}
