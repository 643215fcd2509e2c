// 2:4 sparse GEMM for sm_100a:  D (Ms x N) = A_sparse (Ms x K) * B (K x N)  [+ bias per row] [activation]
//
// The sparse operand is always the tensor-core "A" operand of tcgen05.mma.sp: compressed values are
// staged in shared memory by TMA (128-byte swizzle), its metadata goes shared memory -> tensor memory
// with tcgen05.cp, the dense operand B is staged by TMA, accumulators live in tensor memory and are read
// back with tcgen05.ld by eight epilogue warps.
//
// Warp roles in a CTA of 320 threads: warp 0 = TMA producer (one elected lane), warp 1 = tensor-memory
// allocation + MMA issue (one elected lane), warps 2..9 = epilogue (two per TMEM lane quadrant, half of the
// columns each).
// One CTA computes one 128 x BN output tile; the K loop runs over stages of 128 bytes of compressed A
// per row (logical K 128 for 16-bit types, 256 for 8-bit types) through a STAGES-deep mbarrier ring.
//
// Every wait on an mbarrier is bounded: when a wait gives up, the CTA records a code in *status,
// raises a shared abort flag that cuts all other waits short, drains its own copies in flight (again
// bounded), frees its tensor memory and returns.  Nothing traps.
#include <cuda.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "meta_steps.cuh"
#include "sp24_common.cuh"

namespace sp24 {
namespace {

constexpr int BM = 128;            // rows of the sparse operand per CTA tile (= TMEM lanes)
constexpr int A_STAGE_BYTES = BM * 128;
constexpr uint32_t WAIT_LIMIT = 1u << 22;  // polls of mbarrier.try_wait before a wait gives up

// ------------------------------------------------------------------------------------------------
// PTX wrappers
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when it gave up (limit reached or another role raised the abort flag).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, int code,
                                          uint32_t limit = WAIT_LIMIT) {
    for (uint32_t it = 0; it < limit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 0xFFu) == 0xFFu && *abort_flag) return false;
    }
    *abort_flag = 1;
    if (status) atomicCAS(status, 0, code);
    return false;
}
// The same for a whole warp that goes on to elect a lane: one outcome for all lanes.  Each lane polls for itself, so when a
// wait is given up some lanes may have seen the barrier flip and others not; an elect.sync that names every lane needs them all.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, int code,
                                               uint32_t limit = WAIT_LIMIT) {
    return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, abort_flag, status, code, limit));
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// true in one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_cp_128x128b(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::1.128x128b [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
template <bool F8>
__device__ __forceinline__ void mma_sp(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t e_tmem, uint32_t idesc,
                                       uint32_t accumulate, int int8 = 0) {
    if constexpr (F8) {
        if (int8) {   // signed 8-bit integers, 32-bit integer accumulators; same operand geometry as fp8
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
                "tcgen05.mma.sp.cta_group::1.kind::i8 [%0], %1, %2, [%3], %4, p;\n\t}" ::"r"(d_tmem),
                "l"(adesc), "l"(bdesc), "r"(e_tmem), "r"(idesc), "r"(accumulate)
                : "memory");
        } else {
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
                "tcgen05.mma.sp.cta_group::1.kind::f8f6f4 [%0], %1, %2, [%3], %4, p;\n\t}" ::"r"(d_tmem),
                "l"(adesc), "l"(bdesc), "r"(e_tmem), "r"(idesc), "r"(accumulate)
                : "memory");
        }
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.sp.cta_group::1.kind::f16 [%0], %1, %2, [%3], %4, p;\n\t}" ::"r"(d_tmem),
            "l"(adesc), "l"(bdesc), "r"(e_tmem), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
// shared memory -> global through a tensor map, one element-wise float32 add per element in L2; parts of the box past the tensor are left out
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap *map, int x, int y, uint32_t src) {
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y), "r"(src)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all but the newest N groups of this thread have read their shared memory
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// 16 lanes (the lower or upper half of the warp's quadrant) x 16 columns: register 4 c + 2 h + e of lane L holds row 8 h + L / 4,
// column 8 c + 2 (L % 4) + e
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
// four 8 x 8 matrices of 16-bit values, each written transposed; lane 8 i + j gives the address of row j of matrix i as stored
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared::cta.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
                 : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
// fp32 vector reduction into global memory (sm_90+), address 16-byte aligned
__device__ __forceinline__ void red_add_v4(float *addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte offsets (all >> 4),
// descriptor version 1, swizzle mode in bits 61..63 (0 none, 2 = 128-byte).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t swizzle) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)swizzle << 61;
    return d;
}

struct SpmmParams {
    const void *e_tc;       // metadata in tensor-core atom order
    void *out;
    const void *bias;       // per sparse row (output feature), in the output type, or null
    int64_t ms, n, k;       // sparse rows, dense columns, logical K
    int64_t ld_out;
    int64_t k_atoms;        // number of 128-column metadata atoms per 128-row block (K padded up)
    int *status;
    uint32_t idesc;         // instruction descriptor without the metadata selector bits
    int activation;         // 0 none, 1 relu, 2 silu, 3 gelu (tanh form)
    unsigned long long *trace;  // timing trace of CTA 0: only developer builds (-DSP24_TRACE_BUILD) ever set it
    int int8;               // 8-bit operands are signed integers (kind::i8, int32 accumulators and output)
    int k_splits;           // work units per tile along K (> 1 only for the accumulating fp32 output)
    int mblk_per_tile;      // 128-row blocks per tile: 2 (B staged once per 256 rows) or 1 (more, smaller tiles)
    float alpha;            // float32 outputs: D = alpha * (A * B) (+ bias); 16-bit and integer outputs ignore it
    int bias_f32;           // bias holds float32 values instead of values of the output type
    const float *amax_a, *amax_b;   // float8: absolute maxima of the operands on the device; alpha is the product of their scales
    int bn, stages;         // CTA-pair kernel: tile columns and operand stages
    int accumulate;         // float8, float32 output (ms, n): add alpha * A * B instead of storing it
    int whole_columns;      // CTA-pair weight gradient: map_b is one of make_map_columns
    void *aux;              // fused MLP epilogues (CTA-pair kernel): second tensor shaped and pitched like out
    int64_t ld_aux;
};
// Row sums that the weight-gradient form alone takes along: out[r] (+)= sum over p of parts[p * ms + r]
struct SumsParams {
    const float *parts;
    float *out;
    int64_t n_parts;
    int accumulate;
};

// Epilogue forms of the CTA-pair kernel.  PRE_GELU: aux = h = acc + bias rounded to the output type, out = gelu(h)
// (tanh form, evaluated on the rounded h, so that out is exactly the activation of what aux holds).  DGELU: out =
// acc * gelu'(aux): the input gradient of a layer whose input was gelu(aux), written as the gradient of aux.
enum { EPI_PLAIN = 0, EPI_PRE_GELU = 1, EPI_DGELU = 2 };

__device__ __forceinline__ float tanh_fast(float v) {
    float r;
    asm("tanh.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// GELU, tanh form: 0.5 v (1 + tanh(u)), u = sqrt(2 / pi) (v + 0.044715 v^3); one MUFU per value
__device__ __forceinline__ float gelu_tanh(float v) {
    const float t = tanh_fast(0.7978845608f * fmaf(0.044715f * v * v, v, v));
    return 0.5f * v * (1.f + t);
}
// its derivative: 0.5 (1 + t) + 0.5 v (1 - t^2) sqrt(2 / pi) (1 + 3 * 0.044715 v^2)
__device__ __forceinline__ float gelu_tanh_grad(float v) {
    const float v2 = v * v;
    const float t = tanh_fast(0.7978845608f * fmaf(0.044715f * v2, v, v));
    return 0.5f * (1.f + t) + 0.5f * v * (1.f - t * t) * (0.7978845608f * fmaf(0.134145f, v2, 1.f));
}

template <typename OutT> __device__ __forceinline__ OutT to_out(float v);
template <> __device__ __forceinline__ __half to_out<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 to_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ float to_out<float>(float v) { return v; }
template <> __device__ __forceinline__ int32_t to_out<int32_t>(float v) { return __float_as_int(v); }
template <typename OutT> __device__ __forceinline__ float from_out(OutT v);
template <> __device__ __forceinline__ float from_out<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float from_out<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float from_out<float>(float v) { return v; }
template <> __device__ __forceinline__ float from_out<int32_t>(int32_t) { return 0.f; }   // no bias for integer GEMMs

__device__ __forceinline__ float apply_act(float v, int act) {
    if (act == 1) return v > 0.f ? v : 0.f;
    if (act == 2) return v / (1.f + __expf(-v));
    if (act == 3) {  // GELU, tanh form: v * sigmoid(2 * sqrt(2 / pi) * (v + 0.044715 v^3))
        const float u = 1.5957691216f * (v + 0.044715f * v * v * v);
        return v / (1.f + __expf(-u));
    }
    return v;
}

// The activation is compiled in only for launches that ask for one (template parameter ACT): the plain
// epilogue carries no per-element tests.
template <bool ACT> __device__ __forceinline__ float finish(float v, int act) {
    if constexpr (ACT) return apply_act(v, act);
    return v;
}

// One accumulator word -> one output value.  Integer accumulators pass through untouched: no float operation may
// see their bits (an add of 0.0f would rewrite -0.0 and signalling-NaN patterns, which are ordinary integers).
// float32 outputs are scaled first: alpha * acc + bias in one fused multiply-add (alpha = 1 gives acc + bias exactly).
template <typename OutT, bool ACT, bool SCALED = false> __device__ __forceinline__ OutT emit(uint32_t acc_bits, float bias, int act, float alpha) {
    if constexpr (std::is_same<OutT, int32_t>::value) return (int32_t)acc_bits;
    else if constexpr (SCALED) return to_out<OutT>(finish<ACT>(fmaf(__uint_as_float(acc_bits), alpha, bias), act));
    else if constexpr (std::is_same<OutT, float>::value) return finish<ACT>(fmaf(__uint_as_float(acc_bits), alpha, bias), act);
    else return to_out<OutT>(finish<ACT>(__uint_as_float(acc_bits) + bias, act));
}
// the same, as the 32-bit container of a 4-byte output type
template <typename OutT, bool ACT> __device__ __forceinline__ uint32_t emit_bits(uint32_t acc_bits, float bias, int act, float alpha) {
    if constexpr (std::is_same<OutT, int32_t>::value) return acc_bits;
    else return __float_as_uint(finish<ACT>(fmaf(__uint_as_float(acc_bits), alpha, bias), act));
}

template <typename OutT> __device__ __forceinline__ float load_bias(const SpmmParams &P, int64_t row) {
    return P.bias_f32 ? static_cast<const float *>(P.bias)[row] : from_out<OutT>(static_cast<const OutT *>(P.bias)[row]);
}
// single-CTA kernels: float8 products take a float32 bias, the others one in the output type
template <typename OutT, bool F8> __device__ __forceinline__ float row_bias(const SpmmParams &P, int64_t row) {
    if constexpr (F8) return static_cast<const float *>(P.bias)[row];
    else return from_out<OutT>(static_cast<const OutT *>(P.bias)[row]);
}
// alpha of a float8 product: given, or from the operands' absolute maxima
__device__ __forceinline__ float alpha_of(const SpmmParams &P) {
    return P.amax_a ? (float)(f8_scale(*P.amax_a) * f8_scale(*P.amax_b)) : P.alpha;
}

__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// trace layout: 3 roles x 256 slots of nanosecond timestamps, CTA 0 only.  Compiled out of the shipped library:
// a developer build (-DSP24_TRACE_BUILD) stores through P.trace, which that build takes from the environment.
#ifdef SP24_TRACE_BUILD
#define SP24_TRACE(role, slot) do { if (P.trace && blockIdx.x == 0 && (slot) < 256) P.trace[(role) * 256 + (slot)] = globaltimer(); } while (0)
#else
#define SP24_TRACE(role, slot) do { } while (0)
#endif

__device__ __forceinline__ void epilogue_bar_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// Geometry shared by the kernel and its launcher.
template <int BN, bool F8, bool TRANS_OUT, typename OutT> struct SpmmCfg {
    static constexpr int E_BYTES = F8 ? 4096 : 2048;          // metadata of one 128-row block and one stage
    static constexpr int B_BYTES = BN * 256;                  // two 128-byte K atoms per row of B
    static constexpr int STAGE_BYTES = 2 * A_STAGE_BYTES + B_BYTES + 2 * E_BYTES;
    // transposed output: each accumulator is first copied row by row (16-byte stores) into a staging
    // buffer of 128 rows x STG_COLS columns (+16 bytes of padding per row against bank conflicts), then
    // written out column by column
    static constexpr int STG_COLS = sizeof(OutT) == 4 ? 64 : BN;
    static constexpr int STG_ROW_BYTES = STG_COLS * (int)sizeof(OutT) + 16;
    // 16-bit outputs of wide tiles go through the staging buffer in both output orders (the second accumulator
    // waits in registers, so the tensor memory is free again early); narrow tiles keep a third operand stage
    static constexpr bool STAGED16 = sizeof(OutT) == 2 && (TRANS_OUT || BN > 128);
    static constexpr int STG_BYTES = (TRANS_OUT || STAGED16) ? BM * STG_ROW_BYTES : 0;
    static constexpr int AVAIL = 227 * 1024 - 2048 - STG_BYTES;
    static constexpr int STAGES = AVAIL / STAGE_BYTES >= 4 ? 4 : AVAIL / STAGE_BYTES;
    static constexpr int SMEM = STAGES * STAGE_BYTES + STG_BYTES + 1024;
    static_assert(STAGES >= 2, "tile too large for a two-stage ring");
    static_assert(STAGE_BYTES % 1024 == 0, "stages must keep the 1024-byte swizzle alignment");
};

// Persistent kernel: CTA c processes tiles c, c + gridDim.x, ... ; a tile is (256 sparse rows) x (BN dense
// columns), computed as two 128-row blocks that share every stage of B.  The operand ring keeps filling
// across tile boundaries; the epilogue drains tensor memory into a staging buffer and releases each
// accumulator as soon as it has been read, so the next tile's MMAs overlap the global stores.
template <int BN, bool F8, bool A_MN, bool B_MN, bool TRANS_OUT, typename OutT, bool ACT>
__global__ void __launch_bounds__(320, 1)
spmm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, SpmmParams P) {
    using Cfg = SpmmCfg<BN, F8, TRANS_OUT, OutT>;
    constexpr int STAGES = Cfg::STAGES;
    constexpr int STAGE_BYTES = Cfg::STAGE_BYTES;
    constexpr int E_BYTES = Cfg::E_BYTES;
    constexpr int OFF_B = 2 * A_STAGE_BYTES, OFF_E = OFF_B + Cfg::B_BYTES;
    constexpr int KSTEPS = 4;                 // MMA instructions per stage and row block (32 bytes of compressed A each)
    constexpr uint32_t TMEM_COLS = 512;
    constexpr int E_COL0 = 2 * BN;            // metadata columns behind the two accumulators
    constexpr int E_SLOT = F8 ? 8 : 4;        // metadata columns of one row block and one stage
    // 16-bit operands with a direct fp32 output: the accumulating form (D += A * B), the only one that splits K
    constexpr bool ACCUM = !F8 && !TRANS_OUT && sizeof(OutT) == 4;
    static_assert(E_COL0 + 4 * E_SLOT <= 512, "tensor memory columns exhausted");
    static_assert(BN % 32 == 0 && BN >= 32 && BN <= 256, "invalid tile width");

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t bars[2 * STAGES + 3];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles_n = (int)((P.n + BN - 1) / BN);
    const int n_mblocks = (int)(P.ms / BM);
    const int mpt = P.mblk_per_tile;
    // tile index -> (row tile, column tile) with the row tile varying fastest: the CTAs running at one time
    // cover whole rows of the transposed output (long contiguous runs in DRAM) and share their B tiles in L2
    const int n_tiles_m = (n_mblocks + mpt - 1) / mpt;
    const int n_tiles = n_tiles_n * n_tiles_m;
    // work unit u = (tile u % n_tiles, K slice u / n_tiles); one slice unless the output accumulates
    const int n_units = n_tiles * P.k_splits;
    const int logical_k_per_stage = F8 ? 256 : 128;
    const int k_iters = (int)((P.k + logical_k_per_stage - 1) / logical_k_per_stage);

    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[STAGES]);
    const uint32_t tmem_full = smem_u32(&bars[2 * STAGES]), tmem_empty0 = smem_u32(&bars[2 * STAGES + 1]);

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(tmem_full, 1);
        mbar_init(tmem_empty0, 8);      // one arrival per epilogue warp
        mbar_init(tmem_empty0 + 8, 8);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_base_smem), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;
    chain_enter();

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            int g = 0;  // stages issued so far (ring position across tiles)
            bool ok = true;
            for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
                const int tile = unit % n_tiles, ks = unit / n_tiles;
                const int it0 = (int)((int64_t)ks * k_iters / P.k_splits), it1 = (int)((int64_t)(ks + 1) * k_iters / P.k_splits);
                const int mblk0 = (tile % n_tiles_m) * mpt;
                const int n_mblk = (n_mblocks - mblk0) >= mpt ? mpt : 1;
                const int64_t m0 = (int64_t)mblk0 * BM, n0 = (int64_t)(tile / n_tiles_m) * BN;
                const uint32_t stage_tx = (uint32_t)(n_mblk * (A_STAGE_BYTES + E_BYTES) + Cfg::B_BYTES);
                for (int it = it0; it < it1; ++it, ++g) {
                    const int s = g % STAGES;
                    const uint32_t ph = (g / STAGES) & 1;
                    if (g >= STAGES && !mbar_wait(empty0 + 8 * s, ph ^ 1, &abort_flag, P.status, 1)) { ok = false; break; }
                    const uint32_t sa = smem_u32(smem + (size_t)s * STAGE_BYTES);
                    const uint32_t sb = sa + OFF_B;
                    const uint32_t se = sa + OFF_E;
                    const uint32_t full = full0 + 8 * s;
                    mbar_expect_tx(full, stage_tx);
                    for (int mb = 0; mb < n_mblk; ++mb) {
                        const int mrow = (int)m0 + mb * BM;
                        const uint32_t sam = sa + mb * A_STAGE_BYTES;
                        // compressed A: 128 rows x 128 bytes
                        if constexpr (!A_MN) {
                            tma_load_2d(sam, &map_a, it * (F8 ? 128 : 64), mrow, full);
                        } else {
                            tma_load_2d(sam, &map_a, mrow, it * 64, full);
                            tma_load_2d(sam + 8192, &map_a, mrow + 64, it * 64, full);
                        }
                        // metadata atoms of this 128-row block
                        const uint8_t *e_blk = static_cast<const uint8_t *>(P.e_tc) + (size_t)(mblk0 + mb) * P.k_atoms * 2048;
                        if constexpr (F8) {
                            const MetaAtoms at = meta_atoms_of_step(it, P.k_atoms);
                            bulk_load(se + mb * E_BYTES, e_blk + at.first * 2048, 2048, full);
                            bulk_load(se + mb * E_BYTES + 2048, e_blk + at.second * 2048, 2048, full);
                        } else {
                            bulk_load(se + mb * E_BYTES, e_blk + (size_t)it * 2048, 2048, full);
                        }
                    }
                    // dense B: BN rows x 2 atoms of 128 bytes (K-major) or column blocks of 64 x 128 K-rows (MN-major)
                    if constexpr (!B_MN) {
                        const int kx = it * (F8 ? 256 : 128);
                        tma_load_2d(sb, &map_b, kx, (int)n0, full);
                        tma_load_2d(sb + BN * 128, &map_b, kx + (F8 ? 128 : 64), (int)n0, full);
                    } else {
#pragma unroll
                        for (int j = 0; j < BN / 64; ++j)
                            tma_load_2d(sb + j * 16384, &map_b, (int)n0 + j * 64, it * 128, full);
                    }
                    SP24_TRACE(0, g);
                }
            }
            if (abort_flag) {
                // drain: wait (bounded) for the copies already issued so that none lands after exit
                for (int q = (g > STAGES ? g - STAGES : 0); q < g; ++q) {
                    const int s = q % STAGES;
                    const uint32_t ph = (q / STAGES) & 1;
                    for (uint32_t w = 0; w < WAIT_LIMIT; ++w)
                        if (mbar_try_wait(full0 + 8 * s, ph)) break;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (lane == 0) {
            // K-major, 128-byte swizzle: 8-row groups 1024 bytes apart, 32 (A) / 64 (B) bytes per MMA inside
            // the atom.  MN-major: 64-element column blocks one TMA box apart, 8 K-rows per 1024 bytes.
            constexpr uint32_t A_LBO = A_MN ? 8192 : 16, A_KSTEP = A_MN ? 2048 : 32;
            constexpr uint32_t B_LBO = B_MN ? 16384 : 16, B_KSTEP = B_MN ? 4096 : 64;
            int g = 0, tl = 0;
            bool ok = true;
            for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x, ++tl) {
                const int tile = unit % n_tiles, ks = unit / n_tiles;
                const int it0 = (int)((int64_t)ks * k_iters / P.k_splits), it1 = (int)((int64_t)(ks + 1) * k_iters / P.k_splits);
                const int mblk0 = (tile % n_tiles_m) * mpt;
                const int n_mblk = (n_mblocks - mblk0) >= mpt ? mpt : 1;
                for (int it = it0; it < it1 && ok; ++it, ++g) {
                    const int s = g % STAGES;
                    const uint32_t ph = (g / STAGES) & 1;
                    ok = mbar_wait(full0 + 8 * s, ph, &abort_flag, P.status, 2);
                    if (!ok) break;
                    SP24_TRACE(1, 2 * g);
                    const uint32_t sa = smem_u32(smem + (size_t)s * STAGE_BYTES);
                    const uint32_t sb = sa + OFF_B;
                    const uint32_t se = sa + OFF_E;
                    for (int mb = 0; mb < n_mblk && ok; ++mb) {
                        if (it == it0) {
                            // the epilogue of this CTA's previous tile must have drained this accumulator
                            ok = mbar_wait(tmem_empty0 + 8 * mb, (tl & 1) ^ 1, &abort_flag, P.status, 4);
                            if (!ok) break;
                        }
                        tc_fence_after();
                        const uint32_t e_cols = E_COL0 + ((g & 1) * 2 + mb) * E_SLOT;
                        // metadata: shared memory -> tensor memory, 128 lanes x 16 bytes per atom
                        tc_cp_128x128b(tmem_base + e_cols, make_desc(se + mb * E_BYTES, 16, 128, 0));
                        if constexpr (F8)
                            tc_cp_128x128b(tmem_base + e_cols + 4, make_desc(se + mb * E_BYTES + 2048, 16, 128, 0));
#pragma unroll
                        for (int j = 0; j < KSTEPS; ++j) {
                            const uint64_t adesc = make_desc(sa + mb * A_STAGE_BYTES + j * A_KSTEP, A_LBO, 1024, 2);
                            const uint32_t b_off = B_MN ? j * B_KSTEP : (uint32_t)(j >> 1) * (BN * 128) + (j & 1) * B_KSTEP;
                            const uint64_t bdesc = make_desc(sb + b_off, B_LBO, 1024, 2);
                            const uint32_t ecol = e_cols + (F8 ? 2 * j : j);
                            // 16-bit types: the instruction takes the even column of a pair plus a 1-bit selector
                            const uint32_t e_addr = tmem_base + (F8 ? ecol : (ecol & ~1u));
                            const uint32_t idesc = P.idesc | (F8 ? 0u : (ecol & 1u));
                            mma_sp<F8>(tmem_base + mb * BN, adesc, bdesc, e_addr, idesc, (it > it0 || j > 0) ? 1u : 0u, P.int8);
                        }
                    }
                    tc_commit(empty0 + 8 * s);  // frees the stage when these MMAs have read it
                    SP24_TRACE(1, 2 * g + 1);
                }
                tc_commit(tmem_full);           // accumulators of this tile complete (also arrives after an abort)
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue (warps 2..9)
        // Two warps per tensor-memory lane quadrant, each taking half of the tile's columns.  No early exit
        // here: the eight warps meet at named barrier 1, so after an abort they keep walking the tile list
        // (waits return at once) and simply skip the work.
        const int quad = warp & 3;          // TMEM lane quadrant this warp may read
        const int half = (warp - 2) >> 2;   // which half of the columns
        const int tid = (warp - 2) * 32 + lane;
        OutT *out = static_cast<OutT *>(P.out);
        const float alpha = F8 ? alpha_of(P) : P.alpha;
        OutT *stg = reinterpret_cast<OutT *>(smem + (size_t)STAGES * STAGE_BYTES);
        int tl = 0;
        for (int unit = blockIdx.x; unit < n_units; unit += gridDim.x, ++tl) {
            const int tile = unit % n_tiles;
            const int mblk0 = (tile % n_tiles_m) * mpt;
            const int n_mblk = (n_mblocks - mblk0) >= mpt ? mpt : 1;
            const int64_t m0 = (int64_t)mblk0 * BM, n0 = (int64_t)(tile / n_tiles_m) * BN;
            const bool ok = mbar_wait(tmem_full, tl & 1, &abort_flag, P.status, 3);
            tc_fence_after();
            if (threadIdx.x == 64) SP24_TRACE(2, 4 * tl);
            const bool run = ok && !abort_flag;
            const int row_in_blk = quad * 32 + lane;
            if constexpr (Cfg::STAGED16) {
                // 16-bit output through the staging buffer.  Row r of the staging buffer holds one feature's BN values; its
                // 16-byte pieces are permuted by (r / 8) % 4 so that the column-wise reads below (four groups
                // of eight rows per warp instruction) fall on 32 different banks.
                constexpr int HC = BN / 2;                  // columns per warp
                constexpr int NREG = HC / 2;
                uint8_t *stg_row = reinterpret_cast<uint8_t *>(stg) + (size_t)row_in_blk * Cfg::STG_ROW_BYTES;
                const int swz = 2 * ((row_in_blk >> 3) & 3);
                uint32_t held[NREG];                        // second accumulator, converted, two values per word
                float bias0 = 0.f, bias1 = 0.f;
                if (run && P.bias) {
                    bias0 = row_bias<OutT, F8>(P, m0 + row_in_blk);
                    if (n_mblk == 2) bias1 = row_bias<OutT, F8>(P, m0 + BM + row_in_blk);
                }
                const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16) + half * HC;
                if (run) {
#pragma unroll
                    for (int c = 0; c < HC / 32; ++c) {
                        uint32_t v[32];
                        tmem_ld32(acc + c * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            Vec<OutT, 8> o;
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                o.v[i] = emit<OutT, ACT, F8>(v[q * 8 + i], bias0, P.activation, alpha);
                            const int piece = (half * HC + c * 32) / 8 + q;
                            *reinterpret_cast<uint4 *>(stg_row + ((piece ^ swz) << 4)) = *reinterpret_cast<const uint4 *>(&o);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tmem_empty0);
                if (n_mblk == 2) {
                    if (run) {
#pragma unroll
                        for (int c = 0; c < HC / 32; ++c) {
                            uint32_t v[32];
                            tmem_ld32(acc + BN + c * 32, v);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                Vec<OutT, 2> o;
                                o.v[0] = emit<OutT, ACT, F8>(v[2 * i], bias1, P.activation, alpha);
                                o.v[1] = emit<OutT, ACT, F8>(v[2 * i + 1], bias1, P.activation, alpha);
                                held[c * 16 + i] = *reinterpret_cast<const uint32_t *>(&o);
                            }
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                }
                // both accumulators are in shared memory / registers now: the next tile's MMAs may start
                if (lane == 0) mbar_arrive(tmem_empty0 + 8);
                if (threadIdx.x == 64) SP24_TRACE(2, 4 * tl + 1);
                for (int mb = 0; mb < n_mblk; ++mb) {
                    if (mb == 1) {
                        if (run) {
#pragma unroll
                            for (int q = 0; q < NREG / 4; ++q) {
                                const int piece = (half * HC) / 8 + q;
                                *reinterpret_cast<uint4 *>(stg_row + ((piece ^ swz) << 4)) =
                                    make_uint4(held[4 * q], held[4 * q + 1], held[4 * q + 2], held[4 * q + 3]);
                            }
                        }
                    }
                    epilogue_bar_sync();
                    if (run) {
                        const int64_t mrow0 = m0 + mb * BM;
                        const uint8_t *stg_b = reinterpret_cast<const uint8_t *>(stg);
                        if constexpr (TRANS_OUT) {
                            // thread = two adjacent output rows (dense columns n, n+1) x 8 consecutive features;
                            // a warp instruction covers 8 row pairs x 4 feature groups: 64-byte runs per row
                            for (int i = tid; i < (BN / 2) * (BM / 8); i += 256) {
                                const int mg = (i & 3) + 4 * ((i >> 5) & 3), np = ((i >> 2) & 7) + 8 * (i >> 7);
                                const int word = np ^ ((i & 3) << 3);   // rows mg*8..mg*8+7 share (r / 8) % 4 = mg % 4
                                uint32_t w[8];
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    w[j] = *reinterpret_cast<const uint32_t *>(stg_b + (size_t)(mg * 8 + j) * Cfg::STG_ROW_BYTES + word * 4);
                                uint4 lo, hi;
                                lo.x = __byte_perm(w[0], w[1], 0x5410); hi.x = __byte_perm(w[0], w[1], 0x7632);
                                lo.y = __byte_perm(w[2], w[3], 0x5410); hi.y = __byte_perm(w[2], w[3], 0x7632);
                                lo.z = __byte_perm(w[4], w[5], 0x5410); hi.z = __byte_perm(w[4], w[5], 0x7632);
                                lo.w = __byte_perm(w[6], w[7], 0x5410); hi.w = __byte_perm(w[6], w[7], 0x7632);
                                const int64_t nrow = n0 + 2 * np;
                                OutT *dst = out + nrow * P.ld_out + mrow0 + mg * 8;
                                if (nrow < P.n) *reinterpret_cast<uint4 *>(dst) = lo;
                                if (nrow + 1 < P.n) *reinterpret_cast<uint4 *>(dst + P.ld_out) = hi;
                            }
                        } else {
                            // thread = 8 consecutive columns of one row; a warp writes 512 contiguous bytes
                            constexpr int PIECES = BN / 8;
                            for (int i = tid; i < PIECES * BM; i += 256) {
                                const int row = i / PIECES, piece = i % PIECES;
                                const uint4 v = *reinterpret_cast<const uint4 *>(
                                    stg_b + (size_t)row * Cfg::STG_ROW_BYTES + ((piece ^ (2 * ((row >> 3) & 3))) << 4));
                                const int64_t nb = n0 + piece * 8;
                                OutT *dst = out + (mrow0 + row) * P.ld_out + nb;
                                if (nb + 8 <= P.n) {
                                    *reinterpret_cast<uint4 *>(dst) = v;
                                } else {
                                    const OutT *e = reinterpret_cast<const OutT *>(&v);
                                    for (int j = 0; j < 8; ++j)
                                        if (nb + j < P.n) dst[j] = e[j];
                                }
                            }
                        }
                    }
                    epilogue_bar_sync();
                }
            } else {
                for (int mb = 0; mb < n_mblk; ++mb) {
                    const int64_t mrow0 = m0 + mb * BM;
                    const int64_t m = mrow0 + row_in_blk;
                    float bias = 0.f;
                    if (run && P.bias) bias = row_bias<OutT, F8>(P, m);
                    const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16) + mb * BN;
                    if constexpr (TRANS_OUT) {
                        // 4-byte transposed output, STG_COLS columns at a time; each warp copies its half of a chunk
                        constexpr int CHUNKS = BN / Cfg::STG_COLS;
                        constexpr int HC = Cfg::STG_COLS / 2;
                        static_assert(HC % 32 == 0, "a warp reads whole 32-column pieces");
                        uint8_t *stg_row = reinterpret_cast<uint8_t *>(stg) + (size_t)row_in_blk * Cfg::STG_ROW_BYTES;
#pragma unroll 1
                        for (int ch = 0; ch < CHUNKS; ++ch) {
                            if (run) {
#pragma unroll 1
                                for (int c = 0; c < HC / 32; ++c) {
                                    uint32_t v[32];
                                    const int col = half * HC + c * 32;
                                    tmem_ld32(acc + ch * Cfg::STG_COLS + col, v);
                                    tmem_ld_wait();
#pragma unroll
                                    for (int q = 0; q < 8; ++q) {
                                        float4 o;
                                        o.x = __uint_as_float(emit_bits<OutT, ACT>(v[q * 4 + 0], bias, P.activation, alpha));
                                        o.y = __uint_as_float(emit_bits<OutT, ACT>(v[q * 4 + 1], bias, P.activation, alpha));
                                        o.z = __uint_as_float(emit_bits<OutT, ACT>(v[q * 4 + 2], bias, P.activation, alpha));
                                        o.w = __uint_as_float(emit_bits<OutT, ACT>(v[q * 4 + 3], bias, P.activation, alpha));
                                        *reinterpret_cast<float4 *>(stg_row + (col + q * 4) * 4) = o;
                                    }
                                }
                            }
                            if (ch == CHUNKS - 1) {
                                // this accumulator has been read completely: hand it back to the MMA warp
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) mbar_arrive(tmem_empty0 + 8 * mb);
                                if (threadIdx.x == 64) SP24_TRACE(2, 4 * tl + 1 + mb);
                            }
                            epilogue_bar_sync();
                            if (run) {
                                // thread = one output row x 4 consecutive features; lane pairs cover 8 features of
                                // the same row, so every warp instruction writes whole 32-byte sectors
                                const int64_t nbase = n0 + ch * Cfg::STG_COLS;
                                const uint8_t *stg_b = reinterpret_cast<const uint8_t *>(stg);
                                for (int i = tid; i < Cfg::STG_COLS * (BM / 4); i += 256) {
                                    const int pr = i >> 1;
                                    const int nn = pr % Cfg::STG_COLS, mg = 2 * (pr / Cfg::STG_COLS) + (i & 1);
                                    uint4 o;
                                    o.x = *reinterpret_cast<const uint32_t *>(stg_b + (size_t)(mg * 4 + 0) * Cfg::STG_ROW_BYTES + nn * 4);
                                    o.y = *reinterpret_cast<const uint32_t *>(stg_b + (size_t)(mg * 4 + 1) * Cfg::STG_ROW_BYTES + nn * 4);
                                    o.z = *reinterpret_cast<const uint32_t *>(stg_b + (size_t)(mg * 4 + 2) * Cfg::STG_ROW_BYTES + nn * 4);
                                    o.w = *reinterpret_cast<const uint32_t *>(stg_b + (size_t)(mg * 4 + 3) * Cfg::STG_ROW_BYTES + nn * 4);
                                    if (nbase + nn < P.n)
                                        *reinterpret_cast<uint4 *>(out + (nbase + nn) * P.ld_out + mrow0 + mg * 4) = o;
                                }
                            }
                            epilogue_bar_sync();
                        }
                    } else {
                        constexpr int HC = BN / 2;
                        if (run) {
#pragma unroll 1
                            for (int c = 0; c < HC / 32; ++c) {
                                uint32_t v[32];
                                const int col = half * HC + c * 32;
                                tmem_ld32(acc + col, v);
                                tmem_ld_wait();
                                const int64_t nb = n0 + col;
                                OutT *row = out + m * P.ld_out + nb;
                                if (ACCUM || (F8 && std::is_same<OutT, float>::value && P.accumulate)) {
                                    const float al = F8 ? alpha : 1.f;
#pragma unroll
                                    for (int i = 0; i < 32; ++i)
                                        if constexpr (F8) v[i] = __float_as_uint(__uint_as_float(v[i]) * al);
                                    // D += partial product: fp32 reductions in L2, 16 bytes each, no return value
                                    if (nb + 32 <= P.n) {
#pragma unroll
                                        for (int q = 0; q < 8; ++q)
                                            red_add_v4(reinterpret_cast<float *>(row) + q * 4, __uint_as_float(v[q * 4]), __uint_as_float(v[q * 4 + 1]),
                                                       __uint_as_float(v[q * 4 + 2]), __uint_as_float(v[q * 4 + 3]));
                                    } else {
                                        for (int i = 0; i < 32; ++i)
                                            if (nb + i < P.n) atomicAdd(reinterpret_cast<float *>(row) + i, __uint_as_float(v[i]));
                                    }
                                } else if (nb + 32 <= P.n) {
                                    constexpr int PER = 16 / sizeof(OutT);
#pragma unroll
                                    for (int q = 0; q < 32 / PER; ++q) {
                                        Vec<OutT, PER> o;
#pragma unroll
                                        for (int i = 0; i < PER; ++i)
                                            o.v[i] = emit<OutT, ACT, F8>(v[q * PER + i], bias, P.activation, alpha);
                                        store_vec<OutT, PER>(row + q * PER, o);
                                    }
                                } else {
                                    for (int i = 0; i < 32; ++i)
                                        if (nb + i < P.n)
                                            row[i] = emit<OutT, ACT, F8>(v[i], bias, P.activation, alpha);
                                }
                            }
                        }
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(tmem_empty0 + 8 * mb);
                    }
                }
                if (n_mblk == 1) {
                    // keep the second accumulator's barrier in step with the tile count
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tmem_empty0 + 8);
                }
            }
            if (threadIdx.x == 64) SP24_TRACE(2, 4 * tl + 3);
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------
// Two-CTA form (cluster of 2, tcgen05 cta_group::2) for 16-bit types, B stored (n, k), output (n, ms).
// ------------------------------------------------------------------------------------------------
// A CTA pair computes tiles of 256 sparse rows x BN dense columns (BN up to 240, chosen per problem): every MMA instruction has
// M = 256 (128 rows per CTA) and N = BN, and reads half of its B operand from each CTA's shared memory, so a CTA stages only
// BN / 2 rows of B per stage: 48 KB for 7.9 dense-equivalent MFLOP at 240 columns, where the single-CTA kernel needs 66 KB for
// 6.3 (or 84 KB for two blocks).  One accumulator per tile leaves room for two accumulator buffers in tensor memory, so the
// epilogue of a tile runs entirely under the next tile's MMAs, and four to six operand stages fit.
// Each CTA loads its own A block, metadata and B half with TMA (cta_group::2 form, completing on the leader's
// barrier), drains its own accumulator and reports its release to the leader's barrier.  CTA 0 of the pair
// (the leader) issues all MMAs and metadata copies; its commits arrive on the barriers of both CTAs.  No load
// is multicast.
namespace two {
// Columns of a pair tile: a multiple of 16 (8-bit operands: of 32) in [BN2_MIN, BN2_MAX], chosen per problem (pick_pair_bn).  Two accumulator buffers
// of up to 240 columns start at columns 0 and 256 of tensor memory, the metadata slots sit in the 16 columns between them.
constexpr int BN2_MIN = 32, BN2_MAX = 240, ACC_COL = 256, E_COL = 240;
constexpr int MAX_STAGES2 = 6;
// 8-bit operands: the same bytes per stage (K step 256 instead of 128), twice the metadata.  Stage: A block, metadata, then
// BN / 2 rows of B as two 128-byte K atoms; every part is a multiple of the 1024-byte swizzle period.
constexpr int e2_bytes(bool f8) { return f8 ? 4096 : 2048; }
constexpr int stage2_bytes(bool f8, int bn) { return A_STAGE_BYTES + e2_bytes(f8) + bn * 128; }
// Output staging of the plain epilogue: a chunk is 16 tokens x 32 features of 16 bits, two per epilogue warp.  Four widths have one
// operand stage fewer for it: 16-bit 144 and 208, float8 128 and 192.  Against the direct stores before it the calls
// measured at 208, 128 and 192 lost no more than 1 % (ms 2304, k 3072, n 8192 57.0 -> 57.6 us; float8 ms 768, k 3072, n 8192 15.7 both) but for float8 at width
// 128 with three K steps in one round, 6.4 -> 6.5.  Pieces of 8 tokens, one or two a warp, gave the stages back and were not kept:
// up to 3 % faster at widths 208 and 192 from k 3072 on (57.6 -> 55.4, 15.7 -> 15.4), 1 - 2 % slower at most others.
constexpr int MAX_CHUNKS2 = (BN2_MAX / 16 + 1) / 2;         // of a tile and a warp
constexpr int CHUNK2_BYTES = 16 * 64, STAGING2 = 8 * 2 * CHUNK2_BYTES;
// Barriers and flags behind the staging, at addresses known at run time only.  With the same kernel's barriers in static shared
// memory a K step takes about 30 ns longer where it is bound by latency; us, static -> here: fp16 ms 4096, k 3072, n 16 12.5 -> 11.5;
// ms 1536, k 3072, n 4096 22.8 -> 21.5; float8 ms 256, k 3072, n 16 7.9 -> 7.5; over all shapes 3 % (fp16), 2 % (float8), 1 % (fused).
// Where the stages start makes no difference, so it is the code of the loops.  One place is slower with it: the gelu epilogue at
// k 3072 with 8192 tokens and more, 1 - 8 % (ms 4096, n 16384 229 -> 237; the same with operands of zeros, so not the power limit);
// at k 2048 and 4096 the same sizes are 2 - 5 % faster (197 -> 192, 287 -> 286), at k 768 alike, so no rule on sizes follows.
struct Ctl2 {
    uint64_t bars[2 * MAX_STAGES2 + 6];
    uint32_t tmem_base;
    int abort_flag;
};
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int stages2(bool f8, int bn) {
    const int n = (SMEM_LIMIT - STAGING2 - (int)sizeof(Ctl2)) / stage2_bytes(f8, bn);
    return n < MAX_STAGES2 ? n : MAX_STAGES2;
}
constexpr int smem2(bool f8, int bn) { return stages2(f8, bn) * stage2_bytes(f8, bn) + STAGING2 + (int)sizeof(Ctl2); }
static_assert(stage2_bytes(false, 16) % 1024 == 0 && stage2_bytes(true, 16) % 1024 == 0, "stages must keep the 1024-byte swizzle alignment");
static_assert(stages2(true, BN2_MAX) >= 4, "shared memory budget");
}  // namespace two

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cta address -> shared::cluster address of the same location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar_cluster)
        : "memory");
}
// a box of two 128-byte columns (see make_map_columns), one behind the other in shared memory
__device__ __forceinline__ void tma_load_columns_pair(uint32_t dst, const CUtensorMap *map, int row, int column, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(map), "r"(0), "r"(row), "r"(column), "r"(bar_cluster)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// arrives on the barrier at this shared-memory offset in both CTAs of the pair once the MMAs issued so far are done; first: the
// leader's rank, where the cluster has more than one pair
__device__ __forceinline__ void tc_commit_pair(uint32_t bar, uint32_t first = 0) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)(3u << first))
                 : "memory");
}
__device__ __forceinline__ void tc_cp_128x128b_pair(uint32_t taddr, uint64_t sdesc) {
    asm volatile("tcgen05.cp.cta_group::2.128x128b [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void mma_sp_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t e_tmem, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.sp.cta_group::2.kind::f16 [%0], %1, %2, [%3], %4, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(e_tmem), "r"(idesc), "r"(accumulate)
        : "memory");
}

template <bool F8>
__device__ __forceinline__ void mma_sp_pair_any(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t e_tmem, uint32_t idesc,
                                                uint32_t accumulate) {
    if constexpr (F8)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.sp.cta_group::2.kind::f8f6f4 [%0], %1, %2, [%3], %4, p;\n\t}" ::"r"(d_tmem),
            "l"(adesc), "l"(bdesc), "r"(e_tmem), "r"(idesc), "r"(accumulate)
            : "memory");
    else mma_sp_pair(d_tmem, adesc, bdesc, e_tmem, idesc, accumulate);
}

template <bool A_MN, typename OutT, int EPI, bool F8>
__global__ void __launch_bounds__(320, 1)
spmm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_e, SpmmParams P) {
    using namespace two;
    const int BN = P.bn, STAGES = P.stages;       // see pick_pair_bn
    const int STAGE2_BYTES = stage2_bytes(F8, BN);
    constexpr int OFF_E = A_STAGE_BYTES, OFF_B = OFF_E + e2_bytes(F8);
    constexpr int KE = F8 ? 256 : 128;            // K step of a stage
    constexpr int KSTEPS = 4;
    constexpr uint32_t TMEM_COLS = 512;
    constexpr int E_SLOT = F8 ? 8 : 4;
    static_assert(sizeof(OutT) == 2, "16-bit outputs only");
    static_assert(BN2_MAX <= E_COL && E_COL + 2 * E_SLOT <= ACC_COL && ACC_COL + BN2_MAX <= 512, "tensor memory columns exhausted");

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw;
    if (smem_u32(smem) & 1023) {              // the same in every CTA; the launcher looks first, the swizzled stages depend on it
        chain_enter();
        if (threadIdx.x == 0 && P.status) atomicCAS(P.status, 0, 11);
        return;
    }
    Ctl2 &ctl = *reinterpret_cast<Ctl2 *>(smem + STAGES * STAGE2_BYTES + STAGING2);
    uint64_t *const bars = ctl.bars;
    volatile int &abort_flag = ctl.abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();          // 0 = leader
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int n_tiles_n = (int)((P.n + BN - 1) / BN);
    // 256-row blocks, one 128-row block per CTA.  Where ms is an odd multiple of 128 the last one's second block lies past the operand:
    // its loads give zeros and its results are not stored.
    const int n_tiles_m = (int)((P.ms + 2 * BM - 1) / (2 * BM));
    const int n_tiles = n_tiles_n * n_tiles_m;        // row block varies fastest over the tile index
    const int k_iters = (int)((P.k + KE - 1) / KE);

    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[MAX_STAGES2]);
    const uint32_t tmem_full0 = smem_u32(&bars[2 * MAX_STAGES2]), tmem_empty0 = smem_u32(&bars[2 * MAX_STAGES2 + 2]);
    // Plain form: a pair's last two tiles are complete on barriers of their own.  Before them a warp waits for the tiles of its half only,
    // each of which holds that accumulator back until the warp has read it, so a barrier is never more than one phase from what the
    // warp waits for.  The last two are for all warps, and one that has not waited for the other accumulator before does not know its
    // phase; waiting for every tile instead would stall a warp that two tiles of the other half have passed meanwhile.
    const uint32_t tmem_last0 = smem_u32(&bars[2 * MAX_STAGES2 + 4]);
    auto ends = [&](int tile) { return EPI == EPI_PLAIN && tile + 2 * n_pairs >= n_tiles; };

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);      // used in the leader only: one expect_tx arrival, bytes of both CTAs
            mbar_init(empty0 + 8 * s, 1);     // one commit arrival per CTA
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tmem_full0 + 8 * b, 1);
            mbar_init(tmem_last0 + 8 * b, 1);
            mbar_init(tmem_empty0 + 8 * b, EPI == EPI_PLAIN ? 8 : 16);   // used in the leader only: four or eight epilogue warps of each CTA
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(&ctl.tmem_base), TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                       // the peer's barriers are initialised before anything targets them
    tc_fence_after();
    const uint32_t tmem_base = ctl.tmem_base;
    chain_enter();

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer (one per CTA)
        if (lane == 0) {
            int g = 0, s = 0;
            uint32_t ph = 1;                     // of the empty barriers: the first round passes at once
            bool ok = true;
            const uint32_t cta_tx = (uint32_t)STAGE2_BYTES;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                const int mblk = (tile % n_tiles_m) * 2 + (int)rank;
                const int mrow = mblk * BM;
                const int brow = (tile / n_tiles_m) * BN + (int)rank * (BN / 2);
                for (int it = 0; it < k_iters; ++it, ++g) {
                    if (!mbar_wait(empty0 + 8 * s, ph, &abort_flag, P.status, 1)) { ok = false; break; }
                    const uint32_t sa = smem_u32(smem) + (uint32_t)s * (uint32_t)STAGE2_BYTES;
                    const uint32_t sb = sa + OFF_B;
                    const uint32_t full_leader = map_to_cta(full0 + 8 * s, 0);
                    if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * cta_tx);
                    if constexpr (!A_MN) {
                        tma_load_2d_pair(sa, &map_a, it * (KE / 2), mrow, full_leader);
                    } else {
                        tma_load_columns_pair(sa, &map_a, it * 64, mrow / 64, full_leader);
                    }
                    // metadata of this row block and K step: two rows of 1024 bytes per atom of the table (8-bit: two atoms)
                    tma_load_2d_pair(sa + OFF_E, &map_e, 0, (int)(((int64_t)mblk * P.k_atoms + it * (F8 ? 2 : 1)) * 2), full_leader);
                    // this CTA's half of B: BN / 2 rows x two 128-byte K atoms
                    tma_load_columns_pair(sb, &map_b, brow, 2 * it, full_leader);
                    SP24_TRACE(0, g);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
            if (abort_flag && rank == 0) {
                for (int q = (g > STAGES ? g - STAGES : 0); q < g; ++q) {
                    const int sq = q % STAGES;
                    const uint32_t pq = (q / STAGES) & 1;
                    for (uint32_t w = 0; w < WAIT_LIMIT; ++w)
                        if (mbar_try_wait(full0 + 8 * sq, pq)) break;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer (leader CTA only)
        // All 32 lanes walk the loop together, so that its counters, addresses and descriptors stay in uniform registers
        // (the MMA takes all its operands from there); one elected lane issues.  Descriptors advance by an add to their
        // address field.
        if (rank == 0) {
            constexpr uint32_t A_LBO = A_MN ? 8192 : 16, A_KSTEP = A_MN ? 2048 : 32;
            const uint32_t idesc0 = P.idesc;   // M = 256, N = BN set by the launcher
            const uint32_t smem0 = smem_u32(smem);
            const uint64_t adesc0 = make_desc(smem0, A_LBO, 1024, 2), bdesc0 = make_desc(smem0 + OFF_B, 16, 1024, 2);
            const uint64_t edesc0 = make_desc(smem0 + OFF_E, 16, 128, 0);
            const uint32_t b_atom = (uint32_t)BN * (64 >> 4);       // second K atom of a B half, in descriptor units
            int s = 0, tl = 0;
            uint32_t ph = 0, eslot = 0;
            bool ok = true;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tl) {
                const int buf = tl & 1;
                const uint32_t acc = tmem_base + buf * ACC_COL;
                // the epilogues of both CTAs must have drained this accumulator buffer (two tiles ago)
                ok = mbar_wait_warp(tmem_empty0 + 8 * buf, ((tl >> 1) & 1) ^ 1, &abort_flag, P.status, 4);
                for (int it = 0; it < k_iters && ok; ++it) {
                    ok = mbar_wait_warp(full0 + 8 * s, ph, &abort_flag, P.status, 2);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t off = (uint32_t)s * ((uint32_t)STAGE2_BYTES >> 4);
                    const uint64_t ad = adesc0 + off, bd = bdesc0 + off, ed = edesc0 + off;
                    const uint32_t e_cols = tmem_base + E_COL + eslot;
                    if (elect_one()) {
                        tc_cp_128x128b_pair(e_cols, ed);
                        if constexpr (F8) tc_cp_128x128b_pair(e_cols + 4, ed + (2048 >> 4));
                        // metadata of an MMA: two columns (8-bit), or the even column of a pair plus a 1-bit selector
#pragma unroll
                        for (int j = 0; j < KSTEPS; ++j)
                            mma_sp_pair_any<F8>(acc, ad + j * (A_KSTEP >> 4), bd + ((j >> 1) * b_atom + (j & 1) * (64 >> 4)),
                                                e_cols + (F8 ? 2 * j : (j & ~1)), F8 ? idesc0 : idesc0 | (j & 1), (it > 0 || j > 0) ? 1u : 0u);
                        tc_commit_pair(empty0 + 8 * s);
                    }
                    __syncwarp();
                    eslot ^= E_SLOT;
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (elect_one()) tc_commit_pair((ends(tile) ? tmem_last0 : tmem_full0) + 8 * buf);   // also arrives after an abort
                __syncwarp();
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue (warps 2..9 of both CTAs)
        // Plain form: 16-token chunks of a warp's 32 features, two read and packed to 16 bits while the two before are stored.
        // tcgen05.ld in the 16x256b shape leaves 8 x 8 fragments; stmatrix writes them token-major into the warp's two chunks of shared
        // memory, from where 16-byte stores take them, 8 tokens x 64 bytes an instruction (128-byte rows and TMA stores were no faster).
        // While a later tile will want the accumulator again, the four warps of one half take all of it and the other four the next
        // tile's; of a pair's last two tiles, which nobody waits for, each half takes every other chunk.  With all eight warps on one tile,
        // an accumulator first read whole into registers and then stored, the stores stood still while it was read: 4500 clocks a tile
        // without any operand loads, where stores by themselves take 2640.  us, that -> now: ms 3072, k 768, n 8192 30.4 -> 27.9 (float8
        // 22.6 -> 19.2), n 16384 47.6 -> 46.9; ms 768, n 8192, k 3072 24.6 -> 23.5; ms 4096, n 2043, k 4096 28.2 -> 27.1; ms 1024, n 1024,
        // k 1024 7.4 -> 6.8; ms 512, n 256, k 256 4.8 -> 4.25 (a third of that from the shorter code).  One loop for both cases: 2 - 5 % slower.
        // Fused forms: a warp packs its BN / 2 columns of the accumulator into registers, hands the buffer back, then stores
        // 16-bit values directly; the 32 lanes of a store are 32 consecutive features of one token.
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int HC = BN / 2;                      // fused epilogues: a multiple of 16 up to 96
        constexpr int NREG = 48;
        OutT *out = static_cast<OutT *>(P.out);
        const float alpha = F8 ? alpha_of(P) : 1.f;
        const uint32_t empty_leader0 = map_to_cta(tmem_empty0, 0);
        // plain form: the warp's staging, and where a lane's stmatrix row goes in a chunk: token 8 (lane / 16) + lane % 8 in rows of
        // 64 bytes, features 16 h + 8 (lane / 8 % 2) in 16-byte pieces, permuted by token / 2 % 4 against bank conflicts
        const uint32_t stg = smem_u32(smem) + STAGES * STAGE2_BYTES + (warp - 2) * 2 * CHUNK2_BYTES;
        const uint32_t ld_off = (lane >> 2) * 64 + (((lane & 3) ^ ((lane >> 3) & 3)) << 4);
        uint32_t stm_off[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int tok = 8 * (lane >> 4) + (lane & 7), piece = 2 * h + ((lane >> 3) & 1);
            stm_off[h] = tok * 64 + ((piece ^ ((tok >> 1) & 3)) << 4);
        }
        int tl = 0;
        for (int tile = pair; tile < n_tiles; tile += n_pairs, ++tl) {
            const int buf = tl & 1;
            const bool last = ends(tile);
            if (EPI == EPI_PLAIN && !last && (tl & 1) != half) continue;      // the other half's tile
            const int mrow = ((tile % n_tiles_m) * 2 + (int)rank) * BM + quad * 32;
            const int64_t row0 = (int64_t)(tile / n_tiles_m) * BN;
            const bool ok = mbar_wait((last ? tmem_last0 : tmem_full0) + 8 * buf, last ? 0 : (tl >> 1) & 1, &abort_flag, P.status, 3);
            tc_fence_after();
            if (threadIdx.x == 64) SP24_TRACE(2, 4 * tl);
            const bool run = __all_sync(0xFFFFFFFFu, ok && !abort_flag) && mrow < P.ms;      // the warp reads tensor memory together
            if constexpr (EPI == EPI_PLAIN) {
                const int64_t left = P.n - row0;
                const int limit = left < BN ? (int)left : BN, chunks = (limit + 15) / 16;
                float bias[4] = {0.f, 0.f, 0.f, 0.f};       // of features 8 h + lane / 4
                if (run && P.bias) {
#pragma unroll
                    for (int h = 0; h < 4; ++h) bias[h] = load_bias<OutT>(P, mrow + 8 * h + (lane >> 2));
                }
                const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * ACC_COL;
                const int64_t row = P.ld_out / 8;           // of 16-byte pieces
                auto read = [&](uint32_t column, uint32_t (&v)[2][8]) {      // a chunk past the last one: other columns, read but not stored
                    tmem_ld_16x256b_x2(acc + column, v[0]);
                    tmem_ld_16x256b_x2(acc + (16u << 16) + column, v[1]);
                };
                auto pack = [&](const uint32_t (&v)[2][8], uint32_t (&held)[8]) {      // word 4 h + j: features 16 h + 8 (j % 2), tokens 8 (j / 2)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            Vec<OutT, 2> o;
                            o.v[0] = emit<OutT, false, F8>(v[h][2 * j], bias[2 * h + (j & 1)], 0, alpha);
                            o.v[1] = emit<OutT, false, F8>(v[h][2 * j + 1], bias[2 * h + (j & 1)], 0, alpha);
                            held[4 * h + j] = *reinterpret_cast<const uint32_t *>(&o);
                        }
                };
                auto store = [&](uint32_t at, const uint32_t (&held)[8], uint4 *to, int tokens) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) stmatrix_x4_trans(at + stm_off[h], held[4 * h], held[4 * h + 1], held[4 * h + 2], held[4 * h + 3]);
                    __syncwarp();                           // also: the chunk before the last one has left its half
#pragma unroll
                    for (int h = 0; h < 2; ++h) {           // 8 tokens x 64 bytes an instruction
                        const uint4 o = ld_shared_v4(at + ld_off + h * 512);
                        if (8 * h < tokens) to[8 * h * row] = o;
                    }
                };
                uint4 *const dst = reinterpret_cast<uint4 *>(out + (row0 + (lane >> 2)) * P.ld_out + mrow) + (lane & 3);
                const int mine = limit - (lane >> 2);       // tokens of the tile from this lane's first one on
                uint32_t v[2][2][8], held[2][8];
                if (!last) {
                    // the tile after the next wants this accumulator
                    if (run) {
                        read(0, v[0]);
                        read(16, v[1]);
                    }
#pragma unroll 1
                    for (int c = 0; c < chunks; c += 2) {
                        if (run) {
                            tmem_ld_wait();
                            pack(v[0], held[0]);
                            pack(v[1], held[1]);
                            if (c + 2 < chunks) {
                                read((c + 2) * 16, v[0]);
                                read((c + 3) * 16, v[1]);
                            }
                        }
                        if (c + 2 >= chunks) {          // all read
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cluster(empty_leader0 + 8 * buf);
                        }
                        if (run) {
                            store(stg, held[0], dst + 16 * c * row, mine - 16 * c);
                            if (c + 1 < chunks) store(stg + CHUNK2_BYTES, held[1], dst + 16 * (c + 1) * row, mine - 16 * (c + 1));
                        }
                    }
                    __syncwarp();
                } else {
                    if (run && half < chunks) {
                        read(half * 16, v[0]);
                        read(half * 16 + 32, v[1]);
#pragma unroll
                        for (int i = 0; i < MAX_CHUNKS2; i += 2) {
                            if (half + 2 * i >= chunks) break;
                            tmem_ld_wait();
                            pack(v[0], held[0]);
                            pack(v[1], held[1]);
                            if (i + 2 < MAX_CHUNKS2 && half + 2 * (i + 2) < chunks) {
                                read(half * 16 + 32 * (i + 2), v[0]);
                                read(half * 16 + 32 * (i + 3), v[1]);
                            }
                            uint4 *const to = dst + half * 16 * row;
                            store(stg, held[0], to + 32 * i * row, mine - half * 16 - 32 * i);
                            if (half + 2 * (i + 1) < chunks) store(stg + CHUNK2_BYTES, held[1], to + 32 * (i + 1) * row, mine - half * 16 - 32 * (i + 1));
                        }
                        __syncwarp();
                    }
                    tc_fence_before();
                }
            } else {
                const int64_t tok0 = row0 + half * HC;
                uint32_t held[NREG];
                if (run) {
                    float bias = 0.f;
                    if (P.bias) bias = load_bias<OutT>(P, mrow + lane);
                    const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * ACC_COL + half * HC;
#pragma unroll
                    for (int c = 0; c < NREG / 16; ++c) {
                        if (c * 32 >= HC) break;
                        uint32_t v[32];             // columns past HC belong to other tiles or to the metadata: read, never stored
                        tmem_ld32(acc + c * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            Vec<OutT, 2> o;
                            if constexpr (EPI == EPI_DGELU) {   // no bias; the factor gelu'(aux) is applied at store time
                                o.v[0] = to_out<OutT>(__uint_as_float(v[2 * i]));
                                o.v[1] = to_out<OutT>(__uint_as_float(v[2 * i + 1]));
                            } else {
                                o.v[0] = emit<OutT, false, F8>(v[2 * i], bias, 0, alpha);
                                o.v[1] = emit<OutT, false, F8>(v[2 * i + 1], bias, 0, alpha);
                            }
                            held[c * 16 + i] = *reinterpret_cast<const uint32_t *>(&o);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(empty_leader0 + 8 * buf);
                if (run) {
                    uint16_t *dst = reinterpret_cast<uint16_t *>(out) + tok0 * P.ld_out + mrow + lane;
                    uint16_t *aux = reinterpret_cast<uint16_t *>(P.aux) + tok0 * P.ld_aux + mrow + lane;
                    const bool full = tok0 + HC <= P.n;
                    auto as_f = [](uint16_t bits) { return from_out<OutT>(*reinterpret_cast<const OutT *>(&bits)); };
                    auto as_b = [](float v) { const OutT o = to_out<OutT>(v); return *reinterpret_cast<const uint16_t *>(&o); };
                    // chunks of 16 tokens: all loads of a chunk are issued before the first use, all its stores after
                    constexpr int CHUNK = 8;
#pragma unroll
                    for (int c0 = 0; c0 < NREG; c0 += CHUNK) {
                        if (2 * c0 >= HC) break;
                        uint16_t a[2 * CHUNK];
                        if constexpr (EPI == EPI_DGELU) {
#pragma unroll
                            for (int j = 0; j < 2 * CHUNK; ++j)
                                a[j] = (full || tok0 + 2 * c0 + j < P.n) ? aux[(int64_t)j * P.ld_aux] : (uint16_t)0;
                        }
#pragma unroll
                        for (int j = 0; j < 2 * CHUNK; ++j) {
                            const uint32_t hw = held[c0 + (j >> 1)];
                            const uint16_t h_bits = (j & 1) ? (uint16_t)(hw >> 16) : (uint16_t)(hw & 0xFFFFu);
                            if (full || tok0 + 2 * c0 + j < P.n) {
                                if constexpr (EPI == EPI_PRE_GELU) {
                                    aux[(int64_t)j * P.ld_aux] = h_bits;
                                    dst[(int64_t)j * P.ld_out] = as_b(gelu_tanh(as_f(h_bits)));
                                } else {
                                    dst[(int64_t)j * P.ld_out] = as_b(as_f(h_bits) * gelu_tanh_grad(as_f(a[j])));
                                }
                            }
                        }
                        dst += 2 * CHUNK * P.ld_out;
                        aux += 2 * CHUNK * P.ld_aux;
                        asm volatile("" : "+l"(dst), "+l"(aux));   // running pointers per chunk
                    }
                }
            }
            if (threadIdx.x == 64) SP24_TRACE(2, 4 * tl + 3);
        }
        tc_fence_before();
    }
    // nobody leaves while the peer may still read this CTA's shared memory or signal its barriers
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------
// Few tokens: K cut into slices over the pairs of a cluster.
// ------------------------------------------------------------------------------------------------
// A handful of dense columns gives one tile per 256 rows: 16 pairs of 74 walk 32 K steps each for a 4096 x 4096 weight, and a step
// takes the ring's latency whatever it computes.  Here a cluster of S pairs (S <= 4: eight CTAs) takes one tile, each pair every S-th
// part of K with a ring of its own.  Every pair finishes a share of the tile's columns: all pairs leave their float32 partial sums of
// them in its shared memory, and after one cluster barrier it adds them up in the order of the slices, its own like the others', so
// results repeat bit for bit and equal tokens of a call have equal outputs.
// (One pair finishing the whole tile took 1 us more at 32 columns and 2.5 at 64.)
namespace two {
constexpr int SPLIT_MAX = 4, BN_SPLIT = 64;                 // pairs a cluster at most, the widest tile
// Columns at most.  A training step of the FST and float8 layers has at least 64 tokens (their MVUE compression takes multiples of
// 64) and keeps one order of sums whatever the kernel: an output rounded the other way makes other MVUE draws, which moves a
// model's gradients by several percent.  The bound is not where slices stop gaining: inference, which has no such reason, stops here
// with it (ms 4096, k 4096: n 64 12.7 us, 8.3 in slices; n 128 13.3, 9.5).
constexpr int64_t SPLIT_N = 63, SPLIT_K = 7 * 128;          // K above: see pick_slices
static_assert(SPLIT_N <= BN_SPLIT, "one tile takes all columns");
__host__ __device__ constexpr int share(int bn, int slices) { return (bn + 4 * slices - 1) / (4 * slices) * 4; }     // columns a pair finishes
// a partial share: columns in fours, 128 rows x 16 bytes each, so that a warp's remote store is 512 bytes in one piece
__host__ __device__ constexpr int part_bytes(int bn, int slices) { return share(bn, slices) * BM * 4; }
constexpr int split_stages(int bn, int slices) {
    const int n = (SMEM_LIMIT - slices * part_bytes(bn, slices) - (int)sizeof(Ctl2)) / stage2_bytes(false, bn);
    return n < MAX_STAGES2 ? n : MAX_STAGES2;
}
constexpr int split_smem(int bn, int slices) {
    return split_stages(bn, slices) * stage2_bytes(false, bn) + slices * part_bytes(bn, slices) + (int)sizeof(Ctl2);
}
static_assert(split_stages(BN_SPLIT, SPLIT_MAX) >= 4, "shared memory budget");
}  // namespace two

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

template <bool A_MN, typename OutT>
__global__ void __launch_bounds__(320, 1)
spmm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_e, SpmmParams P) {
    using namespace two;
    const int BN = P.bn, STAGES = P.stages, S = P.k_splits;
    const int STAGE_BYTES = stage2_bytes(false, BN);
    constexpr int OFF_E = A_STAGE_BYTES, OFF_B = OFF_E + e2_bytes(false);
    constexpr uint32_t TMEM_COLS = 512;

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *const smem = smem_raw;                // on 1024 bytes: checked by the launcher, the same in every CTA
    uint8_t *const parts = smem + STAGES * STAGE_BYTES;
    Ctl2 &ctl = *reinterpret_cast<Ctl2 *>(parts + S * part_bytes(BN, S));
    uint64_t *const bars = ctl.bars;
    volatile int &abort_flag = ctl.abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cta = cluster_ctarank(), rank = cta & 1u, leader = cta & ~1u;      // rank in the pair; the pair's first CTA
    const int slice = (int)(cta >> 1);
    const int k_iters = (int)((P.k + 127) / 128), it0 = slice * k_iters / S, it1 = (slice + 1) * k_iters / S;
    const int mblk = (int)blockIdx.x / (2 * S) * 2 + (int)rank;      // a tile: 256 rows, all columns

    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[MAX_STAGES2]), tmem_full = smem_u32(&bars[2 * MAX_STAGES2]);
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(tmem_full, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(&ctl.tmem_base), TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = ctl.tmem_base;
    chain_enter();

    bool run = false;
    const int quad = warp & 3, half = (warp - 2) >> 2, HC = BN / 2, CW = share(BN, S);
    const int mrow = mblk * BM + quad * 32, n = (int)P.n;
    auto owner_of = [&](int col) { return (col >= CW) + (col >= 2 * CW) + (col >= 3 * CW); };      // the pair that finishes a column
    if (warp == 0) {
        if (lane == 0) {
            int s = 0, g = 0;
            uint32_t ph = 1;
            for (int it = it0; it < it1; ++it, ++g) {
                if (!mbar_wait(empty0 + 8 * s, ph, &abort_flag, P.status, 1)) break;
                const uint32_t sa = smem_u32(smem) + (uint32_t)(s * STAGE_BYTES), sb = sa + OFF_B;
                const uint32_t full_leader = map_to_cta(full0 + 8 * s, leader);
                if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * (uint32_t)STAGE_BYTES);
                if constexpr (!A_MN) {
                    tma_load_2d_pair(sa, &map_a, it * 64, mblk * BM, full_leader);
                } else {
                    tma_load_columns_pair(sa, &map_a, it * 64, mblk * 2, full_leader);
                }
                tma_load_2d_pair(sa + OFF_E, &map_e, 0, (int)(((int64_t)mblk * P.k_atoms + it) * 2), full_leader);
                tma_load_columns_pair(sb, &map_b, (int)rank * (BN / 2), 2 * it, full_leader);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            if (abort_flag && rank == 0) {
                for (int q = (g > STAGES ? g - STAGES : 0); q < g; ++q)
                    for (uint32_t w = 0; w < WAIT_LIMIT; ++w)
                        if (mbar_try_wait(full0 + 8 * (q % STAGES), (q / STAGES) & 1)) break;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0) {                       // all lanes in step, one elected lane issues (as in spmm_pair_kernel)
            const uint32_t idesc0 = P.idesc, smem0 = smem_u32(smem);
            constexpr uint32_t A_LBO = A_MN ? 8192 : 16, A_KSTEP = A_MN ? 2048 : 32;
            const uint64_t adesc0 = make_desc(smem0, A_LBO, 1024, 2), bdesc0 = make_desc(smem0 + OFF_B, 16, 1024, 2);
            const uint64_t edesc0 = make_desc(smem0 + OFF_E, 16, 128, 0);
            const uint32_t b_atom = (uint32_t)BN * (64 >> 4);
            int s = 0;
            uint32_t ph = 0, eslot = 0;
            for (int it = it0; it < it1; ++it) {
                if (!mbar_wait_warp(full0 + 8 * s, ph, &abort_flag, P.status, 2)) break;
                tc_fence_after();
                const uint32_t off = (uint32_t)s * ((uint32_t)STAGE_BYTES >> 4), e_cols = tmem_base + E_COL + eslot;
                if (elect_one()) {
                    tc_cp_128x128b_pair(e_cols, edesc0 + off);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        mma_sp_pair(tmem_base, adesc0 + off + j * (A_KSTEP >> 4), bdesc0 + off + ((j >> 1) * b_atom + (j & 1) * (64 >> 4)),
                                    e_cols + (j & ~1), idesc0 | (j & 1), (it > it0 || j > 0) ? 1u : 0u);
                    tc_commit_pair(empty0 + 8 * s, leader);
                }
                __syncwarp();
                eslot ^= 4;
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            if (elect_one()) tc_commit_pair(tmem_full, leader);      // also arrives after an abort
            __syncwarp();
        }
    } else {
        const bool ok = mbar_wait(tmem_full, 0, &abort_flag, P.status, 3);
        tc_fence_after();
        run = __all_sync(0xFFFFFFFFu, ok && !abort_flag);      // the warp reads tensor memory together
        if (run) {
            uint32_t v[32];                    // a lane: one row, 32 columns; those past HC are read, never used
            tmem_ld32(tmem_base + ((uint32_t)(quad * 32) << 16) + half * HC, v);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int col = half * HC + 4 * q, owner = owner_of(col);
                if (4 * q < HC && col < n)
                    st_cluster_v4(map_to_cta(smem_u32(parts + slice * part_bytes(BN, S)) + (col - owner * CW) * BM * 4 + (quad * 32 + lane) * 16,
                                             2 * owner + rank),
                                  v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
        }
        tc_fence_before();
    }
    // the partial tiles have arrived; also: nobody leaves while a peer may still signal its barriers or read its operands
    __syncthreads();
    cluster_sync_all();
    if (warp >= 2 && run && mrow < P.ms) {
        const float bias = P.bias ? load_bias<OutT>(P, mrow + lane) : 0.f;
        const int c0 = half * HC;
        // columns of other pairs read the first 16 bytes instead, so that no load waits for a branch
        const uint32_t from = smem_u32(parts) + (quad * 32 + lane) * 16;
        float sum[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[i] = -0.f;            // plus x: x, whatever its sign
        for (int p = 0; p < S; ++p) {
            uint4 o[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int col = c0 + 4 * q;
                const bool mine = 4 * q < HC && col < n && owner_of(col) == slice;
                o[q] = ld_shared_v4(from + p * part_bytes(BN, S) + (mine ? (col - slice * CW) * BM * 4 : 0));
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                sum[4 * q] += __uint_as_float(o[q].x);
                sum[4 * q + 1] += __uint_as_float(o[q].y);
                sum[4 * q + 2] += __uint_as_float(o[q].z);
                sum[4 * q + 3] += __uint_as_float(o[q].w);
            }
        }
        // this warp's columns, four a branch (a condition for each took 0.1 us more); a store: 32 features of a token
        OutT *dst = static_cast<OutT *>(P.out) + c0 * P.ld_out + mrow + lane;
        const int first = max(slice * CW, c0) - c0, last = min(min((slice + 1) * CW, n), c0 + HC) - c0;
#pragma unroll
        for (int q = 0; q < 8; ++q, dst += 4 * P.ld_out)
            if (4 * q >= first && 4 * q < last) {
                OutT *d = dst;
#pragma unroll
                for (int i = 0; i < 4; ++i, d += P.ld_out)
                    if (4 * q + i < last) *d = to_out<OutT>(sum[4 * q + i] + bias);
            }
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------
// Two-CTA form of the weight-gradient GEMM: D (ms x n, fp32) += A_sparse (ms x k) * B (k x n, stored row-major).
// ------------------------------------------------------------------------------------------------
// Tiles of 256 sparse rows x 256 dense columns per CTA pair (M = 256, N = 256 per instruction); a CTA stages its 128
// rows of A (16 KB), its 128 columns of B as two 64-column boxes of 128 K-rows (32 KB) and 2 KB of metadata per K
// step of 128: 50 KB for 8.4 dense-equivalent MFLOP, four stages.  K is cut into slices (work unit = tile x slice)
// so that the units fill the pairs; every unit adds its partial product with fp32 reductions in L2.  One
// accumulator of 256 columns per CTA: a pair that owns more than one unit drains it before the next unit's MMAs.
//
// Epilogue: tensor memory -> shared memory -> TMA reductions of 16 rows x 32 columns.  Its cost is exposed where a pair has one unit
// (nothing is left to multiply): under 3 us for a few tiles, 7 of 41 with all pairs writing at once (ms 3072, n 768, k 16384, by a
// build without it).  red.global.add.v4 from the registers, 32 rows of 16 bytes an instruction, took 4 us even for one tile (64-byte
// rows: 0.6 us more than 128-byte ones).  us, before -> now, one unit per pair: ms 512, n 256, k 256 9.5 -> 7.8; ms 768, n 768, k 8192
// 15.3 -> 11.8; ms 3072, n 768, k 8192 / 16384 24.6 -> 21.3 / 40.5 -> 37.4; several units (outputs of more tiles than pairs, or given
// slices): ms 3072, n 3072, k 2048 / 8192 31.4 -> 25.4 / 80.6 -> 71.6; ms 4096, n 4096, k 2048 67.2 -> 49.3; ms 512, n 512, k 16384 in
// 40 slices 29.6 -> 21.0.  Barriers at run-time addresses (see Ctl2) made no difference here.
// Where every pair has one unit at most (any output up to 74 tiles) the operand ring is idle by then and holds the whole tile,
// so that no chunk waits for another; a pair with more units stages chunk by chunk beside its ring, which is filling again.
namespace two {
constexpr int BN3 = 256;
constexpr int B3_BYTES = (BN3 / 2) * 256;                  // 128 columns x 128 K-rows x 2 bytes (float8: x 256 x 1)
constexpr int STAGES3 = 4;
constexpr int stage3_bytes(bool f8) { return A_STAGE_BYTES + B3_BYTES + e2_bytes(f8); }   // 51200, float8 53248
// Epilogue staging: a box is 16 rows x 32 columns, 128-byte rows in the 128-byte swizzle of the output's tensor map; a chunk is
// the two boxes of a warp's 32 rows.
constexpr int BOX3_BYTES = 16 * 128, CHUNKS3 = BN3 / 2 / 32;
constexpr int STAGING3 = 8 * BOX3_BYTES;                    // one box per epilogue warp
constexpr int smem3(bool f8) { return STAGES3 * stage3_bytes(f8) + STAGING3 + 1024; }
static_assert(8 * CHUNKS3 * 2 * BOX3_BYTES <= STAGES3 * stage3_bytes(false), "an idle operand ring holds a whole tile");
static_assert(stage3_bytes(false) % 1024 == 0 && stage3_bytes(true) % 1024 == 0, "stages must keep the 1024-byte swizzle alignment");
static_assert(smem3(true) <= SMEM_LIMIT, "shared memory budget");
}  // namespace two

// Float8 (F8): both operands K-major (B stored (n, k)), K step 256, the accumulator times the product of the operands' scales.
template <bool A_MN, bool F8>
__global__ void __launch_bounds__(320, 1)
spmm_pair_acc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const __grid_constant__ CUtensorMap map_e, const __grid_constant__ CUtensorMap map_d, SpmmParams P, SumsParams sums) {
    using namespace two;
    static_assert(!(A_MN && F8), "8-bit operands are K-major");
    constexpr int BN = BN3;
    constexpr int STAGES = STAGES3, STAGE3_BYTES = stage3_bytes(F8), KE = F8 ? 256 : 128;
    constexpr int OFF_B = A_STAGE_BYTES, OFF_E = OFF_B + B3_BYTES;
    constexpr int KSTEPS = 4;
    constexpr uint32_t TMEM_COLS = 512;
    constexpr int E_COL0 = BN, E_SLOT = F8 ? 8 : 4;       // one accumulator, then two metadata slots

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t bars[2 * STAGES + 2];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int n_tiles_n = (int)((P.n + BN - 1) / BN);
    const int n_tiles_m = (int)((P.ms + 2 * BM - 1) / (2 * BM));      // as in spmm_pair_kernel
    const int n_tiles = n_tiles_n * n_tiles_m;
    const int n_units = n_tiles * P.k_splits;     // unit u = (tile u % n_tiles, K slice u / n_tiles)
    const int k_iters = (int)((P.k + KE - 1) / KE);

    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[STAGES]);
    const uint32_t tmem_full = smem_u32(&bars[2 * STAGES]), tmem_empty = smem_u32(&bars[2 * STAGES + 1]);

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(tmem_full, 1);
        mbar_init(tmem_empty, 16);            // used in the leader only: eight epilogue warps of each CTA
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(&tmem_base_smem), TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;
    chain_enter();

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer (one per CTA)
        if (lane == 0) {
            int g = 0;
            bool ok = true;
            constexpr uint32_t cta_tx = STAGE3_BYTES;
            for (int unit = pair; unit < n_units && ok; unit += n_pairs) {
                const int tile = unit % n_tiles, ks = unit / n_tiles;
                const int it0 = (int)((int64_t)ks * k_iters / P.k_splits), it1 = (int)((int64_t)(ks + 1) * k_iters / P.k_splits);
                const int mblk = (tile % n_tiles_m) * 2 + (int)rank;
                const int mrow = mblk * BM;
                const int bcol = (tile / n_tiles_m) * BN + (int)rank * (BN / 2);
                for (int it = it0; it < it1; ++it, ++g) {
                    const int s = g % STAGES;
                    const uint32_t ph = (g / STAGES) & 1;
                    if (g >= STAGES && !mbar_wait(empty0 + 8 * s, ph ^ 1, &abort_flag, P.status, 1)) { ok = false; break; }
                    const uint32_t sa = smem_u32(smem + (size_t)s * STAGE3_BYTES);
                    const uint32_t sb = sa + OFF_B;
                    const uint32_t full_leader = map_to_cta(full0 + 8 * s, 0);
                    if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * cta_tx);
                    if constexpr (!A_MN) {
                        tma_load_2d_pair(sa, &map_a, it * (KE / 2), mrow, full_leader);
                    } else {
                        tma_load_columns_pair(sa, &map_a, it * 64, mrow / 64, full_leader);
                    }
                    tma_load_2d_pair(sa + OFF_E, &map_e, 0, (int)(((int64_t)mblk * P.k_atoms + it * (F8 ? 2 : 1)) * 2), full_leader);
                    // this CTA's 128 columns of B, 32 KB: one request for two columns of 128 bytes (float8: of K; 16 bits: 64 columns x 128
                    // K-rows each), two where the operand's columns are not whole ones (see make_map_columns)
                    if constexpr (F8) {
                        tma_load_columns_pair(sb, &map_b, bcol, 2 * it, full_leader);
                    } else if (P.whole_columns) {
                        tma_load_columns_pair(sb, &map_b, it * 128, bcol / 64, full_leader);
                    } else {
                        tma_load_2d_pair(sb, &map_b, bcol, it * 128, full_leader);
                        tma_load_2d_pair(sb + 16384, &map_b, bcol + 64, it * 128, full_leader);
                    }
                }
            }
            if (abort_flag && rank == 0) {
                for (int q = (g > STAGES ? g - STAGES : 0); q < g; ++q) {
                    const int s = q % STAGES;
                    const uint32_t ph = (q / STAGES) & 1;
                    for (uint32_t w = 0; w < WAIT_LIMIT; ++w)
                        if (mbar_try_wait(full0 + 8 * s, ph)) break;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer (leader CTA only)
        if (rank == 0) {                       // all lanes in step, one elected lane issues (as in spmm_pair_kernel)
            constexpr uint32_t A_LBO = A_MN ? 8192 : 16, A_KSTEP = A_MN ? 2048 : 32;
            const uint32_t idesc0 = P.idesc;   // M = 256, N = 256, operand majors set by the launcher
            const uint32_t smem0 = smem_u32(smem);
            // MN-major B: 64-column blocks 16384 bytes apart, 32 K-rows (4096 bytes) per MMA; K-major: 64 bytes per MMA, two K atoms
            const uint64_t adesc0 = make_desc(smem0, A_LBO, 1024, 2), bdesc0 = make_desc(smem0 + OFF_B, F8 ? 16 : 16384, 1024, 2);
            const uint64_t edesc0 = make_desc(smem0 + OFF_E, 16, 128, 0);
            int s = 0, tl = 0;
            uint32_t ph = 0, eslot = 0;
            bool ok = true;
            for (int unit = pair; unit < n_units && ok; unit += n_pairs, ++tl) {
                const int ks = unit / n_tiles;
                const int it0 = (int)((int64_t)ks * k_iters / P.k_splits), it1 = (int)((int64_t)(ks + 1) * k_iters / P.k_splits);
                // the epilogues of both CTAs must have drained the accumulator of the previous unit
                ok = mbar_wait_warp(tmem_empty, (tl & 1) ^ 1, &abort_flag, P.status, 4);
                for (int it = it0; it < it1 && ok; ++it) {
                    ok = mbar_wait_warp(full0 + 8 * s, ph, &abort_flag, P.status, 2);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t off = (uint32_t)s * (STAGE3_BYTES >> 4);
                    const uint64_t ad = adesc0 + off, bd = bdesc0 + off, ed = edesc0 + off;
                    const uint32_t e_cols = tmem_base + E_COL0 + eslot;
                    if (elect_one()) {
                        tc_cp_128x128b_pair(e_cols, ed);
                        if constexpr (F8) tc_cp_128x128b_pair(e_cols + 4, ed + (2048 >> 4));
#pragma unroll
                        for (int j = 0; j < KSTEPS; ++j)
                            mma_sp_pair_any<F8>(tmem_base, ad + j * (A_KSTEP >> 4),
                                                bd + (F8 ? (j >> 1) * (16384 >> 4) + (j & 1) * (64 >> 4) : j * (4096 >> 4)),
                                                e_cols + (F8 ? 2 * j : (j & ~1)), F8 ? idesc0 : idesc0 | (j & 1),
                                                (it > it0 || j > 0) ? 1u : 0u);
                        tc_commit_pair(empty0 + 8 * s);
                    }
                    __syncwarp();
                    eslot ^= E_SLOT;
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (elect_one()) tc_commit_pair(tmem_full);
                __syncwarp();
            }
        }
    } else {
        // ---------------------------------------------------------------- epilogue (warps 2..9 of both CTAs)
        const int quad = warp & 3, half = (warp - 2) >> 2;
        constexpr int HC = BN / 2;                     // 128 columns per warp
        const uint32_t empty_leader = map_to_cta(tmem_empty, 0);
        const float alpha = F8 ? alpha_of(P) : 1.f;
        const bool idle_ring = n_units <= n_pairs;     // this pair's only unit: the operand ring is free when it is complete
        const uint32_t stg = smem_u32(smem) + (idle_ring ? (warp - 2) * CHUNKS3 * 2 * BOX3_BYTES
                                                         : STAGES3 * STAGE3_BYTES + (warp - 2) * BOX3_BYTES);
        // The row sums that the compression left in parts (the bias gradient), while the first operands are on their way: 32 rows a
        // CTA and turn, in the order of sum_parts_kernel, through the staging that nothing uses yet.  As a launch of its own between
        // the compression and this kernel it took 2.6 us of a replayed step and 4 of an eager one (float8: 3.1, 8192 tokens, 768 -> 3072, 137.5 -> 134.4).
        if (sums.out) {
            float *const part = reinterpret_cast<float *>(smem + STAGES3 * STAGE3_BYTES);
            for (int64_t r = (int64_t)blockIdx.x * 32; r < P.ms; r += (int64_t)gridDim.x * 32) {
                part[(warp - 2) * 32 + lane] = sum_every_eighth(sums.parts + r + lane, sums.n_parts, P.ms, warp - 2);
                epilogue_bar_sync();
                if (warp == 2) {
                    float t = 0.f;
#pragma unroll
                    for (int w = 0; w < 8; ++w) t += part[w * 32 + lane];
                    sums.out[r + lane] = sums.accumulate ? sums.out[r + lane] + t : t;
                }
                epilogue_bar_sync();
            }
        }
        int tl = 0;
        for (int unit = pair; unit < n_units; unit += n_pairs, ++tl) {
            const int tile = unit % n_tiles;
            const int mrow = ((tile % n_tiles_m) * 2 + (int)rank) * BM + quad * 32;
            const int col0 = (tile / n_tiles_m) * BN + half * HC;
            const bool ok = mbar_wait(tmem_full, tl & 1, &abort_flag, P.status, 3);
            tc_fence_after();
            const bool run = __all_sync(0xFFFFFFFFu, ok && !abort_flag) && mrow < P.ms;
            if (run) {
                const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16) + half * HC;
#pragma unroll 1
                for (int c = 0; c < CHUNKS3; ++c) {
                    uint32_t v[32];
                    tmem_ld32(acc + c * 32, v);
                    tmem_ld_wait();
                    if constexpr (F8) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
                    }
                    const int x = col0 + c * 32;
                    // a lane's row of 128 bytes at `row`, its eight 16-byte pieces in the map's 128-byte swizzle
                    auto put = [&](uint32_t row) {
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            st_shared_v4(row + ((q ^ (lane & 7)) << 4), v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
                        fence_proxy_async();
                    };
                    if (idle_ring) {
                        const uint32_t buf = stg + c * 2 * BOX3_BYTES;
                        put(buf + lane * 128);
                        __syncwarp();
                        if (lane == 0 && x < P.n) {
                            tma_reduce_add_2d(&map_d, x, mrow, buf);
                            tma_reduce_add_2d(&map_d, x, mrow + 16, buf + BOX3_BYTES);
                            bulk_commit();
                        }
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (lane == 0) bulk_wait_read<0>();      // the box before has left
                            __syncwarp();
                            if ((lane >> 4) == h) put(stg + (lane & 15) * 128);
                            __syncwarp();
                            if (lane == 0 && x < P.n) {
                                tma_reduce_add_2d(&map_d, x, mrow + 16 * h, stg);
                                bulk_commit();
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(empty_leader);
        }
        if (lane == 0) bulk_wait_read<0>();            // shared memory stays until it has been read
        tc_fence_before();
    }
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------
// metadata: reference (reordered) layout -> tensor-core atom order
// ------------------------------------------------------------------------------------------------
// 16-bit types: atom = 128 rows x 128 logical columns = 2048 bytes, byte 16*L + 4*q + 2*h with
// L = 16*(r/16) + 8*(c%2) + r%8, q = (c/2)%4, h = (r/8)%2 for row r (inside the 128-row block) and
// 16-column metadata word c.  8-bit types: atom = 128 rows x 16 bytes, row-major.
template <int MB>
__global__ void meta_to_tc_kernel(const void *meta_api, uint8_t *e_tc, int64_t m, int64_t ncols, int64_t k_atoms) {
    chain_enter();
    const int64_t words_per_atom = 2048 / MB;
    const int64_t total = (m / 128) * k_atoms * words_per_atom;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int64_t atom = idx / words_per_atom;
    const int w = (int)(idx % words_per_atom);
    const int64_t mb = atom / k_atoms, kb = atom % k_atoms;
    int r, cw;  // row inside the block, metadata word inside the atom's 128 columns
    if constexpr (MB == 2) {
        const int L = w >> 3, q = (w >> 1) & 3, h = w & 1;
        r = 16 * (L >> 4) + 8 * h + (L & 7);
        cw = 2 * q + ((L >> 3) & 1);
    } else {
        r = w >> 2;
        cw = w & 3;
    }
    const int64_t c = kb * (MB == 2 ? 8 : 4) + cw;
    using MetaT = typename VecBytes<MB>::type;
    MetaT val = 0;
    if (c < ncols) val = static_cast<const MetaT *>(meta_api)[meta_offset<MB>(mb * 128 + r, c, m)];
    reinterpret_cast<MetaT *>(e_tc)[idx] = val;
}

CUtensorMapDataType tmap_dtype(int dt) {
    switch (dt) {
        case SP24_F16: return CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
        case SP24_BF16: return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        default: return CU_TENSOR_MAP_DATA_TYPE_UINT8;
    }
}

// cuTensorMapEncodeTiled is looked up through the runtime so that the library has no link-time
// dependency on the driver library (it must load on machines without a GPU driver).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
    static std::atomic<EncodeTiledFn> fn{nullptr};
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// Tensor map over rows of `cols` elements, row_bytes apart; a third dimension where depth is given: depth_bytes apart, box_depth of them a box.
int encode_map(CUtensorMap *map, CUtensorMapDataType type, const void *base, int64_t cols, int64_t rows, int64_t row_bytes, uint32_t box_cols,
               uint32_t box_rows, CUtensorMapSwizzle swizzle, int64_t depth = 0, int64_t depth_bytes = 0, uint32_t box_depth = 0) {
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)depth};
    const cuuint64_t strides[2] = {(cuuint64_t)row_bytes, (cuuint64_t)depth_bytes};
    const cuuint32_t box[3] = {box_cols, box_rows, box_depth};
    const cuuint32_t estr[3] = {1, 1, 1};
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return runtime_error();
    CUresult r = CUDA_SUCCESS;
    for (int attempt = 0; attempt < 2; ++attempt) {
        r = encode(map, type, depth ? 3 : 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_ERROR_INVALID_CONTEXT) break;
        // a host thread that has made no runtime call yet (an autograd worker) has no current context for this
        // driver entry point: let the runtime bind the primary context, then encode again
        cudaFree(nullptr);
    }
    if (r != CUDA_SUCCESS && getenv("SP24_DEBUG"))
        fprintf(stderr, "sparse24_b200: cuTensorMapEncodeTiled failed (%d): base %p rows %lld cols %lld pitch %lld box %u x %u\n",
                (int)r, base, (long long)rows, (long long)cols, (long long)row_bytes, box_cols, box_rows);
    return r == CUDA_SUCCESS ? SP24_OK : SP24_ERR_CUDA;
}

// Operand (rows, cols) with leading dimension ld (elements), 128-byte swizzle.
int make_map(CUtensorMap *map, const void *base, int dt, int64_t rows, int64_t cols, int64_t ld, uint32_t box_cols,
             uint32_t box_rows) {
    return encode_map(map, tmap_dtype(dt), base, cols, rows, ld * dtype_size(dt), box_cols, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

// The same operand as columns of 128 bytes, two a box: one request of an SM's copy engine instead of two, each of which holds the next one up
// (a K step is bound by the requests' latency).  us a launch, two boxes -> one: ms 4096, k 4096, n 16 / 64 / 256 / 2043 7.7 / 13.4 /
// 14.0 / 28.0 -> 7.3 / 12.2 / 13.0 / 27.3; ms 768, n 8192: k 2304 (column-major A) 20.2 -> 18.2, k 3072 23.3 -> 22.0; weight gradient
// ms 2304, n 768, k 8192 20.8 -> 19.5; K of 768, which the epilogue bounds, 0 - 3 %.  cols must fill whole columns: a last one reaching past
// them would read the next row.  An operand of an odd number of columns gets zeros for the second half of its last box.
int make_map_columns(CUtensorMap *map, const void *base, int dt, int64_t rows, int64_t cols, int64_t ld, uint32_t box_rows) {
    const int64_t es = dtype_size(dt), w = 128 / es;
    return encode_map(map, tmap_dtype(dt), base, w, rows, ld * es, (uint32_t)w, box_rows, CU_TENSOR_MAP_SWIZZLE_128B, cols / w, 128, 2);
}

// SP24_SPMM_PAIR=0 in the environment keeps every GEMM on the single-CTA kernels (read once per process)
bool pair_kernels_enabled() {
    static const bool enabled = [] {
        const char *env = getenv("SP24_SPMM_PAIR");
        return !(env && atoi(env) == 0);
    }();
    return enabled;
}

int sm_count_cached() { return sm_count(); }

template <int BN, bool F8, bool A_MN, bool B_MN, bool TRANS, typename OutT>
int launch_spmm(const CUtensorMap &ma, const CUtensorMap &mb, SpmmParams P, cudaStream_t st) {
    using Cfg = SpmmCfg<BN, F8, TRANS, OutT>;
    auto kern = P.activation ? spmm_kernel<BN, F8, A_MN, B_MN, TRANS, OutT, true>
                             : spmm_kernel<BN, F8, A_MN, B_MN, TRANS, OutT, false>;
    static std::atomic<bool> attr_set[64][2];
    int dev = 0;
    cudaGetDevice(&dev);
    const int which = P.activation ? 1 : 0;
    if (dev >= 0 && dev < 64 && !attr_set[dev][which]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM) != cudaSuccess)
            return runtime_error();
        attr_set[dev][which] = true;
    }
    P.idesc |= (uint32_t)(BN >> 3) << 17;
    const int64_t tiles = ((P.n + BN - 1) / BN) * ((P.ms / BM + P.mblk_per_tile - 1) / P.mblk_per_tile) * P.k_splits;
    const int sms = sm_count_cached();
    launch_chained(st, kern, (unsigned)(tiles < sms ? tiles : sms), 320, Cfg::SMEM, ma, mb, P);
    return launch_status();
}

// Metadata atoms as a 2-D tensor for TMA: rows of 1024 bytes (256 int32), two rows per 2048-byte atom, no swizzle.
int make_map_e(CUtensorMap *map, const void *e_tc, int64_t n_atoms, int atoms_per_box = 1) {
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_INT32, e_tc, 256, 2 * n_atoms, 1024, 256, 2 * atoms_per_box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

template <bool A_MN, typename OutT, int EPI = EPI_PLAIN, bool F8 = false>
int launch_spmm_pair(const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &me, SpmmParams P, cudaStream_t st) {
    auto kern = spmm_pair_kernel<A_MN, OutT, EPI, F8>;
    constexpr int SMEM_MAX = two::SMEM_LIMIT;
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        // the kernel takes its dynamic shared memory as it comes: it starts on 1024 bytes only behind none, or whole kilobytes, of
        // static shared memory
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return runtime_error();
        if (fa.sharedSizeBytes % 1024) return SP24_ERR_ALIGN;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX) != cudaSuccess)
            return runtime_error();
        attr_set[dev] = true;
    }
    // M = 256 over the CTA pair, N = bn
    P.idesc = (P.idesc & ~(0x1Fu << 24)) | ((uint32_t)(256 >> 4) << 24) | ((uint32_t)(P.bn >> 3) << 17);
    P.stages = two::stages2(F8, P.bn);
    const int64_t tiles = ((P.n + P.bn - 1) / P.bn) * ((P.ms + 255) / 256);
    const int64_t pairs_max = sm_count_cached() / 2;
    const unsigned pairs = (unsigned)(tiles < pairs_max ? tiles : pairs_max);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * pairs, 1, 1);
    cfg.blockDim = dim3(320, 1, 1);
    cfg.dynamicSmemBytes = two::smem2(F8, P.bn);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_chained
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (cudaLaunchKernelEx(&cfg, kern, ma, mb, me, P) != cudaSuccess) return runtime_error();
    return launch_status();
}

// K slices of the weight gradient on CTA pairs: as many as idle pairs allow.
int64_t pair_slices(int64_t ms, int64_t n, int64_t k, int k_step, int sms) {
    const int64_t tiles = ((n + two::BN3 - 1) / two::BN3) * ((ms + 255) / 256), k_iters = (k + k_step - 1) / k_step;
    return std::max<int64_t>(1, std::min(sms / 2 / tiles, k_iters));
}

template <bool A_MN, bool F8 = false>
int launch_spmm_pair_acc(const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &me, const CUtensorMap &md, SpmmParams P,
                         const SumsParams &sums, int k_splits, cudaStream_t st) {
    auto kern = spmm_pair_acc_kernel<A_MN, F8>;
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, two::smem3(F8)) != cudaSuccess)
            return runtime_error();
        attr_set[dev] = true;
    }
    // M = 256 over the CTA pair, N = 256
    P.idesc = (P.idesc & ~(0x1Fu << 24)) | ((uint32_t)(256 >> 4) << 24) | ((uint32_t)(two::BN3 >> 3) << 17);
    const int64_t tiles = ((P.n + two::BN3 - 1) / two::BN3) * ((P.ms + 255) / 256);
    const int64_t pairs_max = sm_count_cached() / 2;
    constexpr int KE = F8 ? 256 : 128;
    const int64_t splits = k_splits ? std::min<int64_t>(k_splits, (P.k + KE - 1) / KE) : pair_slices(P.ms, P.n, P.k, KE, sm_count_cached());
    P.k_splits = (int)splits;
    const int64_t units = tiles * splits;
    const unsigned pairs = (unsigned)(units < pairs_max ? units : pairs_max);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * pairs, 1, 1);
    cfg.blockDim = dim3(320, 1, 1);
    cfg.dynamicSmemBytes = two::smem3(F8);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_chained
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (cudaLaunchKernelEx(&cfg, kern, ma, mb, me, md, P, sums) != cudaSuccess) return runtime_error();
    return launch_status();
}

// spmm_split_kernel: a cluster of 2 * slices CTAs a tile.
void split_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute (&attr)[2], int slices, int64_t tiles, int smem, cudaStream_t st) {
    cfg.gridDim = dim3((unsigned)(2 * slices * tiles), 1, 1);
    cfg.blockDim = dim3(320, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * slices;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_chained
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
}

// Whether the split kernel can run on the current device at all, worked out on the first call there.
template <bool A_MN, typename OutT> bool split_runs() {
    static bool runs[64], done[64];
    static std::mutex mu;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) runtime_error();
    if (dev < 0 || dev >= 64) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (!done[dev]) {
        auto kern = spmm_split_kernel<A_MN, OutT>;
        cudaFuncAttributes fa{};
        // dynamic shared memory on 1024 bytes, as in launch_spmm_pair
        bool ok = cudaFuncGetAttributes(&fa, kern) == cudaSuccess && fa.sharedSizeBytes % 1024 == 0 &&
                  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, two::SMEM_LIMIT) == cudaSuccess;
        for (int s = 2; s <= two::SPLIT_MAX && ok; ++s) {
            cudaLaunchConfig_t cfg{};
            cudaLaunchAttribute attr[2];
            split_config(cfg, attr, s, 1, two::split_smem(two::BN_SPLIT, s), nullptr);
            int n = 0;
            ok = cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0;
        }
        if (!ok) runtime_error();
        runs[dev] = ok;
        done[dev] = true;
    }
    return runs[dev];
}

// Clusters of this many CTAs, one CTA per SM, that a device of eight GPCs holds at once however its SMs (an even number in each) are
// spread over them: a GPC leaves at most cluster - 2 of its SMs over.  On 148 SMs 33 clusters of four, 20 of six, 13 of eight; the
// device measured here holds 33, 22 and 15.
constexpr int64_t clusters_for_sure(int64_t cluster, int64_t sms) {
    const int64_t used = sms - 8 * (cluster - 2);
    return used > 0 ? (used + cluster - 1) / cluster : 0;
}
static_assert(clusters_for_sure(4, 148) == 33 && clusters_for_sure(6, 148) == 20 && clusters_for_sure(8, 148) == 13, "");

// Slices of K for few columns (1: the pair kernel takes the call): the most that leave every tile a cluster at once, from eight K
// steps (two a slice) on.  They decide the order of the sums, so the rule knows sizes and the number of SMs only: the same bits on every
// device with as many.  us a replayed launch, pair kernel -> here:
//   ms 4096, k 4096: n 1 11.8 -> 6.8, n 33 12.1 -> 7.2; ms 512, k 4096, n 16 11.7 -> 5.6; ms 2304, k 3072, n 16 9.5 -> 5.5
//   ms 1024, k 1024: n 1 5.0 -> 3.5, n 33 5.3 -> 4.0; ms 4096, k 1024, n 16 5.1 -> 4.7; ms 5632, k 4096, n 16 11.8 -> 8.1
// Shorter K keeps the order of sums that the pair and single-CTA kernels share bit for bit; slices would gain 0.1 - 0.6 us there
// (ms 512, n 16, k 512 4.1 -> 3.5).
int pick_slices(int64_t ms, int64_t n, int64_t k, int sms) {
    if (n > two::SPLIT_N || k <= two::SPLIT_K) return 1;
    const int64_t tiles = (ms + 255) / 256;
    for (int s = two::SPLIT_MAX; s >= 2; --s)
        if (tiles <= clusters_for_sure(2 * s, sms)) return s;
    return 1;
}
int split_bn(int64_t n) { return n <= 32 ? 32 : (n <= 48 ? 48 : 64); }

template <bool A_MN, typename OutT>
int launch_spmm_split(const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &me, SpmmParams P, cudaStream_t st) {
    P.idesc = (P.idesc & ~(0x1Fu << 24)) | ((uint32_t)(256 >> 4) << 24) | ((uint32_t)(P.bn >> 3) << 17);
    P.stages = two::split_stages(P.bn, P.k_splits);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    split_config(cfg, attr, P.k_splits, (P.ms + 255) / 256, two::split_smem(P.bn, P.k_splits), st);
    if (cudaLaunchKernelEx(&cfg, spmm_split_kernel<A_MN, OutT>, ma, mb, me, P) != cudaSuccess) return runtime_error();
    return launch_status();
}

// Tile shape: wide / tall tiles stage fewer operand bytes per output, small ones fill the SMs more evenly.
// Cost model per candidate (BN, row blocks per tile): rounds of tiles per CTA x bytes staged per K iteration.
void pick_tile(int64_t ms, int64_t n, int sm_count, int &bn_out, int &mpt_out) {
    const int cand_bn[2] = {192, 128};
    double best_cost = 1e300;
    for (int mpt = 2; mpt >= 1; --mpt) {
        for (int i = 0; i < 2; ++i) {
            const int bn = cand_bn[i];
            const int64_t tiles = ((n + bn - 1) / bn) * ((ms / BM + mpt - 1) / mpt);
            const double rounds = (double)((tiles + sm_count - 1) / sm_count);
            const double cost = rounds * (mpt * (A_STAGE_BYTES + 2048) + bn * 256);
            if (cost < best_cost) { best_cost = cost; bn_out = bn; mpt_out = mpt; }
        }
    }
}

// Columns of a CTA-pair tile: the candidate with the lowest (rounds of tiles per CTA pair) x (bytes staged per CTA and K step).
// The K loop is bound by the operand fill from L2 (about 14 TB/s over the chip whatever the width), so a wide tile pays only
// where it does not leave the last round nearly empty.  The number of stages is left out: one stage of five is worth 3 % at most,
// and no other width makes up for it with the rounds it costs.  fp16, us, at 192 columns -> at the width taken:
//   ms 4096, n 2043, k 4096: 39.3 -> 31.7 (240 columns: two rounds instead of three)
//   ms 3072, n 16384, k 768: 52.2 -> 49.5 (224); ms 768, n 16384, k 3072: 44.5 -> 42.5 (224)
//   ms 768, n 5000, k 1024: 11.8 -> 9.2 (224)
// Few columns: the narrowest tile that still takes one round; single-CTA kernel -> here:
//   ms 4096, k 4096: n 16 19.8 -> 13.2, n 256 20.8 -> 14.6, n 512 21.7 -> 15.5, n 768 24.0 -> 16.2; ms 768, k 3072, n 512 16.4 -> 11.5
// (the single-CTA kernel was never faster, so it keeps what pair_takes_rows leaves it and the other layouts).
// The fused epilogues hold up to 192 columns in registers and take them in chunks of 16 per half tile.  8-bit operands: with
// cta_group::2 and M = 256, kind::f8f6f4 takes N in multiples of 32 (kind::f16, sparse: of 16; the ranges of CUTLASS's
// SM100_MMA_F8F6F4_2x1SM_SS_SPARSE and SM100_MMA_F16BF16_2x1SM_SS_SPARSE).
int pick_pair_bn(int64_t ms, int64_t n, bool plain, bool f8, int sms) {
    const int step = plain && !f8 ? 16 : 32, widest = !plain ? 192 : (f8 ? 224 : two::BN2_MAX);
    const int64_t pairs = sms / 2;
    int best = widest;
    int64_t best_cost = INT64_MAX;
    for (int bn = widest; bn >= two::BN2_MIN; bn -= step) {
        const int64_t tiles = ((n + bn - 1) / bn) * ((ms + 255) / 256);
        const int64_t cost = ((tiles + pairs - 1) / pairs) * two::stage2_bytes(f8, bn);
        if (cost < best_cost) { best_cost = cost; best = bn; }
    }
    return best;
}

// The single-CTA tile of a float8 product with 16-bit results: narrow, since beside the 16-bit staging buffer a wide tile's stages do not
// fit twice.
void pick_f8_tile(int64_t ms, int64_t n, int sms, int &bn, int &mpt) {
    bn = 128;
    mpt = ((n + 127) / 128) * ((ms / BM + 1) / 2) >= sms ? 2 : 1;
}

// Whether the CTA-pair kernel takes an operand of whole or half 256-row blocks.  A half-empty last block costs its MMAs, not its stores, and
// over a map of 9 odd row counts (128 .. 2944), 12 widths (384 .. 16384) and K from 128 to 3072 pairs are faster or alike, us, single CTAs /
// pairs: 1152 x 12000, k 256 16.3 / 12.2; 384 x 12000, k 512 10.3 / 8.0; float8 384 x 12000, k 384 11.7 / 7.6.  Two exceptions.  The one
// block there is is half empty and many tiles are to be written: ms 128, n 16384, k 128 5.1 / 5.8, k 3072 19.6 / 20.5; n 8192 5.3 / 5.5.
// And 16-bit operands of one whole K step whose 128 x 128 tiles fill one round of single CTAs by two thirds or more: n * ms of 1.6 to 2.4
// million, over 9 odd row counts 0 - 12 % slower on pairs, e.g. 384 x 6000 4.3 / 4.8, 896 x 2510 4.29 / 4.64, 2176 x 1011 4.22 / 4.45;
// with fewer tiles or a second round pairs gain again (384 x 2395 4.13 / 3.97, 896 x 2790 4.96 / 4.70).
bool pair_takes_rows(int64_t ms, int64_t n, int64_t k, bool f8, int sms) {
    if (ms % 256 == 0) return true;
    if (!f8 && k == 128) {
        const int64_t tiles = (ms / BM) * ((n + 127) / 128);
        if (tiles <= sms && 3 * tiles >= 2 * sms) return false;
    }
    return ms > BM || n <= 8192;
}

// Row blocks of a tile and K slices of the 16-bit weight gradient on single CTAs.
int single_row_blocks(int64_t ms) { return ms >= 256 ? 2 : 1; }
int64_t single_slices(int64_t ms, int64_t n, int64_t k, int sms) {
    const int64_t bn = n >= 192 ? 192 : 128, mpt = single_row_blocks(ms), k_iters = (k + 127) / 128;
    const int64_t tiles = ((n + bn - 1) / bn) * ((ms / BM + mpt - 1) / mpt);
    return std::max<int64_t>(1, std::min(sms / tiles, k_iters));
}

// Tile and K slices of the float8 weight gradient (added to out with float32 reductions).  At most two slices: two addends on a
// zeroed buffer give the same bits in either order, three do not.  Among these, the fewest bytes staged per CTA.
// ms 3072, n 768, k 8192: 256 x 128 tiles in two slices (144 units) instead of 256 x 192 in three.
void pick_f8_accumulate(int64_t ms, int64_t n, int64_t k, int sms, int &bn_out, int &mpt_out, int &splits_out) {
    const int64_t k_iters = (k + 255) / 256;
    int64_t best = INT64_MAX;
    for (int bn : {192, 128})
        for (int mpt = ms >= 256 ? 2 : 1; mpt >= 1; --mpt)
            for (int splits = 1; splits <= (k_iters > 1 ? 2 : 1); ++splits) {
                const int64_t units = ((n + bn - 1) / bn) * ((ms / BM + mpt - 1) / mpt) * splits;
                const int64_t stage = (int64_t)mpt * (A_STAGE_BYTES + 4096) + bn * 256;
                const int64_t cost = ((units + sms - 1) / sms) * (((k_iters + splits - 1) / splits) * stage);
                if (cost < best) { best = cost; bn_out = bn; mpt_out = mpt; splits_out = splits; }
            }
}

template <bool F8, bool A_MN, bool B_MN, bool TRANS, typename OutT>
int dispatch_bn(int bn, const void *b, int dtype, int64_t n, int64_t k, int64_t ld_b, const CUtensorMap &ma,
                const SpmmParams &P, cudaStream_t st) {
    CUtensorMap mb;
    int rc;
    if (!B_MN) rc = make_map(&mb, b, dtype, n, k, ld_b, F8 ? 128 : 64, (uint32_t)bn);
    else rc = make_map(&mb, b, dtype, k, n, ld_b, 64, 128);
    if (rc) return rc;
    if (bn == 192) return launch_spmm<192, F8, A_MN, B_MN, TRANS, OutT>(ma, mb, P, st);
    return launch_spmm<128, F8, A_MN, B_MN, TRANS, OutT>(ma, mb, P, st);
}

}  // namespace
}  // namespace sp24

using namespace sp24;

extern "C" int sp24_meta_to_tc(const void *meta, int meta_itemsize, int64_t m, int64_t k, void *e_tc, void *stream) {
    if (!meta || !e_tc) return SP24_ERR_ARG;
    if (meta_itemsize != 2 && meta_itemsize != 4) return SP24_ERR_DTYPE;
    if (m <= 0 || k <= 0 || m % 128 || k % (meta_itemsize == 2 ? 64 : 128)) return SP24_ERR_SHAPE;
    if (!aligned16(meta) || !aligned16(e_tc)) return SP24_ERR_ALIGN;
    if (int rc = check_device()) return rc;
    const int64_t k_atoms = (k + 127) / 128;
    const int64_t total = (m / 128) * k_atoms * (2048 / meta_itemsize);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (meta_itemsize == 2)
        launch_chained(st, meta_to_tc_kernel<2>, blocks, 256, 0, meta, static_cast<uint8_t *>(e_tc), m, k / 16, k_atoms);
    else
        launch_chained(st, meta_to_tc_kernel<4>, blocks, 256, 0, meta, static_cast<uint8_t *>(e_tc), m, k / 32, k_atoms);
    return launch_status();
}

extern "C" int64_t sp24_meta_tc_bytes(int64_t m, int64_t k) {
    if (m <= 0 || k <= 0) return 0;
    return ((m + 127) / 128) * ((k + 127) / 128) * 2048;
}

// Argument checks of sp24_spmm (everything except the metadata pointer); no CUDA call.
static int validate_spmm_args(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, int64_t ms, int64_t k,
                              const void *b, int b_mn_major, int64_t ld_b, int64_t n, const void *out, int out_dtype,
                              int trans_out, int64_t ld_out, const void *bias, int activation) {
    if (!a_packed || !b || !out) return SP24_ERR_ARG;
    const bool i8 = dtype == SP24_I8;
    const bool f8 = dtype == SP24_E4M3 || dtype == SP24_E5M2 || i8;   // 8-bit operand geometry
    if (!f8 && dtype != SP24_F16 && dtype != SP24_BF16) return SP24_ERR_DTYPE;
    if (i8 ? out_dtype != SP24_I32 : (f8 ? out_dtype != SP24_F32 : out_dtype != dtype)) return SP24_ERR_DTYPE;
    if (f8 && (a_mn_major || b_mn_major)) return SP24_ERR_DTYPE;  // 8-bit operands are K-major only
    if (i8 && (bias || activation)) return SP24_ERR_ARG;          // integer GEMM: plain product only
    if (activation < 0 || activation > 3) return SP24_ERR_ARG;
    const int esz = f8 ? 1 : 2;
    if (ms <= 0 || n <= 0 || k <= 0 || ms % 128 || k % (f8 ? 128 : 64)) return SP24_ERR_SHAPE;
    // n is free when B is stored (n, k) and the output (n, ms): rows past n are zero-filled on load and skipped
    // on store.  The other layouts have n as a contiguous extent, which must keep 16-byte row pitches.
    if ((b_mn_major || !trans_out) && n % 8) return SP24_ERR_SHAPE;
    const int64_t a_inner = a_mn_major ? ms : k / 2, b_inner = b_mn_major ? n : k, o_inner = trans_out ? ms : n;
    if (ld_a < a_inner || (ld_a * esz) % 16 || ld_b < b_inner || (ld_b * esz) % 16 || ld_out < o_inner) return SP24_ERR_STRIDE;
    if ((ld_out * dtype_size(out_dtype)) % 16) return SP24_ERR_STRIDE;
    if (!aligned16(a_packed) || !aligned16(b) || !aligned16(out)) return SP24_ERR_ALIGN;
    return SP24_OK;
}

static int spmm_impl(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, const void *e_tc, int64_t ms,
                     int64_t k, const void *b, int b_mn_major, int64_t ld_b, int64_t n, void *out, int out_dtype,
                     int trans_out, int64_t ld_out, const void *bias, int activation, float alpha, int *status, void *stream,
                     int bias_f32 = 0, int epi = EPI_PLAIN, void *aux = nullptr, int64_t ld_aux = 0) {
    if (!e_tc) return SP24_ERR_ARG;
    if (int rc = validate_spmm_args(a_packed, dtype, a_mn_major, ld_a, ms, k, b, b_mn_major, ld_b, n, out, out_dtype,
                                    trans_out, ld_out, bias, activation))
        return rc;
    if (!aligned16(e_tc)) return SP24_ERR_ALIGN;
    const bool i8 = dtype == SP24_I8;
    const bool f8 = dtype == SP24_E4M3 || dtype == SP24_E5M2 || i8;   // 8-bit operand geometry
    // CTA-pair kernel: 16-bit types, token-major B and output, no activation; the fused MLP epilogues and the float32 bias exist in
    // that kernel only and for whole 256-row blocks
    const bool pair_layout = !f8 && !b_mn_major && trans_out && activation == 0, pair_ok = pair_layout && ms % 256 == 0;
    if (epi != EPI_PLAIN && (!pair_ok || !aux || ld_aux < ms || (ld_aux * 2) % 16 || !aligned16(aux))) return SP24_ERR_ARG;
    if (bias_f32 && !pair_ok) return SP24_ERR_ARG;
    if (int rc = check_device()) return rc;

    CUtensorMap map_a;
    int rc;

    SpmmParams P{};
    P.e_tc = e_tc; P.out = out; P.bias = bias; P.ms = ms; P.n = n; P.k = k; P.ld_out = ld_out;
    P.k_atoms = (k + 127) / 128; P.status = status; P.activation = activation;
    P.trace = nullptr;
    P.k_splits = 1;
    P.alpha = alpha;
    P.bias_f32 = bias_f32;
    P.aux = aux;
    P.ld_aux = ld_aux;
#ifdef SP24_TRACE_BUILD
    if (const char *env = getenv("SP24_SPMM_TRACE_PTR")) P.trace = reinterpret_cast<unsigned long long *>(strtoull(env, nullptr, 0));
#endif
    // operand format codes: f16 0 / bf16 1; e4m3 0 / e5m2 1; unsigned 0 / signed 1 for the integer kind
    const uint32_t fmt = (dtype == SP24_BF16 || dtype == SP24_E5M2 || i8) ? 1u : 0u;
    // sparse flag, accumulator format (fp32 = 1, int32 = 2), operand formats, operand majors, M = 128 (N is added
    // by the launcher)
    P.int8 = i8 ? 1 : 0;
    P.idesc = (1u << 2) | ((i8 ? 2u : 1u) << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(a_mn_major ? 1 : 0) << 15) |
              ((uint32_t)(b_mn_major ? 1 : 0) << 16) | ((uint32_t)(BM >> 4) << 24);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = sm_count_cached();
    bool pair_form = pair_layout && pair_takes_rows(ms, n, k, false, sms) && pair_kernels_enabled();
    if (epi != EPI_PLAIN || bias_f32) pair_form = true;      // checked above: these forms exist in the pair kernel only
    if (a_mn_major) rc = pair_form ? make_map_columns(&map_a, a_packed, dtype, k / 2, ms, ld_a, 64) : make_map(&map_a, a_packed, dtype, k / 2, ms, ld_a, 64, 64);
    else rc = make_map(&map_a, a_packed, dtype, ms, k / 2, ld_a, f8 ? 128 : 64, 128);
    if (rc) return rc;
    if (pair_form) {
        CUtensorMap map_b, map_e;
        P.bn = pick_pair_bn(ms, n, epi == EPI_PLAIN, false, sms);
        const int slices = epi == EPI_PLAIN && pair_kernels_enabled() ? pick_slices(ms, n, k, sms) : 1;
        if (slices > 1 && (out_dtype == SP24_F16 ? (a_mn_major ? split_runs<true, __half>() : split_runs<false, __half>())
                                                 : (a_mn_major ? split_runs<true, __nv_bfloat16>() : split_runs<false, __nv_bfloat16>()))) {
            P.k_splits = slices;
            P.bn = split_bn(n);
        }
        rc = make_map_columns(&map_b, b, dtype, n, k, ld_b, (uint32_t)P.bn / 2);
        if (rc) return rc;
        rc = make_map_e(&map_e, e_tc, (ms / 128) * P.k_atoms);
        if (rc) return rc;
        if (P.k_splits > 1)
            return out_dtype == SP24_F16 ? (a_mn_major ? launch_spmm_split<true, __half>(map_a, map_b, map_e, P, st)
                                                       : launch_spmm_split<false, __half>(map_a, map_b, map_e, P, st))
                                         : (a_mn_major ? launch_spmm_split<true, __nv_bfloat16>(map_a, map_b, map_e, P, st)
                                                       : launch_spmm_split<false, __nv_bfloat16>(map_a, map_b, map_e, P, st));
#define SP24_PAIR(EPI_) \
        do { \
            if (out_dtype == SP24_F16) \
                return a_mn_major ? launch_spmm_pair<true, __half, EPI_>(map_a, map_b, map_e, P, st) \
                                  : launch_spmm_pair<false, __half, EPI_>(map_a, map_b, map_e, P, st); \
            return a_mn_major ? launch_spmm_pair<true, __nv_bfloat16, EPI_>(map_a, map_b, map_e, P, st) \
                              : launch_spmm_pair<false, __nv_bfloat16, EPI_>(map_a, map_b, map_e, P, st); \
        } while (0)
        if (epi == EPI_PRE_GELU) SP24_PAIR(EPI_PRE_GELU);
        if (epi == EPI_DGELU) SP24_PAIR(EPI_DGELU);
        SP24_PAIR(EPI_PLAIN);
#undef SP24_PAIR
    }
    int bn = 128, mpt = 2;
    pick_tile(ms, n, sms, bn, mpt);
    P.mblk_per_tile = mpt;
#define SP24_GO(F8_, AMN_, BMN_, TR_, OT_) return dispatch_bn<F8_, AMN_, BMN_, TR_, OT_>(bn, b, dtype, n, k, ld_b, map_a, P, st)
    if (i8) {
        if (trans_out) SP24_GO(true, false, false, true, int32_t);
        SP24_GO(true, false, false, false, int32_t);
    }
    if (f8) {
        if (trans_out) SP24_GO(true, false, false, true, float);
        SP24_GO(true, false, false, false, float);
    }
    if (dtype == SP24_F16) {
        if (!a_mn_major && !b_mn_major) { if (trans_out) SP24_GO(false, false, false, true, __half); SP24_GO(false, false, false, false, __half); }
        if (a_mn_major && !b_mn_major) { if (trans_out) SP24_GO(false, true, false, true, __half); SP24_GO(false, true, false, false, __half); }
        if (!a_mn_major && b_mn_major) { if (trans_out) SP24_GO(false, false, true, true, __half); SP24_GO(false, false, true, false, __half); }
        if (trans_out) SP24_GO(false, true, true, true, __half);
        SP24_GO(false, true, true, false, __half);
    }
    if (!a_mn_major && !b_mn_major) { if (trans_out) SP24_GO(false, false, false, true, __nv_bfloat16); SP24_GO(false, false, false, false, __nv_bfloat16); }
    if (a_mn_major && !b_mn_major) { if (trans_out) SP24_GO(false, true, false, true, __nv_bfloat16); SP24_GO(false, true, false, false, __nv_bfloat16); }
    if (!a_mn_major && b_mn_major) { if (trans_out) SP24_GO(false, false, true, true, __nv_bfloat16); SP24_GO(false, false, true, false, __nv_bfloat16); }
    if (trans_out) SP24_GO(false, true, true, true, __nv_bfloat16);
    SP24_GO(false, true, true, false, __nv_bfloat16);
#undef SP24_GO
}


extern "C" int sp24_spmm(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, const void *e_tc, int64_t ms,
                         int64_t k, const void *b, int b_mn_major, int64_t ld_b, int64_t n, void *out, int out_dtype,
                         int trans_out, int64_t ld_out, const void *bias, int activation, int *status, void *stream) {
    return spmm_impl(a_packed, dtype, a_mn_major, ld_a, e_tc, ms, k, b, b_mn_major, ld_b, n, out, out_dtype, trans_out, ld_out,
                     bias, activation, 1.f, status, stream);
}

// The 16-bit GEMM of a transformer MLP with its neighbours fused into the epilogue (CTA-pair kernel): see the header.
extern "C" int sp24_spmm_mlp(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, const void *e_tc, int64_t ms,
                             int64_t k, const void *b, int64_t ld_b, int64_t n, void *out, int64_t ld_out, const void *bias,
                             int bias_is_f32, int epilogue, void *aux, int64_t ld_aux, int *status, void *stream) {
    if (dtype != SP24_F16 && dtype != SP24_BF16) return SP24_ERR_DTYPE;
    if (epilogue < 0 || epilogue > 2) return SP24_ERR_ARG;
    if (epilogue == EPI_DGELU && bias) return SP24_ERR_ARG;
    return spmm_impl(a_packed, dtype, a_mn_major, ld_a, e_tc, ms, k, b, 0, ld_b, n, out, dtype, 1, ld_out, bias, 0, 1.f, status,
                     stream, bias_is_f32 ? 1 : 0, epilogue, aux, ld_aux);
}

extern "C" int sp24_k_slices(int64_t ms, int64_t n, int64_t k, int sms) {
    if (ms <= 0 || ms % 128 || n <= 0 || k <= 0 || k % 64 || sms < 2) return 0;
    return pick_slices(ms, n, k, sms);
}

extern "C" int sp24_pair_tile_columns(int64_t ms, int64_t n, int form, int sms) {
    if (ms <= 0 || ms % 256 || n <= 0 || form < 0 || form > 2 || sms < 2) return 0;
    return pick_pair_bn(ms, n, form != 1, form == 2, sms);
}

// The GEMMs of a float8 layer whose scales stay on the device: D = alpha * (A_sparse * B) [+ float32 bias], alpha = the
// product of the operands' scales, worked out from their absolute maxima (sp24_absmax).
//   trans_out = 1: out (n, ms) in float32, float16 or bfloat16 (rounded once): the layer's output or input gradient
//   without a float32 copy.  16-bit outputs run on CTA pairs (see pair_takes_rows).
//   trans_out = 0: out (ms, n) float32 += alpha * A * B (no bias), K cut into up to two slices: the weight gradient.
static int spmm_f8_impl(const void *a_packed, int dtype, int64_t ld_a, const void *e_tc, int64_t ms, int64_t k, const void *b, int64_t ld_b,
                        int64_t n, void *out, int out_dtype, int trans_out, int64_t ld_out, const float *bias, const float *amax_a,
                        const float *amax_b, const SumsParams &sums, int *status, void *stream) {
    if (dtype != SP24_E4M3 && dtype != SP24_E5M2) return SP24_ERR_DTYPE;
    if (!e_tc || !amax_a || !amax_b || (!trans_out && bias)) return SP24_ERR_ARG;
    if (out_dtype != SP24_F32 && (!trans_out || (out_dtype != SP24_F16 && out_dtype != SP24_BF16))) return SP24_ERR_DTYPE;
    if (int rc = validate_spmm_args(a_packed, dtype, 0, ld_a, ms, k, b, 0, ld_b, n, out, SP24_F32, trans_out, ld_out, bias, 0)) return rc;
    if (!aligned16(e_tc) || (ld_out * dtype_size(out_dtype)) % 16) return SP24_ERR_ALIGN;
    if (int rc = check_device()) return rc;
    CUtensorMap map_a, map_b;
    if (int rc = make_map(&map_a, a_packed, dtype, ms, k / 2, ld_a, 128, 128)) return rc;
    SpmmParams P{};
    P.e_tc = e_tc; P.out = out; P.bias = bias; P.bias_f32 = 1; P.ms = ms; P.n = n; P.k = k; P.ld_out = ld_out;
    P.k_atoms = (k + 127) / 128; P.status = status; P.k_splits = 1; P.alpha = 1.f; P.amax_a = amax_a; P.amax_b = amax_b;
    const uint32_t fmt = dtype == SP24_E5M2 ? 1u : 0u;
    P.idesc = (1u << 2) | (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BM >> 4) << 24);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = sm_count_cached();
    if (trans_out && out_dtype != SP24_F32 && pair_takes_rows(ms, n, k, true, sms) && pair_kernels_enabled()) {
        CUtensorMap map_e;
        P.bn = pick_pair_bn(ms, n, true, true, sms);
        if (int rc = make_map_columns(&map_b, b, dtype, n, k, ld_b, (uint32_t)P.bn / 2)) return rc;
        if (int rc = make_map_e(&map_e, e_tc, (ms / 128) * P.k_atoms, 2)) return rc;
        return out_dtype == SP24_F16 ? launch_spmm_pair<false, __half, EPI_PLAIN, true>(map_a, map_b, map_e, P, st)
                                     : launch_spmm_pair<false, __nv_bfloat16, EPI_PLAIN, true>(map_a, map_b, map_e, P, st);
    }
    int bn = 128, mpt = 2;
    pick_tile(ms, n, sms, bn, mpt);
    if (trans_out && out_dtype != SP24_F32) pick_f8_tile(ms, n, sms, bn, mpt);
    // Weight gradient on CTA pairs: us, single CTAs -> pairs, ms 3072, n 768, k 8192 27.3 -> 13.5; ms 3072, n 3072, k 8192 80.9 -> 45.1;
    // ms 768, n 768, k 8192 15.9 -> 11.3; ms 1280, n 640, k 4096 11.1 -> 8.9; ms 3072, n 640, k 512 10.1 -> 7.5; ms 1024, n 3072, k 256
    // 8.2 -> 7.3.  Below these sizes the pair kernel's longer start counts: ms 1024, n 1024, k 1024 6.8 -> 7.0; ms 2048, n 512, k 512
    // 6.1 -> 6.7; ms 2048, n 1024, k 256 6.1 -> 6.7; ms 256, n 256, k 256 5.6 -> 6.3.
    if (!trans_out && n >= 256 && (k >= 2048 || ms * n >= (k > 256 ? 3 << 19 : 3 << 20)) && pair_kernels_enabled()) {
        CUtensorMap map_e, map_d;
        if (int rc = make_map_columns(&map_b, b, dtype, n, k, ld_b, 128)) return rc;
        if (int rc = make_map_e(&map_e, e_tc, (ms / 128) * P.k_atoms, 2)) return rc;
        if (int rc = encode_map(&map_d, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out, n, ms, ld_out * 4, 32, 16, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
        // slices: what the single-CTA kernel takes at least (the error grows with the length of a float32 accumulation), two at most
        // (two addends on a cleared buffer give the same bits in either order, three do not)
        int bn = 0, mpt = 0, slices = 1;
        pick_f8_accumulate(ms, n, k, sms, bn, mpt, slices);
        if (slices < 2 && pair_slices(ms, n, k, 256, sms) >= 2) slices = 2;
        return launch_spmm_pair_acc<false, true>(map_a, map_b, map_e, map_d, P, sums, slices, st);
    }
    if (sums.out)
        if (int rc = sp24_sum_parts(sums.parts, sums.n_parts, ms, sums.out, sums.accumulate, stream)) return rc;
    if (!trans_out) {
        pick_f8_accumulate(ms, n, k, sms, bn, mpt, P.k_splits);
        P.accumulate = 1;
    }
    P.mblk_per_tile = mpt;
    if (!trans_out) return dispatch_bn<true, false, false, false, float>(bn, b, dtype, n, k, ld_b, map_a, P, st);
    if (out_dtype == SP24_F32) return dispatch_bn<true, false, false, true, float>(bn, b, dtype, n, k, ld_b, map_a, P, st);
    if (int rc = make_map(&map_b, b, dtype, n, k, ld_b, 128, 128)) return rc;
    return out_dtype == SP24_F16 ? launch_spmm<128, true, false, false, true, __half>(map_a, map_b, P, st)
                                 : launch_spmm<128, true, false, false, true, __nv_bfloat16>(map_a, map_b, P, st);
}

extern "C" int sp24_spmm_f8(const void *a_packed, int dtype, int64_t ld_a, const void *e_tc, int64_t ms, int64_t k, const void *b, int64_t ld_b,
                            int64_t n, void *out, int out_dtype, int trans_out, int64_t ld_out, const float *bias, const float *amax_a,
                            const float *amax_b, int *status, void *stream) {
    return spmm_f8_impl(a_packed, dtype, ld_a, e_tc, ms, k, b, ld_b, n, out, out_dtype, trans_out, ld_out, bias, amax_a, amax_b, SumsParams{}, status,
                        stream);
}

extern "C" int sp24_spmm_f8_sums(const void *a_packed, int dtype, int64_t ld_a, const void *e_tc, int64_t ms, int64_t k, const void *b, int64_t ld_b,
                                 int64_t n, float *out, int64_t ld_out, const float *amax_a, const float *amax_b, const float *row_parts,
                                 int64_t n_parts, float *row_sums, int sums_accumulate, int *status, void *stream) {
    if (!row_sums || !row_parts || n_parts <= 0) return SP24_ERR_ARG;
    return spmm_f8_impl(a_packed, dtype, ld_a, e_tc, ms, k, b, ld_b, n, out, SP24_F32, 0, ld_out, nullptr, amax_a, amax_b,
                        SumsParams{row_parts, row_sums, n_parts, sums_accumulate}, status, stream);
}

// The float8 GEMM with the dequantisation folded into the epilogue: D = alpha * (A_sparse * B) [+ bias] [activation],
// alpha = the product of the operands' per-tensor scales.  Float8 operands (float32 output) only.
extern "C" int sp24_spmm_scaled(const void *a_packed, int dtype, int64_t ld_a, const void *e_tc, int64_t ms, int64_t k,
                                const void *b, int64_t ld_b, int64_t n, float *out, int trans_out, int64_t ld_out,
                                const float *bias, int activation, float alpha, int *status, void *stream) {
    if (dtype != SP24_E4M3 && dtype != SP24_E5M2) return SP24_ERR_DTYPE;
    if (!(alpha == alpha)) return SP24_ERR_ARG;
    return spmm_impl(a_packed, dtype, 0, ld_a, e_tc, ms, k, b, 0, ld_b, n, out, SP24_F32, trans_out, ld_out, bias, activation,
                     alpha, status, stream);
}


// ------------------------------------------------------------------------------------------------
// Self-test of the bounded wait: one CTA waits on a barrier that nothing ever signals, with a small
// poll limit.  The wait must give up, record code 9 in *status and let the kernel return normally.  Then the whole-warp form, with
// half of the lanes on a phase that is complete: every lane must learn that the wait was given up (code 10 otherwise).
// ------------------------------------------------------------------------------------------------
namespace sp24 {
namespace {
__global__ void wait_selftest_kernel(int *status, uint32_t limit) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {       // one warp
        abort_flag = 0;
        mbar_init(smem_u32(&bar), 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) mbar_wait(smem_u32(&bar), 0, &abort_flag, status, 9, limit);
    __syncthreads();
    const bool ok = mbar_wait_warp(smem_u32(&bar), threadIdx.x < 16 ? 1 : 0, &abort_flag, status, 9, limit);
    if (__ballot_sync(0xFFFFFFFFu, ok) != 0 && threadIdx.x == 0) *status = 10;
}
}  // namespace
}  // namespace sp24

extern "C" int sp24_selftest_bounded_wait(int *status, int polls, void *stream) {
    if (!status || polls <= 0 || polls > (1 << 20)) return SP24_ERR_ARG;
    if (int rc = check_device()) return rc;
    wait_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(status, (uint32_t)polls);
    return launch_status();
}

// ------------------------------------------------------------------------------------------------
// Sparse GEMM for callers that must not allocate
// ------------------------------------------------------------------------------------------------
// Some hosts of this library cannot call cudaMalloc at the point where they run the GEMM: code replayed
// under a memory plan fixed in advance, a real-time loop that may not touch the allocator, or a plug-in
// whose host application owns all device memory.  sp24_spmm needs one piece of scratch besides its
// inputs and outputs - the metadata re-ordered for the tensor cores - and normally the caller allocates
// it.  This variant keeps that scratch in a fixed array inside the library image instead.  Every GPU
// that loads the library carries the array until the process exits.
constexpr int64_t NOALLOC_SCRATCH_BYTES = 4ll << 20;  // enough for ms * k <= 32 Mi elements
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

namespace sp24 {
namespace {
// Device address of the array, looked up once per device.  In host code the array's name is only a
// handle; the address a kernel can use comes from cudaGetSymbolAddress with that device current.
int noalloc_scratch(void **out) {
    static std::atomic<void *> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return runtime_error();
    if (dev < 0 || dev >= 64) return SP24_ERR_DEVICE;
    if (!cached[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return runtime_error();
        cached[dev] = p;
    }
    *out = cached[dev];
    return SP24_OK;
}
}  // namespace
}  // namespace sp24

extern "C" int64_t sp24_spmm_noalloc_max_bytes(void) { return NOALLOC_SCRATCH_BYTES; }

extern "C" int sp24_spmm_noalloc(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, const void *meta,
                                 int64_t ms, int64_t k, const void *b, int b_mn_major, int64_t ld_b, int64_t n, void *out,
                                 int out_dtype, int trans_out, int64_t ld_out, const void *bias, int activation,
                                 int *status, void *stream) {
    // every check of sp24_spmm comes first: a rejected call launches nothing and leaves the shared array alone
    if (!meta) return SP24_ERR_ARG;
    if (int rc = validate_spmm_args(a_packed, dtype, a_mn_major, ld_a, ms, k, b, b_mn_major, ld_b, n, out, out_dtype,
                                    trans_out, ld_out, bias, activation))
        return rc;
    if (!aligned16(meta)) return SP24_ERR_ALIGN;
    // fp8 and int8 operands carry 32-bit metadata words, the 16-bit types 16-bit words
    const bool f8 = dtype == SP24_E4M3 || dtype == SP24_E5M2 || dtype == SP24_I8;
    if (sp24_meta_tc_bytes(ms, k) > NOALLOC_SCRATCH_BYTES) return SP24_ERR_TOO_LARGE;
    if (int rc = check_device()) return rc;
    void *scratch = nullptr;
    if (int rc = noalloc_scratch(&scratch)) return rc;
    // the conversion rewrites every word the GEMM will read (padding included), so whatever an earlier
    // call left in the array does not matter
    if (int rc = sp24_meta_to_tc(meta, f8 ? 4 : 2, ms, k, scratch, stream)) return rc;
    return sp24_spmm(a_packed, dtype, a_mn_major, ld_a, scratch, ms, k, b, b_mn_major, ld_b, n, out, out_dtype, trans_out,
                     ld_out, bias, activation, status, stream);
}


// D (ms x n, fp32, row-major) += A_sparse (ms x k) * B (k x n, stored row-major): the weight-gradient form.
// K is cut into slices so that tiles x slices fills the SMs; every slice adds its partial product with fp32
// reductions, so the caller zeroes D for a plain product or passes a gradient buffer to accumulate into.
static int spmm_accumulate_impl(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, const void *e_tc, int64_t ms, int64_t k,
                                const void *b, int64_t ld_b, int64_t n, float *out, int64_t ld_out, int k_splits, const float *row_parts,
                                int64_t n_parts, float *row_sums, int sums_accumulate, int *status, void *stream) {
    if (!a_packed || !e_tc || !b || !out || !status) return SP24_ERR_ARG;
    if (dtype != SP24_F16 && dtype != SP24_BF16) return SP24_ERR_DTYPE;
    if (ms <= 0 || n <= 0 || k <= 0 || ms % 128 || k % 64 || n % 8) return SP24_ERR_SHAPE;
    if (k_splits < 0) return SP24_ERR_ARG;
    if (row_sums && (!row_parts || n_parts <= 0)) return SP24_ERR_ARG;
    const int64_t a_inner = a_mn_major ? ms : k / 2;
    if (ld_a < a_inner || (ld_a * 2) % 16 || ld_b < n || (ld_b * 2) % 16 || ld_out < n || (ld_out * 4) % 16) return SP24_ERR_STRIDE;
    if (!aligned16(a_packed) || !aligned16(e_tc) || !aligned16(b) || !aligned16(out)) return SP24_ERR_ALIGN;
    if (int rc = check_device()) return rc;

    SpmmParams P{};
    P.e_tc = e_tc; P.out = out; P.bias = nullptr; P.ms = ms; P.n = n; P.k = k; P.ld_out = ld_out;
    P.k_atoms = (k + 127) / 128; P.status = status; P.activation = 0; P.trace = nullptr;
    P.alpha = 1.f;
    const uint32_t fmt = dtype == SP24_BF16 ? 1u : 0u;
    P.idesc = (1u << 2) | (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(a_mn_major ? 1 : 0) << 15) | (1u << 16) |
              ((uint32_t)(BM >> 4) << 24);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // CTA-pair kernel for at least one full tile of columns
    bool pair_form = n >= 256 && ms > 128 && pair_kernels_enabled();
    if (pair_form && ms % 256) {
        // The last of several 256-row blocks is half empty (a single one lost: ms 128, n 1920, k 6016 13.2 -> 15.3).  The error of a float32
        // accumulation on the tensor cores grows with its length (2176 x 768 over k 8128: 2.4e-6 in two slices, 1.2e-6 in four), so these
        // keep the single-CTA kernel's number of slices at least.  That may make more rounds of pairs than of CTAs, a pair's round being
        // less than half as long: both times are estimated, ns, from rounds and K steps, by a fit to a map of 504 sizes (8 row counts, 9
        // widths, K from 256 to 16384) that they meet by 3.6 % on average, pairs with 6 % added; the row sums would be a launch of their own
        // beside single CTAs.  us, single CTAs / pairs, pairs taken: ms 2944, n 768, k 16384 52.7 / 43.9, ms 2176, n 2304, k 8192 69.0 /
        // 56.8, ms 384, n 256, k 1024 10.7 / 7.6; left alone: ms 384, n 520, k 1984 11.7 / 13.6, ms 1152, n 1024, k 512 11.8 / 12.7.  Against the
        // rounds alone, which decided before, 2 sizes are more than 3 % slower (n 520) and 82 faster, up to 21 %.
        const int sms = sm_count_cached();
        const int64_t k_iters = (k + 127) / 128;
        const int64_t slices = k_splits ? std::min<int64_t>(k_splits, k_iters) : single_slices(ms, n, k, sms);
        if (!k_splits) k_splits = (int)std::max(slices, pair_slices(ms, n, k, 128, sms));
        const int64_t splits = std::min<int64_t>(k_splits, k_iters);
        auto rounds = [&](int64_t columns, int64_t parts, int64_t units) {
            return (((n + columns - 1) / columns) * ((ms + 255) / 256) * parts + units - 1) / units;
        };
        const int64_t pairs = 3250 + rounds(two::BN3, splits, sms / 2) * (4930 + 392 * ((k_iters + splits - 1) / splits));
        const int64_t singles = 6000 + rounds(192, slices, sms) * (6080 + 860 * ((k_iters + slices - 1) / slices)) + (row_sums ? 2600 : 0);
        if (pairs > singles && rounds(two::BN3, splits, sms / 2) > rounds(192, slices, sms)) {
            pair_form = false;
            k_splits = (int)slices;
        }
    }
    CUtensorMap map_a, map_b;
    int rc;
    if (!a_mn_major) rc = make_map(&map_a, a_packed, dtype, ms, k / 2, ld_a, 64, 128);
    else rc = pair_form ? make_map_columns(&map_a, a_packed, dtype, k / 2, ms, ld_a, 64) : make_map(&map_a, a_packed, dtype, k / 2, ms, ld_a, 64, 64);
    if (rc) return rc;
    P.whole_columns = pair_form && n % 64 == 0;
    rc = P.whole_columns ? make_map_columns(&map_b, b, dtype, k, n, ld_b, 128) : make_map(&map_b, b, dtype, k, n, ld_b, 64, 128);
    if (rc) return rc;
    if (pair_form) {
        CUtensorMap map_e;
        rc = make_map_e(&map_e, e_tc, (ms / 128) * P.k_atoms);
        if (rc) return rc;
        CUtensorMap map_d;
        rc = encode_map(&map_d, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out, n, ms, ld_out * 4, 32, 16, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
        const SumsParams sums{row_parts, row_sums, n_parts, sums_accumulate};
        return a_mn_major ? launch_spmm_pair_acc<true>(map_a, map_b, map_e, map_d, P, sums, k_splits, st)
                          : launch_spmm_pair_acc<false>(map_a, map_b, map_e, map_d, P, sums, k_splits, st);
    }
    if (row_sums)
        if (int rc2 = sp24_sum_parts(row_parts, n_parts, ms, row_sums, sums_accumulate, stream)) return rc2;
    // widest tile (least operand traffic per output), then as many K slices as idle SMs allow
    const bool wide = n >= 192;
    P.mblk_per_tile = single_row_blocks(ms);
    P.k_splits = (int)(k_splits ? std::min<int64_t>(k_splits, (k + 127) / 128) : single_slices(ms, n, k, sm_count_cached()));
    // fp16 and bf16 operands share these kernels: the element type only enters through the tensor maps and the
    // instruction descriptor
    if (a_mn_major) return wide ? launch_spmm<192, false, true, true, false, float>(map_a, map_b, P, st)
                                : launch_spmm<128, false, true, true, false, float>(map_a, map_b, P, st);
    return wide ? launch_spmm<192, false, false, true, false, float>(map_a, map_b, P, st)
                : launch_spmm<128, false, false, true, false, float>(map_a, map_b, P, st);
}

extern "C" int sp24_spmm_accumulate_f32(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, const void *e_tc,
                                        int64_t ms, int64_t k, const void *b, int64_t ld_b, int64_t n, float *out,
                                        int64_t ld_out, int k_splits, int *status, void *stream) {
    return spmm_accumulate_impl(a_packed, dtype, a_mn_major, ld_a, e_tc, ms, k, b, ld_b, n, out, ld_out, k_splits, nullptr, 0, nullptr, 0,
                                status, stream);
}

extern "C" int sp24_spmm_accumulate_sums_f32(const void *a_packed, int dtype, int a_mn_major, int64_t ld_a, const void *e_tc, int64_t ms,
                                             int64_t k, const void *b, int64_t ld_b, int64_t n, float *out, int64_t ld_out, int k_splits,
                                             const float *row_parts, int64_t n_parts, float *row_sums, int sums_accumulate, int *status,
                                             void *stream) {
    if (!row_sums) return SP24_ERR_ARG;
    return spmm_accumulate_impl(a_packed, dtype, a_mn_major, ld_a, e_tc, ms, k, b, ld_b, n, out, ld_out, k_splits, row_parts, n_parts, row_sums,
                                sums_accumulate, status, stream);
}
