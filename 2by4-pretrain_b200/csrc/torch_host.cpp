// Native host path of the Python package: argument checks, output allocation, kernel launches through the C ABI and the
// autograd nodes of the layers, in one call from Python each.
//
// A layer step launches half a dozen kernels that take 5 - 60 us each; driven from Python (argument marshalling of 20
// words per launch, tensor views, autograd.Function objects in both directions) its host time was 300 us and bounded
// every step below a few thousand tokens.  Nothing here computes: without the kernel library the module does not load.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/mm.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include "../../include/sparse24_b200.h"

namespace {

using at::Tensor;
using torch::autograd::variable_list;
using OptTensor = c10::optional<Tensor>;
using NoAutograd = at::AutoDispatchBelowADInplaceOrView;

// ---------------------------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------------------------
void check(int rc, const char *what) { TORCH_CHECK(rc == SP24_OK, what, ": ", sp24_strerror(rc), " (code ", rc, ")"); }

int dt(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return SP24_F32;
        case at::kHalf: return SP24_F16;
        case at::kBFloat16: return SP24_BF16;
        case at::kFloat8_e4m3fn: return SP24_E4M3;
        case at::kFloat8_e5m2: return SP24_E5M2;
        case at::kChar: return SP24_I8;
        case at::kInt: return SP24_I32;
        default: TORCH_CHECK(false, "Datatype ", t, " is not supported!");
    }
}
bool is16(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }
bool is_f8(at::ScalarType t) { return t == at::kFloat8_e4m3fn || t == at::kFloat8_e5m2; }

void *cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Every tensor must live on the current device: the kernels run on its current stream and dereference raw addresses.
void on_current_device(const Tensor &t) {
    TORCH_CHECK(t.is_cuda(), "Error tensor.device= ", t.device(), " is not supported! Only CUDA tensors are currently supported.");
    const auto cur = c10::cuda::current_device();
    TORCH_CHECK(t.device().index() == cur, "tensor on ", t.device(), " but the current CUDA device is cuda:", (int)cur,
                ": the sparse24 kernels launch on the current device; wrap the call in torch.cuda.device(tensor.device)");
}
void on_current_device(const OptTensor &t) { if (t.has_value()) on_current_device(*t); }
template <typename... T> void require_cuda(const T &...t) { (on_current_device(t), ...); }

void *ptr(const Tensor &t) { return t.data_ptr(); }
const void *ptr(const OptTensor &t) { return t.has_value() ? t->data_ptr() : nullptr; }
bool aligned(const Tensor &t, uintptr_t a = 16) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % a == 0; }

// Whether somebody wants to see or change what is allocated: a trace, a dispatch mode, a functorch level, memory filled for determinism.
bool allocations_watched() {
    return torch::jit::tracer::isTracing() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) ||
           (at::globalContext().deterministicAlgorithms() && at::globalContext().deterministicFillUninitializedMemory());
}
// Otherwise straight from the allocator: through the dispatcher an allocation took 0.2 us more, and a layer step makes eight.
Tensor empty(c10::IntArrayRef shape, at::ScalarType t, const Tensor &like) {
    if (!like.is_cuda() || allocations_watched()) return at::empty(shape, like.options().dtype(t));
    return at::detail::empty_cuda(shape, t, like.device(), c10::nullopt);
}

// storage order and leading dimension of a 2-D tensor with one unit stride; order -1: neither
struct Layout { int col; int64_t ld; };
Layout layout_of(const Tensor &t) {
    const int64_t rs = t.stride(0), cs = t.stride(1), m = t.size(0), k = t.size(1);
    if (cs == 1 && (rs >= k || m == 1)) return {0, std::max(rs, k)};
    if (rs == 1 && (cs >= m || k == 1)) return {1, std::max(cs, m)};
    return {-1, 0};
}
bool usable(const Tensor &t, const Layout &l) { return l.col >= 0 && aligned(t) && (l.ld * (int64_t)t.element_size()) % 16 == 0; }
// the same logical matrix stored densely in the requested order (no copy when it already is)
Tensor as_layout(const Tensor &t, int col) {
    const Layout l = layout_of(t);
    if (l.col == col && usable(t, l)) return t;
    return col ? t.t().contiguous().t() : t.contiguous();
}

// A view into `base`'s memory with its own type, shape and strides, sharing its version counter (a write through either
// is seen by both) unless given one; byte_off is counted from base's first element.
Tensor carve(const Tensor &base, int64_t byte_off, at::ScalarType t, c10::IntArrayRef shape, c10::IntArrayRef strides,
             const c10::VariableVersion *version = nullptr) {
    auto impl = c10::make_intrusive<c10::TensorImpl>(c10::Storage(base.storage()), base.key_set(), at::scalarTypeToTypeMeta(t));
    impl->set_storage_offset(((int64_t)base.storage_offset() * base.element_size() + byte_off) / (int64_t)c10::elementSize(t));
    impl->set_sizes_and_strides(shape, strides);
    if (!base.is_inference()) impl->set_version_counter(version ? *version : base.unsafeGetTensorImpl()->version_counter());
    return Tensor(std::move(impl));
}

// (rows, last dimension) of a contiguous or reshapeable tensor; sees later in-place writes through its version counter
Tensor rows2d(const Tensor &t) {
    if (t.dim() == 2) return t;
    const int64_t k = t.size(-1);
    if (t.is_contiguous()) return carve(t, 0, t.scalar_type(), {k ? t.numel() / k : 0, k}, {k, 1});
    return t.reshape({-1, k});
}

// The nodes below have no forward-mode derivative: refuse tangents instead of dropping them.
template <typename... T> void no_tangent(const T &...t) {
    TORCH_CHECK_NOT_IMPLEMENTED(!(torch::autograd::isFwGradDefined(t) || ...),
                                "the layers of this package do not implement forward-mode automatic differentiation");
}

// Whether a backward pass is itself recorded (create_graph): what is linear in the incoming gradient through plain torch
// operations then stays a function of it.
bool recorded(const Tensor &grad) { return at::GradMode::is_enabled() && grad.requires_grad(); }

int64_t align256(int64_t v) { return (v + 255) / 256 * 256; }

// Word that a bounded wait of the GEMM kernels reports to, one per device.
struct StatusWords {
    std::vector<Tensor> words = std::vector<Tensor>(64);
    std::mutex mu;
};
StatusWords &status_table() {
    static auto &t = *new StatusWords();                  // never destroyed: the CUDA runtime may be gone at exit
    return t;
}
Tensor &status_word(c10::DeviceIndex dev) {
    auto &t = status_table();
    std::lock_guard<std::mutex> lock(t.mu);
    Tensor &w = t.words.at(dev);
    if (!w.defined()) w = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, dev));
    return w;
}
// the words that exist, by device: those of every device that a GEMM ran on
std::map<int, Tensor> status_words() {
    auto &t = status_table();
    std::lock_guard<std::mutex> lock(t.mu);
    std::map<int, Tensor> out;
    for (size_t i = 0; i < t.words.size(); ++i)
        if (t.words[i].defined()) out[(int)i] = t.words[i];
    return out;
}
int *status_ptr(const Tensor &t) { return static_cast<int *>(status_word(t.device().index()).data_ptr()); }

// Device word added to the Philox offset of the MVUE draws (a step replayed from a CUDA graph bumps it), or none.
OptTensor &rng_offset() {
    static auto &t = *new OptTensor();
    return t;
}

// That word for one conversion: only seeded MVUE draws read it.
const uint64_t *rng_offset_ptr(int64_t mode) {
    const bool draws = mode == SP24_PRUNE_MVUE || mode == SP24_PRUNE_MVUE_FAST;
    return draws && rng_offset().has_value() ? static_cast<const uint64_t *>(rng_offset()->data_ptr()) : nullptr;
}

// Python objects that calls need, held from the module's load on (looked up in a function-local static they could make one
// thread wait for the interpreter lock while another holds it and waits for the static).
struct PyObjects {
    PyObject *getrandbits = nullptr, *bits = nullptr, *weight_grad = nullptr, *dense_weight_grads = nullptr;
} py_objects;

// What random.randint(0, 2**31 - 1) returns, from the same generator state: 32 random bits, drawn again until below 2^31.
// Needs the GIL.
uint64_t python_seed() {
    for (;;) {
        PyObject *r = PyObject_CallOneArg(py_objects.getrandbits, py_objects.bits);
        if (!r) throw py::error_already_set();
        const unsigned long long v = PyLong_AsUnsignedLongLong(r);
        Py_DECREF(r);
        if (v < (1ull << 31)) return v;
    }
}

// ---------------------------------------------------------------------------------------------
// sparse GEMM: input @ dense(weight).T, the contract of sparse.spmm.sparse_linear
// ---------------------------------------------------------------------------------------------
Tensor spmm(const Tensor &input, const Tensor &weight, const Tensor &e_tc, const OptTensor &bias_in, int64_t act, c10::optional<double> alpha,
            bool view_result, bool bias_may_be_f32 = false) {
    TORCH_CHECK(weight.dim() == 2, "_sparse_semi_structured_linear: Expected weight argument to be 2D tensor, got ", weight.dim(), " dims");
    const auto wt = weight.scalar_type();
    TORCH_CHECK(input.scalar_type() == wt, "_sparse_semi_structured_linear: Expected input datatype ", wt, ", but got ", input.scalar_type());
    const int64_t ms = weight.size(0), kh = weight.size(1), k = 2 * kh;
    TORCH_CHECK(input.size(-1) == k, "_sparse_semi_structured_linear: Expected weight argument to have ", input.size(-1) / 2,
                " columns, but got ", kh);
    Tensor x = input.dim() == 2 ? input : input.reshape({-1, k});
    const int64_t n = x.size(0);
    const Layout la = layout_of(weight);
    TORCH_CHECK(la.col >= 0, "_sparse_semi_structured_linear: Invalid strides for weight argument: row stride = ", weight.stride(0),
                ", column stride = ", weight.stride(1));
    Layout lb = layout_of(x);
    if (!usable(x, lb)) {
        x = x.contiguous();
        lb = {0, k};
    }
    // fp8 operands give fp32, int8 operands int32, 16-bit operands their own type
    const bool f8 = is_f8(wt), i8 = wt == at::kChar;
    const auto ot = f8 ? at::kFloat : (i8 ? at::kInt : wt);
    TORCH_CHECK(!i8 || (!bias_in.has_value() && act == 0), "_sparse_semi_structured_linear: the int8 GEMM on sm_100a takes no bias and no activation");
    OptTensor bias = bias_in;
    bool bias_f32 = false;
    if (bias.has_value()) {
        TORCH_CHECK(bias->dim() == 1 && bias->size(0) == ms, "_sparse_semi_structured_linear: Expected bias argument to have ", ms,
                    " elements, but got ", bias->numel());
        if (bias_may_be_f32 && bias->scalar_type() != ot) {
            // the token-major 16-bit GEMM reads a float32 bias in its epilogue; elsewhere it is cast first
            bias_f32 = bias->scalar_type() == at::kFloat && is16(wt) && lb.col == 0 && !view_result && ms % 256 == 0;
            if (!bias_f32) bias = bias->to(ot);
        }
        TORCH_CHECK(bias_f32 || bias->scalar_type() == ot, "two_four_sgemm_cutlass: Expected spars GTEMM bias datatype ", ot, ", but got ",
                    bias->scalar_type());
        bias = bias->contiguous();
    }
    TORCH_CHECK(ms % 128 == 0, "sparse GEMM on sm_100a: number of rows of the sparse matrix must be divisible by 128");
    // k strided in the dense operand (the caller passed B.t()): D (ms, n) row-major, returned as its transposed view
    const bool as_view = lb.col || view_result;
    Tensor out;
    if (as_view) {
        out = empty({ms, n}, ot, weight);
    } else if (input.dim() == 2) {
        out = empty({n, ms}, ot, weight);
    } else {
        auto shape = input.sizes().vec();
        shape.back() = ms;
        out = empty(shape, ot, weight);
    }
    int *status = status_ptr(weight);
    if (alpha.has_value()) {
        TORCH_CHECK(f8 && !la.col && !lb.col, "_sparse_semi_structured_linear: alpha is for float8 operands (both K-major) only");
        check(sp24_spmm_scaled(ptr(weight), dt(wt), la.ld, ptr(e_tc), ms, k, ptr(x), lb.ld, n, static_cast<float *>(ptr(out)), !as_view,
                               as_view ? n : ms, static_cast<const float *>(ptr(bias)), (int)act, (float)*alpha, status, cur_stream()),
              "sp24_spmm_scaled");
    } else if (bias_f32) {
        check(sp24_spmm_mlp(ptr(weight), dt(wt), la.col, la.ld, ptr(e_tc), ms, k, ptr(x), lb.ld, n, ptr(out), ms, ptr(bias), 1, 0, nullptr,
                            ms, status, cur_stream()),
              "sp24_spmm_mlp");
    } else {
        check(sp24_spmm(ptr(weight), dt(wt), la.col, la.ld, ptr(e_tc), ms, k, ptr(x), lb.col, lb.ld, n, ptr(out), dt(ot), !as_view,
                        as_view ? n : ms, ptr(bias), (int)act, status, cur_stream()),
              "sp24_spmm");
    }
    if (!as_view) return out;
    out = out.t();
    if (input.dim() == 2) return out;
    auto shape = input.sizes().vec();
    shape.back() = ms;
    return out.reshape(shape);
}

Tensor sparse_linear(const Tensor &input, const Tensor &weight, const Tensor &e_tc, const OptTensor &bias, int64_t act,
                     c10::optional<double> alpha, bool view_result) {
    NoAutograd guard;
    require_cuda(input, weight, e_tc, bias);
    return spmm(input, weight, e_tc, bias, act, alpha, view_result);
}

// out (ms, n) float32 += sparse @ dense (k, n)
// Row sums that the compressing pass takes along (the bias gradient): `out` is set to them, or increased by them.  `parts` is
// scratch for partial sums (row_parts_bytes), which are added up in a fixed order: a gradient repeats bit for bit.
struct RowSums {
    float *out = nullptr, *parts = nullptr;
    bool add = false;
};
int64_t row_parts_bytes(int64_t m, int64_t k, at::ScalarType packed) { return 4 * m * sp24_row_parts(k, dt(packed)); }
void sum_parts(const RowSums &s, int64_t m, int64_t k, at::ScalarType packed) {
    check(sp24_sum_parts(s.parts, sp24_row_parts(k, dt(packed)), m, s.out, s.add, cur_stream()), "sp24_sum_parts");
}

// sums: the partial row sums of the compressed operand, added up by the same launch
void mm_accumulate(const Tensor &out, const Tensor &weight, const Tensor &e_tc, const Tensor &dense_in, int64_t k_splits,
                   const RowSums &sums = {}) {
    TORCH_CHECK(out.scalar_type() == at::kFloat && out.dim() == 2 && out.stride(1) == 1, "sparse_mm_accumulate_: out must be a row-major fp32 matrix");
    TORCH_CHECK(is16(weight.scalar_type()) && dense_in.scalar_type() == weight.scalar_type(),
                "sparse_mm_accumulate_: expected matching fp16 / bf16 operands, got ", weight.scalar_type(), " and ", dense_in.scalar_type());
    const int64_t ms = weight.size(0), k = 2 * weight.size(1);
    TORCH_CHECK(dense_in.dim() == 2 && dense_in.size(0) == k, "sparse_mm_accumulate_: dense operand must have ", k, " rows, got ", dense_in.sizes());
    const int64_t n = dense_in.size(1);
    TORCH_CHECK(out.size(0) == ms && out.size(1) == n, "sparse_mm_accumulate_: out must be (", ms, ", ", n, "), got ", out.sizes());
    const Layout la = layout_of(weight);
    TORCH_CHECK(la.col >= 0, "sparse_mm_accumulate_: invalid strides for the packed values");
    Tensor dense = dense_in;
    if (dense.stride(1) != 1 || !aligned(dense) || (dense.stride(0) * dense.element_size()) % 16) dense = dense.contiguous();
    if (sums.out) {
        check(sp24_spmm_accumulate_sums_f32(ptr(weight), dt(weight.scalar_type()), la.col, la.ld, ptr(e_tc), ms, k, ptr(dense), dense.stride(0), n,
                                            static_cast<float *>(ptr(out)), out.stride(0), (int)k_splits, sums.parts,
                                            sp24_row_parts(k, dt(weight.scalar_type())), sums.out, sums.add, status_ptr(weight), cur_stream()),
              "sp24_spmm_accumulate_sums_f32");
        return;
    }
    check(sp24_spmm_accumulate_f32(ptr(weight), dt(weight.scalar_type()), la.col, la.ld, ptr(e_tc), ms, k, ptr(dense), dense.stride(0), n,
                                   static_cast<float *>(ptr(out)), out.stride(0), (int)k_splits, status_ptr(weight), cur_stream()),
          "sp24_spmm_accumulate_f32");
}
void sparse_mm_accumulate(const Tensor &out, const Tensor &weight, const Tensor &e_tc, const Tensor &dense, int64_t k_splits) {
    NoAutograd guard;
    require_cuda(out, weight, e_tc, dense);
    mm_accumulate(out, weight, e_tc, dense, k_splits);
}

// ---------------------------------------------------------------------------------------------
// dense -> 2:4
// ---------------------------------------------------------------------------------------------
// clear (fast MVUE of column-major values): a dense tensor that the same launch sets to zero.
// Fills packed / meta from dense; returns the metadata in tensor-core order when it was asked for and the shape allows.
OptTensor prune_into(const Tensor &dense_in, const Tensor &packed, const Tensor &meta, int64_t mode, const OptTensor &mask_in,
                     const OptTensor &uniforms_in, uint64_t seed, uint64_t offset, c10::optional<bool> emit_tc, const RowSums &sums = {},
                     OptTensor e_tc = {}, const Tensor &clear = {}) {
    TORCH_CHECK(dense_in.dim() == 2, "Expected 2-dimensional dense tensor, got ", dense_in.dim(), "-dimensional tensor");
    const int64_t m = dense_in.size(0), k = dense_in.size(1);
    const Layout lp = layout_of(packed);
    TORCH_CHECK(lp.col >= 0, "packed output must be row- or column-major with unit inner stride");
    const Tensor dense = as_layout(dense_in, lp.col);
    OptTensor mask = mask_in, uniforms = uniforms_in;
    int64_t ld_m = 0, ld_u = 0;
    if (mask.has_value()) {
        if (mask->scalar_type() != at::kBool && mask->scalar_type() != at::kByte) mask = mask->ne(0);
        mask = as_layout(*mask, lp.col);
        ld_m = layout_of(*mask).ld;
    }
    if (uniforms.has_value()) {
        uniforms = as_layout(uniforms->to(at::kFloat), lp.col);
        ld_u = layout_of(*uniforms).ld;
    }
    TORCH_CHECK(meta.is_contiguous(), "metadata buffer must be contiguous");
    // 16-bit results with whole 128-row blocks can also get their metadata in the order the GEMM reads, in the same pass.
    // Default: for column-major results (the dY^T operand of the weight-gradient GEMM, consumed at once).
    const bool want_tc = emit_tc.has_value() ? *emit_tc : lp.col == 1;
    if (!e_tc.has_value() && want_tc && packed.element_size() == 2 && m % 128 == 0)
        e_tc = empty({sp24_meta_tc_bytes(m, k)}, at::kByte, packed);
    sp24_prune_extras x{};
    if (!uniforms.has_value()) x.offset_dev = rng_offset_ptr(mode);
    x.e_tc = const_cast<void *>(ptr(e_tc));
    x.row_parts = sums.parts;
    if (clear.defined())
        check(sp24_mvue_compress_clearing(ptr(dense), dt(dense.scalar_type()), m, k, layout_of(dense).ld, ptr(packed), dt(packed.scalar_type()),
                                          lp.ld, ptr(meta), seed, offset, &x, ptr(clear), clear.nbytes(), cur_stream()),
              "sp24_mvue_compress_clearing");
    else
        check(sp24_prune_compress_with(ptr(dense), dt(dense.scalar_type()), m, k, layout_of(dense).ld, lp.col, ptr(packed),
                                       dt(packed.scalar_type()), lp.ld, ptr(meta), (int)mode, ptr(mask), ld_m,
                                       static_cast<const float *>(ptr(uniforms)), ld_u, seed, offset, &x, cur_stream()),
              "sp24_prune_compress");
    if (sums.out) sum_parts(sums, m, k, packed.scalar_type());
    return e_tc;
}
OptTensor prune_compress(const Tensor &dense, const Tensor &packed, const Tensor &meta, int64_t mode, const OptTensor &mask,
                         const OptTensor &uniforms, uint64_t seed, uint64_t offset, c10::optional<bool> emit_tc, const OptTensor &row_sums) {
    NoAutograd guard;
    require_cuda(dense, packed, meta, mask, uniforms, row_sums);
    RowSums sums;
    Tensor scratch;
    if (row_sums.has_value() && dense.dim() == 2) {
        TORCH_CHECK(layout_of(packed).col && row_sums->scalar_type() == at::kFloat && row_sums->numel() == dense.size(0) && row_sums->is_contiguous(),
                    "row_sums: column-major input and a contiguous float32 vector of one value per row");
        scratch = empty({row_parts_bytes(dense.size(0), dense.size(1), packed.scalar_type())}, at::kByte, packed);
        sums = {static_cast<float *>(ptr(*row_sums)), static_cast<float *>(ptr(scratch)), true};
    }
    return prune_into(dense, packed, meta, mode, mask, uniforms, seed, offset, emit_tc, sums);
}

// One allocation of m*k*cf/16 elements: packed values (in the storage order asked for) first, metadata behind.
std::pair<Tensor, Tensor> carve_compressed(int64_t m, int64_t k, at::ScalarType t, bool col, const Tensor &like) {
    const bool b16 = c10::elementSize(t) == 2;
    Tensor buf = empty({m * k * (b16 ? 9 : 10) / 16}, t, like);
    const int64_t kh = k / 2, bytes = m * kh * (int64_t)c10::elementSize(t), mc = k / (b16 ? 16 : 32);
    return {col ? carve(buf, 0, t, {m, kh}, {1, m}) : carve(buf, 0, t, {m, kh}, {kh, 1}),
            carve(buf, bytes, b16 ? at::kShort : at::kInt, {m, mc}, {mc, 1})};
}
// Compression into new buffers, in the storage order of `dense` (row stride > column stride: row-major).
std::tuple<Tensor, Tensor, OptTensor> compress(const Tensor &dense, at::ScalarType t, int64_t mode, const OptTensor &mask, uint64_t seed) {
    NoAutograd guard;
    require_cuda(dense, mask);
    auto [packed, meta] = carve_compressed(dense.size(0), dense.size(1), t, !(dense.stride(0) > dense.stride(1)), dense);
    OptTensor e = prune_into(dense, packed, meta, mode, mask, {}, seed, 0, {});
    return {packed, meta, e};
}

// ---------------------------------------------------------------------------------------------
// mask select + both compressed copies
// ---------------------------------------------------------------------------------------------
// The copies of one (m, k) weight in one allocation: W values | W metadata | W^T values | W^T metadata | both metadata
// copies in tensor-core order (whole 128 x 128 blocks only).
struct Copies {
    Tensor pw, mw, pt, mt, tcw, tct;
    Copies(int64_t m, int64_t k, at::ScalarType t, const Tensor &like) {
        TORCH_CHECK(c10::elementSize(t) == 2, "Datatype ", t, " is not supported!");
        const int64_t vb = m * k, mb = m * k / 8;          // bytes of the values / metadata of one copy
        const bool tc = m % 128 == 0 && k % 128 == 0;
        const int64_t o_mw = vb, o_pt = align256(vb + mb), o_mt = o_pt + vb, o_tw = align256(o_mt + mb), o_tt = o_tw + mb;
        Tensor buf = empty({o_tw + (tc ? 2 * mb : 0)}, at::kByte, like);
        // a version counter for W's tensors and one for W^T's: a write to one copy must not count as a write to the other, which
        // a backward pass may hold
        const c10::VariableVersion of_t(0);
        pw = carve(buf, 0, t, {m, k / 2}, {k / 2, 1});
        mw = carve(buf, o_mw, at::kShort, {m, k / 16}, {k / 16, 1});
        pt = carve(buf, o_pt, t, {k, m / 2}, {1, k}, &of_t);
        mt = carve(buf, o_mt, at::kShort, {k, m / 16}, {m / 16, 1}, &of_t);
        if (tc) {
            tcw = carve(buf, o_tw, at::kByte, {mb}, {1});
            tct = carve(buf, o_tt, at::kByte, {mb}, {1}, &of_t);
        }
    }
};

// (mask, packed_w, meta_w, packed_t, meta_t, tc_w or None, tc_t or None)
py::tuple as_tuple(const Tensor &mask, const Copies &c) {
    auto opt = [](const Tensor &t) { return t.defined() ? py::cast(t) : py::object(py::none()); };
    return py::make_tuple(mask, c.pw, c.mw, c.pt, c.mt, opt(c.tcw), opt(c.tct));
}

// Both copies of one weight, without the GIL; the mask that they follow goes to `mask`.
Copies select_copies(const Tensor &weight, const OptTensor &mask_in, at::ScalarType t, const OptTensor &mask_out, Tensor &mask) {
    NoAutograd guard;
    require_cuda(weight, mask_in, mask_out);
    TORCH_CHECK(weight.dim() == 2, "select_and_compress: expected a 2-D weight");
    const int64_t m = weight.size(0), k = weight.size(1);
    const Tensor w = as_layout(weight, 0);
    const bool select = !mask_in.has_value();
    if (!select) {
        mask = *mask_in;
        if (mask.scalar_type() != at::kBool && mask.scalar_type() != at::kByte) mask = mask.ne(0);
        mask = as_layout(mask, 0);
    } else if (mask_out.has_value()) {
        mask = *mask_out;
        TORCH_CHECK(mask.scalar_type() == at::kBool && mask.dim() == 2 && mask.size(0) == m && mask.size(1) == k && mask.is_contiguous(),
                    "select_and_compress: mask_out must be a contiguous bool tensor of the weight's shape");
    } else {
        mask = empty({m, k}, at::kBool, w);
    }
    Copies c(m, k, t, w);
    const int64_t ldw = layout_of(w).ld, ldm = layout_of(mask).ld;
    if (c.tcw.defined())
        check(sp24_select_dual_compress_tc(ptr(w), dt(w.scalar_type()), m, k, ldw, select, ptr(mask), ldm, ptr(c.pw), dt(t), k / 2, ptr(c.mw),
                                           ptr(c.pt), k, ptr(c.mt), ptr(c.tcw), ptr(c.tct), cur_stream()),
              "sp24_select_dual_compress_tc");
    else
        check(sp24_select_dual_compress(ptr(w), dt(w.scalar_type()), m, k, ldw, select, ptr(mask), ldm, ptr(c.pw), dt(t), k / 2, ptr(c.mw),
                                        ptr(c.pt), k, ptr(c.mt), cur_stream()),
              "sp24_select_dual_compress");
    return c;
}
py::tuple select_compress(const Tensor &weight, const OptTensor &mask_in, at::ScalarType t, const OptTensor &mask_out) {
    Tensor mask;
    c10::optional<Copies> c;
    {
        py::gil_scoped_release nogil;
        c.emplace(select_copies(weight, mask_in, t, mask_out, mask));
    }
    return as_tuple(mask, *c);
}

// Both copies of every weight in one launch; without the GIL.
std::vector<Copies> compress_all(const std::vector<Tensor> &weights, const std::vector<Tensor> &masks, at::ScalarType t, bool reselect) {
    const size_t count = weights.size();
    TORCH_CHECK(masks.size() == count, "select_and_compress_many: one mask per weight");
    std::vector<Copies> copies;
    std::vector<Tensor> keep;
    copies.reserve(count);
    NoAutograd guard;
    std::vector<sp24_dual_desc> descs(count);
    for (size_t i = 0; i < count; ++i) {
        const Tensor &weight = weights[i], &mask = masks[i];
        require_cuda(weight, mask);
        const int64_t m = weight.size(0), k = weight.size(1);
        TORCH_CHECK(m % 128 == 0 && k % 128 == 0, "select_and_compress_many: shape (", m, ", ", k, ") is not a multiple of 128 x 128");
        TORCH_CHECK(weight.scalar_type() == weights[0].scalar_type() && weight.device() == weights[0].device(),
                    "select_and_compress_many: all weights must share dtype and device");
        TORCH_CHECK(mask.scalar_type() == at::kBool && mask.sizes() == weight.sizes() && mask.is_contiguous(),
                    "select_and_compress_many: masks must be contiguous bool tensors of the weights' shapes");
        const Tensor w = as_layout(weight, 0);
        keep.push_back(w);
        copies.emplace_back(m, k, t, w);
        const Copies &c = copies.back();
        descs[i] = {ptr(w), m, k, layout_of(w).ld, ptr(mask), k, ptr(c.pw), k / 2, ptr(c.mw), ptr(c.pt), k, ptr(c.mt), ptr(c.tcw), ptr(c.tct)};
    }
    if (count)
        check(sp24_select_dual_compress_batch(descs.data(), (int)count, dt(weights[0].scalar_type()), dt(t), reselect, cur_stream()),
              "sp24_select_dual_compress_batch");
    return copies;
}

std::vector<py::tuple> select_compress_many(const std::vector<Tensor> &weights, const std::vector<Tensor> &masks, at::ScalarType t, bool reselect) {
    std::vector<Copies> copies;
    {
        py::gil_scoped_release nogil;
        copies = compress_all(weights, masks, t, reselect);
    }
    std::vector<py::tuple> out;
    out.reserve(copies.size());
    for (size_t i = 0; i < copies.size(); ++i) out.push_back(as_tuple(masks[i], copies[i]));
    return out;
}

// ---------------------------------------------------------------------------------------------
// refresh of a model's layers
// ---------------------------------------------------------------------------------------------
// What sparse_ops.refresh_sparse_layers does for layers of the plain class: reads each weight's state, launches once per group and
// installs the copies.  In Python these 20 attribute accesses a layer were more host time than 48 layers' kernel on the GPU (109 us).
// Returns the number of layers refreshed and those it leaves to the caller: any whose class, weight, mask or counters are not plain.
struct LayerNames {
    PyObject *weight, *bias, *parameters, *training, *mode, *cnt, *mask, *counter, *freq, *step, *compressed, *compressed_tc, *weight_sparse, *weight_sparse_T,
        *refreshed, *take, *refresh, *ensure, *tc_copies, *advance, *materialize, *into_grad, *parameter_type;
};
const LayerNames &layer_names() {       // made by the module's load, see PyObjects
    static const LayerNames n = [] {
        auto s = [](const char *t) { return PyUnicode_InternFromString(t); };
        return LayerNames{s("weight"), s("bias"), s("_parameters"), s("training"), s("mode"), s("cnt"), s("mask"), s("counter"), s("freq"), s("step"),
                          s("compressed"), s("compressed_tc"), s("weight_sparse"), s("weight_sparse_T"), s("refreshed"), s("_take"), s("_refresh"),
                          s("_ensure_compressed"), s("_tc_copies"), s("_advance"), s("materialize_sparse_tensors"), s("accumulate_into_grad"),
                          py::module_::import("torch.nn").attr("Parameter").cast<py::object>().release().ptr()};
    }();
    return n;
}
// What an instance holds itself, a new reference or null.
py::object own_dict(PyObject *o) {
    py::object d = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(o, nullptr));
    if (!d) PyErr_Clear();
    return d;
}
PyObject *item(const py::object &dict, PyObject *name) {      // borrowed, null where there is none
    PyObject *v = PyDict_GetItemWithError(dict.ptr(), name);
    if (!v && PyErr_Occurred()) throw py::error_already_set();
    return v;
}
void put(const py::object &dict, PyObject *name, PyObject *v) {
    if (PyDict_SetItem(dict.ptr(), name, v) < 0) throw py::error_already_set();
}
// The dictionary of a weight that is a plain torch.nn.Parameter, whose attributes of this package are kept there and nowhere else.
py::object weight_dict(PyObject *w) { return (PyObject *)Py_TYPE(w) == layer_names().parameter_type ? own_dict(w) : py::object(); }
// c % f == 0 as Python has it; -1 where the two are not plain integers of 64 bits
int due(PyObject *counter, PyObject *freq) {
    if (!counter || !freq || !PyLong_CheckExact(counter) || !PyLong_CheckExact(freq)) return -1;
    int over1 = 0, over2 = 0;
    const long long c = PyLong_AsLongLongAndOverflow(counter, &over1), f = PyLong_AsLongLongAndOverflow(freq, &over2);
    return over1 || over2 || f == 0 ? -1 : (f == -1 || c % f == 0);
}
bool is_sparse_mode(PyObject *mode) { return mode && PyUnicode_CheckExact(mode) && PyUnicode_CompareWithASCIIString(mode, "sparse") == 0; }
// What SparseLinearTranspose._take leaves on the weight, but for the mask.
void install(const py::object &w, const Copies &k) {
    const LayerNames &N = layer_names();
    const py::tuple held = py::make_tuple(k.pw, k.mw, k.pt, k.mt);
    put(w, N.compressed, held.ptr());
    if (k.tcw.defined())
        put(w, N.compressed_tc, py::make_tuple(held, (int64_t)k.mw._version(), (int64_t)k.mt._version(), py::make_tuple(k.tcw, k.tct)).ptr());
    else put(w, N.compressed_tc, Py_None);
    put(w, N.weight_sparse, Py_None);
    put(w, N.weight_sparse_T, Py_None);
}

struct Walk { PyObject *base_modules, *base_named, *modules, *named, *children; };
const Walk &walk_names() {       // made by the module's load, see PyObjects
    static const Walk w = [] {
        auto s = [](const char *t) { return PyUnicode_InternFromString(t); };
        const py::object cls = py::module_::import("torch.nn").attr("Module");
        return Walk{py::object(cls.attr("modules")).release().ptr(), py::object(cls.attr("named_modules")).release().ptr(), s("modules"), s("named_modules"),
                    s("_modules")};
    }();
    return w;
}
// ``model.modules()``, each once and in the same order, or None where a module has a walk of its own: torch's asks every module for its
// ``named_modules``, so one that has another, in its class or on the instance, decides what is below it; ``modules`` counts at the root
// only.  Without a generator per level of nesting, which for 48 layers took as long as the launch that refreshes them (in Python 25 us).
py::object modules(const py::object &model) {
    const Walk &W = walk_names();
    const py::object root = own_dict(model.ptr());
    if (!root || _PyType_Lookup(Py_TYPE(model.ptr()), W.modules) != W.base_modules || item(root, W.modules)) return py::none();
    const py::object seen = py::reinterpret_steal<py::object>(PySet_New(nullptr));
    py::list out;
    std::vector<py::object> stack{model};
    while (!stack.empty()) {
        const py::object mod = std::move(stack.back());
        stack.pop_back();
        if (mod.is_none()) continue;
        const int known = PySet_Contains(seen.ptr(), mod.ptr());
        if (known < 0) throw py::error_already_set();
        if (known) continue;
        PyTypeObject *const cls = Py_TYPE(mod.ptr());
        const py::object dict = own_dict(mod.ptr());
        if (!dict || _PyType_Lookup(cls, W.named) != W.base_named || item(dict, W.named) || _PyType_Lookup(cls, W.children)) return py::none();
        PyObject *const children = item(dict, W.children);
        if (!children || !PyDict_CheckExact(children)) return py::none();
        if (PySet_Add(seen.ptr(), mod.ptr()) < 0) throw py::error_already_set();
        out.append(mod);
        const size_t below = stack.size();
        PyObject *key, *child;
        for (Py_ssize_t at = 0; PyDict_Next(children, &at, &key, &child);) stack.push_back(py::reinterpret_borrow<py::object>(child));
        std::reverse(stack.begin() + below, stack.end());
    }
    return out;
}

std::pair<int64_t, py::list> refresh_layers(const py::list &mods, at::ScalarType t, const py::object &plain) {
    const LayerNames &N = layer_names();
    struct Group { bool reselect; at::ScalarType type; c10::Device device; std::vector<Tensor> weights, masks; std::vector<py::object> owners; };
    std::vector<Group> groups;
    py::list left;
    const py::object materialize = py::reinterpret_steal<py::object>(PyObject_GetAttr(plain.ptr(), N.materialize));
    if (!materialize) throw py::error_already_set();
    const bool plain_class = !PyObject_IsTrue(materialize.ptr());
    for (const py::handle mod : mods) {
        PyObject *params = nullptr, *w = nullptr;
        const py::object dict = plain_class && (PyObject *)Py_TYPE(mod.ptr()) == plain.ptr() ? own_dict(mod.ptr()) : py::object();
        // plain: the weight is the registered parameter, and nothing of its handling is replaced on the instance
        if (dict && !item(dict, N.weight) && !item(dict, N.take) && !item(dict, N.materialize) && (params = item(dict, N.parameters)) && PyDict_Check(params))
            w = item(py::reinterpret_borrow<py::object>(params), N.weight);
        const py::object wd = w && THPVariable_Check(w) ? weight_dict(w) : py::object();
        if (!wd) {
            left.append(mod);
            continue;
        }
        const Tensor &weight = THPVariable_Unpack(w);
        PyObject *mode = item(wd, N.mode), *cnt = item(wd, N.cnt), *mask_o = item(wd, N.mask);
        const int reselect = due(item(wd, N.counter), item(wd, N.freq));
        if (!mode || !PyUnicode_CheckExact(mode) || !cnt || !PyLong_CheckExact(cnt) || !mask_o || !THPVariable_Check(mask_o) || weight.dim() != 2) {
            left.append(mod);
            continue;
        }
        if (!is_sparse_mode(mode) || PyObject_IsTrue(cnt) || !weight.is_cuda()) continue;
        if (weight.size(0) % 128 || weight.size(1) % 128) continue;
        const Tensor &mask = THPVariable_Unpack(mask_o);
        if (mask.device() != weight.device() || mask.scalar_type() != at::kBool || !mask.is_contiguous() || reselect < 0) {
            left.append(mod);
            continue;
        }
        Group *g = nullptr;
        for (Group &have : groups)
            if (have.reselect == (bool)reselect && have.type == weight.scalar_type() && have.device == weight.device()) g = &have;
        if (!g) {
            groups.push_back({(bool)reselect, weight.scalar_type(), weight.device(), {}, {}, {}});
            g = &groups.back();
        }
        g->weights.push_back(weight);
        g->masks.push_back(mask);
        g->owners.push_back(wd);
    }
    int64_t done = 0;
    for (const Group &g : groups) {
        std::vector<Copies> copies;
        {
            py::gil_scoped_release nogil;
            copies = compress_all(g.weights, g.masks, t, g.reselect);
        }
        for (size_t i = 0; i < copies.size(); ++i) {
            install(g.owners[i], copies[i]);
            put(g.owners[i], N.refreshed, Py_True);
            ++done;
        }
    }
    return {done, left};
}

// ---------------------------------------------------------------------------------------------
// masked decay
// ---------------------------------------------------------------------------------------------
// True when done; false when the tensors need what the Python wrapper does for other types, layouts and alignments.
bool masked_add(const Tensor &grad, const Tensor &p, const Tensor &mask, double alpha) {
    if (!grad.is_cuda() || grad.layout() != at::kStrided || p.layout() != at::kStrided || mask.layout() != at::kStrided) return false;
    const auto mt = mask.scalar_type();     // the types whose zero test is the kernel's: bytes, or floats with either sign of zero
    const bool direct = mt == at::kBool || mt == at::kByte || mt == at::kChar || is16(mt) || mt == at::kFloat;
    if (grad.scalar_type() != at::kFloat || p.scalar_type() != at::kFloat || !direct) return false;
    if (grad.sizes() != p.sizes() || grad.sizes() != mask.sizes() || grad.strides() != p.strides() || grad.strides() != mask.strides()) return false;
    if (!grad.is_non_overlapping_and_dense() || !aligned(grad) || !aligned(p) || !aligned(mask, 4 * mask.element_size())) return false;
    const auto cur = c10::cuda::current_device();
    if (grad.device().index() != cur || p.device() != grad.device() || mask.device() != grad.device()) return false;
    check(sp24_masked_add(ptr(grad), ptr(p), ptr(mask), (int)mask.element_size(), grad.numel(), (float)alpha, cur_stream()), "sp24_masked_add");
    return true;
}

// masked_add(grad, p, mask, alpha) as a plain C function of the module: a model's decays are one call a weight, and the general
// argument conversion was a tenth of each.
PyObject *py_masked_add(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n == 4 && THPVariable_Check(args[0]) && THPVariable_Check(args[1]) && THPVariable_Check(args[2]),
                     "masked_add: expected three tensors and a number");
    const double alpha = PyFloat_AsDouble(args[3]);
    if (alpha == -1.0 && PyErr_Occurred()) return nullptr;
    const Tensor &grad = THPVariable_Unpack(args[0]), &p = THPVariable_Unpack(args[1]), &mask = THPVariable_Unpack(args[2]);
    bool done;
    {
        py::gil_scoped_release nogil;
        done = masked_add(grad, p, mask, alpha);
    }
    return PyBool_FromLong(done);
    END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------
// FST layer
// ---------------------------------------------------------------------------------------------
bool accumulable(const Tensor &grad) { return grad.defined() && grad.scalar_type() == at::kFloat && grad.is_contiguous(); }

// The layer's option for an exact weight gradient is a Python attribute of the weight and its GEMM is torch's.
bool wants_dense_weight_grad(const Tensor &weight) {
    py::object w = py::reinterpret_steal<py::object>(THPVariable_Wrap(weight));
    PyObject *v = PyObject_GetAttr(w.ptr(), py_objects.weight_grad);
    if (!v) {
        PyErr_Clear();
        return false;
    }
    const bool dense = PyUnicode_Check(v) && PyUnicode_CompareWithASCIIString(v, "dense") == 0;
    Py_DECREF(v);
    return dense;
}

// dW = MVUE24(g^T) x and db = g.sum(0); g (tokens, out_features) and x (tokens, in_features) in 16 bits.  One pass over g
// compresses it and takes the bias gradient.  into_grad: both are added to existing float32 .grad buffers and come back
// undefined.
std::pair<Tensor, Tensor> fst_weight_grads(const Tensor &g_in, const Tensor &x, const Tensor &weight, const Tensor &bias, bool into_grad,
                                           bool need_w, bool need_b) {
    need_b = need_b && bias.defined();
    uint64_t seed = 0;
    if (need_w) {
        py::gil_scoped_acquire gil;
        if (wants_dense_weight_grad(weight)) {
            TORCH_CHECK(py_objects.dense_weight_grads, "set_dense_weight_grads has not been called");
            py::object r = py::reinterpret_borrow<py::object>(py_objects.dense_weight_grads)(g_in, x, weight, bias.defined() ? py::cast(bias) : py::object(py::none()),
                                                                  into_grad, need_w, need_b);
            py::tuple t(r);
            return {t[0].is_none() ? Tensor() : py::cast<Tensor>(t[0]), t[1].is_none() ? Tensor() : py::cast<Tensor>(t[1])};
        }
        seed = python_seed();
    }
    Tensor gw, gb;
    if (need_b && recorded(g_in)) {
        gb = g_in.sum({0}, false, at::kFloat);
        need_b = false;
    }
    NoAutograd guard;
    if (need_w) {
        const Tensor g = g_in.contiguous();
        const int64_t tokens = g.size(0), out_f = g.size(1), in_f = x.size(1);
        TORCH_CHECK(out_f % 32 == 0 && tokens % 64 == 0, "gradient of shape (", tokens, ", ", out_f,
                    "): features % 32 == 0 and tokens % 64 == 0 required");
        const bool f32 = weight.scalar_type() == at::kFloat && in_f % 8 == 0;
        const bool into = into_grad && f32 && accumulable(weight.grad());
        Tensor sums, acc;
        if (into) {
            acc = weight.grad();
            if (need_b && accumulable(bias.grad())) sums = bias.grad();
        } else if (f32) {
            acc = gw = empty({out_f, in_f}, at::kFloat, g);      // the compression clears it for the GEMM that adds to it
            if (need_b && bias.scalar_type() == at::kFloat) sums = gb = empty({out_f}, at::kFloat, g);
        }
        // packed values, metadata, its tensor-core copy and partial bias sums, all consumed by the next launches
        const int64_t vb = out_f * tokens, mb = out_f * tokens / 8;
        const bool tc = out_f % 128 == 0;
        const int64_t o_tc = align256(vb + mb), o_parts = align256(o_tc + (tc ? sp24_meta_tc_bytes(out_f, tokens) : 0));
        Tensor buf = empty({o_parts + (sums.defined() ? row_parts_bytes(out_f, tokens, g.scalar_type()) : 0)}, at::kByte, g);
        const Tensor gp = carve(buf, 0, g.scalar_type(), {out_f, tokens / 2}, {1, out_f});
        const Tensor gm = carve(buf, vb, at::kShort, {out_f, tokens / 16}, {tokens / 16, 1});
        OptTensor e;
        if (tc) e = carve(buf, o_tc, at::kByte, {sp24_meta_tc_bytes(out_f, tokens)}, {1});
        RowSums rs;
        if (sums.defined()) rs = {static_cast<float *>(ptr(sums)), reinterpret_cast<float *>(static_cast<char *>(ptr(buf)) + o_parts), into};
        prune_into(g.t(), gp, gm, SP24_PRUNE_MVUE_FAST, {}, {}, seed, 0, false, {nullptr, rs.parts, false}, e, gw);
        if (sums.defined()) need_b = false;
        TORCH_CHECK(tc, "sparse GEMM on sm_100a: number of rows of the sparse matrix must be divisible by 128");
        if (acc.defined()) mm_accumulate(acc, gp, *e, x, 0, rs);
        else gw = spmm(x.t(), gp, *e, {}, 0, {}, false).t();
    }
    if (need_b) gb = g_in.sum(0);
    return {gw, gb};
}

struct FstBackward : torch::autograd::Node {
    torch::autograd::SavedVariable x_, pt_, tct_;
    Tensor weight_, bias_;
    std::vector<int64_t> shape_;
    bool into_grad_ = false, released_ = false;

    std::string name() const override { return "FstLinearBackward"; }
    void release_variables() override {
        x_.reset_data();
        pt_.reset_data();
        tct_.reset_data();
        released_ = true;
    }
    variable_list apply(variable_list &&grads) override {
        TORCH_CHECK(!released_, torch::autograd::ERR_BACKWARD_TWICE);
        variable_list out(3);
        Tensor g = grads[0];
        if (!g.defined()) return out;
        const Tensor x = x_.unpack(), pt = pt_.unpack(), tct = tct_.unpack();
        {
            c10::optional<NoAutograd> guard;
            if (!recorded(g)) guard.emplace();
            // the gradient of a plain sum arrives as one expanded value; the reference layer replaces it by ones
            if (g.dim() == 3 && g.stride(0) == 0 && g.stride(1) == 0 && g.stride(2) == 0) g = at::ones_like(g);
            if (g.dim() != 2) g = g.reshape({-1, g.size(-1)});
            if (g.scalar_type() != pt.scalar_type()) g = g.to(pt.scalar_type());
            if (task_should_compute_output(0)) {
                if (!guard) guard.emplace();
                Tensor dx = spmm(g, pt, tct, {}, 0, {}, false);
                out[0] = dx.dim() == (int64_t)shape_.size() ? dx : dx.view(shape_);
            }
        }
        if (task_should_compute_output(1) || task_should_compute_output(2)) {
            auto [gw, gb] = fst_weight_grads(g, x, weight_, bias_, into_grad_, task_should_compute_output(1), task_should_compute_output(2));
            out[1] = gw;
            out[2] = gb;
        }
        return out;
    }
};

Tensor unpack(PyObject *o) {
    TORCH_CHECK(THPVariable_Check(o), "expected a tensor");
    return THPVariable_Unpack(o);
}

// y = x W_s^T + b on the compressed copies
Tensor fst_product(const Tensor &input, const Tensor &weight, const OptTensor &bias, const Tensor &pw, const Tensor &pt, const Tensor &tcw, const Tensor &tct,
                   bool into_grad) {
    require_cuda(input, pw, pt, tcw, tct, bias);
    no_tangent(input, weight, bias);
    Tensor x, y;
    {
        NoAutograd guard;
        x = rows2d(input);
        if (x.scalar_type() != pw.scalar_type()) x = x.to(pw.scalar_type());
        y = spmm(x, pw, tcw, bias, 0, {}, false, true);
        if (input.dim() != 2) {
            auto shape = input.sizes().vec();
            shape.back() = pw.size(0);
            y = y.view(shape);
        }
    }
    const Tensor b = bias.has_value() ? *bias : Tensor();
    if (torch::autograd::compute_requires_grad(input, weight, b)) {
        auto node = std::shared_ptr<FstBackward>(new FstBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(input, weight, b));
        node->x_ = torch::autograd::SavedVariable(x, false);
        node->pt_ = torch::autograd::SavedVariable(pt, false);
        node->tct_ = torch::autograd::SavedVariable(tct, false);
        node->weight_ = weight;
        node->bias_ = b;
        node->shape_ = input.sizes().vec();
        node->into_grad_ = into_grad;
        torch::autograd::set_history(y, node);
    }
    return y;
}
// copies: (packed_w, meta_w, packed_t, meta_t); tc = their metadata in tensor-core order.
Tensor fst_linear(const Tensor &input, const Tensor &weight, const OptTensor &bias, const py::tuple &copies, const py::tuple &tc, bool into_grad) {
    const Tensor pw = unpack(copies[0].ptr()), pt = unpack(copies[2].ptr()), tcw = unpack(tc[0].ptr()), tct = unpack(tc[1].ptr());
    py::gil_scoped_release nogil;
    return fst_product(input, weight, bias, pw, pt, tcw, tct, into_grad);
}

// The class whose forward fst_forward knows, and its five methods that take part: replaced ones are called by Python instead.
struct LayerClass {
    PyTypeObject *type = nullptr;
    PyObject *methods[5] = {};
} layer_class;
void set_layer_class(const py::object &cls) {
    const LayerNames &N = layer_names();
    PyObject *const names[5] = {N.take, N.refresh, N.ensure, N.tc_copies, N.advance};
    for (int i = 0; i < 5; ++i) {
        layer_class.methods[i] = PyObject_GetAttr(cls.ptr(), names[i]);
        if (!layer_class.methods[i]) throw py::error_already_set();
    }
    layer_class.type = (PyTypeObject *)cls.inc_ref().ptr();
}
bool layer_class_untouched() {
    const LayerNames &N = layer_names();
    PyObject *const names[5] = {N.take, N.refresh, N.ensure, N.tc_copies, N.advance};
    for (int i = 0; i < 5; ++i)
        if (_PyType_Lookup(layer_class.type, names[i]) != layer_class.methods[i]) return false;
    return _PyType_Lookup(layer_class.type, N.materialize) == Py_False;
}
void add_one(const py::object &dict, PyObject *name, PyObject *v) {
    const py::object one = py::reinterpret_steal<py::object>(PyLong_FromLong(1)), sum = py::reinterpret_steal<py::object>(PyNumber_Add(v, one.ptr()));
    if (!sum) throw py::error_already_set();
    put(dict, name, sum.ptr());
}

// fst_forward(layer, x): SparseLinearTranspose.forward of a plain layer in sparse mode, state and all; None where anything about the call is
// not plain, before anything was changed: the class's own Python takes the call then.  In Python the attributes, tuples and frames
// of a call were a third of a small layer's forward.
PyObject *py_fst_forward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const LayerNames &N = layer_names();
    if (n != 2 || Py_TYPE(args[0]) != layer_class.type || !THPVariable_Check(args[1]) || torch::jit::tracer::isTracing() || !layer_class_untouched())
        Py_RETURN_NONE;
    const py::object dict = own_dict(args[0]);
    if (!dict || item(dict, N.weight) || item(dict, N.bias) || item(dict, N.take) || item(dict, N.refresh) || item(dict, N.ensure) ||
        item(dict, N.tc_copies) || item(dict, N.advance) || item(dict, N.materialize))
        Py_RETURN_NONE;
    PyObject *const params_o = item(dict, N.parameters), *const training = item(dict, N.training);
    if (!params_o || !PyDict_Check(params_o) || (training != Py_True && training != Py_False)) Py_RETURN_NONE;
    const py::object params = py::reinterpret_borrow<py::object>(params_o);
    PyObject *const w_o = item(params, N.weight), *const b_o = item(params, N.bias);
    if (!w_o || !THPVariable_Check(w_o) || !b_o || (b_o != Py_None && !THPVariable_Check(b_o))) Py_RETURN_NONE;
    const py::object wd = weight_dict(w_o);
    if (!wd) Py_RETURN_NONE;
    PyObject *const cnt = item(wd, N.cnt), *const mask_o = item(wd, N.mask), *const step = item(wd, N.step), *const counter = item(wd, N.counter);
    if (!is_sparse_mode(item(wd, N.mode)) || !cnt || !PyLong_CheckExact(cnt) || !step || !PyLong_CheckExact(step) || !counter || !PyLong_CheckExact(counter) ||
        !mask_o || !THPVariable_Check(mask_o))
        Py_RETURN_NONE;
    const Tensor weight = THPVariable_Unpack(w_o), mask = THPVariable_Unpack(mask_o), x = THPVariable_Unpack(args[1]);
    const OptTensor bias = b_o == Py_None ? OptTensor() : OptTensor(THPVariable_Unpack(b_o));
    if (mask.device() != weight.device()) Py_RETURN_NONE;
    PyObject *into = item(dict, N.into_grad);
    if (!into) into = _PyType_Lookup(layer_class.type, N.into_grad);
    if (into != Py_True && into != Py_False) Py_RETURN_NONE;
    const bool first = PyObject_IsTrue(cnt) == 0;
    PyObject *const refreshed = item(wd, N.refreshed);
    if (refreshed && refreshed != Py_True && refreshed != Py_False) Py_RETURN_NONE;
    const bool compress_now = first && refreshed != Py_True;

    Tensor pw, pt, tcw, tct;
    if (compress_now) {
        const int reselect = due(counter, item(wd, N.freq));
        // whole 128 x 128 blocks: the launch leaves the metadata in the GEMM's order too
        if (reselect < 0 || weight.dim() != 2 || weight.size(0) % 128 || weight.size(1) % 128) Py_RETURN_NONE;
        // a reselected mask overwrites the existing buffer, so that it keeps one address for the whole run
        const bool reuse = reselect && mask.is_cuda() && mask.is_contiguous() && mask.scalar_type() == at::kBool;
        const bool bf16 = at::autocast::is_autocast_enabled(at::kCUDA) && at::autocast::get_autocast_dtype(at::kCUDA) == at::kBFloat16;
        Tensor used;
        c10::optional<Copies> c;
        {
            py::gil_scoped_release nogil;
            c.emplace(select_copies(weight, reselect ? OptTensor() : OptTensor(mask), bf16 ? at::kBFloat16 : at::kHalf,
                                    reuse ? OptTensor(mask) : OptTensor(), used));
        }
        if (!used.is_same(mask)) put(wd, N.mask, py::cast(used).ptr());
        install(wd, *c);
        pw = c->pw;
        pt = c->pt;
        tcw = c->tcw;
        tct = c->tct;
    } else {
        // the copies at hand and their metadata in the GEMM's order, if both are still what the compression left
        PyObject *const held = item(wd, N.compressed), *const tc = item(wd, N.compressed_tc);
        if (!held || !PyTuple_CheckExact(held) || PyTuple_GET_SIZE(held) != 4 || !tc || !PyTuple_CheckExact(tc) || PyTuple_GET_SIZE(tc) != 4 ||
            PyTuple_GET_ITEM(tc, 0) != held)
            Py_RETURN_NONE;
        for (int i = 0; i < 4; ++i)
            if (!THPVariable_Check(PyTuple_GET_ITEM(held, i))) Py_RETURN_NONE;
        PyObject *const order = PyTuple_GET_ITEM(tc, 3);
        auto version = [](const Tensor &t, PyObject *v) { return !t.is_inference() && PyLong_CheckExact(v) && PyLong_AsLongLong(v) == (long long)t._version(); };
        if (!PyTuple_CheckExact(order) || PyTuple_GET_SIZE(order) != 2 || !THPVariable_Check(PyTuple_GET_ITEM(order, 0)) ||
            !THPVariable_Check(PyTuple_GET_ITEM(order, 1)) || !version(THPVariable_Unpack(PyTuple_GET_ITEM(held, 1)), PyTuple_GET_ITEM(tc, 1)) ||
            !version(THPVariable_Unpack(PyTuple_GET_ITEM(held, 3)), PyTuple_GET_ITEM(tc, 2)))
            Py_RETURN_NONE;
        pw = THPVariable_Unpack(PyTuple_GET_ITEM(held, 0));
        pt = THPVariable_Unpack(PyTuple_GET_ITEM(held, 2));
        tcw = THPVariable_Unpack(PyTuple_GET_ITEM(order, 0));
        tct = THPVariable_Unpack(PyTuple_GET_ITEM(order, 1));
        if (first) put(wd, N.refreshed, Py_False);
    }
    Tensor y;
    {
        py::gil_scoped_release nogil;
        y = fst_product(x, weight, bias, pw, pt, tcw, tct, into == Py_True);
    }
    if (training == Py_True) {
        // read again: a saved-tensor hook may have run Python since
        PyObject *const c = item(wd, N.cnt), *const s = item(wd, N.step), *const o = item(wd, N.counter);
        if (!c || !s || !o) {
            PyErr_SetString(PyExc_AttributeError, "the weight's counters are gone");
            return nullptr;
        }
        if (PyObject_IsTrue(c) == 0) add_one(wd, N.counter, o);
        add_one(wd, N.step, s);
        add_one(wd, N.cnt, c);
    }
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------
// float8 FST layer: the per-tensor scales never leave the device
// ---------------------------------------------------------------------------------------------
Tensor absmax(const Tensor &x, const Tensor &mask = {}) {
    Tensor a = empty({1}, at::kFloat, x);
    check(sp24_absmax(ptr(x), dt(x.scalar_type()), x.numel(), mask.defined() ? ptr(mask) : nullptr, static_cast<float *>(ptr(a)), cur_stream()),
          "sp24_absmax");
    return a;
}
// contiguous and on a 16-byte boundary (a view into a larger buffer may start anywhere)
Tensor quantizable(const Tensor &t) {
    const Tensor c = (t.scalar_type() == at::kFloat || is16(t.scalar_type()) ? t : t.to(at::kFloat)).contiguous();
    return aligned(c) ? c : c.clone();
}

struct Q8 {
    Tensor packed, meta, tc;
    RowSums sums;
    // room for the compressed (m, k) matrix, `extra` bytes behind the result
    Tensor make(int64_t m, int64_t k, int64_t extra, const Tensor &like) {
        const int64_t vb = m * k / 2, mb = m * k / 8, tb = m % 128 == 0 ? sp24_meta_tc_bytes(m, k) : 0;
        const int64_t end = align256(align256(vb) + align256(mb) + tb);
        const Tensor buf = empty({end + extra}, at::kByte, like);
        packed = carve(buf, 0, at::kFloat8_e4m3fn, {m, k / 2}, {k / 2, 1});
        meta = carve(buf, align256(vb), at::kInt, {m, k / 32}, {k / 32, 1});
        if (tb) tc = carve(buf, align256(vb) + align256(mb), at::kByte, {tb}, {1});
        return carve(buf, end, at::kByte, {extra}, {1});
    }
};
// e4m3 2:4 compression of the logical (m, k) matrix `dense` under the scale of *amax, packed values row-major.
// row_sums: o.sums says how the next launch gets them; its parts live as long as o.packed.
Q8 compress_q8(const Tensor &dense_in, int mode, const OptTensor &mask_in, const Tensor &amax, uint64_t seed, const Tensor &row_sums,
               const Tensor &q_dense, const Tensor &clear = {}) {
    const int64_t m = dense_in.size(0), k = dense_in.size(1);
    TORCH_CHECK(m % 32 == 0 && k % 128 == 0, "compress_q8: shape (", m, ", ", k, "): rows % 32 == 0 and columns % 128 == 0 required");
    Tensor dense = dense_in;
    Layout l = layout_of(dense);
    if (!usable(dense, l)) {
        dense = dense.contiguous();
        l = {0, k};
    }
    OptTensor mask = mask_in;
    int64_t ld_m = 0;
    if (mask.has_value()) {
        mask = as_layout(*mask, l.col);
        ld_m = layout_of(*mask).ld;
    }
    Q8 o;
    const Tensor parts = o.make(m, k, row_sums.defined() ? row_parts_bytes(m, k, at::kFloat8_e4m3fn) : 0, dense);
    sp24_prune_extras x{};
    x.amax = static_cast<const float *>(ptr(amax));
    x.offset_dev = rng_offset_ptr(mode);
    x.packed_row_major = 1;
    if (o.tc.defined()) x.e_tc = ptr(o.tc);
    if (row_sums.defined()) {
        o.sums = {static_cast<float *>(ptr(row_sums)), static_cast<float *>(ptr(parts)), false};
        x.row_parts = o.sums.parts;
    }
    if (q_dense.defined()) {
        x.q_dense = ptr(q_dense);
        x.ld_q = q_dense.size(1);
    }
    if (clear.defined() && l.col)
        check(sp24_mvue_compress_clearing(ptr(dense), dt(dense.scalar_type()), m, k, l.ld, ptr(o.packed), SP24_E4M3, k / 2, ptr(o.meta), seed, 0,
                                          &x, ptr(clear), clear.nbytes(), cur_stream()),
              "sp24_mvue_compress_clearing");
    else {
        if (clear.defined()) check(sp24_zero(ptr(clear), clear.nbytes(), cur_stream()), "sp24_zero");
        check(sp24_prune_compress_with(ptr(dense), dt(dense.scalar_type()), m, k, l.ld, l.col, ptr(o.packed), SP24_E4M3, k / 2, ptr(o.meta),
                                       mode, ptr(mask), ld_m, nullptr, 0, seed, 0, &x, cur_stream()),
              "sp24_prune_compress_q8");
    }
    return o;
}

// (absolute maximum of the masked weight, W: packed, meta, tc, W^T: packed, meta, tc)
py::tuple fp8_weight(const Tensor &w, const Tensor &mask_in) {
    Tensor amax;
    Q8 a, b;
    {
        py::gil_scoped_release nogil;
        NoAutograd guard;
        require_cuda(w, mask_in);
        const Tensor mask = mask_in.scalar_type() == at::kBool ? mask_in : mask_in.ne(0);
        const bool direct = w.scalar_type() == at::kFloat && w.is_contiguous() && mask.is_contiguous() && w.sizes() == mask.sizes() &&
                            w.numel() % 4 == 0 && aligned(w) && aligned(mask);
        amax = direct ? absmax(w, mask) : absmax(quantizable(at::where(mask, w, at::zeros({}, w.options()))));
        const int64_t m = w.size(0), k = w.size(1);
        const Layout l = layout_of(w);
        // one read for both where W is row-major in whole 128 x 128 blocks
        if (l.col == 0 && usable(w, l) && (w.scalar_type() == at::kFloat || is16(w.scalar_type())) && mask.is_contiguous() && aligned(mask, 4) &&
            mask.sizes() == w.sizes() && m % 128 == 0 && k % 128 == 0 && m <= 64 * 65535 && m && k) {
            a.make(m, k, 0, w);
            b.make(k, m, 0, w);
            check(sp24_dual_compress_f8(ptr(w), dt(w.scalar_type()), m, k, l.ld, ptr(mask), k, static_cast<const float *>(ptr(amax)), ptr(a.packed),
                                        ptr(a.meta), ptr(a.tc), ptr(b.packed), ptr(b.meta), ptr(b.tc), cur_stream()),
                  "sp24_dual_compress_f8");
        } else {
            a = compress_q8(w, SP24_PRUNE_MASK, mask, amax, 0, {}, {});
            b = compress_q8(w.t(), SP24_PRUNE_MASK, mask.t(), amax, 0, {}, {});
        }
    }
    auto opt = [](const Tensor &t) { return t.defined() ? py::cast(t) : py::object(py::none()); };
    return py::make_tuple(amax, a.packed, a.meta, opt(a.tc), b.packed, b.meta, opt(b.tc));
}

// input (n, k) e4m3 times the compressed weight, as (n, ms) in `out_t`
Tensor spmm_f8(const Tensor &packed, const Tensor &tc, const Tensor &amax_w, const Tensor &xq, const Tensor &amax_x, const Tensor &bias,
               at::ScalarType out_t) {
    const int64_t ms = packed.size(0), k = 2 * packed.size(1), n = xq.size(0);
    TORCH_CHECK(xq.size(1) == k, "_sparse_semi_structured_linear: Expected weight argument to have ", xq.size(1) / 2, " columns, but got ", k / 2);
    TORCH_CHECK(tc.defined(), "sparse GEMM on sm_100a: number of rows of the sparse matrix must be divisible by 128");
    const auto kt = is16(out_t) ? out_t : at::kFloat;
    Tensor out = empty({n, ms}, kt, xq);
    check(sp24_spmm_f8(ptr(packed), SP24_E4M3, packed.stride(0), ptr(tc), ms, k, ptr(xq), xq.stride(0), n, ptr(out), dt(kt), 1, ms,
                       bias.defined() ? static_cast<const float *>(ptr(bias)) : nullptr, static_cast<const float *>(ptr(amax_w)),
                       static_cast<const float *>(ptr(amax_x)), status_ptr(xq), cur_stream()),
          "sp24_spmm_f8");
    return kt == out_t ? out : out.to(out_t);
}

struct Fp8Backward : torch::autograd::Node {
    torch::autograd::SavedVariable xq_t_;
    Tensor amax_x_, amax_w_, pt_, tct_;
    bool has_bias_ = false;
    std::vector<int64_t> shape_;
    at::ScalarType dtype_ = at::kFloat;

    std::string name() const override { return "Fp8LinearBackward"; }
    void release_variables() override {
        xq_t_.reset_data();
        pt_.reset();
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(3);
        if (!grads[0].defined()) return out;
        TORCH_CHECK(pt_.defined(), torch::autograd::ERR_BACKWARD_TWICE);
        const bool need_x = task_should_compute_output(0), need_w = task_should_compute_output(1);
        bool need_b = has_bias_ && task_should_compute_output(2);
        uint64_t seed = 0;
        if (need_w) {
            py::gil_scoped_acquire gil;
            seed = python_seed();
        }
        if (need_b && recorded(grads[0])) {
            out[2] = grads[0].reshape({-1, grads[0].size(-1)}).sum({0}, false, at::kFloat);
            need_b = false;
        }
        NoAutograd guard;
        const Tensor g = quantizable(grads[0].reshape({-1, grads[0].size(-1)}));
        const int64_t n = g.size(0), of = g.size(1);
        const Tensor amax = absmax(g);
        Tensor gq;
        if (need_x) gq = empty({n, of}, at::kFloat8_e4m3fn, g);
        if (need_w) {
            // one pass over dY: the MVUE compression of dY^T, the quantised dY and the bias gradient
            const Tensor xq_t = xq_t_.unpack();
            const int64_t in_f = xq_t.size(0);
            Tensor gw = empty({of, in_f}, at::kFloat, g), gb = need_b ? empty({of}, at::kFloat, g) : Tensor();
            const Q8 c = compress_q8(g.t(), SP24_PRUNE_MVUE_FAST, {}, amax, seed, gb, gq, gw);
            TORCH_CHECK(c.tc.defined(), "sparse GEMM on sm_100a: number of rows of the sparse matrix must be divisible by 128");
            const float *scale_g = static_cast<const float *>(ptr(amax)), *scale_x = static_cast<const float *>(ptr(amax_x_));
            if (c.sums.out)
                check(sp24_spmm_f8_sums(ptr(c.packed), SP24_E4M3, n / 2, ptr(c.tc), of, n, ptr(xq_t), n, in_f, static_cast<float *>(ptr(gw)), in_f,
                                        scale_g, scale_x, c.sums.parts, sp24_row_parts(n, SP24_E4M3), c.sums.out, c.sums.add, status_ptr(g),
                                        cur_stream()),
                      "sp24_spmm_f8_sums");
            else
                check(sp24_spmm_f8(ptr(c.packed), SP24_E4M3, n / 2, ptr(c.tc), of, n, ptr(xq_t), n, in_f, ptr(gw), SP24_F32, 0, in_f, nullptr, scale_g,
                                   scale_x, status_ptr(g), cur_stream()),
                      "sp24_spmm_f8");
            out[1] = gw;
            if (need_b) out[2] = gb;
            need_b = false;
        } else if (need_x) {
            check(sp24_quantize_f8(ptr(g), dt(g.scalar_type()), n, of, of, static_cast<const float *>(ptr(amax)), ptr(gq), nullptr, 0, cur_stream()),
                  "sp24_quantize_f8");
        }
        if (need_x) out[0] = spmm_f8(pt_, tct_, amax_w_, gq, amax, {}, dtype_).view(shape_);
        if (need_b) out[2] = g.sum(0);
        return out;
    }
};

Tensor fp8_linear(const Tensor &input, const Tensor &weight, const OptTensor &bias_in, const Tensor &amax_w, const Tensor &pw,
                  const OptTensor &tcw, const Tensor &pt, const OptTensor &tct) {
    require_cuda(input, pw, pt, bias_in);
    no_tangent(input, weight, bias_in);
    const Tensor bias = bias_in.has_value() ? *bias_in : Tensor();
    const bool tape = torch::autograd::compute_requires_grad(input, weight, bias);
    Tensor y, xq_t, amax;
    {
        NoAutograd guard;
        const Tensor x = quantizable(rows2d(input));
        const int64_t n = x.size(0), k = x.size(1);
        amax = absmax(x);
        Tensor xq = empty({n, k}, at::kFloat8_e4m3fn, x);
        if (tape && weight.requires_grad()) xq_t = empty({k, n}, at::kFloat8_e4m3fn, x);
        check(sp24_quantize_f8(ptr(x), dt(x.scalar_type()), n, k, k, static_cast<const float *>(ptr(amax)), ptr(xq),
                               xq_t.defined() ? ptr(xq_t) : nullptr, n, cur_stream()),
              "sp24_quantize_f8");
        const Tensor b = bias.defined() ? bias.to(at::kFloat).contiguous() : Tensor();
        if (b.defined())
            TORCH_CHECK(b.dim() == 1 && b.size(0) == pw.size(0), "_sparse_semi_structured_linear: Expected bias argument to have ", pw.size(0),
                        " elements, but got ", b.numel());
        y = spmm_f8(pw, tcw.has_value() ? *tcw : Tensor(), amax_w, xq, amax, b, input.scalar_type());
        if (input.dim() != 2) {
            auto shape = input.sizes().vec();
            shape.back() = pw.size(0);
            y = y.view(shape);
        }
    }
    if (tape) {
        auto node = std::shared_ptr<Fp8Backward>(new Fp8Backward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(input, weight, bias));
        node->xq_t_ = torch::autograd::SavedVariable(xq_t, false);
        node->amax_x_ = amax;
        node->amax_w_ = amax_w;
        node->pt_ = pt;
        node->tct_ = tct.has_value() ? *tct : Tensor();
        node->has_bias_ = bias.defined();
        node->shape_ = input.sizes().vec();
        node->dtype_ = input.scalar_type();
        torch::autograd::set_history(y, node);
    }
    return y;
}

// ---------------------------------------------------------------------------------------------
// S-STE layer: forward on the sparse tensor cores, both gradients dense (the soft-threshold mask is 2:4 along the rows
// of W only, so W_s^T has no sparse form, and the weight gradient is the straight-through dY^T X)
// ---------------------------------------------------------------------------------------------
struct SoftThresholdBackward : torch::autograd::Node {
    torch::autograd::SavedVariable x_, packed_, meta_;
    bool released_ = false, has_bias_ = false, w_f32_ = false;
    std::vector<int64_t> shape_;

    std::string name() const override { return "SoftThresholdLinearBackward"; }
    void release_variables() override {
        x_.reset_data();
        packed_.reset_data();
        meta_.reset_data();
        released_ = true;
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(3);
        if (!grads[0].defined()) return out;
        TORCH_CHECK(!released_, torch::autograd::ERR_BACKWARD_TWICE);
        const Tensor x = x_.unpack(), packed = packed_.unpack(), meta = meta_.unpack();
        const int64_t m = packed.size(0), k = 2 * packed.size(1);
        Tensor w;
        if (task_should_compute_output(0)) {
            NoAutograd guard;
            w = empty({m, k}, packed.scalar_type(), packed);
            check(sp24_to_dense(ptr(packed), dt(w.scalar_type()), m, k, k / 2, ptr(meta), ptr(w), k, cur_stream()), "sp24_to_dense");
        }
        if (recorded(grads[0])) {
            // all three are linear in dY; the products of 16-bit values are taken on float32 copies, exact operands either way
            const Tensor g = grads[0].reshape({-1, grads[0].size(-1)}).to(packed.scalar_type());
            if (w.defined()) out[0] = at::mm(g, w).view(shape_);
            if (task_should_compute_output(1)) out[1] = w_f32_ ? at::mm(g.t().to(at::kFloat), x.to(at::kFloat)) : at::mm(g.t(), x);
            if (has_bias_ && task_should_compute_output(2)) out[2] = g.sum({0}, false, at::kFloat);
            return out;
        }
        NoAutograd guard;
        const Tensor g = grads[0].reshape({-1, grads[0].size(-1)}).to(packed.scalar_type());
        if (w.defined()) out[0] = at::mm(g, w).view(shape_);
        if (task_should_compute_output(1)) out[1] = w_f32_ ? at::mm(g.t(), x, at::kFloat) : at::mm(g.t(), x);
        if (has_bias_ && task_should_compute_output(2)) {
            if (g.is_contiguous() && g.size(1) % 8 == 0 && aligned(g)) {
                Tensor s = empty({g.size(1)}, at::kFloat, g);
                check(sp24_column_sums_set(ptr(g), dt(g.scalar_type()), g.size(0), g.size(1), g.size(1), static_cast<float *>(ptr(s)), cur_stream()),
                      "sp24_column_sums_set");
                out[2] = s;
            } else {
                out[2] = g.sum(0);
            }
        }
        return out;
    }
};

// (packed, meta, tc or none) of S(weight) * scale
std::tuple<Tensor, Tensor, OptTensor> soft_threshold_compress(const Tensor &weight, c10::optional<double> scale, at::ScalarType t) {
    NoAutograd guard;
    require_cuda(weight);
    TORCH_CHECK(weight.dim() == 2, "Expected 2-dimensional dense tensor, got ", weight.dim(), "-dimensional tensor");
    TORCH_CHECK(is16(t), "soft_threshold24_compress: packed dtype must be float16 or bfloat16, got ", t);
    const int64_t m = weight.size(0), k = weight.size(1);
    TORCH_CHECK(m % 32 == 0 && k % 64 == 0, "soft_threshold24_compress: shape (", m, ", ", k, "): rows % 32 == 0 and columns % 64 == 0 required");
    const Tensor w = as_layout(weight, 0);
    auto [packed, meta] = carve_compressed(m, k, t, false, w);
    OptTensor e;
    if (m % 128 == 0) e = empty({sp24_meta_tc_bytes(m, k)}, at::kByte, w);
    check(sp24_soft_threshold24_compress(ptr(w), dt(w.scalar_type()), m, k, layout_of(w).ld, 0, ptr(packed), dt(t), k / 2, ptr(meta),
                                         scale.has_value(), (float)scale.value_or(0.0), const_cast<void *>(ptr(e)), cur_stream()),
          "sp24_soft_threshold24_compress");
    return {packed, meta, e};
}

Tensor soft_threshold_linear(const Tensor &input, const Tensor &weight, const OptTensor &bias, double scale, at::ScalarType t) {
    no_tangent(input, weight, bias);
    auto [packed, meta, e] = soft_threshold_compress(weight.detach(), scale, t);
    TORCH_CHECK(e.has_value(), "sparse GEMM on sm_100a: number of rows of the sparse matrix must be divisible by 128");
    require_cuda(input, bias);
    Tensor x, y;
    {
        NoAutograd guard;
        x = rows2d(input).to(t);
        y = spmm(x, packed, *e, bias, 0, {}, false, true);
        if (input.dim() != 2) {
            auto shape = input.sizes().vec();
            shape.back() = packed.size(0);
            y = y.view(shape);
        }
    }
    const Tensor b = bias.has_value() ? *bias : Tensor();
    if (torch::autograd::compute_requires_grad(input, weight, b)) {
        auto node = std::shared_ptr<SoftThresholdBackward>(new SoftThresholdBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(input, weight, b));
        node->x_ = torch::autograd::SavedVariable(x, false);
        node->packed_ = torch::autograd::SavedVariable(packed, false);
        node->meta_ = torch::autograd::SavedVariable(meta, false);
        node->has_bias_ = b.defined();
        node->w_f32_ = weight.scalar_type() == at::kFloat;
        node->shape_ = input.sizes().vec();
        torch::autograd::set_history(y, node);
    }
    return y;
}

// ---------------------------------------------------------------------------------------------
// trainer ops around the GEMMs
// ---------------------------------------------------------------------------------------------
// Where a backward kernel adds two parameter gradients: straight into existing float32 .grad buffers (autograd then
// receives nothing), or into a zeroed temporary of shape (2, d).
struct AffineGrads {
    Tensor g, b, rg, rb;
    AffineGrads(const Tensor &weight, const Tensor &bias, bool into, int64_t d, const Tensor &like) {
        if (into && accumulable(weight.grad()) && accumulable(bias.grad())) {
            g = weight.grad();
            b = bias.grad();
            return;
        }
        Tensor buf = empty({2 * d}, at::kFloat, like);
        check(sp24_zero(ptr(buf), 2 * d * 4, cur_stream()), "sp24_zero");
        g = rg = carve(buf, 0, at::kFloat, {d}, {1});
        b = rb = carve(buf, d * 4, at::kFloat, {d}, {1});
    }
};

struct LayerNormBackward : torch::autograd::Node {
    torch::autograd::SavedVariable x_, stats_;
    Tensor weight_, bias_;
    std::vector<int64_t> shape_;
    at::ScalarType x_dtype_ = at::kFloat;
    bool into_grad_ = false, released_ = false;

    std::string name() const override { return "SparseLayerNormBackward"; }
    void release_variables() override {
        x_.reset_data();
        stats_.reset_data();
        released_ = true;
    }
    variable_list apply(variable_list &&grads) override {
        TORCH_CHECK(!released_, torch::autograd::ERR_BACKWARD_TWICE);
        variable_list out(3);
        if (!grads[0].defined()) return out;
        const Tensor x = x_.unpack(), stats = stats_.unpack();
        NoAutograd guard;
        const int64_t rows = x.size(0), d = x.size(1);
        Tensor dy = grads[0].reshape({rows, d});
        if (dy.scalar_type() != at::kFloat && !is16(dy.scalar_type())) dy = dy.to(at::kFloat);
        dy = dy.contiguous();
        Tensor dx = at::empty_like(x);
        AffineGrads t(weight_, bias_, into_grad_, d, x);
        const float *st = static_cast<const float *>(ptr(stats));
        check(sp24_layernorm_bwd(ptr(dy), dt(dy.scalar_type()), static_cast<const float *>(ptr(x)), static_cast<const float *>(ptr(weight_)), st,
                                 st + rows, static_cast<float *>(ptr(dx)), static_cast<float *>(ptr(t.g)), static_cast<float *>(ptr(t.b)), rows, d,
                                 cur_stream()),
              "sp24_layernorm_bwd");
        out[0] = dx.view(shape_).to(x_dtype_);
        out[1] = t.rg;
        out[2] = t.rb;
        return out;
    }
};

Tensor layer_norm(const Tensor &input, const Tensor &weight, const Tensor &bias, double eps, at::ScalarType out_t, bool into_grad) {
    require_cuda(input, weight, bias);
    no_tangent(input, weight, bias);
    Tensor x, out, stats;
    {
        NoAutograd guard;
        const int64_t d = input.size(-1);
        x = rows2d(input);
        if (x.scalar_type() != at::kFloat) x = x.to(at::kFloat);
        x = x.contiguous();
        const int64_t rows = x.size(0);
        out = empty(input.sizes(), out_t, x);
        stats = empty({2 * rows}, at::kFloat, x);             // mean, then reciprocal standard deviation
        float *st = static_cast<float *>(ptr(stats));
        check(sp24_layernorm_fwd(static_cast<const float *>(ptr(x)), static_cast<const float *>(ptr(weight)), static_cast<const float *>(ptr(bias)),
                                 ptr(out), dt(out_t), st, st + rows, rows, d, (float)eps, cur_stream()),
              "sp24_layernorm_fwd");
    }
    if (torch::autograd::compute_requires_grad(input, weight, bias)) {
        auto node = std::shared_ptr<LayerNormBackward>(new LayerNormBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(input, weight, bias));
        node->x_ = torch::autograd::SavedVariable(x, false);
        node->stats_ = torch::autograd::SavedVariable(stats, false);
        node->weight_ = weight;
        node->bias_ = bias;
        node->shape_ = input.sizes().vec();
        node->x_dtype_ = input.scalar_type();
        node->into_grad_ = into_grad;
        torch::autograd::set_history(out, node);
    }
    return out;
}

// (x + delta, layer_norm(x + delta)); backward: the gradient arriving along the residual stream is added to the norm's
// input gradient and the sum goes to both inputs (float32 for x, delta's type for delta).
struct AddLayerNormBackward : torch::autograd::Node {
    torch::autograd::SavedVariable res_, stats_;
    Tensor weight_, bias_;
    std::vector<int64_t> shape_;
    at::ScalarType delta_dtype_ = at::kFloat;
    bool into_grad_ = false, released_ = false;

    std::string name() const override { return "SparseAddLayerNormBackward"; }
    void release_variables() override {
        res_.reset_data();
        stats_.reset_data();
        released_ = true;
    }
    variable_list apply(variable_list &&grads) override {
        TORCH_CHECK(!released_, torch::autograd::ERR_BACKWARD_TWICE);
        variable_list out(4);
        const Tensor &grad_res = grads[0];
        Tensor grad_out = grads[1];
        if (!grad_res.defined() && !grad_out.defined()) return out;
        const Tensor res = res_.unpack(shared_from_this()), stats = stats_.unpack();
        NoAutograd guard;
        const int64_t d = shape_.back(), rows = res.numel() / d;
        if (!grad_out.defined()) grad_out = at::zeros(shape_, res.options().dtype(delta_dtype_));   // the normalised output was not used
        const Tensor dy = grad_out.reshape({rows, d}).contiguous();
        Tensor dres;
        if (grad_res.defined()) {
            dres = grad_res.reshape({rows, d});
            if (dres.scalar_type() != at::kFloat || !dres.is_contiguous()) dres = dres.to(at::kFloat).contiguous();
        }
        Tensor dx = empty(shape_, at::kFloat, res), ddelta = empty(shape_, dy.scalar_type(), res);
        AffineGrads t(weight_, bias_, into_grad_, d, res);
        const float *st = static_cast<const float *>(ptr(stats));
        check(sp24_add_layernorm_bwd(ptr(dy), dt(dy.scalar_type()), dres.defined() ? static_cast<const float *>(ptr(dres)) : nullptr,
                                     static_cast<const float *>(ptr(res)), static_cast<const float *>(ptr(weight_)), st, st + rows,
                                     static_cast<float *>(ptr(dx)), ptr(ddelta), static_cast<float *>(ptr(t.g)), static_cast<float *>(ptr(t.b)),
                                     rows, d, cur_stream()),
              "sp24_add_layernorm_bwd");
        out[0] = dx;
        out[1] = ddelta;
        out[2] = t.rg;
        out[3] = t.rb;
        return out;
    }
};

std::pair<Tensor, Tensor> add_layer_norm(const Tensor &x, const Tensor &delta, const Tensor &weight, const Tensor &bias, double eps, bool into_grad) {
    require_cuda(x, delta, weight, bias);
    no_tangent(x, delta, weight, bias);
    Tensor res, out, stats;
    {
        NoAutograd guard;
        const int64_t d = x.size(-1), rows = x.numel() / d;
        res = empty(x.sizes(), at::kFloat, x);
        out = empty(x.sizes(), delta.scalar_type(), x);
        stats = empty({2 * rows}, at::kFloat, x);
        float *st = static_cast<float *>(ptr(stats));
        check(sp24_add_layernorm_fwd(static_cast<const float *>(ptr(x)), ptr(delta), static_cast<float *>(ptr(res)), static_cast<const float *>(ptr(weight)),
                                     static_cast<const float *>(ptr(bias)), ptr(out), dt(out.scalar_type()), st, st + rows, rows, d, (float)eps,
                                     cur_stream()),
              "sp24_add_layernorm_fwd");
    }
    if (torch::autograd::compute_requires_grad(x, delta, weight, bias)) {
        auto node = std::shared_ptr<AddLayerNormBackward>(new AddLayerNormBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(x, delta, weight, bias));
        node->stats_ = torch::autograd::SavedVariable(stats, false);
        node->weight_ = weight;
        node->bias_ = bias;
        node->shape_ = x.sizes().vec();
        node->delta_dtype_ = delta.scalar_type();
        node->into_grad_ = into_grad;
        torch::autograd::set_history(res, node);
        torch::autograd::set_history(out, node);
        node->res_ = torch::autograd::SavedVariable(res, true);
    }
    return {res, out};
}

// Mean cross entropy whose gradient for an upstream gradient of 1 is written by the forward launch; backward rescales it
// on the device only when the upstream gradient is not 1.
struct CrossEntropyBackward : torch::autograd::Node {
    torch::autograd::SavedVariable dlogits_;
    bool consumed_ = false;
    std::string name() const override { return "SparseCrossEntropyBackward"; }
    void release_variables() override {
        dlogits_.reset_data();
        consumed_ = true;
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(1);
        if (!grads[0].defined()) return out;
        TORCH_CHECK(!consumed_, "cross_entropy: the fused gradient buffer was already handed out by an earlier backward pass");
        const Tensor g = dlogits_.unpack();                // handed out once
        release_variables();
        NoAutograd guard;
        const Tensor up = grads[0].reshape({1}).to(at::kFloat).contiguous();
        check(sp24_scale_unless_one(ptr(g), dt(g.scalar_type()), static_cast<const float *>(ptr(up)), g.numel(), cur_stream()), "sp24_scale_unless_one");
        out[0] = g;
        return out;
    }
};

Tensor cross_entropy(const Tensor &logits, const Tensor &targets) {
    require_cuda(logits, targets);
    no_tangent(logits);
    Tensor loss, dlogits;
    {
        NoAutograd guard;
        const int64_t rows = logits.size(0), v = logits.size(1);
        Tensor both = empty({2 * rows}, at::kFloat, logits);   // log-sum-exp, then the rows' losses
        dlogits = empty({rows, v}, logits.scalar_type(), logits);
        float *lse = static_cast<float *>(ptr(both));
        check(sp24_cross_entropy_fused(ptr(logits), dt(logits.scalar_type()), static_cast<const int64_t *>(ptr(targets)), lse, lse + rows,
                                       (float)(1.0 / rows), ptr(dlogits), rows, v, logits.stride(0), v, cur_stream()),
              "sp24_cross_entropy_fused");
        loss = carve(both, rows * 4, at::kFloat, {rows}, {1}).mean();
    }
    auto node = std::shared_ptr<CrossEntropyBackward>(new CrossEntropyBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(logits));
    node->dlogits_ = torch::autograd::SavedVariable(dlogits, false);
    torch::autograd::set_history(loss, node);
    return loss;
}

struct EmbedBackward : torch::autograd::Node {
    torch::autograd::SavedVariable ids_;
    Tensor wte_, wpe_;
    bool into_grad_ = false, released_ = false;
    std::string name() const override { return "SparseEmbedTokensBackward"; }
    void release_variables() override {
        ids_.reset_data();
        released_ = true;
    }
    variable_list apply(variable_list &&grads) override {
        variable_list out(2);
        if (!grads[0].defined()) return out;
        TORCH_CHECK(!released_, torch::autograd::ERR_BACKWARD_TWICE);
        const Tensor ids = ids_.unpack();
        NoAutograd guard;
        Tensor dx = grads[0];
        if (dx.scalar_type() != at::kFloat || !dx.is_contiguous()) dx = dx.to(at::kFloat).contiguous();
        Tensor gw = wte_.grad(), gp = wpe_.grad();
        const bool into = into_grad_ && accumulable(gw) && accumulable(gp);
        if (!into) {
            gw = at::zeros(wte_.sizes(), wte_.options().dtype(at::kFloat));
            gp = at::zeros(wpe_.sizes(), wpe_.options().dtype(at::kFloat));
        }
        const int64_t b = ids.size(0), t = ids.size(1);
        check(sp24_embedding_bwd(static_cast<const float *>(ptr(dx)), static_cast<const int64_t *>(ptr(ids)), static_cast<float *>(ptr(gw)),
                                 static_cast<float *>(ptr(gp)), b * t, t, wte_.size(1), wte_.size(0), cur_stream()),
              "sp24_embedding_bwd");
        if (!into) {
            out[0] = gw;
            out[1] = gp;
        }
        return out;
    }
};

Tensor embed_tokens(const Tensor &ids_in, const Tensor &wte, const Tensor &wpe, bool into_grad) {
    no_tangent(wte, wpe);
    Tensor ids, out;
    {
        NoAutograd guard;
        ids = ids_in.contiguous();
        const int64_t b = ids.size(0), t = ids.size(1), d = wte.size(1);
        out = empty({b, t, d}, at::kFloat, wte);
        check(sp24_embedding_fwd(static_cast<const int64_t *>(ptr(ids)), static_cast<const float *>(ptr(wte)), static_cast<const float *>(ptr(wpe)),
                                 static_cast<float *>(ptr(out)), b * t, t, d, wte.size(0), cur_stream()),
              "sp24_embedding_fwd");
    }
    if (torch::autograd::compute_requires_grad(wte, wpe)) {
        auto node = std::shared_ptr<EmbedBackward>(new EmbedBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(wte, wpe));
        node->ids_ = torch::autograd::SavedVariable(ids, false);
        node->wte_ = wte;
        node->wpe_ = wpe;
        node->into_grad_ = into_grad;
        torch::autograd::set_history(out, node);
    }
    return out;
}

struct GeluBackward : torch::autograd::Node {
    torch::autograd::SavedVariable x_;
    bool released_ = false;
    std::string name() const override { return "SparseGeluBackward"; }
    void release_variables() override {
        x_.reset_data();
        released_ = true;
    }
    variable_list apply(variable_list &&grads) override {
        TORCH_CHECK(!released_, torch::autograd::ERR_BACKWARD_TWICE);
        variable_list out(1);
        if (!grads[0].defined()) return out;
        const Tensor x = x_.unpack();
        NoAutograd guard;
        Tensor dy = grads[0].contiguous();
        if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
        Tensor dx = at::empty_like(x);
        check(sp24_gelu(ptr(x), ptr(dy), ptr(dx), dt(x.scalar_type()), x.numel(), cur_stream()), "sp24_gelu");
        out[0] = dx;
        return out;
    }
};

Tensor gelu(const Tensor &input) {
    require_cuda(input);
    no_tangent(input);
    Tensor x, out;
    {
        NoAutograd guard;
        x = input.contiguous();
        out = at::empty_like(x);
        check(sp24_gelu(ptr(x), nullptr, ptr(out), dt(x.scalar_type()), x.numel(), cur_stream()), "sp24_gelu");
    }
    if (torch::autograd::compute_requires_grad(input)) {
        auto node = std::shared_ptr<GeluBackward>(new GeluBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(input));
        node->x_ = torch::autograd::SavedVariable(x, false);
        torch::autograd::set_history(out, node);
    }
    return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    using nogil = py::call_guard<py::gil_scoped_release>;
    py_objects.getrandbits = py::object(py::module_::import("random").attr("getrandbits")).release().ptr();
    py_objects.bits = PyLong_FromLong(32);
    py_objects.weight_grad = PyUnicode_InternFromString("weight_grad");
    m.def("set_dense_weight_grads", [](py::object fn) {
        Py_XDECREF(py_objects.dense_weight_grads);
        py_objects.dense_weight_grads = fn.release().ptr();
    });
    m.def("sparse_linear", &sparse_linear, nogil());
    m.def("sparse_mm_accumulate", &sparse_mm_accumulate, nogil());
    m.def("prune_compress", &prune_compress, nogil());
    m.def("compress", &compress, nogil());
    m.def("select_compress", &select_compress);
    m.def("select_compress_many", &select_compress_many);
    layer_names();
    walk_names();
    m.def("modules", &modules);
    m.def("refresh_layers", &refresh_layers);
    static PyMethodDef calls[] = {{"masked_add", (PyCFunction)(void (*)(void))py_masked_add, METH_FASTCALL, nullptr},
                                  {"fst_forward", (PyCFunction)(void (*)(void))py_fst_forward, METH_FASTCALL, nullptr},
                                  {nullptr, nullptr, 0, nullptr}};
    if (PyModule_AddFunctions(m.ptr(), calls) < 0) throw py::error_already_set();
    m.def("set_layer_class", &set_layer_class);
    m.def("fst_linear", &fst_linear);
    m.def("fst_weight_grads",
          [](const Tensor &g, const Tensor &x, const Tensor &w, const OptTensor &b, bool into, bool nw, bool nb) {
              auto [gw, gb] = fst_weight_grads(g, x, w, b.has_value() ? *b : Tensor(), into, nw, nb);
              return std::make_pair(gw.defined() ? OptTensor(gw) : OptTensor(), gb.defined() ? OptTensor(gb) : OptTensor());
          },
          nogil());
    m.def("soft_threshold_compress", &soft_threshold_compress, nogil());
    m.def("soft_threshold_linear", &soft_threshold_linear, nogil());
    m.def("fp8_weight", &fp8_weight);
    m.def("fp8_linear", &fp8_linear, nogil());
    m.def("layer_norm", &layer_norm, nogil());
    m.def("add_layer_norm", &add_layer_norm, nogil());
    m.def("cross_entropy", &cross_entropy, nogil());
    m.def("embed_tokens", &embed_tokens, nogil());
    m.def("gelu", &gelu, nogil());
    m.def("python_seed", &python_seed);
    m.def("set_rng_offset", [](const OptTensor &t) { rng_offset() = t; });
    m.def("status_words", &status_words);
    m.def("status_word", [](int dev) { return status_word((c10::DeviceIndex)dev); });
}
