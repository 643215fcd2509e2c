"""CTA-pair GEMMs whose last 256-row block is half empty (an odd multiple of 128 rows of the sparse operand): results against float64
and nothing written past the last row or column of the output's window, on both sides of the rule that picks the kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ROUND = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}
SIZES = [(128, 17, 192), (128, 5200, 1088), (384, 1, 64), (384, 2600, 512), (640, 300, 640), (896, 1984, 1152)]


def _window(rows, cols, dtype):
    buf = torch.randn(rows + 2, cols + 16, device=DEV).to(dtype)
    return buf, buf.clone(), buf[1:-1, 8:-8]


def _check(buf, before, out, ref, bound):
    assert bool(((out.double() - ref).abs() <= bound).all())
    out.copy_(before[1:-1, 8:-8])
    assert torch.equal(buf, before)


@pytest.mark.parametrize("dtype", list(ROUND), ids=["f16", "bf16"])
@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n,k", SIZES)
def test_products(ms, n, k, col, dtype):
    import sparse
    from sparse import _ext, spmm
    g = torch.Generator(device=DEV).manual_seed(ms + n)
    w = torch.randn(ms, k, device=DEV, generator=g).to(dtype)
    sp = sparse.to_sparse_semi_structured(w.t().contiguous().t() if col else w, dtype=dtype)
    x = torch.randn(n, k, device=DEV, generator=g).to(dtype)
    b = torch.randn(ms, device=DEV, generator=g).to(dtype)
    buf, before, out = _window(n, ms, dtype)
    p, e, status = sp.sparse_tensor_cutlass, spmm.tc_metadata(sp.meta_tensor_cutlass, ms, k), spmm._status_word(torch.device(DEV))
    dt = _ext.dt(dtype)
    _ext.check(_ext.lib().sp24_spmm(p.data_ptr(), dt, int(col), ms if col else k // 2, e.data_ptr(), ms, k, x.data_ptr(), 0, k, n,
                                    out.data_ptr(), dt, 1, ms + 16, b.data_ptr(), 0, status.data_ptr(), _ext.stream()), "spmm")
    spmm.check_status()
    a = sp.to_dense().double()
    ref = x.double() @ a.t() + b.double()
    mag = x.double().abs() @ a.abs().t() + b.double().abs()
    _check(buf, before, out, ref, ROUND[dtype] * ref.abs() * 1.01 + (k + 2) * 2.0 ** -24 * mag)      # float32 sums, one rounding


@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n,k", [(1152, 8200, 576), (640, 16390, 1088)])
def test_products_of_more_tiles_than_pairs(ms, n, k, col):
    """About 185 and 210 tiles on 74 pairs: the persistent loop, the second accumulator and a half-empty block that hands both back early."""
    test_products(ms, n, k, col, torch.float16)


@pytest.mark.parametrize("dtype", list(ROUND), ids=["f16", "bf16"])
@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n", [(384, 4096), (384, 4097), (384, 6272), (384, 6273), (1152, 2048), (1152, 2049)])
def test_products_of_one_k_step(ms, n, col, dtype):
    """96 and 99, 147 and 150, 144 and 153 tiles of 128 x 128: either side of what single CTAs take in one round of 148."""
    test_products(ms, n, 128, col, dtype)


@pytest.mark.parametrize("ms,n,k,splits", [(128, 256, 192, 0), (384, 264, 1088, 3), (1152, 1152, 1984, 0), (384, 520, 1024, 0), (640, 264, 1088, 0), (384, 264, 64, 5)])
@pytest.mark.parametrize("col", [False, True])
def test_weight_gradient(ms, n, k, splits, col):
    import sparse
    from sparse.spmm import check_status, sparse_mm_accumulate_
    g = torch.Generator(device=DEV).manual_seed(ms + n + k)
    w = torch.randn(ms, k, device=DEV, generator=g).half()
    sp = sparse.to_sparse_semi_structured(w.t().contiguous().t() if col else w, dtype=torch.float16)
    x = torch.randn(k, n, device=DEV, generator=g).half()
    buf, before, out = _window(ms, n, torch.float32)
    sparse_mm_accumulate_(out, sp.sparse_tensor_cutlass, sp.meta_tensor_cutlass, x, k_splits=splits)
    check_status()
    a, start = sp.to_dense().double(), before[1:-1, 8:-8].double()
    _check(buf, before, out, start + a @ x.double(), (k + 16) * 2.0 ** -24 * (start.abs() + a.abs() @ x.double().abs()))


@pytest.mark.parametrize("ms,n,k", [(128, 17, 384), (128, 5200, 1152), (384, 2600, 512), (640, 300, 640)])
def test_float8_products(ms, n, k):
    """Exact products of e4m3 values, float32 sums, one rounding: against the single-CTA kernel's float32 result, rounded."""
    from sparse import _ext, fp8, spmm
    g = torch.Generator(device=DEV).manual_seed(ms + n)
    w, x = torch.randn(ms, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    sw, (xq, sx) = fp8.scale_of(w), fp8.quantize(x)
    aw, ax = w.abs().amax().reshape(1), x.abs().amax().reshape(1)
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MSE, scale=sw)
    buf, before, out = _window(n, ms, torch.float16)
    tc, status = spmm.tc_metadata(meta, ms, k), spmm._status_word(torch.device(DEV))
    _ext.check(_ext.lib().sp24_spmm_f8(packed.data_ptr(), _ext.E4M3, k // 2, tc.data_ptr(), ms, k, xq.data_ptr(), k, n, out.data_ptr(),
                                       _ext.F16, 1, ms + 16, None, aw.data_ptr(), ax.data_ptr(), status.data_ptr(), _ext.stream()), "spmm_f8")
    spmm.check_status()
    ref = spmm.sparse_linear(xq, packed, meta, alpha=sw * sx)
    _check(buf, before, out, ref.half().double(), torch.zeros(1, device=DEV, dtype=torch.float64))


@pytest.mark.parametrize("ms,n,k", [(1152, 8200, 640), (640, 16390, 1152)])
def test_float8_products_of_more_tiles_than_pairs(ms, n, k):
    test_float8_products(ms, n, k)
