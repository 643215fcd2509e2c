"""The CTA-pair GEMM's plain epilogue over several tiles a pair: accumulators that are wanted again (all columns by four warps) and a pair's
last two (every other chunk by eight), widths of an odd and an even number of chunks, last tiles of one and of seventeen tokens, a bias, a
half-empty row block, inside the output's window."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ROUND = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


# tiles a pair: 3 to 6, 12, 2 and 1
@pytest.mark.parametrize("dtype", list(ROUND), ids=["f16", "bf16"])
@pytest.mark.parametrize("ms,n,k", [(3072, 8193, 64), (2304, 8081, 128), (768, 16385, 192), (3072, 16384, 64), (1152, 8225, 320), (512, 8191, 64), (256, 17, 64)])
def test_several_tiles_a_pair(ms, n, k, dtype):
    import sparse
    from sparse import _ext, spmm
    g = torch.Generator(device=DEV).manual_seed(ms + n + k)
    sp = sparse.to_sparse_semi_structured(torch.randn(ms, k, device=DEV, generator=g).to(dtype), dtype=dtype)
    x, bias = torch.randn(n, k, device=DEV, generator=g).to(dtype), torch.randn(ms, device=DEV, generator=g).to(dtype)
    buf = torch.randn(n + 2, ms + 16, device=DEV, generator=g).to(dtype)
    before, out = buf.clone(), buf[1:-1, 8:-8]
    p, e, status = sp.sparse_tensor_cutlass, spmm.tc_metadata(sp.meta_tensor_cutlass, ms, k), spmm._status_word(torch.device(DEV))
    dt = _ext.dt(dtype)
    for b in (bias, None):
        _ext.check(_ext.lib().sp24_spmm(p.data_ptr(), dt, 0, k // 2, e.data_ptr(), ms, k, x.data_ptr(), 0, k, n, out.data_ptr(), dt, 1, ms + 16,
                                        _ext.ptr(b), 0, status.data_ptr(), _ext.stream()), "spmm")
        spmm.check_status()
        a = sp.to_dense().double()
        ref, mag = x.double() @ a.t(), x.double().abs() @ a.abs().t()
        if b is not None:
            ref, mag = ref + b.double(), mag + b.double().abs()
        # float32 sums, one rounding
        assert bool(((out.double() - ref).abs() <= ROUND[dtype] * ref.abs() * 1.01 + (k + 2) * 2.0 ** -24 * mag).all())
    out.copy_(before[1:-1, 8:-8])
    assert torch.equal(buf, before)


@pytest.mark.parametrize("ms,n,k", [(128, 8192, 64), (128, 8200, 64), (384, 12008, 128), (1408, 4100, 256)])
def test_either_side_of_the_rule_for_odd_row_blocks(ms, n, k):
    test_several_tiles_a_pair(ms, n, k, torch.float16)


# one K step a tile, where the MMAs of two tiles are shortest against a warp's stores: five and nine tiles a pair of 16 to 240 columns
@pytest.mark.parametrize("ms,n,k", [(94720, 16, 64), (94720, 48, 64), (94720, 112, 128), (170240, 33, 64), (3072, 16384, 128), (4096, 20011, 64)])
def test_short_tiles_again_and_again(ms, n, k):
    test_several_tiles_a_pair(ms, n, k, torch.float16)


# float8: a K step is 256 long
@pytest.mark.parametrize("dtype", list(ROUND), ids=["f16", "bf16"])
@pytest.mark.parametrize("ms,n,k", [(3072, 16384, 128), (3072, 8193, 256), (768, 30011, 128), (94720, 48, 128), (1152, 12001, 384)])
def test_float8_tiles(ms, n, k, dtype):
    """Against the single-CTA kernel's float32 result, rounded: exact products, float32 sums in the same order."""
    from sparse import _ext, fp8, spmm
    g = torch.Generator(device=DEV).manual_seed(ms + n)
    w, x = torch.randn(ms, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    (xq, sx), aw, ax = fp8.quantize(x), w.abs().amax().reshape(1), x.abs().amax().reshape(1)
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MSE, scale=fp8.scale_of(w))
    tc, status = spmm.tc_metadata(meta, ms, k), spmm._status_word(torch.device(DEV))
    buf = torch.randn(n + 2, ms + 16, device=DEV, generator=g).to(dtype)
    before, out = buf.clone(), buf[1:-1, 8:-8]
    for _ in range(3):
        out.fill_(float("nan"))
        _ext.check(_ext.lib().sp24_spmm_f8(packed.data_ptr(), _ext.E4M3, k // 2, tc.data_ptr(), ms, k, xq.data_ptr(), k, n, out.data_ptr(),
                                           _ext.dt(dtype), 1, ms + 16, None, aw.data_ptr(), ax.data_ptr(), status.data_ptr(), _ext.stream()), "spmm_f8")
        spmm.check_status()
        ref = spmm.sparse_linear(xq, packed, meta, alpha=fp8.scale_of(w) * sx)
        assert torch.equal(out, ref.to(dtype))
    out.copy_(before[1:-1, 8:-8])
    assert torch.equal(buf, before)


@pytest.mark.parametrize("sums", [False, True])
@pytest.mark.parametrize("ms,n,k", [(896, 1152, 1984), (2176, 640, 4096), (384, 520, 1984), (2944, 2944, 384), (1920, 1152, 8192)])
def test_weight_gradients_of_odd_row_blocks(ms, n, k, sums):
    """With fewer and more units than pairs, on pairs and on single CTAs, against float64; the row sums with them or on their own."""
    import sparse
    from sparse import _ext, spmm
    lib, g = _ext.lib(), torch.Generator(device=DEV).manual_seed(ms + n + k)
    sp = sparse.to_sparse_semi_structured(torch.randn(ms, k, device=DEV, generator=g).half().t().contiguous().t(), dtype=torch.float16)
    x, parts = torch.randn(k, n, device=DEV, generator=g).half(), torch.randn(3, ms, device=DEV, generator=g)
    p, e, status = sp.sparse_tensor_cutlass, spmm.tc_metadata(sp.meta_tensor_cutlass, ms, k), spmm._status_word(torch.device(DEV))
    out, got = torch.zeros(ms, n, device=DEV), torch.zeros(ms, device=DEV)
    a = (p.data_ptr(), _ext.F16, 1, ms, e.data_ptr(), ms, k, x.data_ptr(), n, n, out.data_ptr(), n, 0)
    if sums:
        _ext.check(lib.sp24_spmm_accumulate_sums_f32(*a, parts.data_ptr(), 3, got.data_ptr(), 0, status.data_ptr(), _ext.stream()), "spmm")
        assert bool(((got.double() - parts.double().sum(0)).abs() <= 4 * 2.0 ** -24 * parts.double().abs().sum(0)).all())
    else:
        _ext.check(lib.sp24_spmm_accumulate_f32(*a, status.data_ptr(), _ext.stream()), "spmm")
    spmm.check_status()
    d = sp.to_dense().double()
    assert bool(((out.double() - d @ x.double()).abs() <= (k + 16) * 2.0 ** -24 * (d.abs() @ x.double().abs())).all())
