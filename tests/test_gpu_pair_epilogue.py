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
