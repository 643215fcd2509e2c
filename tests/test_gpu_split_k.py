"""The GEMM for few columns, K cut into slices over the pairs of a cluster: two to four slices, tiles of 32, 48 and 64 columns with ragged
ends, odd row blocks, K that ends inside a step, and a K too short and a width too large for it: against float64, inside the output's window, and the same
bits every time."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
ROUND = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("dtype", list(ROUND), ids=["f16", "bf16"])
@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n,k", [(256, 1, 1024), (512, 17, 960), (384, 33, 1152), (128, 63, 4096), (1024, 48, 1088), (640, 49, 2048),
                                    (2304, 32, 1600), (4096, 8, 1088), (6144, 63, 1024), (2048, 64, 1024), (512, 16, 896)])
def test_few_columns(ms, n, k, col, dtype):
    import sparse
    from sparse import _ext, spmm
    g = torch.Generator(device=DEV).manual_seed(ms + n)
    w = torch.randn(ms, k, device=DEV, generator=g).to(dtype)
    sp = sparse.to_sparse_semi_structured(w.t().contiguous().t() if col else w, dtype=dtype)
    x, b = torch.randn(n, k, device=DEV, generator=g).to(dtype), torch.randn(ms, device=DEV, generator=g).to(dtype)
    buf = torch.randn(n + 2, ms + 16, device=DEV, generator=g).to(dtype)
    before, out = buf.clone(), buf[1:-1, 8:-8]
    p, e, status = sp.sparse_tensor_cutlass, spmm.tc_metadata(sp.meta_tensor_cutlass, ms, k), spmm._status_word(torch.device(DEV))
    dt, results = _ext.dt(dtype), []
    for _ in range(3):
        _ext.check(_ext.lib().sp24_spmm(p.data_ptr(), dt, int(col), ms if col else k // 2, e.data_ptr(), ms, k, x.data_ptr(), 0, k, n,
                                        out.data_ptr(), dt, 1, ms + 16, b.data_ptr(), 0, status.data_ptr(), _ext.stream()), "spmm")
        results.append(out.clone())
    spmm.check_status()
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])
    a = sp.to_dense().double()
    ref, mag = x.double() @ a.t() + b.double(), x.double().abs() @ a.abs().t() + b.double().abs()
    # k + 4 float32 additions and one rounding
    assert bool(((out.double() - ref).abs() <= ROUND[dtype] * ref.abs() * 1.01 + (k + 4) * 2.0 ** -24 * mag).all())
    out.copy_(before[1:-1, 8:-8])
    assert torch.equal(buf, before)


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("ms", [512, 4096, 7168])      # four, three and two slices of K
def test_equal_tokens_have_equal_outputs(ms, bias):
    """Products of 2^24, -2^24, 0.5 and 0.25 in different slices: every token's sum is 0.75 where the first two slices are added
    up first, and one of the small products is lost where another slice comes between them.  Random tokens beside them: equal ones give the same bits."""
    import sparse
    from sparse import spmm
    k, n = 4096, 63
    w = torch.zeros(ms, k, device=DEV)
    w[:, 0], w[:, 12 * 128], w[:, 22 * 128], w[:, 28 * 128] = 4096.0, -4096.0, 1.0, 1.0
    x = torch.zeros(1, k, device=DEV)
    x[:, 0], x[:, 12 * 128], x[:, 22 * 128], x[:, 28 * 128] = 4096.0, 4096.0, 0.5, 0.25
    b = torch.zeros(ms, device=DEV).half() if bias else None
    sp = sparse.to_sparse_semi_structured(w.half(), dtype=torch.float16)
    y = spmm.sparse_linear(x.half().expand(n, k).contiguous(), sp.sparse_tensor_cutlass, sp.meta_tensor_cutlass, bias=b)
    assert bool((y == 0.75).all())
    sp = sparse.to_sparse_semi_structured(torch.randn(ms, k, device=DEV).half(), dtype=torch.float16)
    x = torch.randn(1, k, device=DEV).half()
    y = spmm.sparse_linear(x.expand(n, k).contiguous(), sp.sparse_tensor_cutlass, sp.meta_tensor_cutlass, bias=b)
    spmm.check_status()
    assert torch.equal(y, y[:1].expand(n, ms))
