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
