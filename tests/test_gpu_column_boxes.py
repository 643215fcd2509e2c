"""Operands that the CTA-pair GEMMs fetch two 128-byte columns a request: windows of larger buffers whose surroundings are NaN, an odd number
of columns, and the widths of the weight gradient that keep one request a column."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _window(rows, cols, pad, g):
    buf = torch.full((rows + 2, cols + 2 * pad), float("nan"), device=DEV, dtype=torch.float16)
    buf[1:-1, pad:pad + cols] = torch.randn(rows, cols, device=DEV, generator=g).half()
    return buf[1:-1, pad:pad + cols]


def _sparse(ms, k, col, g):
    import sparse
    w = torch.randn(ms, k, device=DEV, generator=g).half()
    return sparse.to_sparse_semi_structured(w.t().contiguous().t() if col else w, dtype=torch.float16)


@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n,k", [(256, 40, 64), (384, 300, 192), (512, 17, 1088), (256, 300, 320)])
def test_products(ms, n, k, col):
    from sparse import spmm
    g = torch.Generator(device=DEV).manual_seed(ms + n + k)
    sp, x = _sparse(ms, k, col, g), _window(n, k, 24, g)
    y = spmm.sparse_linear(x, sp.sparse_tensor_cutlass, sp.meta_tensor_cutlass).double()
    spmm.check_status()
    a = sp.to_dense().double()
    ref, mag = x.double() @ a.t(), x.double().abs() @ a.abs().t()
    assert bool(((y - ref).abs() <= 2.0 ** -11 * ref.abs() * 1.01 + (k + 4) * 2.0 ** -24 * mag).all())      # float32 sums, one rounding


@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n,k", [(256, 256, 64), (384, 320, 192), (512, 264, 192), (256, 376, 320), (512, 640, 1088)])
def test_weight_gradient(ms, n, k, col):
    from sparse.spmm import check_status, sparse_mm_accumulate_
    g = torch.Generator(device=DEV).manual_seed(ms + n + k)
    sp, x = _sparse(ms, k, col, g), _window(k, n, 40, g)
    out = torch.zeros(ms, n, device=DEV)
    sparse_mm_accumulate_(out, sp.sparse_tensor_cutlass, sp.meta_tensor_cutlass, x)
    check_status()
    a = sp.to_dense().double()
    assert bool(((out.double() - a @ x.double()).abs() <= (k + 16) * 2.0 ** -24 * (a.abs() @ x.double().abs())).all())
