"""The CTA-pair weight-gradient GEMM's epilogue (shared memory, then TMA reductions) at the ends of its tiles and chunks: one unit per
pair and several, columns that end inside a box of 32, inside a warp's half and inside a tile, K slices, and an output that is a
window of a larger buffer."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# ms, n, k, k_splits: 74 pairs; 12 x 7 tiles are two rounds, 2 tiles x 40 slices too
SIZES = [(256, 256, 128, 0), (512, 264, 192, 0), (256, 504, 320, 2), (256, 392, 4096, 0), (3072, 1544, 192, 0), (512, 256, 5120, 40),
         (256, 520, 6400, 30)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n,k,splits", SIZES)
def test_pair_weight_gradient(dtype, col, ms, n, k, splits):
    """Against float64: exact products, then float32 additions in any order: K + slices roundings of 2^-24 on the sums of magnitudes."""
    import sparse
    from sparse.spmm import check_status, sparse_mm_accumulate_
    g = torch.Generator(device=DEV).manual_seed(ms + n + k)
    w = torch.randn(ms, k, device=DEV, generator=g).to(dtype)
    sp = sparse.to_sparse_semi_structured(w.t().contiguous().t() if col else w, dtype=dtype)
    x = torch.randn(k, n, device=DEV, generator=g).to(dtype)
    buf = torch.randn(ms + 2, n + 16, device=DEV, generator=g)
    before = buf.clone()
    out = buf[1:-1, 8:8 + n]
    sparse_mm_accumulate_(out, sp.sparse_tensor_cutlass, sp.meta_tensor_cutlass, x, k_splits=splits)
    check_status()
    a = sp.to_dense().double()
    ref = before[1:-1, 8:8 + n].double() + a @ x.double()
    mag = before[1:-1, 8:8 + n].double().abs() + a.abs() @ x.double().abs()
    assert bool(((out.double() - ref).abs() <= (k + splits + 2) * 2.0 ** -24 * mag).all())
    buf[1:-1, 8:8 + n] = before[1:-1, 8:8 + n]
    assert torch.equal(buf, before)
