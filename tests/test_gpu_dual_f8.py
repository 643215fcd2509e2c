"""Both float8 copies of a weight from one read: the bits of the two conversions of W and W.T (which a column-major weight takes), for masks
of two kept in every group, of any number, and values at the ends of e4m3's range."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind", ["transposable", "any"])
@pytest.mark.parametrize("m,k,pad", [(128, 128, 0), (128, 640, 0), (384, 128, 8), (256, 384, 16), (2304, 768, 0)])
def test_same_bits_as_two_conversions(m, k, pad, kind, dtype):
    import sparse
    g = torch.Generator(device=DEV).manual_seed(m + k)
    buf = torch.randn(m, k + pad, device=DEV, generator=g).to(dtype)
    w = buf[:, :k]
    w[0, 0], w[1, 1], w[2, 5], w[3, 3] = 0.0, -0.0, 300.0, float("inf") if kind == "any" else -300.0
    mask = sparse.mask_select(w.contiguous())[1] if kind == "transposable" else torch.rand(m, k, device=DEV, generator=g) < 0.5
    if kind == "any":
        mask[3, 3] = False
    a = sparse.fp8.Fp8SparseWeight(w, mask)
    b = sparse.fp8.Fp8SparseWeight(w.t().contiguous().t(), mask)
    for name in ("amax", "pw", "mw", "tcw", "pt", "mt", "tct"):
        x, y = getattr(a, name), getattr(b, name)
        assert x.shape == y.shape and x.dtype == y.dtype and torch.equal(x.view(torch.uint8), y.view(torch.uint8)), name


def test_refusals():
    from sparse import _ext
    lib, w = _ext.lib(), torch.zeros(256, 256, device=DEV)
    p = w.data_ptr()

    def call(m=256, k=256, ld=256, ld_mask=256, dtype=_ext.F32, at=p, out=p):
        return lib.sp24_dual_compress_f8(at, dtype, m, k, ld, p, ld_mask, p, out, p, p, p, p, p, _ext.stream())
    assert call(at=None) < 0 and call(m=192) < 0 and call(k=64) < 0 and call(ld=128) < 0 and call(ld=258) < 0 and call(ld_mask=258) < 0
    assert call(dtype=_ext.E4M3) < 0 and call(at=p + 4) < 0 and call(out=p + 8) < 0
