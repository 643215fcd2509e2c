"""The float8 weight-gradient GEMM, D += alpha * A_sparse * B, on CTA pairs and on single CTAs: against float64 at ragged columns, odd
row blocks and both sides of the rule that picks the kernel, inside its window, and the same bits every time on a cleared buffer."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("ms,n,k", [(256, 256, 128), (256, 256, 2048), (384, 264, 2176), (128, 512, 2304), (1920, 1024, 384), (3072, 512, 128),
                                    (3072, 1032, 256), (2944, 1016, 256), (2944, 2056, 384), (3072, 3080, 2176)])      # 108 and 156 units on 74 pairs: chunks beside a ring in use
def test_float8_weight_gradient(ms, n, k):
    from sparse import _ext, fp8, spmm
    from sparse._semi_structured_conversions import sparse_semi_structured_to_dense
    g = torch.Generator(device=DEV).manual_seed(ms + n + k)
    w, x = torch.randn(ms, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    sw, (xq, sx) = fp8.scale_of(w), fp8.quantize(x)
    aw, ax = w.abs().amax().reshape(1), x.abs().amax().reshape(1)
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MSE, scale=sw)
    tc, status = spmm.tc_metadata(meta, ms, k), spmm._status_word(torch.device(DEV))

    def add_to(out):
        _ext.check(_ext.lib().sp24_spmm_f8(packed.data_ptr(), _ext.E4M3, k // 2, tc.data_ptr(), ms, k, xq.data_ptr(), k, n, out.data_ptr(),
                                           _ext.F32, 0, out.stride(0), None, aw.data_ptr(), ax.data_ptr(), status.data_ptr(), _ext.stream()),
                   "spmm_f8")
        spmm.check_status()

    buf = torch.randn(ms + 2, n + 16, device=DEV, generator=g)
    before, out = buf.clone(), buf[1:-1, 8:-8]
    add_to(out)
    a = sparse_semi_structured_to_dense(packed, meta).double()
    start = before[1:-1, 8:-8].double()
    ref = start + sw * sx * (a @ xq.double().t())
    mag = start.abs() + sw * sx * (a.abs() @ xq.double().abs().t())
    # exact products; k float32 additions, the factor (one rounding of it, one of the product) and two additions to D
    assert bool(((out.double() - ref).abs() <= (k + 8) * 2.0 ** -24 * mag).all())
    out.copy_(before[1:-1, 8:-8])
    assert torch.equal(buf, before)
    first, again = torch.zeros(ms, n, device=DEV), torch.zeros(ms, n, device=DEV)
    add_to(first)
    add_to(again)
    assert torch.equal(first, again)
