"""Row sums that the float8 weight-gradient GEMM takes along, on CTA pairs (one unit a pair and several) and on single CTAs: the bits of the
launch of its own, and the product unchanged."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("ms,n,k", [(256, 256, 2048), (384, 264, 2176), (3072, 1032, 256), (2944, 1080, 128), (128, 512, 256), (256, 128, 384)])
def test_row_sums(ms, n, k, accumulate):
    from sparse import _ext, fp8, spmm
    lib, g = _ext.lib(), torch.Generator(device=DEV).manual_seed(ms + n + k)
    w, x = torch.randn(ms, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    (xq, _), sw = fp8.quantize(x), fp8.scale_of(w)
    aw, ax = w.abs().amax().reshape(1), x.abs().amax().reshape(1)
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MSE, scale=sw)
    tc, status = spmm.tc_metadata(meta, ms, k), torch.zeros(1, dtype=torch.int32, device=DEV)
    n_parts = lib.sp24_row_parts(k, _ext.E4M3)
    parts, start = torch.randn(n_parts, ms, device=DEV, generator=g), torch.randn(ms, device=DEV, generator=g)
    want, got = start.clone(), start.clone()
    d0, d1 = torch.zeros(ms, n, device=DEV), torch.zeros(ms, n, device=DEV)
    a = (packed.data_ptr(), _ext.E4M3, k // 2, tc.data_ptr(), ms, k, xq.data_ptr(), k, n)
    assert lib.sp24_sum_parts(parts.data_ptr(), n_parts, ms, want.data_ptr(), accumulate, _ext.stream()) == 0
    assert lib.sp24_spmm_f8(*a, d0.data_ptr(), _ext.F32, 0, n, None, aw.data_ptr(), ax.data_ptr(), status.data_ptr(), _ext.stream()) == 0
    assert lib.sp24_spmm_f8_sums(*a, d1.data_ptr(), n, aw.data_ptr(), ax.data_ptr(), parts.data_ptr(), n_parts, got.data_ptr(), accumulate,
                                 status.data_ptr(), _ext.stream()) == 0
    assert int(status) == 0 and torch.equal(got, want) and torch.equal(d0, d1)
    assert lib.sp24_spmm_f8_sums(*a, d1.data_ptr(), n, aw.data_ptr(), ax.data_ptr(), None, n_parts, got.data_ptr(), accumulate,
                                 status.data_ptr(), _ext.stream()) < 0
