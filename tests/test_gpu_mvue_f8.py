"""Float8 MVUE compression of column-major 16-bit gradients by persistent blocks, against the kernel that float32 gradients take: the same
values give the same bits everywhere (stored values, both metadata orders, the quantised tensor) and row sums within their rounding, for
half-empty last row tiles, one and many tiles a block, pitches, and without each of the extras."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _compress(g, amax, out, extras):
    from sparse import _ext
    lib = _ext.lib()
    k, m = g.shape
    ld = g.stride(0)
    dt8 = _ext.dt(out)
    packed = torch.full((m, k // 2 + 16), 77, dtype=torch.uint8, device=DEV)
    meta = torch.empty(m, k // 32, dtype=torch.int32, device=DEV)
    tc = torch.empty(lib.sp24_meta_tc_bytes(m, k), dtype=torch.uint8, device=DEV) if extras and m % 128 == 0 else None
    q = torch.full((k, m + 16), 77, dtype=torch.uint8, device=DEV) if extras else None
    parts = torch.empty(lib.sp24_row_parts(k, dt8), m, device=DEV) if extras else None
    x = _ext.PruneExtras()
    x.packed_row_major, x.amax, x.e_tc, x.row_parts, x.q_dense, x.ld_q = 1, amax.data_ptr(), _ext.ptr(tc), _ext.ptr(parts), _ext.ptr(q), m + 16
    _ext.check(lib.sp24_prune_compress_with(g.data_ptr(), _ext.dt(g.dtype), m, k, ld, 1, packed.data_ptr(), dt8, k // 2 + 16, meta.data_ptr(),
                                            _ext.PRUNE_MVUE_FAST, None, 0, None, 0, 1234567, 3, x, _ext.stream()), "prune_compress_with")
    return (packed, meta, tc, q), parts


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("out", [torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("m,k,pad", [(32, 128, 0), (96, 256, 8), (128, 384, 0), (160, 1152, 24), (1024, 4224, 0), (3072, 2048, 0)])
def test_same_bits_as_float32_input(m, k, pad, out, dtype):
    gen = torch.Generator(device=DEV).manual_seed(m + k)
    g = (torch.randn(k, m + pad, device=DEV, generator=gen) * torch.where(torch.rand(k, m + pad, device=DEV, generator=gen) < 0.01, 100.0, 1.0)).to(dtype)[:, :m]
    g[0, 0], g[1, 1] = 0.0, -0.0
    amax = g.float().abs().amax().reshape(1)
    for extras in (True, False):
        got, parts = _compress(g, amax, out, extras)
        want, want_parts = _compress(g.float(), amax, out, extras)
        for a, b in zip(got, want):
            assert (a is None) == (b is None) and (a is None or torch.equal(a, b))
        if extras:
            ref, mag = g.double().view(-1, 128, m).sum(1), g.double().abs().view(-1, 128, m).sum(1)
            for p in (parts, want_parts):
                assert bool(((p.double() - ref).abs() <= 128 * 2.0 ** -24 * mag).all())
