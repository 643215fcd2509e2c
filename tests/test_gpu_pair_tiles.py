"""Widths of the CTA-pair GEMM's tiles, bit for bit against the single-CTA kernel (reached through the activation, which the pair
kernel does not have): fixed sizes at ragged ends and over several rounds, and per form one size for every width the rule takes."""
import pytest
import torch

from _pair_tiles import FLOAT8, FUSED, PLAIN, WIDTHS, shapes

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _operand(ms, k, dtype, seed, col):
    import sparse
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = torch.randn(ms, k, device=DEV, generator=g).to(dtype)
    sp = sparse.to_sparse_semi_structured(w.t().contiguous().t() if col else w, dtype=dtype)
    return sp.sparse_tensor_cutlass, sp.meta_tensor_cutlass, g


# (ms, n): one round (n alone decides where ms is small), several rounds, and the ragged ends of tiles
SIZES = [(256, n) for n in (1, 15, 16, 17, 31, 33, 2368, 2369, 3553, 17760, 17761)] + \
        [(2048, n) for n in (9, 257, 288, 289, 433, 721, 1297)] + [(3072, 1100), (768, 5000), (4096, 1023)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("col", [False, True])
@pytest.mark.parametrize("ms,n", SIZES)
def test_every_tile_width_has_the_single_cta_bits(dtype, col, ms, n):
    """Both kernels accumulate each output in the same K order: no tolerance."""
    from sparse.spmm import check_status, sparse_linear
    k = 832 if n < 2000 else 192
    p, e, g = _operand(ms, k, dtype, ms + n, col)
    x = torch.randn(n, k, device=DEV, generator=g).to(dtype)
    b = torch.randn(ms, device=DEV, generator=g).to(dtype)
    for sign in (1, -1):          # both signs of every output pass the relu once
        assert torch.equal(sparse_linear(x * sign, p, e, b * sign).clamp(min=0), sparse_linear(x * sign, p, e, b * sign, "relu"))
    check_status()


@pytest.mark.parametrize("ms,n", [(256, 1), (512, 33), (2048, 289), (1024, 1023), (768, 5000), (3072, 2369)])
def test_fused_epilogues_at_every_width(ms, n):
    """The kept pre-activation has the plain product's bits; the activation's derivative stays within two bf16 roundings."""
    import torch.nn.functional as F
    from sparse.spmm import sparse_linear, sparse_linear_mlp
    p, e, g = _operand(ms, 192, torch.bfloat16, n, False)
    x = torch.randn(n, 192, device=DEV, generator=g).bfloat16()
    b = torch.randn(ms, device=DEV, generator=g).bfloat16()
    plain = sparse_linear(x, p, e, b)
    act, pre = sparse_linear_mlp(x, p, e, bias=b, epilogue="gelu")
    assert torch.equal(pre, plain)
    ref = F.gelu(pre.float(), approximate="tanh")
    assert float((act.float() - ref).abs().max() / ref.abs().max()) <= 2 ** -8
    d = sparse_linear_mlp(x, p, e, epilogue="dgelu", aux=pre)
    q = pre.float().requires_grad_(True)
    F.gelu(q, approximate="tanh").backward(sparse_linear(x, p, e).float())
    assert float((d.float() - q.grad).abs().max() / q.grad.abs().max()) <= 2 ** -7


@pytest.mark.parametrize("ms,n", [(256, 128), (512, 256), (768, 1152), (256, 17792)])
def test_float8_pair_products(ms, n):
    """e4m3 products with the scales taken on the device, 16-bit result against float64 of the same operands: one rounding to
    bf16 (2^-9 of the value) over float32 sums."""
    import sparse
    k = 256
    g = torch.Generator(device=DEV).manual_seed(n)
    w = torch.randn(ms, k, device=DEV, generator=g)
    mask = sparse.mask_select(w)[1]
    w8 = sparse.fp8.Fp8SparseWeight(w, mask)
    x = torch.randn(n, k, device=DEV, generator=g).bfloat16()
    y = sparse.fp8.sparse_linear_transpose_fp8.apply(x, w, w8, None)
    sw, sx = float((w * mask).abs().max()) / 448, float(x.abs().max()) / 448
    wq = ((w * mask) * (1 / sw)).to(torch.float8_e4m3fn).double() * sw
    xq = sparse.fp8.quantize(x)[0].double() * sx
    ref = xq @ wq.t()
    assert float((y.double() - ref).norm() / ref.norm()) <= 2 ** -8


def _size(form, width):
    """(ms, n) of ``width`` on this GPU."""
    return shapes(form, torch.cuda.get_device_properties(0).multi_processor_count)[width]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("width", sorted(WIDTHS[PLAIN]))
def test_plain_products_at_each_width(width, dtype):
    test_every_tile_width_has_the_single_cta_bits(dtype, width % 32 == 0, *_size(PLAIN, width))


@pytest.mark.parametrize("width", sorted(WIDTHS[FUSED]))
def test_fused_epilogues_at_each_width(width):
    test_fused_epilogues_at_every_width(*_size(FUSED, width))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("width", sorted(WIDTHS[FLOAT8]))
@pytest.mark.parametrize("k", [256, 640])
def test_float8_products_at_each_width(width, k, dtype):
    """16-bit results of the pair kernel against the float32 results of the single-CTA kernel, rounded."""
    from sparse import _ext, fp8, spmm
    ms, n = _size(FLOAT8, width)
    lib = _ext.lib()
    g = torch.Generator(device=DEV).manual_seed(width)
    w, x = torch.randn(ms, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    bias = torch.randn(ms, device=DEV, generator=g)
    sw, (xq, sx) = fp8.scale_of(w), fp8.quantize(x)
    aw, ax = w.abs().amax().reshape(1), x.abs().amax().reshape(1)
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MSE, scale=sw)
    tc, status = spmm.tc_metadata(meta, ms, k), spmm._status_word(torch.device(DEV))
    out = torch.empty(n, ms, dtype=dtype, device=DEV)
    _ext.check(lib.sp24_spmm_f8(packed.data_ptr(), _ext.E4M3, k // 2, tc.data_ptr(), ms, k, xq.data_ptr(), k, n, out.data_ptr(),
                                _ext.dt(dtype), 1, ms, bias.data_ptr(), aw.data_ptr(), ax.data_ptr(), status.data_ptr(), _ext.stream()),
               "spmm_f8")
    assert torch.equal(out, spmm.sparse_linear(xq, packed, meta, bias=bias, alpha=sw * sx).to(dtype))
    spmm.check_status()


def _window(n, ms, dtype):
    """A pre-filled buffer with a row more above and below and 8 values more on either side, its bits, and the (n, ms) window."""
    buf = torch.randn(n + 2, ms + 16, device=DEV).to(dtype)
    return buf, buf.view(torch.int16).clone(), buf[1:-1, 8:-8]


def _only_the_window_changed(buf, before, window, result):
    assert torch.equal(window, result)
    window.view(torch.int16).copy_(before[1:-1, 8:-8])
    assert torch.equal(buf.view(torch.int16), before)


@pytest.mark.parametrize("ms,n", [(256, 1), (256, 7), (512, 17), (1024, 33)] + [(0, w) for w in sorted(WIDTHS[PLAIN])])
def test_plain_products_stay_in_their_window(ms, n):
    """16-byte stores of a pitched output at few tokens and at each width's ragged end (ms 0: the shape of that width)."""
    from sparse import _ext, spmm
    ms, n = (ms, n) if ms else _size(PLAIN, n)
    k = 192
    p, e, g = _operand(ms, k, torch.bfloat16, ms + n, False)
    x = torch.randn(n, k, device=DEV, generator=g).bfloat16()
    b = torch.randn(ms, device=DEV, generator=g).bfloat16()
    buf, before, out = _window(n, ms, torch.bfloat16)
    status = spmm._status_word(torch.device(DEV))
    _ext.check(_ext.lib().sp24_spmm(p.data_ptr(), _ext.BF16, 0, k // 2, spmm.tc_metadata(e, ms, k).data_ptr(), ms, k, x.data_ptr(), 0, k, n,
                                    out.data_ptr(), _ext.BF16, 1, ms + 16, b.data_ptr(), 0, status.data_ptr(), _ext.stream()), "spmm")
    _only_the_window_changed(buf, before, out, spmm.sparse_linear(x, p, e, b))
    spmm.check_status()


@pytest.mark.parametrize("ms,n", [(256, 1), (256, 7), (512, 17)] + [(0, w) for w in sorted(WIDTHS[FLOAT8])])
def test_float8_products_stay_in_their_window(ms, n):
    from sparse import _ext, fp8, spmm
    ms, n = (ms, n) if ms else _size(FLOAT8, n)
    k = 384
    g = torch.Generator(device=DEV).manual_seed(ms + n)
    w, x = torch.randn(ms, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    sw, (xq, sx) = fp8.scale_of(w), fp8.quantize(x)
    aw, ax = w.abs().amax().reshape(1), x.abs().amax().reshape(1)
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MSE, scale=sw)
    buf, before, out = _window(n, ms, torch.float16)
    tc, status = spmm.tc_metadata(meta, ms, k), spmm._status_word(torch.device(DEV))
    _ext.check(_ext.lib().sp24_spmm_f8(packed.data_ptr(), _ext.E4M3, k // 2, tc.data_ptr(), ms, k, xq.data_ptr(), k, n, out.data_ptr(),
                                       _ext.F16, 1, ms + 16, None, aw.data_ptr(), ax.data_ptr(), status.data_ptr(), _ext.stream()), "spmm_f8")
    _only_the_window_changed(buf, before, out, spmm.sparse_linear(xq, packed, meta, alpha=sw * sx).half())
    spmm.check_status()
