"""Kernels of the float8 layer whose scales stay on the device, and the column sums: against torch on the same inputs, at
the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
E4M3 = torch.float8_e4m3fn


def _lib():
    from sparse import _ext
    return _ext.lib(), _ext


def _rand(shape, dtype, seed, std=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, device=DEV, generator=g) * std).to(dtype)


def _amax(x, mask=None):
    lib, _ext = _lib()
    a = torch.full((1,), -1.0, device=DEV)
    _ext.check(lib.sp24_absmax(x.data_ptr(), _ext.dt(x.dtype), x.numel(), _ext.ptr(mask), a.data_ptr(), _ext.stream()), "absmax")
    return a


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 8), (3, 1000), (1025, 1024), (4096, 2056)])
def test_absmax_is_exact(dtype, shape):
    x = _rand(shape, dtype, 1)
    assert torch.equal(_amax(x)[0], x.abs().amax().float())
    assert float(_amax(torch.zeros_like(x))) == 0.0
    if dtype == torch.float32:
        mask = torch.rand(*shape, device=DEV) < 0.5
        assert torch.equal(_amax(x, mask)[0], torch.where(mask, x, 0.0).abs().amax())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (127, 72), (128, 64), (160, 1000), (1056, 136)])
def test_quantize_matches_torch_and_transposes(dtype, rows, cols):
    from sparse import fp8
    lib, _ext = _lib()
    x = _rand((rows, cols), dtype, 2)
    q, q_t = torch.empty(rows, cols, dtype=E4M3, device=DEV), torch.empty(cols, rows, dtype=E4M3, device=DEV)
    a = _amax(x)
    _ext.check(lib.sp24_quantize_f8(x.data_ptr(), _ext.dt(dtype), rows, cols, cols, a.data_ptr(), q.data_ptr(), q_t.data_ptr(), rows,
                                    _ext.stream()), "quantize")
    want, _ = fp8.quantize(x)
    assert torch.equal(q.view(torch.uint8), want.view(torch.uint8))
    assert torch.equal(q_t.view(torch.uint8), want.view(torch.uint8).t().contiguous())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("top", [5.1875, 5.28125, 4.75, 7.125])
def test_quantize_of_exact_ties(dtype, top):
    """Maxima at which 16-bit values land exactly between two e4m3 values (x / scale = 84, 42, ...): the plain pass, the pass
    beside the compression and ``fp8.quantize`` take the same side."""
    from sparse import fp8, spmm
    lib, _ext = _lib()
    m, k = 256, 256
    x = _rand((k, m), dtype, 12, 1.5).clamp(-top, top)
    x[0, 0] = top
    x[1] = top * 3 / 16
    want, s = fp8.quantize(x)
    a = _amax(x)
    q, gq = torch.empty(k, m, dtype=E4M3, device=DEV), torch.empty(k, m, dtype=E4M3, device=DEV)
    _ext.check(lib.sp24_quantize_f8(x.data_ptr(), _ext.dt(dtype), k, m, m, a.data_ptr(), q.data_ptr(), None, 0, _ext.stream()), "quantize")
    packed, meta = fp8.compress_q8(x.t(), mode=_ext.PRUNE_MSE, scale=s)
    p2, m2 = torch.empty_like(packed), torch.empty_like(meta)
    _ext.check(lib.sp24_prune_compress_q8_dev(x.data_ptr(), _ext.dt(dtype), m, k, m, 1, p2.data_ptr(), _ext.E4M3, k // 2, m2.data_ptr(),
                                              _ext.PRUNE_MSE, None, 0, a.data_ptr(), 0, 0, None, None, gq.data_ptr(), m, _ext.stream()),
               "compress")
    assert torch.equal(q.view(torch.uint8), want.view(torch.uint8))
    assert torch.equal(gq.view(torch.uint8), want.view(torch.uint8))
    assert torch.equal(p2.view(torch.uint8), packed.view(torch.uint8)) and torch.equal(m2, meta)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k", [(128, 128), (384, 256), (256, 1152)])
def test_compress_with_device_scale_equals_host_scale(dtype, m, k):
    """dY^T: the same packed values and metadata as with the scale read back; the extras against torch."""
    from sparse import fp8, spmm
    lib, _ext = _lib()
    g = _rand((k, m), dtype, 3, 1e-3)
    s = fp8.scale_of(g)
    packed, meta = fp8.compress_q8(g.t(), mode=_ext.PRUNE_MVUE_FAST, scale=s, seed=11)
    p2, m2 = torch.empty_like(packed), torch.empty_like(meta)
    tc = torch.zeros(spmm.tc_bytes(m, k), dtype=torch.uint8, device=DEV)
    sums = torch.ones(m, device=DEV)
    gq = torch.empty(k, m, dtype=E4M3, device=DEV)
    a = _amax(g)
    _ext.check(lib.sp24_prune_compress_q8_dev(g.data_ptr(), _ext.dt(dtype), m, k, m, 1, p2.data_ptr(), _ext.E4M3, k // 2, m2.data_ptr(),
                                              _ext.PRUNE_MVUE_FAST, None, 0, a.data_ptr(), 11, 0, tc.data_ptr(), sums.data_ptr(),
                                              gq.data_ptr(), m, _ext.stream()), "compress")
    assert torch.equal(p2.view(torch.uint8), packed.view(torch.uint8)) and torch.equal(m2, meta)
    assert torch.equal(tc, spmm.tc_metadata(meta, m, k))
    assert torch.equal(gq.view(torch.uint8), fp8.quantize(g)[0].view(torch.uint8))
    # float32 sums of k values: k ulps of the sum of magnitudes
    want = 1.0 + g.double().sum(0)
    assert float((sums.double() - want).abs().max()) <= k * 2 ** -24 * float(1 + g.double().abs().sum(0).max())
    # row-major source (a weight): metadata in tensor-core order as well
    w = _rand((m, k), torch.float32, 4)
    mask = torch.zeros(m, k, dtype=torch.bool, device=DEV)
    mask[:, 0::4] = mask[:, 3::4] = True
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MASK, mask=mask, scale=fp8.scale_of(w))
    aw = _amax(w)
    _ext.check(lib.sp24_prune_compress_q8_dev(w.data_ptr(), _ext.F32, m, k, k, 0, p2.data_ptr(), _ext.E4M3, k // 2, m2.data_ptr(),
                                              _ext.PRUNE_MASK, mask.data_ptr(), k, aw.data_ptr(), 0, 0, tc.data_ptr(), None, None, 0,
                                              _ext.stream()), "compress")
    assert torch.equal(p2.view(torch.uint8), packed.view(torch.uint8)) and torch.equal(m2, meta)
    assert torch.equal(tc, spmm.tc_metadata(meta, m, k))


@pytest.mark.parametrize("ms,k,n", [(128, 128, 1), (128, 384, 200), (256, 256, 1024), (512, 640, 1100), (768, 128, 2048)])
def test_f8_gemm_with_device_scales(ms, k, n):
    """All output forms against the float32 product of the dequantised operands; 16-bit outputs are one rounding away."""
    from sparse import fp8, spmm
    lib, _ext = _lib()
    w, x, bias = _rand((ms, k), torch.float32, 5), _rand((n, k), torch.float32, 6), _rand((ms,), torch.float32, 7)
    sw, (xq, sx) = fp8.scale_of(w), fp8.quantize(x)
    packed, meta = fp8.compress_q8(w, mode=_ext.PRUNE_MSE, scale=sw)
    tc = spmm.tc_metadata(meta, ms, k)
    aw, ax = _amax(w), _amax(x)
    ref = spmm.sparse_linear(xq, packed, meta, bias=bias, alpha=sw * sx)
    status = spmm._status_word(torch.device(DEV))

    def call(out, trans, b):
        _ext.check(lib.sp24_spmm_f8(packed.data_ptr(), _ext.E4M3, k // 2, tc.data_ptr(), ms, k, xq.data_ptr(), k, n, out.data_ptr(),
                                    _ext.dt(out.dtype), trans, out.shape[1], _ext.ptr(b), aw.data_ptr(), ax.data_ptr(), status.data_ptr(),
                                    _ext.stream()), "spmm_f8")
        return out

    assert torch.equal(call(torch.empty(n, ms, device=DEV), 1, bias), ref)
    for dtype in (torch.float16, torch.bfloat16):
        assert torch.equal(call(torch.empty(n, ms, dtype=dtype, device=DEV), 1, bias), ref.to(dtype))
    if n % 8 == 0:
        acc = call(torch.ones(ms, n, device=DEV), 0, None)
        want = 1.0 + spmm.sparse_linear(xq, packed, meta, alpha=sw * sx).t()
        # slices of K are added in float32: a few ulps of the largest partial sum
        assert float((acc - want).abs().max() / want.abs().max()) <= 1e-5
    spmm.check_status()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 264), (257, 256), (4096, 1000)])
def test_column_sums(dtype, rows, cols):
    lib, _ext = _lib()
    x = _rand((rows, cols), dtype, 8)
    out = torch.full((cols,), 2.0, device=DEV)
    _ext.check(lib.sp24_column_sums(x.data_ptr(), _ext.dt(dtype), rows, cols, cols, out.data_ptr(), _ext.stream()), "column_sums")
    want = 2.0 + x.double().sum(0)
    assert float((out.double() - want).abs().max()) <= (rows + 1) * 2 ** -24 * float(2 + x.double().abs().sum(0).max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_float8_draws_follow_the_device_counter(dtype):
    """A step replayed from a graph keeps its seed; the installed counter moves the draws of the layer and of ``compress_q8``, and
    a counter of c gives what an offset of c gives."""
    import random
    import sparse
    from sparse import fp8, _ext
    from sparse._semi_structured_conversions import set_device_rng_offset
    tokens, in_f, out_f = 256, 256, 128
    x, dy = _rand((tokens, in_f), dtype, 21).requires_grad_(True), _rand((tokens, out_f), dtype, 22, 1e-3)
    w = torch.nn.Parameter(_rand((out_f, in_f), torch.float32, 23))
    w8 = fp8.Fp8SparseWeight(w, sparse.mask_select(w.detach())[1])

    def grad():
        w.grad = x.grad = None
        random.seed(9)
        fp8.sparse_linear_transpose_fp8.apply(x, w, w8, None).backward(dy)
        return w.grad

    scale = fp8.scale_of(dy)
    counter = torch.zeros(1, dtype=torch.int64, device=DEV)
    plain = grad()
    try:
        set_device_rng_offset(counter)
        at0 = grad()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            grad()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            held = grad()
        replays = []
        for c in (0, 3, 5):
            counter.fill_(c)
            graph.replay()
            replays.append(held.clone())
        counter.fill_(3)
        eager3, q3 = grad(), fp8.compress_q8(dy.t(), mode=_ext.PRUNE_MVUE_FAST, scale=scale, seed=9)
    finally:
        set_device_rng_offset(None)
    want3 = fp8.compress_q8(dy.t(), mode=_ext.PRUNE_MVUE_FAST, scale=scale, seed=9, offset=3)
    assert torch.equal(at0, plain) and torch.equal(replays[0], plain) and torch.equal(replays[1], eager3)
    assert torch.equal(q3[0].view(torch.uint8), want3[0].view(torch.uint8)) and torch.equal(q3[1], want3[1])
    assert not torch.equal(replays[0], replays[1]) and not torch.equal(replays[1], replays[2])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("off", [1, 3])
def test_float8_layer_takes_any_alignment(dtype, off):
    """An input and a gradient that start off a 16-byte boundary give what their aligned copies give."""
    import random
    import sparse
    from sparse import fp8
    tokens, in_f, out_f = 256, 128, 256

    def shifted(t):
        v = torch.empty(t.numel() + off, dtype=t.dtype, device=DEV)[off:].view(t.shape)
        return v.copy_(t)

    w, b = (torch.nn.Parameter(_rand(s, torch.float32, 30)) for s in ((out_f, in_f), (out_f,)))
    w8 = fp8.Fp8SparseWeight(w, sparse.mask_select(w.detach())[1])
    x, dy = _rand((tokens, in_f), dtype, 31), _rand((tokens, out_f), dtype, 32, 1e-3)
    res = []
    for put in (torch.clone, shifted):
        w.grad = b.grad = None
        random.seed(3)
        t = put(x).requires_grad_(True)
        y = fp8.sparse_linear_transpose_fp8.apply(t, w, w8, b)
        y.backward(put(dy))
        res.append((y.detach(), t.grad, w.grad, b.grad))
    assert put(x).data_ptr() % 16 and all(torch.equal(p, q) for p, q in zip(*res))


def test_quantize_takes_any_number_of_rows():
    """More rows than 65535 tiles hold."""
    from sparse import fp8
    lib, _ext = _lib()
    rows, cols = 65535 * 128 + 200, 8
    x = _rand((rows, cols), torch.float16, 33)
    q, q_t, a = torch.empty(rows, cols, dtype=E4M3, device=DEV), torch.empty(cols, rows, dtype=E4M3, device=DEV), _amax(x)
    _ext.check(lib.sp24_quantize_f8(x.data_ptr(), _ext.dt(x.dtype), rows, cols, cols, a.data_ptr(), q.data_ptr(), q_t.data_ptr(), rows,
                                    _ext.stream()), "quantize")
    want = fp8.quantize(x)[0].view(torch.uint8)
    assert torch.equal(q.view(torch.uint8), want) and torch.equal(q_t.view(torch.uint8), want.t().contiguous())
