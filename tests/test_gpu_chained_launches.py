"""Kernels of the library in plain stream order, whatever runs around them: their input is written directly before and overwritten directly
after by foreign kernels or by the library's own, on one stream, across two streams with events, and in a captured graph with a fork and a
join.  Results are those of calls with everything waited for in between, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(*shape, seed, dtype=torch.float16):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)).to(dtype)


def _mvue(buf):
    """Compression of buf^T to float16: the sparse operand of a weight gradient."""
    from sparse import _ext
    from sparse._semi_structured_conversions import prune_compress
    k, m = buf.shape
    packed, meta = torch.empty(k // 2, m, dtype=torch.float16, device=DEV).t(), torch.empty(m, k // 16, dtype=torch.int16, device=DEV)
    prune_compress(buf.t(), packed, meta, mode=_ext.PRUNE_MVUE_FAST, seed=5)
    return packed, meta


def _select(buf):
    import sparse
    mask, w, wt = sparse.select_and_compress(buf, dtype=torch.float16)
    return (mask, *w, *wt)


def _decay(buf):
    import sparse
    grad, mask = torch.zeros_like(buf), torch.zeros(buf.shape, dtype=torch.bool, device=DEV)
    sparse.masked_add_(grad, buf, mask, alpha=0.5)
    sparse.masked_add_(grad, grad, mask, alpha=0.25)
    return (grad,)


def _product(ms):
    import sparse
    from sparse import spmm
    w = sparse.to_sparse_semi_structured(_rand(ms, 1024, seed=9), dtype=torch.float16)
    p, e = w.sparse_tensor_cutlass, w.meta_tensor_cutlass
    spmm.tc_metadata(e, ms, 1024)

    def op(buf):
        y = spmm.sparse_linear(buf, p, e)
        out = torch.zeros(ms, 1024, device=DEV)
        spmm.sparse_mm_accumulate_(out, *_mvue(y), buf, k_splits=1)
        return y, out
    return op


def _few_tokens():
    import sparse
    from sparse import spmm
    w = sparse.to_sparse_semi_structured(_rand(2048, 2048, seed=8), dtype=torch.float16)
    p, e = w.sparse_tensor_cutlass, w.meta_tensor_cutlass
    spmm.tc_metadata(e, 2048, 2048)

    def op(buf):
        y = buf
        for _ in range(4):
            y = spmm.sparse_linear(y, p, e) * 0.02
        return (y,)
    return op


def _float8(buf):
    from sparse import _ext
    amax, q = torch.full((1,), 9.0, device=DEV), torch.empty(buf.shape, dtype=torch.uint8, device=DEV)
    rows, cols = buf.shape
    _ext.check(_ext.lib().sp24_absmax(buf.data_ptr(), _ext.dt(buf.dtype), buf.numel(), None, amax.data_ptr(), _ext.stream()), "absmax")
    _ext.check(_ext.lib().sp24_quantize_f8(buf.data_ptr(), _ext.dt(buf.dtype), rows, cols, cols, amax.data_ptr(), q.data_ptr(), None, 0,
                                           _ext.stream()), "quantize")
    return amax, q


def _norm_backward(buf):
    """gamma comes from the library's own optimizer kernel, directly before."""
    import sparse
    from sparse import _ext
    rows, d = buf.shape
    gamma, m, v = torch.ones(d, device=DEV), torch.zeros(d, device=DEV), torch.zeros(d, device=DEV)
    x, mean, rstd = torch.ones(rows, d, device=DEV), torch.zeros(rows, device=DEV), torch.ones(rows, device=DEV)
    dx, dg, db = torch.empty_like(x), torch.zeros(d, device=DEV), torch.zeros(d, device=DEV)
    sparse.adamw_masked_decay_(gamma, buf[0].float().contiguous(), m, v, step=1, lr=0.5)
    _ext.check(_ext.lib().sp24_layernorm_bwd(buf.data_ptr(), _ext.dt(buf.dtype), x.data_ptr(), gamma.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                                             dx.data_ptr(), dg.data_ptr(), db.data_ptr(), rows, d, _ext.stream()), "layernorm_bwd")
    return gamma, dx


# name -> (operation, shape and type of its input)
OPS = {
    "mvue": lambda: (_mvue, (2048, 1024), torch.float16),
    "mvue float32": lambda: (_mvue, (2048, 1024), torch.float32),
    "select": lambda: (_select, (1024, 1024), torch.float16),
    "decay": lambda: (_decay, (2048, 1024), torch.float32),
    "products": lambda: (_product(1024), (2048, 1024), torch.float16),
    "products odd rows": lambda: (_product(896), (2048, 1024), torch.float16),
    "few tokens": lambda: (_few_tokens(), (16, 2048), torch.float16),
    "float8": lambda: (_float8, (2048, 1024), torch.bfloat16),
    "norm backward": lambda: (_norm_backward, (2048, 768), torch.bfloat16),
}


def _setup(name):
    op, shape, dtype = OPS[name]()
    values = [_rand(*shape, seed=s, dtype=dtype) for s in (1, 2)]
    want = []
    for v in values:
        torch.cuda.synchronize()
        want.append([t.clone() for t in op(v)])
        torch.cuda.synchronize()
    assert any(not torch.equal(a, b) for a, b in zip(*want))
    return op, values, want


def _same(got, want):
    torch.cuda.synchronize()
    from sparse.spmm import check_status
    check_status()
    return all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("name", list(OPS))
def test_one_stream(name):
    op, values, want = _setup(name)
    buf, got = torch.empty_like(values[0]), []
    for r in range(8):
        buf.copy_(values[r % 2])            # written by a foreign kernel
        got.append(op(buf))
        buf.fill_(float("nan"))             # and overwritten by another
    assert all(_same(g, want[r % 2]) for r, g in enumerate(got))


def _two_streams(op, values, buf, side, rounds):
    """The rounds alternate between the current stream and ``side``, each of which waits for the other's last round."""
    main, got = torch.cuda.current_stream(), []
    for r in range(rounds):
        here, there = (main, side) if r % 2 == 0 else (side, main)
        with torch.cuda.stream(here):
            buf.copy_(values[r % 2])
            got.append(op(buf))
            buf.zero_()
        there.wait_stream(here)
    main.wait_stream(side)
    return got


@pytest.mark.parametrize("name", list(OPS))
def test_two_streams(name):
    op, values, want = _setup(name)
    got = _two_streams(op, values, torch.empty_like(values[0]), torch.cuda.Stream(), 6)
    assert all(_same(g, want[r % 2]) for r, g in enumerate(got))


@pytest.mark.parametrize("name", list(OPS))
def test_captured_fork_and_join(name):
    op, values, want = _setup(name)
    buf, side = torch.empty_like(values[0]), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _two_streams(op, values, buf, side, 4)
    for _ in range(3):
        for g in got:
            for t in g:
                t.zero_()
        graph.replay()
        assert all(_same(g, want[r % 2]) for r, g in enumerate(got))
