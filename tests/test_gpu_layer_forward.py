"""SparseLinearTranspose.forward in native code: results, gradients and the state on the weight of a run are those of the class's own Python
(which a subclass takes), through new masks, accumulation windows, a batched refresh, evaluation, edited copies and replaced methods."""
import gc
import random

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
STATE = ("mode", "cnt", "counter", "freq", "step", "weight_sparse", "weight_sparse_T")


@pytest.fixture(autouse=True)
def _nothing_left():
    """Caught exceptions hold layers in cycles; other tests count the memory in use."""
    yield
    gc.collect()


def _pair(i, o, bias=True):
    import sparse

    class Sub(sparse.SparseLinearTranspose):
        pass

    torch.manual_seed(5)
    a, b = sparse.SparseLinearTranspose(i, o, bias=bias).to(DEV), Sub(i, o, bias=bias).to(DEV)
    b.load_state_dict(a.state_dict())
    for m in (a, b):
        m.weight.mask = sparse.mask_select(m.weight.detach())[1]
        m.weight.freq = 3
    return a, b


def _same(a, b):
    w, v = a.weight, b.weight
    assert all(getattr(w, n) == getattr(v, n) for n in STATE) and getattr(w, "refreshed", False) == getattr(v, "refreshed", False)
    assert torch.equal(w.mask, v.mask) and (w.compressed is None) == (v.compressed is None)
    if w.compressed is not None:
        assert all(torch.equal(x, y) and x.stride() == y.stride() and x._version == y._version for x, y in zip(w.compressed, v.compressed))
        assert w.compressed_tc[0] is w.compressed and w.compressed_tc[1:3] == v.compressed_tc[1:3]
        assert all(torch.equal(x, y) for x, y in zip(w.compressed_tc[3], v.compressed_tc[3]))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, None])
@pytest.mark.parametrize("i,o,bias,shape", [(128, 256, True, (64,)), (384, 128, False, (2, 64)), (256, 384, True, (128,))])
def test_a_run_leaves_the_same_state(i, o, bias, shape, dtype):
    import sparse
    a, b = _pair(i, o, bias)
    x = torch.randn(*shape, i, device=DEV, requires_grad=True)
    seen = a.weight.mask.data_ptr()

    def one(layer):
        random.seed(3)
        with torch.autocast("cuda", dtype=dtype or torch.float16, enabled=dtype is not None):
            y = layer(x)
        grads = torch.autograd.grad(y.float().square().mean(), [x] + list(layer.parameters()))
        return (y, *grads)
    for step in range(7):
        for m in (a, b):
            m.weight.cnt = 0
            m.train(step != 5)
        if step == 4:
            for m in (a, b):
                with torch.autocast("cuda", dtype=dtype or torch.float16, enabled=dtype is not None):
                    assert sparse.refresh_sparse_layers(torch.nn.ModuleList([m])) == 1
        for micro in range(2):
            for p, q in zip(one(a), one(b)):
                assert p.dtype == q.dtype and torch.equal(p, q)
            _same(a, b)
        with torch.no_grad():
            for m in (a, b):
                m.weight.mul_(1.0 + 0.25 * torch.randn(o, i, device=DEV, generator=torch.Generator(device=DEV).manual_seed(step)))
    assert a.weight.mask.data_ptr() == seen and a.weight.step == 12


def test_what_is_not_plain_goes_to_python(monkeypatch):
    import sparse
    from sparse import _ext
    a, b = _pair(128, 256)
    x = torch.randn(64, 128, device=DEV)
    native = _ext.host.fst_forward
    assert native(b, x) is None and native(a, 3) is None and b.weight.step == 0
    y = native(a, x)
    assert a.weight.step == 1 and torch.equal(y, b(x))
    assert native(a, x) is not None
    a.weight.compressed[1].add_(0)                 # metadata written to: its order for the GEMM is made anew
    assert native(a, x) is None and a.weight.step == 2 and torch.equal(a(x), y)
    a.weight.cnt = 0
    a._refresh = lambda reselect: (_ for _ in ()).throw(KeyError("mine"))
    assert native(a, x) is None
    with pytest.raises(KeyError):
        a(x)
    del a._refresh
    a.weight.mask = a.weight.mask.cpu()
    assert native(a, x) is None and torch.equal(a(x), y)
    monkeypatch.setattr(sparse.SparseLinearTranspose, "_advance", lambda self: None)
    assert native(a, x) is None
    step = a.weight.step
    a(x)
    assert a.weight.step == step
    monkeypatch.undo()
    monkeypatch.setattr(sparse.SparseLinearTranspose, "materialize_sparse_tensors", True)
    assert native(a, x) is None


def test_odd_shapes_refuse_as_before():
    import sparse
    layer = sparse.SparseLinearTranspose(128, 192).to(DEV)
    with pytest.raises(RuntimeError, match="divisible by 128"):
        layer(torch.randn(64, 128, device=DEV))
