"""Autograd nodes of the native host path: saved tensors pass through the saved-tensor hooks, a forward-mode tangent is
refused, and a weight's copies changed in place between the passes are noticed.  And the linear layer's unpadded route."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layers():
    import sparse
    from sparse import train_ops
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(128, 256, device=DEV, generator=g).half()
    fst = sparse.SparseLinearTranspose(256, 128, bias=True).cuda()
    sste = sparse.SoftThresholdLinear(256, 128, bias=True, device=DEV, spmm=True)
    sste.init_scale()
    norm = train_ops.LayerNorm(256).cuda()
    mask = sparse.mask_select(fst.weight.detach())[1]

    def fp8(t):
        return sparse.fp8.sparse_linear_transpose_fp8.apply(t, fst.weight, sparse.fp8.Fp8SparseWeight(fst.weight, mask), fst.bias)

    def auto(layer):
        def call(t):
            with torch.autocast("cuda", torch.float16):
                return layer(t)
        return call
    return x, {"fst": auto(fst), "sste": sste, "fp8": fp8, "norm": auto(norm), "gelu": train_ops.gelu,
               "add_norm": auto(lambda t: train_ops.add_layer_norm(t.float(), t, norm)[1]),
               "cross_entropy": lambda t: train_ops.cross_entropy(t, torch.arange(128, device=DEV))}


NAMES = ["fst", "sste", "fp8", "norm", "gelu", "add_norm", "cross_entropy"]


@pytest.mark.parametrize("name", NAMES)
def test_saved_tensors_pass_through_hooks(name):
    """Packed to the host and back, the gradient has the same bits; every node hands at least one tensor to the hooks."""
    import random
    x, calls = _layers()
    packed, grads = [], []
    for hooked in (False, True):
        random.seed(5)
        t = x.clone().requires_grad_(True)
        if hooked:
            def pack(v):
                packed.append(v.shape)
                return v.stride(), v.cpu()

            def unpack(p):
                return torch.empty_strided(p[1].shape, p[0], dtype=p[1].dtype, device=DEV).copy_(p[1])
            with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
                y = calls[name](t)
        else:
            y = calls[name](t)
        y.backward(torch.ones_like(y) * 0.5)
        grads.append(t.grad)
    assert packed
    assert torch.equal(grads[0], grads[1])


@pytest.mark.parametrize("name", NAMES)
def test_forward_mode_is_refused(name):
    x, calls = _layers()
    with fwAD.dual_level(), pytest.raises(NotImplementedError):
        calls[name](fwAD.make_dual(x, torch.ones_like(x)))


def test_changed_copies_are_noticed():
    import sparse
    x, _ = _layers()
    layer = sparse.SparseLinearTranspose(256, 128, bias=False).cuda()
    with torch.autocast("cuda", torch.float16):
        y = layer(x.requires_grad_(True))
    layer.weight.compressed[2].mul_(2)
    with pytest.raises(RuntimeError, match="inplace"):
        y.backward(torch.ones_like(y))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tokens", [1, 7, 8, 127, 129, 255, 257, 1025])
def test_ragged_tokens_equal_padded_ones(dtype, tokens):
    """A ragged number of token-major rows is not padded; each row's result has the bits it has among padded rows.  The
    same kernel accumulates every row in the same K order, wherever the last tile is cut."""
    import sparse
    g = torch.Generator(device=DEV).manual_seed(tokens)
    w = sparse.to_sparse_semi_structured(torch.randn(256, 512, device=DEV, generator=g).to(dtype), dtype=dtype)
    b = torch.randn(256, device=DEV, generator=g).to(dtype)
    full = torch.randn((tokens + 7) // 8 * 8, 512, device=DEV, generator=g).to(dtype)
    x = full[:tokens].clone()
    with torch.inference_mode():
        assert torch.equal(F.linear(x, w, b), F.linear(full, w, b)[:tokens])
        assert torch.equal(F.linear(x, w), F.linear(full, w)[:tokens])
        assert torch.equal(F.linear(full[:tokens].unsqueeze(0), w, b)[0], F.linear(full, w, b)[:tokens])


class _Call(torch.nn.Module):
    """``fn(module, x)`` as a module: a trace takes the module's parameters for parameters, not for constants."""

    def __init__(self, fn, module=None):
        super().__init__()
        self.fn, self.module = fn, module

    def forward(self, t):
        with torch.autocast("cuda", torch.float16):
            return self.fn(self.module, t)


def _traceable(name):
    import sparse
    from sparse import train_ops
    if name in ("fst", "fst dense", "fp8"):
        layer = sparse.SparseLinearTranspose(256, 128, bias=True).cuda()
        if name == "fst dense":
            layer.weight.weight_grad = "dense"
        if name != "fp8":
            return _Call(lambda m, t: m(t), layer)
        w8 = sparse.fp8.Fp8SparseWeight(layer.weight, sparse.mask_select(layer.weight.detach())[1])
        return _Call(lambda m, t: sparse.fp8.sparse_linear_transpose_fp8.apply(t, m.weight, w8, m.bias), layer)
    if name == "sste":
        layer = sparse.SoftThresholdLinear(256, 128, bias=True, device=DEV, spmm=True)
        layer.init_scale()
        return _Call(lambda m, t: m(t), layer)
    if name == "gelu":
        return _Call(lambda m, t: train_ops.gelu(t))
    if name == "cross_entropy":
        targets = torch.arange(128, device=DEV)
        return _Call(lambda m, t: train_ops.cross_entropy(t, targets))
    norm = train_ops.LayerNorm(256).cuda()
    if name == "norm":
        return _Call(lambda m, t: m(t), norm)
    return _Call(lambda m, t: train_ops.add_layer_norm(t.float(), t, m)[1], norm)


@pytest.mark.parametrize("name", NAMES + ["fst dense"])
def test_traced_layers_replay(name):
    """``torch.jit.trace`` records a layer as a call: other inputs give their own results and gradients, not what the trace's
    output buffer happens to hold."""
    import random
    torch.manual_seed(6)
    layer = _traceable(name)
    first, second = (torch.randn(128, 256, device=DEV).half() for _ in range(2))
    layer(first)                               # an FST layer compresses its weight before it is traced
    traced = torch.jit.trace(layer, (first.clone().requires_grad_(True),), check_trace=False)
    grads = []
    for f in (layer, traced):
        t = second.clone().requires_grad_(True)
        layer.zero_grad(set_to_none=True)
        random.seed(4)
        y = f(t)
        torch.manual_seed(7)
        y.backward(torch.randn_like(y))
        grads.append([y.detach(), t.grad] + [p.grad for p in layer.parameters()])
    assert len(grads[0]) == len(grads[1])
    for a, b in zip(*grads):
        assert a.dtype == b.dtype and float((a.float() - b.float()).norm()) <= 1e-6 * float(a.float().norm())     # sums in any order


def test_traced_embedding_replays():
    from sparse import train_ops
    wte, wpe = torch.randn(64, 32, device=DEV), torch.randn(16, 32, device=DEV)
    first, second = (torch.randint(0, 64, (2, 16), device=DEV) for _ in range(2))
    traced = torch.jit.trace(lambda t: train_ops.embed_tokens(t, wte, wpe), (first,), check_trace=False)
    assert torch.equal(traced(second), train_ops.embed_tokens(second, wte, wpe))


def _dense_of(name, layer):
    """The weight that the layer's input gradient multiplies by, float64."""
    return layer.get_sparse_weights().detach().half().double() if name == "sste" else None


@pytest.mark.parametrize("name", ["sste", "fst", "fst dense", "fp8"])
def test_gradients_stay_functions_of_the_incoming_one(name):
    """Under ``create_graph`` whatever is a plain torch operation on dY keeps its graph (a gradient penalty differentiates it):
    all three gradients of the S-STE layer, the bias sums of the others.  (The dense option's weight gradient has a graph too, but
    torch's product with a float32 result has no derivative and says so.)"""
    torch.manual_seed(8)
    call = _traceable(name)
    layer = call.module
    x = torch.randn(128, 256, device=DEV).half().requires_grad_(True)
    v = (torch.randn(128, 128, device=DEV) * 0.1).requires_grad_(True)
    wanted = {"sste": [x, layer.weight, layer.bias], "fst dense": [layer.weight, layer.bias]}.get(name, [layer.bias])
    y = call(x)
    got = torch.autograd.grad(y, wanted, v.half(), create_graph=True)
    assert all(g.requires_grad for g in got)
    penalised = [(t, g) for t, g in zip(wanted, got) if name != "fst dense" or t is layer.bias]
    plain = torch.autograd.grad(call(x), wanted, v.detach().half())
    for a, b in zip(got, plain):
        assert a.dtype == b.dtype and float((a - b).float().norm()) <= 1e-3 * float(b.float().norm())
    # penalty = sum of squares of the gradients; its derivative in dY, in 64 bits
    torch.autograd.backward(sum((g.float() ** 2).sum() for _, g in penalised))
    v64, want = v.detach().half().double(), 0
    for t, _ in penalised:
        if t is x:
            w = _dense_of(name, layer)
            want = want + 2 * (v64 @ w) @ w.t()
        elif t is layer.weight:
            want = want + 2 * x.detach().double() @ (v64.t() @ x.detach().double()).t()
        else:
            want = want + 2 * v64.sum(0).expand_as(v64)
    assert float((v.grad.double() - want).norm() / want.norm()) <= 4e-3       # fp16 roundings of the two products


@pytest.mark.parametrize("dtype", [torch.uint16, torch.uint32, torch.int16, torch.int32, torch.float8_e4m3fn, torch.float8_e5m2, torch.float16,
                                   torch.bfloat16, torch.float32, torch.int8, torch.uint8])
def test_masked_add_takes_a_mask_for_what_its_type_says(dtype):
    """Zero is decided by the mask's type: -0.0 is zero in every floating type, the top bit alone is not in an integer."""
    import sparse
    n = 96
    if dtype.is_floating_point:
        m = torch.tensor([0.0, -0.0, 1.0, -2.0] * (n // 4), device=DEV).to(dtype)
        zero = torch.tensor([True, True, False, False] * (n // 4), device=DEV)
    else:
        top = torch.iinfo(dtype).min or torch.iinfo(dtype).max // 2 + 1
        m = torch.tensor([0, top, 1, 0] * (n // 4)).to(dtype).to(DEV)
        zero = torch.tensor([True, False, False, True] * (n // 4), device=DEV)
    g, p = torch.randn(n, device=DEV), torch.randn(n, device=DEV)
    want = torch.where(zero, g + p * 0.5, g)
    sparse.masked_add_(g, p, m, alpha=0.5)
    assert torch.equal(g, want)


def test_copies_of_w_and_of_its_transpose_are_written_apart():
    """The copies live in one allocation; a write to W's between the passes is no write to W^T's, which the backward pass holds."""
    import sparse
    x, _ = _layers()
    layer = sparse.SparseLinearTranspose(256, 128, bias=False).cuda()
    t = x.clone().requires_grad_(True)
    with torch.autocast("cuda", torch.float16):
        y = layer(t)
    y.backward(torch.ones_like(y), retain_graph=True)
    want, before = t.grad.clone(), layer.weight.compressed[3]._version
    t.grad = None
    layer.weight.compressed[0].mul_(2)
    layer.weight.compressed[1].add_(0)
    assert layer.weight.compressed[3]._version == before
    y.backward(torch.ones_like(y))
    assert torch.equal(t.grad, want)


@pytest.mark.parametrize("dtype", [torch.int8, torch.float8_e4m3fn])
@pytest.mark.parametrize("tokens", [1, 7, 17, 129, 255])
def test_ragged_tokens_of_8_bit_operands(dtype, tokens):
    """The unpadded route with 8-bit operands: each row has the bits it has among rows padded to a multiple of 32."""
    import sparse
    g = torch.Generator(device=DEV).manual_seed(tokens)
    dense = torch.randint(-9, 9, (256, 512), device=DEV, generator=g).to(torch.int8 if dtype == torch.int8 else torch.float32)
    if dtype == torch.int8:
        w = sparse.to_sparse_semi_structured(dense, dtype=dtype)
    else:
        w = sparse.to_sparse_semi_structured(dense.half(), dtype=dtype)
    full = torch.randint(-9, 9, ((tokens + 31) // 32 * 32, 512), device=DEV, generator=g).to(dtype)
    x = full[:tokens].clone()
    with torch.inference_mode():
        want = F.linear(full, w)[:tokens]
        assert torch.equal(F.linear(x, w), want)
        assert torch.equal(F.linear(x.unsqueeze(0), w)[0], want)
    ref = x.double() @ _kept(w, dense).double().t()
    assert torch.equal(want.double(), ref)             # integers of at most 9 * 9 * 512: exact in float32 and int32


def _kept(w, dense):
    from sparse import spmm
    eye = torch.eye(dense.shape[1], device=DEV).to(w.sparse_tensor_cutlass.dtype)
    return spmm.sparse_linear(eye, w.sparse_tensor_cutlass, w.meta_tensor_cutlass).t()
