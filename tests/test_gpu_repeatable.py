"""Gradients that repeat bit for bit: the sums behind them are taken in a fixed order, not by atomics."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _gradient(tokens, features, dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    d = torch.randn(tokens, features, device=DEV, generator=g) * 1e-3
    d.mul_(torch.where(torch.rand(tokens, features, device=DEV, generator=g) < 0.01, 100.0, 1.0))
    return d.to(dtype)


def _step(kind, tokens, in_f, out_f, dtype, into=False):
    """Gradients (dw, db) of one layer step whose state is the same on every call."""
    import sparse
    torch.manual_seed(1)
    random.seed(1)
    x = torch.randn(tokens, in_f, device=DEV).to(dtype).requires_grad_(True)
    dy = _gradient(tokens, out_f, dtype, 2)
    if kind == "sste":
        layer = sparse.SoftThresholdLinear(in_f, out_f, bias=True, device=DEV, spmm=True, spmm_dtype=dtype)
        layer.init_scale()
    else:
        layer = sparse.SparseLinearTranspose(in_f, out_f, bias=True).cuda()
    if into:
        layer.accumulate_into_grad = True
        layer.weight.grad, layer.bias.grad = torch.zeros_like(layer.weight), torch.ones_like(layer.bias)
    if kind == "fp8":
        w8 = sparse.fp8.Fp8SparseWeight(layer.weight, sparse.mask_select(layer.weight.detach())[1])
        y = sparse.fp8.sparse_linear_transpose_fp8.apply(x, layer.weight, w8, layer.bias)
    else:
        with torch.autocast("cuda", dtype):
            y = layer(x)
    y.backward(dy)
    return layer.weight.grad, layer.bias.grad, dy


# (tokens, in, out): one partial sum, a ragged number of them, and enough blocks to finish in any order
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind,into", [("fst", False), ("fst", True), ("fp8", False), ("sste", False)])
@pytest.mark.parametrize("tokens,in_f,out_f", [(256, 256, 256), (768, 128, 384), (16384, 256, 1024)])
def test_bias_gradient_repeats(kind, into, tokens, in_f, out_f, dtype):
    """The same bits every time, and float32 sums: within ``tokens`` roundings of the sum of magnitudes."""
    _, db, dy = _step(kind, tokens, in_f, out_f, dtype, into)
    for _ in range(4):
        assert torch.equal(_step(kind, tokens, in_f, out_f, dtype, into)[1], db)
    want = dy.double().sum(0) + (1.0 if into else 0.0)
    assert float((db.double() - want).abs().max()) <= (tokens + 1) * 2 ** -24 * float(1 + dy.double().abs().sum(0).max())


@pytest.mark.parametrize("n_parts,m", [(1, 32), (7, 96), (8, 33), (9, 1), (131, 1000)])
def test_sum_of_parts(n_parts, m):
    from sparse import _ext
    parts = torch.randn(n_parts, m, device=DEV)
    out = torch.full((m,), 3.0, device=DEV)
    for add in (1, 0):
        _ext.check(_ext.lib().sp24_sum_parts(parts.data_ptr(), n_parts, m, out.data_ptr(), add, _ext.stream()), "sum_parts")
        want = parts.double().sum(0) + 3.0 * add
        assert float((out.double() - want).abs().max()) <= (n_parts + 1) * 2 ** -24 * float(3 + parts.double().abs().sum(0).max())


# (tokens, in, out): one tile, tiles that would leave room for four and for three slices of K, more tiles than SMs
@pytest.mark.parametrize("tokens,in_f,out_f", [(256, 256, 128), (4096, 512, 512), (8192, 768, 3072), (1024, 3072, 2048)])
def test_float8_weight_gradient_repeats(tokens, in_f, out_f):
    from sparse.spmm import check_status
    dw = _step("fp8", tokens, in_f, out_f, torch.bfloat16)[0]
    for _ in range(4):
        assert torch.equal(_step("fp8", tokens, in_f, out_f, torch.bfloat16)[0], dw)
    check_status()
