"""Workloads on which the speed of this framework is measured, each one a call sequence of a user's program.

``listed()`` names the fixed workloads, ``draw(rng)`` gives further ones from the same ranges.  ``prepare(case, seed)``
makes what the program holds before the call, ``run(state)`` is one pass through the public entry points, ``work(case)``
the bytes and operations the pass cannot do without, ``tolerance(case)`` how far two correct implementations may differ.

Kinds of workload:
  fst      one training step of a ``SparseLinearTranspose`` layer right after an optimizer step: the compressed copies of
           the weight are rebuilt (a new mask on every 40th step), forward, backward to input, weight and bias
  fp8      the same layer step on e4m3 operands (``sparse.fp8``), the weight compressed anew
  linear   inference: ``F.linear`` with a weight that was converted once by ``to_sparse_semi_structured``
  upkeep   what a step does to a model's sparse weights between backward and forward: masked decay of every gradient,
           then the compressed copies of all layers
  select   a mask refresh of whole weights: transposable 4x4 masks and both compressed copies
  mvue     gradient pruning: MVUE 2:4 compression of dY^T
  sste     one training step of the S-STE layer, forward on the sparse tensor cores
  gpt2     forward and backward pass of the GPT-2 trainer's model, launched eagerly or replayed from a CUDA graph
"""
import os
import random
import sys

import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.getcwd(), "2by4-pretrain_b200"))      # the tree being measured is the working folder

import sparse  # noqa: E402
import train_gpt2  # noqa: E402

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
ALPHA = 2e-4            # masked decay of the reference recipe


def listed():
    return [
        # a layer of a test-size model: launches and host time are all there is
        {"name": "fst small", "kind": "fst", "tokens": 256, "in": 256, "out": 512, "dtype": "fp16", "bias": True},
        # MLP up-projection of GPT-2 on 16 sequences of 1024 tokens, the layer the GEMM benchmark is quoted on
        {"name": "fst mlp 16k tokens", "kind": "fst", "tokens": 16384, "in": 768, "out": 3072, "dtype": "fp16", "bias": True},
        # sizes off every tile: odd multiples of 128 features, a ragged number of tokens, no bias, bf16
        {"name": "fst ragged", "kind": "fst", "tokens": 1984, "in": 1152, "out": 896, "dtype": "bf16", "bias": False},
        # float8 form of the up-projection on 8 sequences of 1024 tokens
        {"name": "fp8 mlp", "kind": "fp8", "tokens": 8192, "in": 768, "out": 3072, "dtype": "bf16", "bias": True},
        # token-by-token decoding of a small batch
        {"name": "linear decode", "kind": "linear", "tokens": 16, "in": 4096, "out": 4096, "dtype": "fp16"},
        # a prompt of odd length
        {"name": "linear prefill", "kind": "linear", "tokens": 2043, "in": 4096, "out": 4096, "dtype": "bf16"},
        # all 48 sparse weights of GPT-2 124M, every optimizer step
        {"name": "upkeep gpt2", "kind": "upkeep", "layers": 12, "d": 768, "dtype": "bf16"},
        # mask refresh of eight 4096 x 4096 weights, the conversion benchmark's matrices
        {"name": "select 4096", "kind": "select", "count": 8, "m": 4096, "k": 4096, "dtype": "fp16"},
        # gradient of 8192 tokens x 4096 features
        {"name": "mvue gradient", "kind": "mvue", "tokens": 8192, "features": 4096, "dtype": "bf16"},
        # S-STE recipe on the attention projection
        {"name": "sste layer", "kind": "sste", "tokens": 4096, "in": 768, "out": 2304, "dtype": "fp16", "bias": True},
        # a test-size transformer launched from Python, as while developing a model
        {"name": "gpt2 tiny eager", "kind": "gpt2", "layers": 2, "d": 256, "heads": 4, "batch": 4, "seq": 128, "vocab": 512,
         "graph": False},
        # the pre-training step at GPT-2 124M's width and vocabulary on 8192 tokens, replayed from a graph.  Four of the twelve
        # blocks and 512 positions: in deeper stacks and longer sequences the unordered sums of the attention's backward pass
        # alone move the gradients by several percent (other roundings make other MVUE draws)
        {"name": "gpt2 wide graph", "kind": "gpt2", "layers": 4, "d": 768, "heads": 12, "batch": 16, "seq": 512, "vocab": 50304,
         "graph": True},
    ]


def _log(rng, lo, hi, step):
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["fst", "fst", "fp8", "linear", "linear", "upkeep", "select", "mvue", "sste", "gpt2"])
    dtype = rng.choice(["fp16", "bf16"])
    bias = rng.random() < 0.7
    if kind == "fst":
        return {"kind": kind, "tokens": _log(rng, 128, 16384, 64), "in": _log(rng, 256, 3072, 128),
                "out": _log(rng, 256, 3072, 128), "dtype": dtype, "bias": bias}
    if kind == "fp8":
        return {"kind": kind, "tokens": _log(rng, 256, 8192, 128), "in": _log(rng, 256, 3072, 128),
                "out": _log(rng, 256, 3072, 128), "dtype": dtype, "bias": bias}
    if kind == "linear":
        return {"kind": kind, "tokens": _log(rng, 1, 4096, 1), "in": _log(rng, 512, 4096, 64), "out": _log(rng, 512, 4096, 128),
                "dtype": dtype}
    if kind == "upkeep":
        return {"kind": kind, "layers": rng.randint(2, 12), "d": _log(rng, 256, 1024, 128), "dtype": dtype}
    if kind == "select":
        return {"kind": kind, "count": rng.randint(1, 8), "m": _log(rng, 256, 4096, 128), "k": _log(rng, 256, 4096, 128),
                "dtype": rng.choice(["fp16", "bf16", "fp32"])}
    if kind == "mvue":
        return {"kind": kind, "tokens": _log(rng, 128, 16384, 64), "features": _log(rng, 256, 4096, 128), "dtype": dtype}
    if kind == "sste":
        return {"kind": kind, "tokens": _log(rng, 128, 8192, 8), "in": _log(rng, 256, 3072, 64), "out": _log(rng, 256, 3072, 128),
                "dtype": dtype, "bias": bias}
    heads = rng.choice([2, 4, 6, 8])
    return {"kind": kind, "layers": rng.randint(1, 4), "d": 128 * heads // 2, "heads": heads, "batch": 2 ** rng.randint(0, 3),
            "seq": _log(rng, 64, 512, 64), "vocab": _log(rng, 256, 16384, 64), "graph": rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------------------------------------------------
def _randn(gen, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(dtype)


def _gradient(gen, *shape, dtype):
    """Gradients: small, with one entry in a hundred a hundred times larger."""
    g = torch.randn(*shape, device="cuda", generator=gen) * 1e-3
    g.mul_(torch.where(torch.rand(*shape, device="cuda", generator=gen) < 0.01, 100.0, 1.0))
    return g.to(dtype)


def _set_weight(layer, gen, bias):
    with torch.no_grad():
        layer.weight.copy_(_randn(gen, *layer.weight.shape, std=0.02))
        if bias:
            layer.bias.copy_(_randn(gen, layer.bias.shape[0], std=0.02))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    random.seed(seed)                  # MVUE seeds come from Python's generator
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "gpt2":
        return _prepare_gpt2(case, seed, gen, s)
    dtype = DTYPES[case["dtype"]]
    s["dtype"] = dtype
    if kind in ("fst", "fp8", "sste"):
        t, i, o, bias = case["tokens"], case["in"], case["out"], case["bias"]
        s["x"] = _randn(gen, t, i, dtype=dtype).requires_grad_(True)
        s["dy"] = _gradient(gen, t, o, dtype=dtype)
        if kind == "sste":
            s["layer"] = sparse.SoftThresholdLinear(i, o, bias=bias, device="cuda", spmm=True, spmm_dtype=dtype)
            _set_weight(s["layer"], gen, bias)
            s["layer"].init_scale()
        else:
            s["layer"] = sparse.SparseLinearTranspose(i, o, bias=bias).cuda()
            _set_weight(s["layer"], gen, bias)
            if kind == "fp8":
                s["mask"] = sparse.mask_select(s["layer"].weight.detach())[1]
    elif kind == "linear":
        w = _randn(gen, case["out"], case["in"], std=0.02, dtype=dtype)
        s["w"] = sparse.to_sparse_semi_structured(w, dtype=dtype)
        s["b"] = _randn(gen, case["out"], std=0.02, dtype=dtype)
        s["x"] = _randn(gen, case["tokens"], case["in"], dtype=dtype)
    elif kind == "upkeep":
        d = case["d"]
        mods = []
        flat = _randn(gen, 12 * d * d * case["layers"], std=1e-3)      # all gradients, as a trainer's flat buffer
        at = 0
        for _ in range(case["layers"]):
            for o, i in ((3 * d, d), (d, d), (4 * d, d), (d, 4 * d)):
                with torch.device("cuda"):
                    mod = sparse.SparseLinearTranspose(i, o)
                _set_weight(mod, gen, False)
                mod.weight.mask = sparse.mask_select(mod.weight.detach())[1]
                mod.weight.grad = flat[at:at + o * i].view(o, i)
                at += o * i
                mod.weight.counter = 1
                mods.append(mod)
        s["model"], s["flat"] = torch.nn.ModuleList(mods), flat
    elif kind == "select":
        s["w"] = [_randn(gen, case["m"], case["k"], std=0.02, dtype=dtype) for _ in range(case["count"])]
        s["masks"] = [torch.ones(case["m"], case["k"], dtype=torch.bool, device="cuda") for _ in s["w"]]
    else:
        s["g"] = _gradient(gen, case["tokens"], case["features"], dtype=dtype)
    return s


def _prepare_gpt2(case, seed, gen, s):
    with torch.device("cuda"):         # parameters are drawn on the GPU
        model = train_gpt2.build("sparse", "cuda", layers=case["layers"], d=case["d"], heads=case["heads"], seq=case["seq"],
                                 vocab=case["vocab"], seed=seed)
    s["model"] = model
    s["weights"] = [p for p in model.parameters() if hasattr(p, "mask")]
    tok = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), device="cuda", generator=gen)
    s["x"], s["y"] = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    s["graph"] = None
    if case["graph"]:
        # the graph trainer's way: gradients in one flat buffer, kernels add into it; the mask is selected before
        params = list(model.parameters())
        flat = torch.zeros(sum((p.numel() + 3) // 4 * 4 for p in params), device="cuda")
        at = 0
        for p in params:
            p.grad = flat[at:at + p.numel()].view_as(p)
            at += (p.numel() + 3) // 4 * 4
        for mod in model.modules():
            if hasattr(mod, "accumulate_into_grad"):
                mod.accumulate_into_grad = True
        # the output head's share of the tied embedding's gradient goes to a buffer of its own
        model.head_grad = torch.zeros_like(model.wte.weight, dtype=torch.bfloat16)

        def step(reselect):
            flat.zero_()
            for p in s["weights"]:
                p.cnt, p.counter = 0, 0 if reselect else 1
            return _forward_backward(s)

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step(True)
            step(False)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            loss = step(False)
        s["graph"], s["flat"], s["loss"] = graph, flat, loss
    return s


def _forward_backward(s):
    with torch.autocast(device_type="cuda", dtype=torch.bfloat16):
        sparse.refresh_sparse_layers(s["model"])
        loss = s["model"](s["x"], s["y"])
    loss.backward()
    return loss.detach()


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def run(s):
    return _RUN[s["kind"]](s)


def _grads(s, y):
    layer, x = s["layer"], s["x"]
    out = {"y": y.detach(), "dx": x.grad, "dw": layer.weight.grad}
    if layer.bias is not None:
        out["db"] = layer.bias.grad
    return out


def _run_fst(s):
    layer, x = s["layer"], s["x"]
    x.grad = None
    layer.zero_grad(set_to_none=True)
    layer.weight.cnt = 0               # what the training loop does after an optimizer step
    with torch.autocast(device_type="cuda", dtype=s["dtype"]):
        y = layer(x)
    y.backward(s["dy"])
    return _grads(s, y)


def _run_fp8(s):
    layer, x = s["layer"], s["x"]
    x.grad = None
    layer.zero_grad(set_to_none=True)
    w8 = sparse.fp8.Fp8SparseWeight(layer.weight, s["mask"])
    y = sparse.fp8.sparse_linear_transpose_fp8.apply(x, layer.weight, w8, layer.bias)
    y.backward(s["dy"])
    return _grads(s, y)


def _run_linear(s):
    with torch.inference_mode():
        return F.linear(s["x"], s["w"], s["b"])


def _run_upkeep(s):
    for mod in s["model"]:
        w = mod.weight
        sparse.masked_add_(w.grad, w.data, w.mask, alpha=ALPHA)
        w.cnt = 0
    with torch.autocast(device_type="cuda", dtype=s["dtype"]):
        sparse.refresh_sparse_layers(s["model"])
    # every gradient, and the copies of three blocks: all of them would be four tensors a layer
    return s["flat"], [mod.weight.compressed for mod in list(s["model"])[-12:]]


def _run_select(s):
    if len(s["w"]) == 1:
        return sparse.select_and_compress(s["w"][0], dtype=_packed_dtype(s))
    return sparse.select_and_compress_many(s["w"], s["masks"], dtype=_packed_dtype(s), reselect=True)


def _packed_dtype(s):
    return torch.bfloat16 if s["dtype"] == torch.float32 else s["dtype"]


def _run_mvue(s):
    c = sparse.to_sparse_semi_structured(s["g"].t(), MVUE24=True, dtype=s["dtype"])
    return c.values(), c.indices()


def _run_sste(s):
    layer, x = s["layer"], s["x"]
    x.grad = None
    layer.zero_grad(set_to_none=True)
    with torch.autocast(device_type="cuda", dtype=s["dtype"]):
        y = layer(x)
    y.backward(s["dy"])
    return _grads(s, y)


def _run_gpt2(s):
    if s["graph"] is not None:
        s["graph"].replay()
        return {"loss": s["loss"], "grads": s["flat"], "head": s["model"].head_grad}
    model = s["model"]
    model.zero_grad(set_to_none=True)
    loss = _forward_backward(s)
    train_gpt2.masked_decay_(model, ALPHA)
    return {"loss": loss, "grads": [p.grad for p in model.parameters()]}


_RUN = {"fst": _run_fst, "fp8": _run_fp8, "linear": _run_linear, "upkeep": _run_upkeep, "select": _run_select, "mvue": _run_mvue,
        "sste": _run_sste, "gpt2": _run_gpt2}


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def work(case):
    """Each input read once, each output written once; a 2:4 product counts the operations on kept values only."""
    kind = case["kind"]
    compressed = 2 / 2 + 1 / 8         # bytes of a dense element in one 16-bit compressed copy
    if kind in ("fst", "fp8", "sste"):
        t, i, o = case["tokens"], case["in"], case["out"]
        # x, dx, y, dy in 16 bits; weight in, its gradient out in 32 bits; the mask
        io = 2 * 2 * t * (i + o) + 8 * i * o + (i * o if kind != "sste" else 0)
        products = 3 if kind != "sste" else 5      # three sparse products; S-STE: one sparse, two dense
        return {"bytes": io, "flops": products * t * i * o}
    if kind == "linear":
        t, i, o = case["tokens"], case["in"], case["out"]
        return {"bytes": 2 * t * (i + o) + compressed * i * o, "flops": t * i * o}
    if kind == "upkeep":
        n = 12 * case["d"] ** 2 * case["layers"]
        return {"bytes": n * (4 + 4 + 4 + 1 + 2 * compressed), "flops": n}
    if kind == "select":
        n = case["count"] * case["m"] * case["k"]
        return {"bytes": n * ((4 if case["dtype"] == "fp32" else 2) + 1 + 2 * compressed), "flops": 8 * n}
    if kind == "mvue":
        n = case["tokens"] * case["features"]
        return {"bytes": n * (2 + compressed), "flops": 10 * n}
    d, t = case["d"], case["batch"] * case["seq"]
    blocks, table = 12 * d * d * case["layers"], (case["vocab"] + case["seq"]) * d
    attention = case["layers"] * 3 * 2 * t * case["seq"] * d       # causal: half of the score matrix, both products
    return {"bytes": 8 * (blocks + table) + blocks + 16 * t, "flops": 3 * t * blocks + 6 * t * case["vocab"] * d + attention}


def tolerance(case):
    kind = case["kind"]
    if kind in ("upkeep", "select"):
        return "exact"                 # masks, kept values and metadata; the decay has two defined roundings
    if kind == "gpt2":
        return {"rel": 0.03}           # bf16 activations through every layer and back
    if kind == "fp8":
        return {"rel": 0.01}           # 16-bit results of e4m3 operands: values at a rounding boundary may fall either way
    if kind == "mvue":
        return {"rel": 0.01 if case["dtype"] == "bf16" else 0.002, "differ": 1e-4}     # draws on the boundary of an interval
    return {"rel": 0.01 if case["dtype"] == "bf16" else 0.002}
