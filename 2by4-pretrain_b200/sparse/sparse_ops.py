"""Autograd linear layers of the 2:4 training recipes.

``SparseLinearTranspose`` / ``sparse_linear_transpose`` are the FST layer the reference only lists in
its README (README.md:125-200 of the reference): forward Y = X W_s^T with the weight compressed under
a transposable 2:4 mask, backward dX = dY W_s through the separately compressed W^T, and
dW = MVUE24(dY^T) X with the gradient compressed on the fly.  ``MyLinear`` / ``SparseLinear`` are the
older dense-GEMM variants of sparse/sparse_ops.py:8-87 of the reference.
"""
import torch
import torch.nn.functional as F
from torch import autograd, nn
from torch.amp import custom_fwd, custom_bwd

from . import _ext
from ._ext import host as _host
from .semi_structured import SparseSemiStructuredTensor, to_sparse_semi_structured
from .transposable_semi_structured import TransposableSparse
from .triton_ops import MVUE24_approx_triton
from .spmm import sparse_linear as _spmm, sparse_linear_mlp as _spmm_mlp, register_tc_metadata, tc_metadata


def _dense_linear(name, dx_weight, doc):
    """Builds the autograd function of a dense linear layer, y = x W^T (+ b), whose input gradient is
    dY @ ``dx_weight(W)``.  The two dense layers of the reference differ only in that factor
    (sparse/sparse_ops.py:8-87 of the reference): W itself, or a fresh MVUE 2:4 estimate of it."""

    def forward(ctx, input, weight, bias):
        ctx.save_for_backward(input, weight)
        ctx.lead = input.shape[:-1]
        y = input.reshape(-1, input.shape[-1]).mm(weight.t()).view(*ctx.lead, weight.shape[0])
        return y if bias is None else y + bias

    def backward(ctx, grad_output):
        input, weight = ctx.saved_tensors
        want_x, want_w, want_b = ctx.needs_input_grad
        g = grad_output.reshape(-1, weight.shape[0])
        gx = g.mm(dx_weight(weight)).view(*ctx.lead, weight.shape[1]) if want_x else None
        gw = g.t().mm(input.reshape(-1, weight.shape[1])) if want_w else None
        gb = g.sum(0) if want_b else None
        return gx, gw, gb

    return type(name, (autograd.Function,), {
        "__doc__": doc,
        "forward": staticmethod(custom_fwd(device_type='cuda')(forward)),
        "backward": staticmethod(custom_bwd(device_type='cuda')(backward)),
    })


my_linear = _dense_linear("my_linear", lambda w: w, "Plain dense linear layer as a custom autograd function.")
sparse_linear = _dense_linear(
    "sparse_linear", lambda w: MVUE24_approx_triton(w.t()).t(),
    "Dense GEMMs; the input gradient multiplies dY with an MVUE 2:4 estimate of the weight, drawn along its "
    "output-feature axis on every backward pass.")


class MyLinear(nn.Linear):
    def forward(self, x):
        return my_linear.apply(x, self.weight, self.bias)


class SparseLinear(nn.Linear):
    def forward(self, x):
        return sparse_linear.apply(x, self.weight, self.bias)


class sparse_linear_transpose(autograd.Function):
    """README.md:169-200 of the reference.  Three sparse GEMMs per layer and micro-step."""

    @staticmethod
    @custom_fwd(device_type='cuda', cast_inputs=torch.float16)
    def forward(ctx, input, weight, weight_sparse, weight_sparse_T, bias):
        ctx.save_for_backward(input, weight_sparse_T, bias)
        ctx.shape = input.shape
        input = input.reshape(-1, input.shape[-1])
        # same product as torch.mm(input, weight_sparse.t()); calling the GEMM wrapper directly skips the
        # Python-level tensor-subclass dispatch; the bias is added in the GEMM epilogue (one rounding instead of
        # the listing's two)
        b = None if bias is None else bias.to(input.dtype)
        output = _spmm(input, weight_sparse.sparse_tensor_cutlass, weight_sparse.meta_tensor_cutlass, bias=b)
        return output.view(*ctx.shape[:-1], -1)

    @staticmethod
    @custom_bwd(device_type='cuda')
    def backward(ctx, grad_output):
        input, weight_T, bias = ctx.saved_tensors
        grad_input = grad_weight = grad_bias = None
        if grad_output.dim() == 3 and grad_output.stride() == (0, 0, 0):
            grad_output = torch.ones_like(grad_output, device=grad_output.device, dtype=grad_output.dtype)
        grad_output = grad_output.reshape(-1, grad_output.shape[-1])
        if ctx.needs_input_grad[0]:
            # torch.mm(grad_output, weight_T.t())
            grad_input = _spmm(grad_output, weight_T.sparse_tensor_cutlass, weight_T.meta_tensor_cutlass).view(ctx.shape)
        if ctx.needs_input_grad[1]:
            input = input.reshape(-1, input.shape[-1])
            # torch.mm(to_sparse_semi_structured(grad_output.t(), MVUE24=True), input)
            gs = to_sparse_semi_structured(grad_output.t(), MVUE24=True, dtype=grad_output.dtype)
            grad_weight = _spmm(input.t(), gs.sparse_tensor_cutlass, gs.meta_tensor_cutlass).t()
        if ctx.needs_input_grad[4]:
            grad_bias = grad_output.sum(0)
        return grad_input, grad_weight, None, None, grad_bias


def _mm_f32(a, b, acc=None):
    """a @ b (16-bit operands) with a float32 result; added into ``acc`` in the GEMM's epilogue when given."""
    try:
        if acc is not None:
            return torch.addmm(acc, a, b, out_dtype=torch.float32, out=acc)
        return torch.mm(a, b, out_dtype=torch.float32)
    except (TypeError, RuntimeError):             # a torch without the out_dtype argument on this overload
        r = torch.mm(a, b).float()
        return r if acc is None else acc.add_(r)


def _dense_weight_grads(g, x, weight, bias, into_grad, need_w, need_b):
    """The exact dW = g^T x as a dense GEMM with float32 output (the option ``weight_grad = "dense"`` of the layer).
    Same contract as the native ``fst_weight_grads``: (grad_weight,
    grad_bias), each None where it went straight into a ``.grad`` buffer."""
    grad_weight = grad_bias = None
    into = into_grad and weight.grad is not None and weight.grad.dtype == torch.float32 and weight.grad.is_contiguous()
    if need_w:
        if into:
            _mm_f32(g.t(), x, weight.grad)
        else:
            gw = _mm_f32(g.t(), x)
            grad_weight = gw if weight.dtype == torch.float32 else gw.to(weight.dtype)
    if bias is not None and need_b:
        if into and need_w and bias.grad is not None and bias.grad.dtype == torch.float32:
            bias.grad.add_(g.sum(0, dtype=torch.float32))
        else:
            grad_bias = g.sum(0)
    return grad_weight, grad_bias


class _fst_mlp(autograd.Function):
    """Transformer MLP, proj(gelu(fc(x))), on two FST layers with the element-wise work folded into the GEMM epilogues:
    the up-projection writes both the pre-activation h and gelu(h); in the backward pass the down-projection's input
    gradient is multiplied by gelu'(h) in its epilogue, so the gradient of h is written directly.  Saves four passes
    over the (tokens, 4 d) activations per layer and step (GELU forward, its backward, and the tensors between them).
    ``fc`` / ``proj`` are (weight, bias, (pw, mw, pt, mt), into_grad)."""

    @staticmethod
    def forward(ctx, input, w_fc, b_fc, w_proj, b_proj, comp_fc, comp_proj, into_grad):
        pw1, mw1, pt1, mt1 = comp_fc
        pw2, mw2, pt2, mt2 = comp_proj
        x = input.reshape(-1, input.shape[-1])
        if x.dtype != pw1.dtype:
            x = x.to(pw1.dtype)
        act, pre = _spmm_mlp(x, pw1, mw1, bias=b_fc, epilogue="gelu")
        out = _spmm_mlp(act, pw2, mw2, bias=b_proj)
        ctx.save_for_backward(x, act, pre, pt1, mt1, pt2, mt2)
        ctx.shape = input.shape
        ctx.params = (w_fc, b_fc, w_proj, b_proj, into_grad)
        return out.view(*input.shape[:-1], -1)

    @staticmethod
    def backward(ctx, grad_output):
        x, act, pre, pt1, mt1, pt2, mt2 = ctx.saved_tensors
        w_fc, b_fc, w_proj, b_proj, into_grad = ctx.params
        g = grad_output.reshape(-1, grad_output.shape[-1])
        if g.dtype != pt2.dtype:
            g = g.to(pt2.dtype)
        g = g.contiguous()
        need = ctx.needs_input_grad
        d_pre = _spmm_mlp(g, pt2, mt2, epilogue="dgelu", aux=pre)           # gradient of fc's output, (tokens, 4 d)
        gw2, gb2 = _ext.host.fst_weight_grads(g, act, w_proj, b_proj, into_grad, need[3], need[4])
        grad_input = _spmm(d_pre, pt1, mt1).view(ctx.shape) if need[0] else None
        gw1, gb1 = _ext.host.fst_weight_grads(d_pre, x, w_fc, b_fc, into_grad, need[1], need[2])
        return grad_input, gw1, gb1, gw2, gb2, None, None, None


def fst_mlp(x, fc, proj):
    """proj(gelu(fc(x), approximate="tanh")) for two ``SparseLinearTranspose`` layers.  Runs the fused epilogues when
    both layers are in sparse mode, their compressed copies are 16-bit and their shapes allow it; otherwise exactly
    the three separate calls.  Counters of both layers advance as in their own ``forward``."""
    w1, w2 = fc.weight, proj.weight
    ok = w1.mode == 'sparse' and w2.mode == 'sparse' and w1.is_cuda and w1.shape[0] % 256 == 0 and w2.shape[0] % 256 == 0 \
        and fc.bias is not None and proj.bias is not None
    if not ok:
        return proj(F.gelu(fc(x), approximate="tanh"))
    for layer in (fc, proj):
        layer._ensure_compressed()
        _, mw, _, mt = layer.weight.compressed
        tcw, tct = layer._tc_copies()
        register_tc_metadata(mw, tcw)
        register_tc_metadata(mt, tct)
    y = _fst_mlp.apply(x, w1, fc.bias, w2, proj.bias, w1.compressed, w2.compressed,
                       fc.accumulate_into_grad and proj.accumulate_into_grad)
    fc._advance()
    proj._advance()
    return y


class SparseLinearTranspose(nn.Linear):
    """Drop-in for ``nn.Linear`` that trains with 2:4 sparse GEMMs (FST).

    State lives on ``self.weight`` as in the reference listing: ``freq`` (mask refresh period in
    optimizer steps), ``cnt`` (micro-steps since the last optimizer step; the training loop resets it
    to 0 after each optimizer step), ``counter`` (optimizer steps), ``step`` (forward calls),
    ``mask`` (bool, transposable 2:4), ``weight_sparse`` / ``weight_sparse_T`` and ``mode``
    ('sparse' or 'dense').  When both the mask and the compressed copies are due, one fused kernel
    produces all three from a single read of the weight.

    ``materialize_sparse_tensors`` (class attribute, default False): when True the compressed copies are
    also wrapped as ``SparseSemiStructuredTensor`` objects in ``weight.weight_sparse`` /
    ``weight.weight_sparse_T`` after every refresh, as in the listing; the layer itself works on the raw
    buffers (``weight.compressed`` = (packed_w, meta_w, packed_t, meta_t)) to keep the host cost low.
    """

    materialize_sparse_tensors = False
    # How the weight gradient is formed (``weight.weight_grad``, set per layer from this class attribute).  "mvue": the
    # reference recipe, dW = MVUE24(dY^T) X on the sparse tensor cores (README.md:190-192 of the reference).  "dense":
    # the exact dW = dY^T X as a dense GEMM: no estimator noise, and on B200 the faster of the two (the MVUE pass plus
    # the sparse GEMM take longer than the dense GEMM they replace).
    weight_grad = "mvue"
    # True: the weight-gradient GEMM adds straight into an existing fp32 ``weight.grad`` (a trainer that owns flat
    # gradient buffers and needs no autograd hook on the weight, e.g. the graph-replayed one); False: autograd gets it
    accumulate_into_grad = False

    def __init__(self, in_features: int, out_features: int, bias: bool = True, func=lambda step: 'dense', **kwargs):
        super().__init__(in_features, out_features, bias=bias, **kwargs)
        self.weight.freq = 40  # update freq

        self.weight.cnt = 0  # how many steps after an optim step
        self.weight.counter = 0  # how many optim steps
        self.weight.step = 0  # total training step

        self.weight.mask = torch.ones_like(self.weight, dtype=torch.bool)
        self.weight.weight_sparse = None
        self.weight.weight_sparse_T = None
        self.weight.compressed = None
        self.weight.compressed_tc = None
        self.weight.mode = 'sparse'
        self.weight.weight_grad = self.weight_grad
        self.func = func

        self.transposable_sparse = TransposableSparse(abs=True)
        SparseSemiStructuredTensor._FORCE_CUTLASS = True  # kept for parity with the reference; has no effect

    def _refresh(self, reselect: bool):
        w = self.weight
        # a reselected mask overwrites the existing buffer, so w.mask keeps one address for the whole run
        reuse = w.mask if (reselect and w.mask.is_cuda and w.mask.is_contiguous() and w.mask.dtype == torch.bool) else None
        # compressed copies in the autocast dtype when it is bf16 (no cast passes over the activations);
        # fp16 otherwise, like the reference layer (custom_fwd(cast_inputs=torch.float16))
        dtype = torch.float16
        if torch.is_autocast_enabled('cuda') and torch.get_autocast_dtype('cuda') == torch.bfloat16:
            dtype = torch.bfloat16
        self._take(_ext.host.select_compress(w.detach(), None if reselect else w.mask, dtype, reuse), dtype)

    def _take(self, copies, dtype, w=None):
        """Install (mask, packed_w, meta_w, packed_t, meta_t, tc_w, tc_t) as the compressed copies of the weight."""
        if w is None:
            w = self.weight
        w.mask, pw, mw, pt, mt, tcw, tct = copies
        w.compressed = (pw, mw, pt, mt)
        # the metadata in tensor-core order, good for exactly these metadata tensors as they are now
        w.compressed_tc = (w.compressed, mw._version, mt._version, (tcw, tct)) if tcw is not None else None
        if not self.materialize_sparse_tensors:
            w.weight_sparse = w.weight_sparse_T = None
            return
        if tcw is not None:
            register_tc_metadata(mw, tcw)
            register_tc_metadata(mt, tct)
        out_f, in_f = w.shape
        w.weight_sparse = SparseSemiStructuredTensor(
            None, original_shape=torch.Size([out_f, in_f]), sparse_tensor_cutlass=pw, meta_tensor_cutlass=mw,
            dtype=dtype)
        w.weight_sparse_T = SparseSemiStructuredTensor(
            None, original_shape=torch.Size([in_f, out_f]), sparse_tensor_cutlass=pt, meta_tensor_cutlass=mt,
            dtype=dtype)

    def _tc_copies(self):
        """Both metadata copies in tensor-core order: what the compressing kernel wrote, or converted when it could not,
        when the copies were replaced by hand or when their metadata was written to since."""
        w = self.weight
        pw, mw, pt, mt = w.compressed
        held = w.compressed_tc
        if held is not None and held[0] is w.compressed and held[1] == mw._version and held[2] == mt._version:
            return held[3]
        return tc_metadata(mw, pw.shape[0], 2 * pw.shape[1]), tc_metadata(mt, pt.shape[0], 2 * pt.shape[1])

    def _ensure_compressed(self):
        """Rebuild the mask and / or the compressed copies when this forward pass is due to (first micro-step after an
        optimizer step; every ``freq`` optimizer steps with a new mask)."""
        w = self.weight
        if w.mask.device != w.device:
            w.mask = w.mask.to(device=w.device)
        if w.cnt == 0:
            if getattr(w, 'refreshed', False):
                w.refreshed = False      # refresh_sparse_layers has just rebuilt the copies of this step
            else:
                self._refresh(reselect=(w.counter % w.freq == 0))
        elif w.compressed is None:   # state restored in the middle of an accumulation window
            self._refresh(reselect=False)

    def _advance(self):
        w = self.weight
        if self.training:
            if w.cnt == 0:
                w.counter += 1
            w.step += 1
            w.cnt += 1

    def forward(self, x):
        w = self.weight
        if w.mode == 'dense':
            x = F.linear(x, w, self.bias)
        else:
            y = _host.fst_forward(self, x)   # all of what follows and _advance for a plain layer; None where anything is not plain
            if y is not None:
                return y
            self._ensure_compressed()
            x = _ext.call_layer(_ext.host.fst_linear, x, w, self.bias, w.compressed, self._tc_copies(), self.accumulate_into_grad)
        self._advance()
        return x


def _modules(model: nn.Module):
    """``list(model.modules())``, walked by native code where no module has a walk of its own."""
    return _host.modules(model) or list(model.modules())


def refresh_sparse_layers(model: nn.Module) -> int:
    """What every ``SparseLinearTranspose`` of ``model`` would do at the start of its next forward pass when a
    refresh is due (``cnt`` == 0): reselect the mask if ``counter % freq == 0`` and rebuild the compressed copies
    of W and W^T; done here for all those layers with one kernel launch per 48 weights instead of one per layer.
    Call it right before the forward pass, under the same autocast context.  Layers whose shapes are not
    multiples of 128 are left to refresh themselves.  Returns the number of layers refreshed."""
    dtype = torch.float16
    if torch.is_autocast_enabled('cuda') and torch.get_autocast_dtype('cuda') == torch.bfloat16:
        dtype = torch.bfloat16
    layers = [mod for mod in _modules(model) if isinstance(mod, SparseLinearTranspose)]
    done, layers = _host.refresh_layers(layers, dtype, SparseLinearTranspose)
    groups = {}
    for mod in layers:                       # those with a class, weight, mask or counters of their own
        w = mod.weight                       # the attribute: a subclass or a parametrization may answer for the parameter
        if w.mode != 'sparse' or w.cnt != 0 or not w.is_cuda:
            continue
        shape = w.shape                      # rows decide first: a trainer's flat shard of odd size is passed over too
        if shape[0] % 128 or shape[1] % 128:
            continue
        mask, device = w.mask, w.device
        if mask.device != device:
            w.mask = mask = mask.to(device=device)
        if mask.dtype != torch.bool or not mask.is_contiguous():
            w.mask = mask = mask.to(torch.bool).contiguous()
        key = (w.counter % w.freq == 0, w.dtype, device)
        group = groups.get(key)
        if group is None:
            group = groups[key] = ([], [], [])
        group[0].append(mod)
        group[1].append(w)
        group[2].append(mask)
    for (reselect, _, _), (mods, weights, masks) in groups.items():
        res = _ext.host.select_compress_many(weights, masks, dtype, reselect)
        for mod, w, copies in zip(mods, weights, res):
            mod._take(copies, dtype, w)
            w.refreshed = True
            done += 1
    return done


def sparse_state(model: nn.Module) -> dict:
    """Training state the FST layers keep outside ``state_dict()``: per sparse weight its mask, counters,
    refresh period and mode, keyed by parameter name.  Save it next to the checkpoint."""
    out = {}
    for name, p in model.named_parameters():
        if hasattr(p, 'mask'):
            out[name] = {'mask': p.mask.detach().cpu(), 'cnt': p.cnt, 'counter': p.counter, 'step': p.step,
                         'freq': p.freq, 'mode': p.mode}
    return out


def load_sparse_state(model: nn.Module, state: dict) -> None:
    """Inverse of ``sparse_state``; call after ``load_state_dict``.  The compressed copies are dropped,
    so the next forward pass of a layer in the middle of an accumulation window (``cnt`` != 0)
    rebuilds them from the restored weight under the restored mask."""
    params = dict(model.named_parameters())
    for name, st in state.items():
        if name not in params or not hasattr(params[name], 'mask'):
            raise RuntimeError(f"load_sparse_state: {name} is not a sparse weight of this model")
        p = params[name]
        if tuple(st['mask'].shape) != tuple(p.shape):
            raise RuntimeError(f"load_sparse_state: mask of {name} has shape {tuple(st['mask'].shape)}, expected {tuple(p.shape)}")
        p.mask = st['mask'].to(device=p.device, dtype=torch.bool)
        p.cnt, p.counter, p.step, p.freq, p.mode = st['cnt'], st['counter'], st['step'], st['freq'], st['mode']
        p.compressed = p.compressed_tc = None
        p.weight_sparse = p.weight_sparse_T = None
