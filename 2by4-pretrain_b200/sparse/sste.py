"""S-STE training layer: continuous 2:4 pruning by soft thresholding with a frozen per-tensor scale.

The reference lists these classes only in its README (README.md:233-267 of the reference); here they are
real.  ``SoftThreshold`` prunes with ``soft_threshold24_triton`` and passes the gradient straight
through; ``SoftThresholdLinear`` is the ``nn.Linear`` replacement (the README calls it ``SparseLinear``,
a name the package already uses for the MVUE layer of sparse/sparse_ops.py:86-87).  The scale is folded
into the pruning kernel's store, and with ``spmm=True`` the forward GEMM runs on the 2:4 sparse tensor
cores from a compressed copy of the pruned weight.
"""
import torch
import torch.nn.functional as F
from torch import autograd, nn

from . import _ext
from .spmm import register_tc_metadata
from .triton_ops import soft_threshold24_triton


class SoftThreshold(autograd.Function):
    """weight -> soft_threshold24(weight) * scale; d/dweight = identity (straight-through)."""

    @staticmethod
    def forward(ctx, weight, scale):
        s = float(scale) if not isinstance(scale, float) else scale
        sparse, _ = soft_threshold24_triton(weight.detach(), scale=s)
        return sparse

    @staticmethod
    def backward(ctx, grad_output):
        return grad_output, None


def soft_threshold24_compress(weight: torch.Tensor, scale=None, dtype: torch.dtype = torch.float16):
    """One pass over ``weight``: S-STE soft threshold (times ``scale`` if given) and 2:4 compression to ``dtype``.
    Returns (packed (m, k/2), reordered metadata (m, k/16) int16), the operands of ``sparse_linear``; the
    tensor-core order of the metadata is written by the same kernel when m is a multiple of 128.  Bit-identical to
    ``soft_threshold24_triton(weight, scale=scale)``, a cast and ``to_sparse_semi_structured(..., mask=mask)``."""
    packed, meta, e_tc = _ext.host.soft_threshold_compress(weight.detach(), None if scale is None else float(scale), dtype)
    if e_tc is not None:
        register_tc_metadata(meta, e_tc)
    return packed, meta


class SoftThresholdLinear(nn.Linear):
    """``nn.Linear`` whose weight passes through the S-STE pruning function on every forward.

    ``init_scale()`` freezes ``scale = <w, S(w)> / <S(w), S(w)>`` (S = soft threshold) once, before
    training, as in the README listing; the value is kept as a buffer (checkpointed) and as a Python
    float so that the forward pass needs no device-to-host read.
    """

    def __init__(self, in_features: int, out_features: int, bias: bool = True, device=None, dtype=None,
                 spmm: bool = False, spmm_dtype: torch.dtype = torch.float16):
        super().__init__(in_features, out_features, bias=bias, device=device, dtype=dtype)
        self.register_buffer('scale', torch.tensor(0.))
        self._scale_value = None
        self.spmm = spmm
        self.spmm_dtype = spmm_dtype

    def _scale(self) -> float:
        if self._scale_value is None:      # e.g. after load_state_dict
            self._scale_value = float(self.scale)
        return self._scale_value

    def _load_from_state_dict(self, *args, **kwargs):
        super()._load_from_state_dict(*args, **kwargs)
        self._scale_value = None

    def get_sparse_weights(self):
        return SoftThreshold.apply(self.weight, self._scale())

    @torch.no_grad()
    def init_scale(self):
        weight = self.weight.detach()
        weight_sparse, _ = soft_threshold24_triton(weight)
        w, ws = weight.flatten().float(), weight_sparse.flatten().float()
        value = torch.dot(w, ws) / torch.dot(ws, ws)
        self.scale.copy_(value)
        self._scale_value = float(value)
        self.weight.scale = self.scale

    def forward(self, x):
        if self.spmm:
            # one kernel soft-thresholds, scales and compresses the weight; both gradients are dense GEMMs (README.md:233-267
            # of the reference): the mask is 2:4 along the rows of W only, and dW is the straight-through dY^T X
            return _ext.call_layer(_ext.host.soft_threshold_linear, x, self.weight, self.bias, self._scale(), self.spmm_dtype)
        return F.linear(x, self.get_sparse_weights(), self.bias)
