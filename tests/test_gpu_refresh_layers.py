"""The refresh of a model's sparse layers, native for plain layers: the state that each layer's own refresh leaves, for layers it takes and
layers it leaves to Python (own class, own mask type, copies wanted as tensors), in one model."""
import copy

import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"



def _model():
    import sparse

    class Sub(sparse.SparseLinearTranspose):
        pass

    class Wrapped(sparse.SparseLinearTranspose):
        materialize_sparse_tensors = True

    torch.manual_seed(3)
    layers = [sparse.SparseLinearTranspose(128, 256), sparse.SparseLinearTranspose(384, 128), Sub(128, 128), Wrapped(128, 256),
              sparse.SparseLinearTranspose(128, 128), sparse.SparseLinearTranspose(256, 128), sparse.SparseLinearTranspose(128, 192)]
    model = nn.ModuleList(layers).to(DEV)
    for i, layer in enumerate(layers):
        layer.weight.mask = sparse.mask_select(layer.weight.detach())[1] if i != 6 else layer.weight.mask.to(DEV)
        layer.weight.counter = 40 if i in (1, 4) else 3
    layers[4].weight.mask = layers[4].weight.mask.to(torch.uint8)       # not bool: converted by the Python path
    layers[5].weight.cnt = 1                                            # not due
    return model


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_state_is_that_of_each_layers_own_refresh(dtype):
    import sparse
    model = _model()
    own = copy.deepcopy(model)
    for a, b in zip(model, own):          # deepcopy keeps parameters, not the attributes on them
        for name in ("mode", "cnt", "counter", "freq", "step", "weight_grad", "weight_sparse", "weight_sparse_T", "compressed", "compressed_tc"):
            setattr(b.weight, name, getattr(a.weight, name))
        b.weight.mask = a.weight.mask.clone()
    with torch.autocast(device_type="cuda", dtype=dtype):
        assert sparse.refresh_sparse_layers(model) == 5
        assert sparse.refresh_sparse_layers(nn.ModuleList()) == 0
        for i, layer in enumerate(own):
            if i not in (5, 6):
                layer._ensure_compressed()
    for i, (a, b) in enumerate(zip(model, own)):
        w, v = a.weight, b.weight
        if i in (5, 6):
            assert w.compressed is None and not getattr(w, "refreshed", False)
            continue
        assert w.refreshed and w.mask.dtype == torch.bool and torch.equal(w.mask, v.mask.bool())
        for x, y in zip(w.compressed, v.compressed):
            assert x.dtype == y.dtype and x.stride() == y.stride() and torch.equal(x, y)
        assert w.compressed_tc[0] is w.compressed and w.compressed_tc[1:3] == v.compressed_tc[1:3]
        assert all(torch.equal(x, y) for x, y in zip(a._tc_copies(), b._tc_copies()))
        assert (w.weight_sparse is None) == (v.weight_sparse is None) == (i != 3)
    x = torch.randn(64, 128, device=DEV)
    with torch.autocast(device_type="cuda", dtype=dtype):
        assert torch.equal(model[0](x), own[0](x))
    assert not model[0].weight.refreshed
