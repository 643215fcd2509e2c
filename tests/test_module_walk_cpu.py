"""The walk over a model's modules that the batched refresh of sparse layers makes: what ``modules()`` yields, in its order."""
from types import SimpleNamespace

import pytest
import torch
from torch import nn


def _nested():
    shared = nn.Linear(4, 4)
    model = nn.Sequential(nn.ModuleList([shared, nn.Sequential(nn.ReLU(), shared)]), nn.ModuleDict({"a": nn.Identity(), "b": shared}), shared)
    model.register_module("absent", None)
    model[0][1].back = shared
    return model


class _Narrow(nn.Module):
    def __init__(self):
        super().__init__()
        self.a, self.b = nn.Linear(2, 2), nn.Linear(2, 2)

    def modules(self):
        yield self.a


class _Hides(nn.Module):
    """A module that shows one of its two children to a walk."""
    def __init__(self):
        super().__init__()
        self.shown, self.hidden = nn.Linear(2, 2), nn.Linear(2, 2)

    def named_modules(self, memo=None, prefix="", remove_duplicate=True):
        yield prefix, self
        yield prefix + ".shown", self.shown


def _own(name, value):
    """A module with ``name`` of its own on the instance, not in the class."""
    model = nn.Sequential(nn.Linear(2, 2), nn.ReLU())
    model.__dict__[name] = lambda *a, **k: iter(value(model))
    return model


def test_same_modules_in_the_same_order():
    from sparse.sparse_ops import _modules
    own_modules, own_named = _own("modules", lambda m: [m[0]]), _own("named_modules", lambda m: [("", m), ("1", m[1])])
    for model in (nn.Linear(2, 2), _nested(), _Narrow(), nn.ModuleList(), _Hides(), nn.Sequential(nn.ReLU(), nn.ModuleList([_Hides()])),
                  nn.Sequential(_Narrow(), nn.ReLU()), own_modules, own_named, nn.Sequential(own_modules, own_named)):
        assert [id(m) for m in _modules(model)] == [id(m) for m in model.modules()]


def test_parametrized_weight_is_found():
    """A weight that is no plain parameter is read as an attribute; on the CPU nothing is refreshed."""
    import sparse
    layer = sparse.SparseLinearTranspose(128, 128)
    w = layer.weight
    del layer._parameters["weight"]
    layer.__dict__["weight"] = w
    assert sparse.refresh_sparse_layers(nn.ModuleList([layer])) == 0
    assert torch.equal(layer.weight.mask, torch.ones(128, 128, dtype=torch.bool))


def _gpu_weight(shape, counter=1):
    """What the refresh reads of a weight on the GPU."""
    return SimpleNamespace(mode="sparse", cnt=0, counter=counter, freq=40, is_cuda=True, shape=torch.Size(shape), dtype=torch.float32,
                           device=torch.device("cpu"), mask=torch.ones(shape, dtype=torch.bool))


@pytest.fixture
def refreshed(monkeypatch):
    """The weights that reach the native call, by the refresh's option ``reselect``."""
    import sparse.sparse_ops as ops
    calls = {}

    def native(weights, masks, dtype, reselect):
        calls[reselect] = list(weights)
        return [(m, *[torch.empty(0)] * 4, None, None) for m in masks]

    monkeypatch.setattr(ops, "_ext", SimpleNamespace(host=SimpleNamespace(select_compress_many=native)))
    return calls


def test_refresh_takes_the_weight_that_the_layer_uses(refreshed):
    """A plain parameter, an attribute in the place of a parameter that was taken out (what a parametrization leaves), one that
    hides the parameter, and a subclass that answers itself."""
    import sparse

    class Viewed(sparse.SparseLinearTranspose):
        def __getattribute__(self, name):
            if name == "weight" and "seen" in object.__getattribute__(self, "__dict__"):
                return self.seen
            return super().__getattribute__(name)

    plain, replaced, hidden = (sparse.SparseLinearTranspose(128, 128) for _ in range(3))
    viewed = Viewed(128, 128)
    del replaced._parameters["weight"]
    weights = [_gpu_weight((128, 256), c) for c in (1, 40, 1)]
    replaced.__dict__["weight"], hidden.__dict__["weight"], viewed.__dict__["seen"] = weights
    assert sparse.refresh_sparse_layers(nn.ModuleList([plain, replaced, hidden, viewed])) == 3        # `plain` is on the CPU
    assert [id(w) for w in refreshed[False]] == [id(weights[0]), id(weights[2])] and refreshed[True] == [weights[1]]
    assert all(w.refreshed for w in weights) and torch.equal(plain.weight.mask, torch.ones(128, 128, dtype=torch.bool))


@pytest.mark.parametrize("shape", [(100,), (130, 128), (128, 130), (2, 128, 128)])
def test_refresh_leaves_other_shapes_alone(refreshed, shape):
    """Sizes off 128, and shards that a trainer keeps flat: left to the layer itself."""
    import sparse
    layer = sparse.SparseLinearTranspose(128, 128)
    layer.__dict__["weight"] = _gpu_weight(shape)
    assert sparse.refresh_sparse_layers(layer) == 0 and not refreshed
