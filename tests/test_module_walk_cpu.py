"""The walk over a model's modules that the batched refresh of sparse layers makes: what ``modules()`` yields, in its order."""
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
