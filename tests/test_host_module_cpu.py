"""CPU test of the native host module: it loads without a GPU and draws MVUE seeds from Python's generator exactly as
``random.randint(0, 2**31 - 1)`` does (users seed runs through ``random``)."""
import random


def test_native_seed_equals_randint_stream():
    from sparse import _ext
    random.seed(7)
    want = [random.randint(0, 2 ** 31 - 1) for _ in range(500)]
    after = random.getstate()
    random.seed(7)
    assert [_ext.host.python_seed() for _ in range(500)] == want
    assert random.getstate() == after


def test_check_status_sees_every_device(monkeypatch):
    """A wait that gave up is reported whichever device it ran on; asking for one device looks at that one only."""
    from types import SimpleNamespace

    import pytest
    import torch
    from sparse import _ext, spmm
    words = {0: torch.zeros(1, dtype=torch.int32), 1: torch.tensor([2], dtype=torch.int32)}
    monkeypatch.setattr(_ext, "host", SimpleNamespace(status_words=lambda: words, status_word=lambda i: words[i]))
    spmm.check_status(torch.device("cuda", 0))
    with pytest.raises(RuntimeError, match="role code 2.*cuda:1"):
        spmm.check_status()
    assert int(words[1]) == 0                  # reported once
    spmm.check_status()
    words[1].fill_(4)
    with pytest.raises(RuntimeError, match="role code 4"):
        spmm.check_status(device=torch.device("cuda", 1))


def test_package_under_another_name():
    """The package may be vendored: the dense weight-gradient option finds its Python part relative to the package."""
    import os
    import subprocess
    import sys
    root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2by4-pretrain_b200", "sparse")
    code = f"""
import importlib.util, sys
spec = importlib.util.spec_from_file_location("vendored24", {root!r} + "/__init__.py", submodule_search_locations=[{root!r}])
sys.modules["vendored24"] = mod = importlib.util.module_from_spec(spec)
spec.loader.exec_module(mod)
import torch
from vendored24 import _ext
w = torch.nn.Parameter(torch.zeros(4, 8))
w.weight_grad = "dense"
g, x = torch.randn(16, 4, dtype=torch.bfloat16), torch.randn(16, 8, dtype=torch.bfloat16)
gw, gb = _ext.host.fst_weight_grads(g, x, w, w[:, 0], False, True, True)
assert gw.dtype == torch.float32 and (gw - g.float().t() @ x.float()).abs().max() < 0.1 and gb.shape == (4,)
assert "sparse" not in sys.modules
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd="/")
