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
