"""CPU check of what programmatic dependent launch asks of the kernels: a kernel may be resident while the one before it still writes, so
it waits before its first access and takes no load that promises read-only data, which the wait does not hold back."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2by4-pretrain_b200", "csrc")


def _code(path):
    src = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", src)


def _sources():
    return {os.path.basename(p): _code(p) for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def test_no_load_promises_read_only_data():
    found = [(name, w) for name, src in _sources().items() for w in ("__ldg", "ld.global.nc", ".nc.", "__restrict__", "__ldcs") if w in src]
    assert not found


def test_every_kernel_waits_for_the_one_before():
    seen = 0
    for name, src in _sources().items():
        for part in re.split(r"\b__global__\b", src)[1:]:
            kernel = re.search(r"(\w+_kernel)\s*\(", part).group(1)
            body = part[part.index("{"):]
            if kernel != "wait_selftest_kernel":         # launched by itself, in plain stream order
                assert "chain_enter();" in body, (name, kernel)
            seen += 1
    assert seen >= 25
