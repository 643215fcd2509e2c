"""CPU check, by reading the sources, of what happens to the CUDA runtime's error when a call of it fails: it is taken out of the runtime on
the spot, so that the next entry point, whose own launch succeeds, does not report it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2by4-pretrain_b200", "csrc")


def _lines():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = re.sub(r"//[^\n]*", "", open(path).read()).replace("\\\n", "\n")
        yield os.path.basename(path), src


def test_failed_calls_leave_nothing_behind():
    found = 0
    for name, src in _lines():
        for m in re.finditer(r"!= cudaSuccess\b([^;]*);", src):
            found += 1
            assert "runtime_error()" in m.group(1), (name, m.group(0))
    assert found >= 15


def test_the_error_code_comes_from_one_place():
    """Anything else that returns it is the driver API, which keeps no error, or the two functions that take the error out."""
    spots = [(name, line.strip()) for name, src in _lines() for line in src.splitlines() if "SP24_ERR_CUDA" in line]
    allowed = {("abi_core.cu", "return SP24_ERR_CUDA;"), ("abi_core.cu", 'case SP24_ERR_CUDA: return "the CUDA runtime reported an error";'),
               ("spmm_sm100.cu", "return r == CUDA_SUCCESS ? SP24_OK : SP24_ERR_CUDA;")}
    assert set(spots) == allowed and len([s for s in spots if s[0] == "abi_core.cu"]) == 3
