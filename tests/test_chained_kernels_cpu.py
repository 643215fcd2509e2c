"""CPU check of what programmatic dependent launch asks of the kernels: a kernel may be resident while the one before it still writes, so
it waits before its first access and takes no load that promises read-only data, which the wait does not hold back.  One exception: the
masked decay asks L2 for its operands before the wait, which reads no value."""
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


def _before_the_wait():
    """Every kernel's code in front of its wait (a refusal that waits and returns taken out), with its parameters."""
    for name, src in _sources().items():
        for part in re.split(r"\b__global__\b", src)[1:]:
            kernel, params = re.search(r"(\w+_kernel)\s*\(([^{]*)\)", part).groups()
            body, depth, end = part[part.index("{"):], 0, 0
            for end, c in enumerate(body):
                depth += (c == "{") - (c == "}")
                if depth == 0:
                    break
            body = re.sub(r"\{\s*chain_enter\(\);[^{}]*return;\s*\}", "{}", body[:end])
            if "chain_enter();" in body:
                yield kernel, params, body[1:body.index("chain_enter();")]


def test_nothing_is_accessed_before_the_wait():
    gemm = _sources()["spmm_sm100.cu"]
    pointers = set()
    for struct in ("SpmmParams", "SumsParams"):
        text = re.search(r"struct %s \{(.*?)\n\};" % struct, gemm, re.S).group(1)
        for decl in text.split(";"):
            pointers.update(re.findall(r"\*\s*(?:const\s+)?(\w+)", decl))
    assert {"out", "bias", "status", "parts"} <= pointers
    seen = set()
    for kernel, params, head in _before_the_wait():
        if kernel == "masked_add_kernel":
            rest = re.sub(r"prefetch_l2\([^;]*\);", "", head)
            assert "prefetch_l2(" in head and not re.search(r"\b(grad|p|mask)\b", re.sub(r"\bahead\.\w+", "", rest)), rest
        elif kernel.startswith("spmm_"):        # barriers and tensor memory are set up from sizes alone
            used = set(re.findall(r"\b(?:P|sums)\.(\w+)", head))
            assert not used & pointers and not re.search(r"\bmap_\w+|\bsums\b|prefetch_l2|atomic|ld_global|tma_load", head), (kernel, used)
        else:
            assert not head.strip(), (kernel, head)
        seen.add(kernel)
    assert len(seen) >= 25 and {"masked_add_kernel", "spmm_pair_kernel", "spmm_pair_acc_kernel"} <= seen
