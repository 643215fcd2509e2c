"""CPU check, by reading the sources, of what the library keeps between calls: each device's answers (an SM count, an attribute that was
set) are atomic, a thread's own or under a lock, since entry points are called from several threads."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2by4-pretrain_b200", "csrc")


def test_kept_answers_are_atomic_or_locked():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"^\s+static (?!const|__device__|inline|__global__)([^;(]*?)(?:\{[^;]*|= [^;]*)?;", src, flags=re.M):
            after = src[m.start():m.start() + 200]
            found.append((os.path.basename(path), m.group(1).strip(), "std::atomic" in m.group(1) or "thread_local" in m.group(1) or "static std::mutex" in after))
    assert len(found) >= 9 and all(ok for _, _, ok in found), found
