"""CPU check of the metadata that each K step of the sparse GEMM stages: every load inside the buffer of sp24_meta_tc_bytes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include <cstdio>
#include "meta_steps.cuh"
int main() {
    // k_atoms atoms per 128-row block, 256 columns (two atoms) a step, as the kernel walks them
    for (int64_t k_atoms = 1; k_atoms <= 65; ++k_atoms) {
        const int64_t steps = (k_atoms * 128 + 255) / 256;
        for (int64_t s = 0; s < steps; ++s) {
            const sp24::MetaAtoms a = sp24::meta_atoms_of_step(s, k_atoms);
            std::printf("%lld %lld %lld %lld\n", (long long)k_atoms, (long long)s, (long long)a.first, (long long)a.second);
        }
    }
}
"""


def test_every_metadata_load_stays_in_its_row_block(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "2by4-pretrain_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    seen = {}
    for line in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines():
        k_atoms, step, first, second = map(int, line.split())
        assert 0 <= first < k_atoms and 0 <= second < k_atoms
        assert first == 2 * step and second == (first + 1 if first + 1 < k_atoms else first)
        seen.setdefault(k_atoms, set()).update((first, second))
    assert all(atoms == set(range(k)) for k, atoms in seen.items()) and len(seen) == 65
