// Which metadata a K step of the single-CTA sparse GEMM stages.  Plain C++, so that the arithmetic can be checked on the CPU.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define SP24_HD __host__ __device__ __forceinline__
#else
#define SP24_HD inline
#endif

namespace sp24 {

// The metadata of a 128-row block is a run of 2048-byte atoms, one per 128 columns of K, and the buffer ends with the last
// block's run.  8-bit operands take 256 columns a step, so the last step of a run of odd length has one atom only: it is staged
// twice, the second copy goes with columns that the operands' tensor maps fill with zeros.
struct MetaAtoms { int64_t first, second; };
SP24_HD MetaAtoms meta_atoms_of_step(int64_t step, int64_t atoms_per_block) {
    const int64_t a = 2 * step;
    return {a, a + 1 < atoms_per_block ? a + 1 : a};
}

}  // namespace sp24
