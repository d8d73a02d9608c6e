// Roots of unity that are powers of two, and the output order of the in-register DFTs (dft3.cuh).
#pragma once
#include <cstdint>

namespace vdft {

// w_R = 2^root_exp(log2 R): the reference's root_of_unity(R) = 7^((p-1)/R) for R = 2..64.
__host__ __device__ constexpr int root_exp(int logr) {
    return logr == 1 ? 96 : logr == 2 ? 48 : logr == 3 ? 120 : logr == 4 ? 156 : logr == 5 ? 78 : 39;
}

__host__ __device__ constexpr int brev(int x, int bits) {
    int r = 0;
    for (int i = 0; i < bits; ++i) r |= ((x >> i) & 1) << (bits - 1 - i);
    return r;
}

}  // namespace vdft
