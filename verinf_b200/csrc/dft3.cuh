// In-register radix-2^k DFT butterflies on three-limb values (gl3.cuh); every twiddle is a power of two.
#pragma once
#include "dft_reg.cuh"
#include "gl3.cuh"

namespace vd3 {

using vg3::T3;

template <int LOGR, int LOGLEN, int I, bool INV>
__device__ __forceinline__ void dif_level(T3* v) {
    constexpr int R = 1 << LOGR, LEN = 1 << LOGLEN, HALF = LEN / 2;
    if constexpr (I < R / 2) {
        constexpr int k = I % HALF, lo = (I / HALF) * LEN + k, hi = lo + HALF;
        constexpr int s0 = (vdft::root_exp(LOGLEN) * k) % 192, s = INV ? (192 - s0) % 192 : s0;
        const T3 d = s >= 96 ? vg3::sub3(v[hi], v[lo]) : vg3::sub3(v[lo], v[hi]);   // 2^96 = -1
        v[lo] = vg3::add3(v[lo], v[hi]);
        v[hi] = vg3::shl3<s % 96>(d);
        dif_level<LOGR, LOGLEN, I + 1, INV>(v);
    }
}
template <int LOGR, int LOGLEN, bool INV>
__device__ __forceinline__ void dif_levels(T3* v) {
    if constexpr (LOGLEN >= 1) {
        dif_level<LOGR, LOGLEN, 0, INV>(v);
        dif_levels<LOGR, LOGLEN - 1, INV>(v);
    }
}
// Decimation-in-frequency DFT of R = 2^LOGR three-limb values, X[c] = v[bitrev(c)] in [0, 2^64).  Top limbs that start
// in {-2 .. 2} grow to at most 2^6 in magnitude for R <= 16, and each level's shifts leave room for them: a shift of
// 2^28 occurs on the first level only, where differences stay within {-5 .. 4}.
template <int LOGR, bool INV>
__device__ __forceinline__ void dif(T3* t, uint64_t* v) {
    dif_levels<LOGR, LOGR, INV>(t);
#pragma unroll
    for (int i = 0; i < (1 << LOGR); ++i) v[i] = vg3::norm3(t[i]);
}
template <int LOGR, bool INV>
__device__ __forceinline__ void dif(uint64_t* v) {
    T3 t[1 << LOGR];
#pragma unroll
    for (int i = 0; i < (1 << LOGR); ++i) t[i] = vg3::widen(v[i]);
    dif<LOGR, INV>(t, v);
}

}  // namespace vd3
