// Goldilocks arithmetic on unreduced values: any 64-bit word stands for its residue, and the sums inside a butterfly
// are kept as three limbs.
//
// With phi = 2^32: phi^2 = phi - 1 and phi^3 = -1 (mod p), so a limb at 2^64 is worth 2^32 - 1 and a limb at 2^96 is
// worth -1.  The canonical form of gl.cuh costs a conditional correction per addition (7 instructions) and subtraction
// (5) and a comparison with p per product; here an addition or subtraction is one carry chain of 3, a multiplication
// by a power of two 7-9, and a product (17) stops anywhere in [0, 2^64).
//
// What the sequences are shaped by, measured on B200 (issue slots per warp instruction, 1 = the scheduler's rate):
// carry-chain adds, shifts and logic run on the ALU pipe at 2, 32-bit multiply-adds on the other integer pipe at 2,
// 64-bit-result multiplies at 4 there whether or not they carry (so mad.lo.cc + madc.hi of the same operands, one
// instruction, costs as much as a plain wide multiply).  A multiply-add can take a carry in, so the last limb of a
// chain is written as a multiply by one (madc.lo) to level the two pipes; it cannot give a carry out.
// Radix-16 DFT of registers 60 -> 43 slots per element, product 49 -> 32, both in sequence 102 -> 72.
#pragma once
#include <cstdint>

#include "gl.cuh"

namespace vg3 {

using vgl::pack;

// x2*2^64 + x1*2^32 + x0 with a signed top limb
struct T3 { uint32_t x0, x1; int32_t x2; };

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t lo32(uint64_t a) { return (uint32_t)a; }
__device__ __forceinline__ uint32_t hi32(uint64_t a) { return (uint32_t)(a >> 32); }

// r + k*(2^32 - 1) mod 2^64, k in {-1, 0, 1}
__device__ __forceinline__ uint64_t add_k_eps(uint64_t r, int32_t k) {
    uint32_t r0 = lo32(r), r1 = hi32(r);
    asm("{\n\t.reg .u32 s;\n\t"
        "shr.s32 s, %2, 31;\n\t"
        "sub.cc.u32 %0, %0, %2;\n\t"
        "subc.u32 %1, %1, s;\n\t"
        "mad.lo.u32 %1, %2, %3, %1;\n\t}"
        : "+r"(r0), "+r"(r1) : "r"(k), "r"(vgl::VGL_ONE));
    return pack(r0, r1);
}

// (p3:p2:p1:p0) mod p into [0, 2^64): p0 + p1 phi + p2 (phi - 1) - p3.  With k the multiple of 2^64 that the two chains
// leave, the value less k*2^64 is at most 2^64 - 2^33 (k = 1) or at least 2^64 - 2^32 + 1 (k = -1): the last step fits.
__device__ __forceinline__ uint64_t reduce(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3) {
    uint32_t r0, r1; int32_t k;
    asm("{\n\t.reg .u32 e0, e1, m;\n\t.reg .b64 e;\n\t"
        "sub.cc.u32 %0, %3, %6;\n\t"
        "subc.cc.u32 %1, %4, 0;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "mul.wide.u32 e, %5, %7;\n\t"
        "mov.b64 {e0, e1}, e;\n\t"
        "add.cc.u32 %0, %0, e0;\n\t"
        "addc.cc.u32 %1, %1, e1;\n\t"
        "madc.lo.u32 %2, m, %8, 0;\n\t}"
        : "=&r"(r0), "=&r"(r1), "=&r"(k)
        : "r"(p0), "r"(p1), "r"(p2), "r"(p3), "r"(vgl::VGL_M1), "r"(vgl::VGL_ONE));
    return add_k_eps(pack(r0, r1), k);
}

// 128-bit product: the second middle product is added to the first as it is formed (multiply-add with carry out)
__device__ __forceinline__ void mul128(uint64_t a, uint64_t b, uint32_t& p0, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    asm("{\n\t.reg .u32 m0, m1;\n\t.reg .b64 t, w, m;\n\t"
        "mul.wide.u32 t, %4, %6;\n\t"
        "mul.wide.u32 w, %5, %7;\n\t"
        "mul.wide.u32 m, %4, %7;\n\t"
        "mov.b64 {m0, m1}, m;\n\t"
        "mov.b64 {%0, %1}, t;\n\t"
        "mov.b64 {%2, %3}, w;\n\t"
        "mad.lo.cc.u32 m0, %5, %6, m0;\n\t"
        "madc.hi.cc.u32 m1, %5, %6, m1;\n\t"
        "madc.lo.u32 %3, %3, %8, 0;\n\t"
        "add.cc.u32 %1, %1, m0;\n\t"
        "addc.cc.u32 %2, %2, m1;\n\t"
        "madc.lo.u32 %3, %3, %8, 0;\n\t}"
        : "=&r"(p0), "=&r"(p1), "=&r"(p2), "=&r"(p3)
        : "r"(lo32(a)), "r"(hi32(a)), "r"(lo32(b)), "r"(hi32(b)), "r"(vgl::VGL_ONE));
}

// a*b mod p into [0, 2^64), for any 64-bit a and b
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) {
    uint32_t p0, p1, p2, p3;
    mul128(a, b, p0, p1, p2, p3);
    return reduce(p0, p1, p2, p3);
}

// [0, 2^64) -> [0, p): r >= p exactly when the high half is 2^32 - 1 and the low half is not 0; then r - p = low - 1
__device__ __forceinline__ uint64_t canon(uint64_t r) {
    uint32_t r0 = lo32(r), r1 = hi32(r);
    asm("{\n\t.reg .pred q;\n\t"
        "setp.eq.u32 q, %1, 0xffffffff;\n\t"
        "setp.ne.and.u32 q, %0, 0, q;\n\t"
        "@q mov.u32 %1, 0;\n\t"
        "@q add.u32 %0, %0, 0xffffffff;\n\t}"
        : "+r"(r0), "+r"(r1));
    return pack(r0, r1);
}

__device__ __forceinline__ T3 widen(uint64_t a) { return T3{lo32(a), hi32(a), 0}; }
__device__ __forceinline__ T3 add3(T3 a, T3 b) {
    T3 r;
    asm("add.cc.u32 %0, %3, %6;\n\t"
        "addc.cc.u32 %1, %4, %7;\n\t"
        "madc.lo.u32 %2, %5, %9, %8;"
        : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
        : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(b.x0), "r"(b.x1), "r"(b.x2), "r"(vgl::VGL_ONE));
    return r;
}
__device__ __forceinline__ T3 sub3(T3 a, T3 b) {
    T3 r;
    asm("sub.cc.u32 %0, %3, %6;\n\t"
        "subc.cc.u32 %1, %4, %7;\n\t"
        "subc.u32 %2, %5, %8;"
        : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
        : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(b.x0), "r"(b.x1), "r"(b.x2));
    return r;
}

// (x1:x0) + x2*(2^32 - 1), any signed x2, as three limbs with a top limb in {-1, 0, 1}
__device__ __forceinline__ T3 fold3(uint32_t x0, uint32_t x1, int32_t x2) {
    T3 r;
    asm("sub.cc.u32 %0, %3, %5;\n\t"       // - x2, sign-extended
        "subc.cc.u32 %1, %4, %6;\n\t"
        "subc.u32 %2, 0, 0;\n\t"           // - borrow (the two sign words at 2^64 cancel)
        "add.cc.u32 %1, %1, %5;\n\t"       // + x2*2^32
        "madc.lo.u32 %2, %2, %7, 0;"
        : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2)
        : "r"(x0), "r"(x1), "r"(x2), "r"(x2 >> 31), "r"(vgl::VGL_ONE));
    return r;
}
// three limbs -> [0, 2^64)
__device__ __forceinline__ uint64_t norm3(T3 a) {
    const T3 r = fold3(a.x0, a.x1, a.x2);
    return add_k_eps(pack(r.x0, r.x1), r.x2);
}

// a * 2^S, 0 <= S < 192, as three limbs with a top limb in {-2 .. 2}; needs |a.x2| < 2^(31 - S % 32).
// (l2:l1:l0) = a << (S % 32), then S / 32 multiplications by phi; 2^96 = -1 gives the second half of the range.
template <int S>
__device__ __forceinline__ T3 shl3(T3 a) {
    static_assert(S >= 0 && S < 192, "shift out of range");
    if constexpr (S == 0) {
        return a;
    } else if constexpr (S == 96) {
        return sub3(T3{0, 0, 0}, a);
    } else {
        constexpr int V = S % 32, U = (S % 96) / 32;
        constexpr bool NEG = S >= 96;
        uint32_t l0 = a.x0, l1 = a.x1; int32_t l2 = a.x2;
        if constexpr (V != 0) {
            l2 = (int32_t)__funnelshift_l(a.x1, (uint32_t)a.x2, V);
            l1 = __funnelshift_l(a.x0, a.x1, V);
            l0 = a.x0 << V;
        }
        const int32_t s = l2 >> 31;
        T3 r;
        if constexpr (U == 0 && !NEG) {
            return fold3(l0, l1, l2);
        } else if constexpr (U == 0) {          // l2 - (l1:l0) - l2 phi
            asm("sub.cc.u32 %0, %5, %3;\n\t"
                "subc.cc.u32 %1, %6, %4;\n\t"
                "subc.u32 %2, 0, 0;\n\t"
                "sub.cc.u32 %1, %1, %5;\n\t"
                "subc.u32 %2, %2, 0;"
                : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2) : "r"(l0), "r"(l1), "r"(l2), "r"(s));
            return r;
        } else if constexpr (U == 1 && !NEG) {  // l0 phi + l1 (phi - 1) - l2
            // The one chain here that changes direction: madc reads the flag that subc.cc left.  PTX calls that flag the
            // borrow; the assembler for sm_100a keeps one carry flag, set when there is NO borrow, and this counts on it (the
            // -1 ahead stands for the borrow).  Nothing in the PTX document promises it: bench_int_pipes.cu checks it against
            // 128-bit arithmetic, and every transform of 16 points and more against the oracle would be wrong without it.
            // Both forms that stay inside the document are slower (last pass of the encode 3 and 4 %, middle pass 0.5 and 0.6 %).
            asm("{\n\t.reg .u32 e0, e1;\n\t.reg .b64 e;\n\t"
                "mul.wide.u32 e, %4, %7;\n\t"
                "mov.b64 {e0, e1}, e;\n\t"
                "add.cc.u32 %1, e1, %3;\n\t"
                "addc.u32 %2, 0xffffffff, 0;\n\t"      // carry - 1
                "sub.cc.u32 %0, e0, %5;\n\t"
                "subc.cc.u32 %1, %1, %6;\n\t"
                "madc.lo.u32 %2, %6, %7, %2;\n\t}"
                : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2) : "r"(l0), "r"(l1), "r"(l2), "r"(s), "r"(vgl::VGL_M1));
            return r;
        } else if constexpr (U == 1) {          // l2 - l1 (phi - 1) - l0 phi
            asm("{\n\t.reg .u32 e0, e1;\n\t.reg .b64 e;\n\t"
                "mul.wide.u32 e, %4, %7;\n\t"
                "mov.b64 {e0, e1}, e;\n\t"
                "sub.cc.u32 %0, %5, e0;\n\t"
                "subc.cc.u32 %1, %6, e1;\n\t"
                "subc.u32 %2, %6, 0;\n\t"
                "sub.cc.u32 %1, %1, %3;\n\t"
                "subc.u32 %2, %2, 0;\n\t}"
                : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2) : "r"(l0), "r"(l1), "r"(l2), "r"(s), "r"(vgl::VGL_M1));
            return r;
        } else if constexpr (!NEG) {            // l0 (phi - 1) - l1 - l2 phi
            asm("{\n\t.reg .u32 e0, e1;\n\t.reg .b64 e;\n\t"
                "mul.wide.u32 e, %3, %7;\n\t"
                "mov.b64 {e0, e1}, e;\n\t"
                "sub.cc.u32 %0, e0, %4;\n\t"
                "subc.cc.u32 %1, e1, %5;\n\t"
                "subc.u32 %2, 0, %6;\n\t}"
                : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2) : "r"(l0), "r"(l1), "r"(l2), "r"(s), "r"(vgl::VGL_M1));
            return r;
        } else {                                // l1 + l2 phi - l0 (phi - 1)
            asm("{\n\t.reg .u32 e0, e1;\n\t.reg .b64 e;\n\t"
                "mul.wide.u32 e, %3, %7;\n\t"
                "mov.b64 {e0, e1}, e;\n\t"
                "sub.cc.u32 %0, %4, e0;\n\t"
                "subc.cc.u32 %1, %5, e1;\n\t"
                "subc.u32 %2, %6, 0;\n\t}"
                : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2) : "r"(l0), "r"(l1), "r"(l2), "r"(s), "r"(vgl::VGL_M1));
            return r;
        }
    }
}
#endif  // __CUDACC__

}  // namespace vg3
