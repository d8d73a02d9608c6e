// Integer-pipe and field-primitive microbenchmarks for sm_100a.
//
// The hot path is bound by integer issue rates that no vendor peak figure covers, so the
// denominators are measured: register-resident kernels, 8 independent chains per thread, one
// instruction kind (or one field primitive) per kernel, timed with CUDA events.  Under
// `ncu --metrics smsp__inst_executed.sum,sm__inst_executed_pipe_alu.sum,sm__inst_executed_pipe_fma.sum
// --clock-control none` the same binary gives instructions per primitive.
// Build and run: python bench.py --micro int_pipes   (binary: build/int_pipes)
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

#include "verinf_b200/csrc/dft3.cuh"
#include "verinf_b200/csrc/dft_reg.cuh"
#include "verinf_b200/csrc/gl.cuh"

// The canonical form of the power-of-two shifts and of the in-register DFT, which the library had before gl3.cuh: what
// the three-limb form is timed and checked against.
namespace vgl {
#ifdef __CUDA_ARCH__
// (l1:l0) + h*(2^32-1) mod p, canonical; (l1:l0) is any u64, h any u32: 12 instructions
__device__ __forceinline__ uint64_t add_mul_eps(uint32_t l0, uint32_t l1, uint32_t h) {
    uint32_t r0, r1;
#if VGL_FMA_CARRY & 4
    asm("{\n\t.reg .u32 c, e0, e1;\n\t.reg .b64 e;\n\t.reg .pred q;\n\t"
        "mul.wide.u32 e, %4, %5;\n\t"          // e = h*EPS (FMA pipe)
        "mov.b64 {e0, e1}, e;\n\t"
        "add.cc.u32 %0, %2, e0;\n\t"
        "addc.cc.u32 %1, %3, e1;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "mad.lo.cc.u32 %0, c, %5, %0;\n\t"     // += carry ? EPS : 0 (FMA pipe)
        "madc.lo.u32 %1, c, %6, %1;\n\t"
        "setp.eq.u32 q, %1, 0xffffffff;\n\t"
        "setp.ne.and.u32 q, %0, 0, q;\n\t"
        "@q mov.u32 %1, 0;\n\t"
        "@q add.u32 %0, %0, 0xffffffff;\n\t}"
        : "=&r"(r0), "=&r"(r1) : "r"(l0), "r"(l1), "r"(h), "r"(VGL_M1), "r"(VGL_ZERO));
    return pack(r0, r1);
#endif
    asm("{\n\t.reg .u32 m, e0, e1;\n\t.reg .pred q;\n\t"
        "sub.cc.u32 e0, 0, %4;\n\t"
        "subc.u32 e1, %4, 0;\n\t"
        "add.cc.u32 %0, %2, e0;\n\t"
        "addc.cc.u32 %1, %3, e1;\n\t"
        "addc.u32 m, 0, 0;\n\t"
        "neg.s32 m, m;\n\t"
        "add.cc.u32 %0, %0, m;\n\t"
        "addc.u32 %1, %1, 0;\n\t"
        "setp.eq.u32 q, %1, 0xffffffff;\n\t"
        "setp.ne.and.u32 q, %0, 0, q;\n\t"
        "@q mov.u32 %1, 0;\n\t"
        "@q add.u32 %0, %0, 0xffffffff;\n\t}"
        : "=&r"(r0), "=&r"(r1) : "r"(l0), "r"(l1), "r"(h));
    return pack(r0, r1);
}
#endif

// x * 2^S mod p for a compile-time 0 <= S < 96 (x canonical -> canonical).
// Every 2^k-th root of unity with k <= 6 is a power of two in this field
// (2 has order 192), so radix-<=64 butterflies multiply by shifts only.
// With phi = 2^32 (phi^2 = phi - 1, phi^3 = -1) and (l2:l1:l0) = x << (S mod 32):
//   S <  32: (l1:l0) + l2*(2^32-1)
//   S <  64: the general 128-bit reduction of (l2:l1:l0:0)
//   S >= 64: l0*(2^32-1) - (l2:l1)
// (Issuing the limb shifts as wide multiplies on the FMA pipe, or building the 64-bit sums from
// mad.wide plus a 64-bit compare instead of carry chains, was measured slower on B200: radix-16
// butterfly throughput 2004 and 1250 G element-stages/s against 2091 for this form.)
template <int S>
__device__ __forceinline__ uint64_t mul_pow2(uint64_t x) {
    static_assert(S >= 0 && S < 96, "shift out of range");
#ifdef __CUDA_ARCH__
    if constexpr (S == 0) {
        return x;
    } else {
        constexpr int V = S % 32, U = S / 32;
        // (l2:l1:l0) = x << V as three 32-bit limbs
        uint32_t l0 = (uint32_t)x, l1 = (uint32_t)(x >> 32), l2 = 0;
        if constexpr (V != 0) {
            l2 = l1 >> (32 - V); l1 = (l1 << V) | (l0 >> (32 - V)); l0 <<= V;
        }
        if constexpr (U == 0) {
            // l0 + l1 phi + l2 phi^2 = (l1:l0) + l2*(2^32-1)
            return add_mul_eps(l0, l1, l2);
        } else if constexpr (U == 1) {
            // l0 phi + l1 phi^2 + l2 phi^3: the 128-bit value (hi = (l2:l1), lo = (l0:0))
            return reduce128(pack(0, l0), pack(l1, l2));
        } else {
            // l0 phi^2 + l1 phi^3 + l2 phi^4 = l0*(2^32-1) - (l2:l1); (l2:l1) < 2^63 is canonical
#if VGL_FMA_CARRY & 4
            uint64_t e;
            asm("mul.wide.u32 %0, %1, %2;" : "=l"(e) : "r"(l0), "r"(VGL_M1));     // FMA pipe
            return sub(e, pack(l1, l2));
#else
            uint32_t e0, e1;
            asm("sub.cc.u32 %0, 0, %2;\n\t"
                "subc.u32 %1, %2, 0;"
                : "=&r"(e0), "=&r"(e1) : "r"(l0));
            return sub(pack(e0, e1), pack(l1, l2));
#endif
        }
    }
#else
    return x;
#endif
}

}  // namespace vgl

namespace vdft {

using vgl::add;
using vgl::sub;

template <int LOGLEN, int K, bool INV>
__device__ __forceinline__ void bfly(uint64_t& a, uint64_t& b) {
    constexpr int s0 = (root_exp(LOGLEN) * K) % 192;
    constexpr int s = INV ? (192 - s0) % 192 : s0;
    uint64_t t = add(a, b);
    uint64_t d = (s >= 96) ? sub(b, a) : sub(a, b);   // 2^96 = -1
    a = t;
    b = vgl::mul_pow2<s % 96>(d);
}

template <int LOGR, int LOGLEN, int I, bool INV>
__device__ __forceinline__ void dif_level(uint64_t* v) {
    constexpr int R = 1 << LOGR, LEN = 1 << LOGLEN, HALF = LEN / 2;
    if constexpr (I < R / 2) {
        constexpr int blk = I / HALF, k = I % HALF;
        bfly<LOGLEN, k, INV>(v[blk * LEN + k], v[blk * LEN + k + HALF]);
        dif_level<LOGR, LOGLEN, I + 1, INV>(v);
    }
}
// In-register decimation-in-frequency DFT of R = 2^LOGR values: X[c] = v[bitrev(c)].
template <int LOGR, int LOGLEN, bool INV>
__device__ __forceinline__ void dif(uint64_t* v) {
    if constexpr (LOGLEN >= 1) {
        dif_level<LOGR, LOGLEN, 0, INV>(v);
        dif<LOGR, LOGLEN - 1, INV>(v);
    }
}

}  // namespace vdft

namespace {
constexpr int ITERS = 1024, CHAINS = 8, GRID = 148 * 8, BLOCK = 256;

template <int OP>
__global__ void __launch_bounds__(BLOCK) k_raw(uint32_t* out, uint32_t a0, uint32_t m) {
    uint32_t x[CHAINS], y[CHAINS];
    uint64_t z[CHAINS];
#pragma unroll
    for (int i = 0; i < CHAINS; ++i) { x[i] = a0 + threadIdx.x + i; y[i] = a0 * 3 + i; z[i] = ((uint64_t)x[i] << 32) | y[i]; }
    for (int it = 0; it < ITERS; ++it) {
#pragma unroll
        for (int i = 0; i < CHAINS; ++i) {
            if (OP == 0) asm volatile("add.u32 %0, %0, %1;" : "+r"(x[i]) : "r"(y[i]));
            if (OP == 1) asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(x[i]) : "r"(m), "r"(y[i]));
            if (OP == 2) asm volatile("mad.wide.u32 %0, %1, %2, %0;" : "+l"(z[i]) : "r"(x[i]), "r"(m));
            if (OP == 3) asm volatile("shf.r.wrap.b32 %0, %0, %0, %1;" : "+r"(x[i]) : "r"(m));
            if (OP == 4) asm volatile("prmt.b32 %0, %0, %0, 0x1032;" : "+r"(x[i]));
            if (OP == 5) asm volatile("add.cc.u32 %0, %0, %2; addc.u32 %1, %1, %3;" : "+r"(x[i]), "+r"(y[i]) : "r"(m), "r"(a0));
            if (OP == 7) asm volatile("mad.wide.s32 %0, %1, %2, %0;" : "+l"(z[i]) : "r"(x[i]), "r"(m));
            if (OP == 8) {      // wide product, then a 64-bit add of an independent value (no fused accumulate)
                uint64_t t;
                asm volatile("mul.wide.s32 %0, %1, %2;" : "=l"(t) : "r"(x[i]), "r"(m));
                asm volatile("add.s64 %0, %0, %1;" : "+l"(z[i]) : "l"(t));
            }
            if (OP == 9) asm volatile("mad.lo.s32 %0, %1, %2, %0;" : "+r"(y[i]) : "r"(x[i]), "r"(m));
            if (OP == 6) {
                asm volatile("add.u32 %0, %0, %1;" : "+r"(x[i]) : "r"(m));
                asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(y[i]) : "r"(m), "r"(a0));
            }
        }
    }
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < CHAINS; ++i) acc ^= x[i] ^ y[i] ^ (uint32_t)z[i] ^ (uint32_t)(z[i] >> 32);
    out[blockIdx.x * BLOCK + threadIdx.x] = acc;
}

template <int OP>
__global__ void __launch_bounds__(BLOCK) k_field(uint64_t* out, uint64_t seed) {
    using namespace vgl;
    uint64_t v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = (seed * (threadIdx.x + 1 + i * 977) + i) % P;
    for (int it = 0; it < ITERS / 4; ++it) {
        if (OP == 0) vdft::dif<4, 4, false>(v);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (OP == 1) v[i] = sub(v[i], v[(i + 1) & 15]);
            if (OP == 2) v[i] = add(v[i], v[(i + 1) & 15]);
            if (OP == 3) v[i] = mul(v[i], v[(i + 1) & 15]);
            if (OP == 4) v[i] = mul_pow2<12>(v[i]);
            if (OP == 5) v[i] = mul_pow2<48>(v[i]);
            if (OP == 6) v[i] = mul_pow2<72>(v[i]);
        }
    }
    uint64_t acc = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) acc ^= v[i];
    out[blockIdx.x * BLOCK + threadIdx.x] = acc;
}

// unreduced three-limb form (gl3.cuh): products and radix-16 DFTs of words in [0, 2^64)
template <int OP>
__global__ void __launch_bounds__(BLOCK) k_three(uint64_t* out, uint64_t seed) {
    uint64_t v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = (seed * (threadIdx.x + 1 + i * 977) + i) % vgl::P;
    for (int it = 0; it < ITERS / 4; ++it) {
        if (OP == 0) vd3::dif<4, false>(v);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (OP == 1) v[i] = vg3::mul(v[i], v[(i + 1) & 15]);
            if (OP == 2) v[i] = vg3::norm3(vg3::shl3<12>(vg3::widen(v[i])));
        }
    }
    uint64_t acc = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) acc ^= v[i];
    out[blockIdx.x * BLOCK + threadIdx.x] = acc;
}


// ---- self-check of the device field primitives against 128-bit integer arithmetic ----------
template <int S> __device__ bool chk_pow2(uint64_t x) {
    unsigned __int128 v = (unsigned __int128)x;
    for (int i = 0; i < S; ++i) { v <<= 1; if (v >= vgl::P) v -= vgl::P; }
    return vgl::mul_pow2<S>(x) == (uint64_t)v;
}
__device__ uint64_t edge_or_rand(uint64_t i, uint64_t salt) {
    const uint64_t P = vgl::P;
    const uint64_t edges[12] = {0, 1, 2, P - 1, P - 2, 0xFFFFFFFFull, 0x100000000ull, 0xFFFFFFFF00000000ull,
                                0x8000000000000000ull, 0xFFFFFFFEFFFFFFFFull, 0x00000000FFFFFFFEull, P - 0xFFFFFFFFull};
    if ((i & 7) == 0) return edges[(i >> 3) % 12];
    uint64_t z = (i + salt) * 0x9E3779B97F4A7C15ull; z ^= z >> 31; z *= 0xBF58476D1CE4E5B9ull; z ^= z >> 29;
    return z % P;
}
__global__ void k_selfcheck(unsigned long long* bad) {
    using namespace vgl;
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint64_t a = edge_or_rand(i, 1), b = edge_or_rand(i / 3 + (i & 7) * 11, 7);
    unsigned __int128 A = a, B = b;
    int f = 0;
    if (add(a, b) != (uint64_t)((A + B) % P)) f |= 1;
    if (sub(a, b) != (uint64_t)((A + P - B) % P)) f |= 2;
    if (mul(a, b) != (uint64_t)((A * B) % P)) f |= 4;
    uint64_t hi = edge_or_rand(i * 5 + 3, 99) | (i & 1 ? 0xFFFFFFFF00000000ull : 0), lo = a | (i & 2 ? 0xFFFFFFFF00000000ull : 0);
    unsigned __int128 W = ((unsigned __int128)hi << 64) | lo;
    if (reduce128(lo, hi) != (uint64_t)(W % P)) f |= 8;
    if (sub(a, P) != a) f |= 16;
    if (!(chk_pow2<1>(a) && chk_pow2<12>(a) && chk_pow2<24>(a) && chk_pow2<31>(a) && chk_pow2<32>(a) && chk_pow2<36>(a) &&
          chk_pow2<48>(a) && chk_pow2<60>(a) && chk_pow2<63>(a) && chk_pow2<64>(a) && chk_pow2<72>(a) && chk_pow2<84>(a) &&
          chk_pow2<95>(a))) f |= 32;
    {   // three-limb form against the canonical one: any 64-bit words, edges included
        const uint64_t x = a + (i & 8 ? 0xFFFFFFFFull : 0), y = b | (i & 4 ? 0xFFFFFFFF00000000ull : 0);
        if (vg3::canon(vg3::mul(x, y)) != (uint64_t)(((unsigned __int128)x * y) % P)) f |= 64;
        uint64_t v[16], u[16];
        for (int k = 0; k < 16; ++k) { u[k] = edge_or_rand(i * 16 + k, 5) | (k & i & 1 ? 0xFFFFFFFF00000000ull : 0); v[k] = u[k] % P; }
        vdft::dif<4, 4, false>(v); vd3::dif<4, false>(u);
        for (int k = 0; k < 16; ++k) if (vg3::canon(u[k]) != v[k]) f |= 128;
        for (int k = 0; k < 16; ++k) { u[k] = edge_or_rand(i * 16 + k, 6) | (k & i & 1 ? 0xFFFFFFFF00000000ull : 0); v[k] = u[k] % P; }
        vdft::dif<4, 4, true>(v); vd3::dif<4, true>(u);
        for (int k = 0; k < 16; ++k) if (vg3::canon(u[k]) != v[k]) f |= 256;
        const vg3::T3 t = vg3::sub3(vg3::widen(a), vg3::widen(b));
        const uint64_t d = sub(a, b);
        if (vg3::canon(vg3::norm3(vg3::shl3<12>(t))) != mul_pow2<12>(d) || vg3::canon(vg3::norm3(vg3::shl3<39>(t))) != mul_pow2<39>(d) ||
            vg3::canon(vg3::norm3(vg3::shl3<32>(t))) != mul_pow2<32>(d) || vg3::canon(vg3::norm3(vg3::shl3<36>(t))) != mul_pow2<36>(d) ||
            vg3::canon(vg3::norm3(vg3::shl3<48>(t))) != mul_pow2<48>(d) || vg3::canon(vg3::norm3(vg3::shl3<60>(t))) != mul_pow2<60>(d) ||
            vg3::canon(vg3::norm3(vg3::shl3<78>(t))) != mul_pow2<78>(d) || vg3::canon(vg3::norm3(vg3::shl3<96>(t))) != sub(0, d) ||
            vg3::canon(vg3::norm3(vg3::shl3<117>(t))) != sub(0, mul_pow2<21>(d)) ||
            vg3::canon(vg3::norm3(vg3::shl3<156>(t))) != sub(0, mul_pow2<60>(d)) ||
            vg3::canon(vg3::norm3(vg3::shl3<162>(t))) != sub(0, mul_pow2<66>(d))) f |= 512;
    }
    if (f) atomicOr(bad, (unsigned long long)f);
}

template <class F>
float time_ms(F launch) {
    cudaEvent_t a, b;
    cudaEventCreate(&a); cudaEventCreate(&b);
    launch(); cudaDeviceSynchronize();
    cudaEventRecord(a); launch(); cudaEventRecord(b); cudaEventSynchronize(b);
    float ms = 0; cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a); cudaEventDestroy(b);
    return ms;
}
}  // namespace

int main(int argc, char**) {      // any argument: the self-check alone
    void* d = nullptr;
    if (cudaMalloc(&d, (size_t)GRID * BLOCK * 8) != cudaSuccess) { printf("no CUDA device\n"); return 1; }
    {
        unsigned long long* bad; cudaMalloc(&bad, 8); cudaMemset(bad, 0, 8);
        k_selfcheck<<<4096, 256>>>(bad);
        unsigned long long h = 0; cudaMemcpy(&h, bad, 8, cudaMemcpyDeviceToHost);
        printf("self-check of add/sub/mul/reduce128/mul_pow2 and the three-limb form vs 128-bit arithmetic: %s (flags %llu) %s\n",
               h ? "MISMATCH" : "ok", h, cudaGetErrorString(cudaGetLastError()));
        cudaFree(bad);
        if (argc > 1) return h != 0 || cudaGetLastError() != cudaSuccess;
    }
    int khz = 0; cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, 0);
    const double threads = (double)GRID * BLOCK;
    auto raw = [&](const char* name, int per, float ms) {
        double ops = threads * ITERS * CHAINS * per;
        printf("%-28s %8.3f ms %9.1f Gop/s %7.1f ops/clk/SM\n", name, ms, ops / ms / 1e6, ops / (ms * 1e-3) / 148 / (khz * 1e3));
    };
    raw("add.u32", 1, time_ms([&] { k_raw<0><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("mad.lo.u32", 1, time_ms([&] { k_raw<1><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("mad.wide.u32", 1, time_ms([&] { k_raw<2><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("shf.r.wrap", 1, time_ms([&] { k_raw<3><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("prmt", 1, time_ms([&] { k_raw<4><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("add.cc + addc", 2, time_ms([&] { k_raw<5><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("add.u32 + mad.lo.u32", 2, time_ms([&] { k_raw<6><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("mad.wide.s32", 1, time_ms([&] { k_raw<7><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("mul.wide.s32 + add.s64", 1, time_ms([&] { k_raw<8><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    raw("mad.lo.s32", 1, time_ms([&] { k_raw<9><<<GRID, BLOCK>>>((uint32_t*)d, 12345, 77); }));
    auto fld = [&](const char* name, int per, float ms) {
        double ops = threads * (ITERS / 4) * per;
        printf("%-28s %8.3f ms %9.1f Gop/s\n", name, ms, ops / ms / 1e6);
    };
    fld("radix-16 DFT element-stage", 64, time_ms([&] { k_field<0><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("gl sub", 16, time_ms([&] { k_field<1><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("gl add", 16, time_ms([&] { k_field<2><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("gl mul", 16, time_ms([&] { k_field<3><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("gl mul_pow2<12>", 16, time_ms([&] { k_field<4><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("gl mul_pow2<48>", 16, time_ms([&] { k_field<5><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("gl mul_pow2<72>", 16, time_ms([&] { k_field<6><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("three-limb radix-16 DFT element-stage", 64, time_ms([&] { k_three<0><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("three-limb mul", 16, time_ms([&] { k_three<1><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    fld("three-limb shl3<12> + norm", 16, time_ms([&] { k_three<2><<<GRID, BLOCK>>>((uint64_t*)d, 12345); }));
    cudaFree(d);
    return 0;
}
