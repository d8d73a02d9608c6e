// Sumcheck proofs from the caller's own tables to finished round polynomials on the host.
//
// What it replaces in the reference: prove_terms_gpu with fold_t and gl_sum (layergkr/gpu.py:326-410; CPU twin
// layergkr/sumcheck.py:153-226).  sumcheck.cu keeps the per-round entry points whose samples stay on the device (for
// sharded proofs); here the tables are read in place (or copied as the first round of a session sums them), folds write the
// work buffer, and the last block of each
// round hands its sums to the host through mapped memory, so a round is one launch and no copy, and a queued proof waits
// for the device once.
//
// What bounds it: large tables the integer pipes (a pair of entries costs 2 products per sample point), small ones the
// chain of rounds.  Against both:
//  * With the challenges known a kernel does two rounds per pass: it reads four entries per table and index, sums both
//    rounds' polynomials and writes one entry.  A 3 x 2^24 proof moves 0.67 GB instead of 1.6 and is launched 8 times.
//  * A round polynomial of degree d is summed at 0, infinity, -1 and 2 instead of 0..d: the value at infinity is the
//    product of the differences, -1 is one subtraction away from 0, and the value at 1 follows from the round before.
//    The host turns sums into coefficients and evaluates them (a few products per round).
//  * Sums stay unreduced: 160-bit sums of 128-bit products where the term structure is a single product.
//  * Tables of at most 2^11 entries finish in one block that holds them in shared memory, one barrier per round.
#include <atomic>
#include <cstring>
#include <mutex>
#include <new>

#include "../../include/verinf_b200.h"
#include "common.cuh"
#include "gl3.cuh"

namespace {

using vg3::T3;

constexpr int MAX_TABLES = 8, MAX_TERMS = 8, MAX_FAC = 4;
constexpr int NPT = 5;                  // sums per round: at 0, 1, infinity, -1, 2
constexpr int BLOCK = 256;
constexpr int MAX_GRID = 148 * 4;
constexpr int TAIL_LOG = 11;            // table length from which one block does the remaining rounds
constexpr int TAIL_BLOCK = 512;
constexpr int MAX_ROUNDS = 48;
constexpr int ROW = 8;                  // words per round in the host buffer

struct Terms {
    int n, deg;
    uint32_t count[MAX_TERMS];          // multiplicity of table k in bits 4k .. 4k+3
    int nfac[MAX_TERMS];
    int sign[MAX_TERMS];                // coefficient 1, -1 (added or taken away as it is) or general (0)
    uint64_t coef[MAX_TERMS];
};
struct Tables { const uint64_t* in[MAX_TABLES]; uint64_t* out[MAX_TABLES]; };
// where the sums of a launch go: per-block sums and a ticket on the device, the totals in mapped host memory
struct Sink {
    uint64_t* partials;                 // (grid, 2 * NPT)
    unsigned* ticket;                   // zero between launches
    volatile uint64_t* row0;            // totals of the first and second round of the launch
    volatile uint64_t* row1;
    volatile uint64_t* flag;            // set to `stamp` behind the totals when not null
    uint64_t stamp;
};

// ---- arithmetic on canonical table entries ------------------------------------------------------------------------
__device__ __forceinline__ uint64_t sub(uint64_t a, uint64_t b) { return vgl::sub(a, b); }
// a + m for canonical a and any m: at most one carry, because a + m < 2^64 + p
__device__ __forceinline__ uint64_t add_any(uint64_t a, uint64_t m) {
    uint32_t r0, r1, k;
    asm("add.cc.u32 %0, %3, %5;\n\taddc.cc.u32 %1, %4, %6;\n\taddc.u32 %2, 0, 0;"
        : "=&r"(r0), "=&r"(r1), "=r"(k) : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)m), "r"((uint32_t)(m >> 32)));
    uint64_t r = vgl::pack(r0, r1);
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(r) : "r"(k), "r"(vgl::VGL_M1));
    return r;
}
// a + r (b - a), canonical
__device__ __forceinline__ uint64_t fold(uint64_t a, uint64_t b, uint64_t r) {
    return vg3::canon(add_any(a, vg3::mul(r, sub(b, a))));
}

// Sum of words (three limbs, the top one signed) or of unreduced products (five limbs)
struct Acc {
    uint32_t x[5];
    __device__ __forceinline__ void clear() { x[0] = x[1] = x[2] = x[3] = x[4] = 0; }
    __device__ __forceinline__ void add_word(uint64_t v) {
        asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]) : "r"((uint32_t)v), "r"((uint32_t)(v >> 32)));
    }
    // a term with coefficient -1: words of any kind can be taken away, while p - v is a word only for v <= p
    __device__ __forceinline__ void sub_word(uint64_t v) {
        asm("sub.cc.u32 %0, %0, %3;\n\tsubc.cc.u32 %1, %1, %4;\n\tsubc.u32 %2, %2, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]) : "r"((uint32_t)v), "r"((uint32_t)(v >> 32)));
    }
    __device__ __forceinline__ void add_product(uint64_t a, uint64_t b) {
        uint32_t p0, p1, p2, p3;
        vg3::mul128(a, b, p0, p1, p2, p3);
        asm("add.cc.u32 %0, %0, %5;\n\taddc.cc.u32 %1, %1, %6;\n\taddc.cc.u32 %2, %2, %7;\n\taddc.cc.u32 %3, %3, %8;\n\taddc.u32 %4, %4, 0;"
            : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]) : "r"(p0), "r"(p1), "r"(p2), "r"(p3));
    }
    // [0, 2^64); 2^128 = -2^32, and fewer than 2^31 words or products are summed
    __device__ __forceinline__ uint64_t value(bool products) const {
        if (!products) return vg3::norm3(T3{x[0], x[1], (int32_t)x[2]});
        const uint64_t r = vg3::reduce(x[0], x[1], x[2], x[3]);
        return vg3::norm3(vg3::sub3(vg3::widen(r), T3{0, x[4], 0}));
    }
};

// One product term structure: SIMPLE = the product of all NT tables, else sums of terms over them.
template <int NT, bool SIMPLE>
__device__ __forceinline__ void add_point(Acc& acc, const uint64_t (&f)[NT], const Terms& tm, bool leading) {
    if constexpr (SIMPLE) {
        if constexpr (NT == 1) acc.add_word(f[0]);
        else {
            uint64_t p = f[0];
#pragma unroll
            for (int k = 1; k + 1 < NT; ++k) p = vg3::mul(p, f[k]);
            acc.add_product(p, f[NT - 1]);
        }
    } else {
        for (int t = 0; t < tm.n; ++t) {
            if (leading && tm.nfac[t] != tm.deg) continue;       // at infinity only the terms of full degree count
            const int sg = tm.sign[t];
            uint64_t p = tm.coef[t];
            bool have = sg == 0;
#pragma unroll
            for (int k = 0; k < NT; ++k) {
                const uint32_t c = (tm.count[t] >> (4 * k)) & 15u;
                for (uint32_t m = 0; m < c; ++m) {
                    if (have) p = vg3::mul(p, f[k]);
                    else { p = f[k]; have = true; }
                }
            }
            if (sg < 0) acc.sub_word(p); else acc.add_word(p);
        }
    }
}
template <int NT, bool SIMPLE> constexpr bool sums_products() { return SIMPLE && NT > 1; }

// sums of one pair (lo, hi) per table; FIRST: the value at 1 as well.  Points beyond the degree are left out.
template <int NT, bool SIMPLE>
__device__ __forceinline__ void add_pair(Acc (&acc)[NPT], const uint64_t (&lo)[NT], const uint64_t (&hi)[NT], const Terms& tm, bool first) {
    const int deg = SIMPLE ? NT : tm.deg;
    add_point<NT, SIMPLE>(acc[0], lo, tm, false);
    if (first) add_point<NT, SIMPLE>(acc[1], hi, tm, false);
    if (deg < 2) return;
    uint64_t d[NT], f[NT];
#pragma unroll
    for (int k = 0; k < NT; ++k) d[k] = sub(hi[k], lo[k]);
    add_point<NT, SIMPLE>(acc[2], d, tm, true);
    if (deg < 3) return;
#pragma unroll
    for (int k = 0; k < NT; ++k) f[k] = sub(lo[k], d[k]);
    add_point<NT, SIMPLE>(acc[3], f, tm, false);
    if (deg < 4) return;
#pragma unroll
    for (int k = 0; k < NT; ++k) f[k] = add_any(hi[k], d[k]);
    add_point<NT, SIMPLE>(acc[4], f, tm, false);
}

// ---- sums over a block and over the grid --------------------------------------------------------------------------
// A word is summed over a warp as pieces of 22, 22 and 20 bits by the integer reduction unit; pieces of all warps of a
// block stay below 2^32.
__device__ __forceinline__ void put_pieces(uint32_t* dst, uint64_t v, int lane) {
    const uint32_t a = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0x3fffffu);
    const uint32_t b = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 22) & 0x3fffffu);
    const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 44));
    if (lane == 0) { dst[0] = a; dst[1] = b; dst[2] = c; }
}
template <int WARPS, int N>
__device__ __forceinline__ uint64_t sum_pieces(const uint32_t (*red)[N * 3], int x) {      // total of value x
    uint32_t p[3] = {0, 0, 0};
#pragma unroll
    for (int w = 0; w < WARPS; ++w)
#pragma unroll
        for (int i = 0; i < 3; ++i) p[i] += red[w][3 * x + i];
    const uint64_t a = p[0] + ((uint64_t)p[1] << 22), b = (uint64_t)p[2] << 44, s = a + b;
    return vg3::norm3(T3{(uint32_t)s, (uint32_t)(s >> 32), (int32_t)((p[2] >> 20) + (s < a ? 1u : 0u))});
}

// Per-thread sums v[0..N) -> totals over the grid in the sink's rows (the first NPT values in row0, the rest in row1).
template <int N>
__device__ __forceinline__ void finish(const uint64_t (&v)[N], const Sink& sk) {
    constexpr int WARPS = BLOCK / 32;
    __shared__ uint32_t red[WARPS][N * 3];
    __shared__ uint64_t tot[WARPS][16];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll
    for (int x = 0; x < N; ++x) put_pieces(&red[wid][3 * x], v[x], lane);
    __syncthreads();
    uint64_t s = 0;
    if (tid < N) s = sum_pieces<WARPS, N>(red, tid);
    if (gridDim.x > 1) {
        if (tid < N) {
            __stcg(reinterpret_cast<unsigned long long*>(sk.partials) + (int64_t)blockIdx.x * N + tid, (unsigned long long)s);
            __threadfence();
        }
        __syncwarp();
        if (tid == 0) last = atomicInc(sk.ticket, gridDim.x - 1) == gridDim.x - 1;       // wraps to zero for the next launch
        __syncthreads();
        if (!last) return;
        __threadfence();
        // 16 values wide: thread (b, x) adds the blocks b, b + 16, ... of value x
        T3 t{0, 0, 0};
        const int x = tid & 15;
        if (x < N)
            for (int b = tid >> 4; b < (int)gridDim.x; b += BLOCK / 16)
                t = vg3::add3(t, vg3::widen(__ldcg(reinterpret_cast<const unsigned long long*>(sk.partials) + (int64_t)b * N + x)));
        uint64_t u = vg3::norm3(t);
        t = vg3::add3(vg3::widen(u), vg3::widen(__shfl_xor_sync(0xffffffffu, u, 16)));
        u = vg3::norm3(t);
        if (lane < 16) tot[wid][lane] = u;
        __syncthreads();
        if (tid < N) {
            t = T3{0, 0, 0};
#pragma unroll
            for (int w = 0; w < WARPS; ++w) t = vg3::add3(t, vg3::widen(tot[w][tid]));
            s = vg3::norm3(t);
        }
    }
    if (tid < N) {
        if (tid < NPT) sk.row0[tid] = s; else sk.row1[tid - NPT] = s;
        __threadfence_system();
    }
    if (tid < 32) {
        __syncwarp();
        if (tid == 0 && sk.flag) *sk.flag = sk.stamp;
    }
}

// ---- kernels ------------------------------------------------------------------------------------------------------
// One round: FOLD = with the challenge r of the round before (size -> size/2, written to out, which may be in), then the
// sums.  Without FOLD the entries are copied to out where there is one.
template <int NT, bool SIMPLE, bool FOLD>
__global__ void __launch_bounds__(BLOCK) k_round(Tables tb, Terms tm, int64_t size, uint64_t r, Sink sk) {
    const int64_t q = FOLD ? size / 4 : size / 2;
    Acc acc[NPT];
#pragma unroll
    for (int x = 0; x < NPT; ++x) acc[x].clear();
    for (int64_t i = (int64_t)blockIdx.x * BLOCK + threadIdx.x; i < q; i += (int64_t)gridDim.x * BLOCK) {
        uint64_t lo[NT], hi[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) {
            const uint64_t* f = tb.in[k];
            if constexpr (FOLD) {
                lo[k] = fold(f[i], f[i + 2 * q], r);
                hi[k] = fold(f[i + q], f[i + 3 * q], r);
                tb.out[k][i] = lo[k];
                tb.out[k][i + q] = hi[k];
            } else {
                lo[k] = f[i];
                hi[k] = f[i + q];
                if (tb.out[0]) {
                    tb.out[k][i] = lo[k];
                    tb.out[k][i + q] = hi[k];
                }
            }
        }
        add_pair<NT, SIMPLE>(acc, lo, hi, tm, !FOLD);
    }
    uint64_t v[NPT];
#pragma unroll
    for (int x = 0; x < NPT; ++x) v[x] = acc[x].value(sums_products<NT, SIMPLE>());
    finish<NPT>(v, sk);
}

// Two rounds with known challenges r0, r1: sums of the tables as they are (first: the very first round), fold with r0,
// sums again, fold with r1; size -> size/4.
template <int NT, bool SIMPLE>
__global__ void __launch_bounds__(BLOCK, 2) k_round2(Tables tb, Terms tm, int64_t size, uint64_t r0, uint64_t r1, int first, Sink sk) {
    const int64_t q = size / 4;
    Acc acc[2][NPT];
#pragma unroll
    for (int x = 0; x < NPT; ++x) { acc[0][x].clear(); acc[1][x].clear(); }
    for (int64_t i = (int64_t)blockIdx.x * BLOCK + threadIdx.x; i < q; i += (int64_t)gridDim.x * BLOCK) {
        uint64_t a[NT], b[NT], c[NT], d[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) {
            const uint64_t* f = tb.in[k];
            a[k] = f[i]; b[k] = f[i + q]; c[k] = f[i + 2 * q]; d[k] = f[i + 3 * q];
        }
        add_pair<NT, SIMPLE>(acc[0], a, c, tm, first);
        add_pair<NT, SIMPLE>(acc[0], b, d, tm, first);
#pragma unroll
        for (int k = 0; k < NT; ++k) { a[k] = fold(a[k], c[k], r0); b[k] = fold(b[k], d[k], r0); }
        add_pair<NT, SIMPLE>(acc[1], a, b, tm, false);
#pragma unroll
        for (int k = 0; k < NT; ++k) tb.out[k][i] = fold(a[k], b[k], r1);
    }
    uint64_t v[2 * NPT];
#pragma unroll
    for (int x = 0; x < NPT; ++x) {
        v[x] = acc[0][x].value(sums_products<NT, SIMPLE>());
        v[NPT + x] = acc[1][x].value(sums_products<NT, SIMPLE>());
    }
    finish<2 * NPT>(v, sk);
}

// All remaining rounds (tables of at most 2^TAIL_LOG entries) in one block.  A thread folds into the entry that it alone
// reads, and the warp sums of a round go to one of two buffers, so one barrier per round separates everything.
struct Coins { uint64_t c[TAIL_LOG]; };
template <int NT, bool SIMPLE>
__global__ void __launch_bounds__(TAIL_BLOCK) k_tail(Tables tb, Terms tm, int size, const __grid_constant__ Coins coins,
                                                     int first, Sink sk) {
    constexpr int WARPS = TAIL_BLOCK / 32;
    extern __shared__ uint64_t tab[];                   // [table][entry]
    __shared__ uint32_t red[2][WARPS][NPT * 3];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int e = tid; e < size; e += TAIL_BLOCK)
#pragma unroll
        for (int k = 0; k < NT; ++k) tab[k * size + e] = tb.in[k][e];
    __syncthreads();
    int rnd = 0;
    for (int half = size / 2; half >= 1; half >>= 1, ++rnd) {
        const uint64_t r = coins.c[rnd];
        const bool one = first && rnd == 0;
        Acc acc[NPT];
#pragma unroll
        for (int x = 0; x < NPT; ++x) acc[x].clear();
        for (int i = tid; i < half; i += TAIL_BLOCK) {
            uint64_t lo[NT], hi[NT];
#pragma unroll
            for (int k = 0; k < NT; ++k) { lo[k] = tab[k * size + i]; hi[k] = tab[k * size + i + half]; }
            add_pair<NT, SIMPLE>(acc, lo, hi, tm, one);
#pragma unroll
            for (int k = 0; k < NT; ++k) tab[k * size + i] = fold(lo[k], hi[k], r);
        }
        if (wid * 32 < half || wid == 0) {
#pragma unroll
            for (int x = 0; x < NPT; ++x)
                put_pieces(&red[rnd & 1][wid][3 * x], acc[x].value(sums_products<NT, SIMPLE>()), lane);
        } else if (lane < NPT * 3) {
            red[rnd & 1][wid][lane] = 0;
        }
        __syncthreads();
        if (tid < NPT) sk.row0[(int64_t)rnd * ROW + tid] = sum_pieces<WARPS, NPT>(red[rnd & 1], tid);
    }
    if (tid < 32) {
        __threadfence_system();
        __syncwarp();
        if (tid == 0 && sk.flag) *sk.flag = sk.stamp;
    }
}


// ---- host side ----------------------------------------------------------------------------------------------------
// Mapped host memory for the sums and a device word for the ticket, each owned by one proof at a time and kept between
// proofs, at most SLOTS_KEPT idle ones per device: a proof of hundreds of tables has a session for every eight of them.
// release_sumcheck_slots() returns them to the driver.  (In blocks of 32 the first 130 sessions took 424 ms instead of 49: a
// pinned allocation of 100 KB takes far longer than 32 of 3 KB.)
struct Slot {
    int device;
    uint64_t* host;          // MAX_ROUNDS rows, then the flag
    uint64_t* dev;           // its device address
    unsigned* ticket;
    uint64_t stamp;
    Slot* next;              // in the list of idle ones
};
constexpr size_t SLOT_WORDS = (size_t)MAX_ROUNDS * ROW + 8;
constexpr int SLOTS_KEPT = 256;
std::mutex g_slot_mu;
Slot* g_slots = nullptr;

void free_slot(Slot* s) {
    cudaFreeHost(s->host);
    cudaFree(s->ticket);
    delete s;
}
int take_slot(Slot** out) {
    int dev;
    VI_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lk(g_slot_mu);
        for (Slot** at = &g_slots; *at; at = &(*at)->next)
            if ((*at)->device == dev) {
                *out = *at;
                *at = (*at)->next;
                return VI_OK;
            }
    }
    Slot* s = new (std::nothrow) Slot{dev, nullptr, nullptr, nullptr, 0, nullptr};
    if (!s) return vi::fail(VI_ERR_CUDA, "sumcheck: out of host memory");
    cudaError_t e = cudaHostAlloc((void**)&s->host, SLOT_WORDS * 8, cudaHostAllocMapped | cudaHostAllocPortable);
    if (e == cudaSuccess) { memset(s->host, 0, SLOT_WORDS * 8); e = cudaHostGetDevicePointer((void**)&s->dev, s->host, 0); }
    if (e == cudaSuccess) e = cudaMalloc((void**)&s->ticket, 256);
    if (e == cudaSuccess) e = cudaMemset(s->ticket, 0, 256);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();      // the clear is ordered before launches on any stream
    if (e != cudaSuccess) {
        if (s->host) cudaFreeHost(s->host);
        if (s->ticket) cudaFree(s->ticket);
        delete s;
        return vi::fail(VI_ERR_CUDA, "sumcheck: result buffer: %s", cudaGetErrorString(e));
    }
    *out = s;
    return VI_OK;
}
void give_slot(Slot* s) {
    {
        std::lock_guard<std::mutex> lk(g_slot_mu);
        int n = 0;
        for (Slot* o = g_slots; o; o = o->next) n += o->device == s->device;
        if (n < SLOTS_KEPT) { s->next = g_slots; g_slots = s; return; }
    }
    free_slot(s);
}

// Waits for the stamp: polls the flag (a launch's sums are some microseconds away), then lets the driver wait.
int wait_stamp(Slot* s, cudaStream_t st) {
    auto* flag = reinterpret_cast<std::atomic<uint64_t>*>(s->host + (size_t)MAX_ROUNDS * ROW);
    for (int i = 0; i < 200000; ++i) {
        if (flag->load(std::memory_order_acquire) == s->stamp) return VI_OK;
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
    }
    VI_CUDA(cudaStreamSynchronize(st));
    if (flag->load(std::memory_order_acquire) == s->stamp) return VI_OK;
    return vi::fail(VI_ERR_CUDA, "sumcheck: the launch ended without its sums");
}

struct Problem {
    Terms tm;
    Tables tb;
    int nt;
    bool simple;
};

int make_problem(Problem& pb, const uint64_t* const* tabs, int n_tables, int n_terms, const uint64_t* coefs, const int32_t* nfac,
                 const int32_t* fac) {
    VI_REQUIRE(n_tables >= 1 && n_tables <= MAX_TABLES, "sumcheck: 1..%d tables supported (got %d)", MAX_TABLES, n_tables);
    VI_REQUIRE(n_terms >= 1 && n_terms <= MAX_TERMS, "sumcheck: 1..%d terms supported (got %d)", MAX_TERMS, n_terms);
    VI_REQUIRE(tabs && coefs && nfac && fac, "sumcheck: null pointer");
    memset(&pb, 0, sizeof(pb));
    pb.nt = n_tables;
    for (int k = 0; k < n_tables; ++k) {
        VI_REQUIRE(tabs[k] != nullptr, "sumcheck: null table");
        pb.tb.in[k] = tabs[k];
    }
    Terms& tm = pb.tm;
    tm.n = n_terms;
    for (int t = 0; t < n_terms; ++t) {
        VI_REQUIRE(nfac[t] >= 1 && nfac[t] <= MAX_FAC, "sumcheck: a term needs 1..%d factors", MAX_FAC);
        VI_REQUIRE(coefs[t] < vgl::P, "sumcheck: coefficient not canonical");
        tm.coef[t] = coefs[t];
        tm.sign[t] = coefs[t] == 1 ? 1 : coefs[t] == vgl::P - 1 ? -1 : 0;
        tm.nfac[t] = nfac[t];
        if (nfac[t] > tm.deg) tm.deg = nfac[t];
        for (int j = 0; j < nfac[t]; ++j) {
            const int k = fac[t * MAX_FAC + j];
            VI_REQUIRE(k >= 0 && k < n_tables, "sumcheck: factor index out of range");
            tm.count[t] += 1u << (4 * k);
        }
    }
    pb.simple = n_terms == 1 && coefs[0] == 1 && nfac[0] == n_tables && tm.count[0] == 0x11111111u >> (32 - 4 * n_tables);
    return VI_OK;
}

int grid_for(int64_t items, int cap) {
    const int64_t g = (items + BLOCK - 1) / BLOCK;
    return (int)(g < 1 ? 1 : g < cap ? g : cap);
}

enum { K_ROUND, K_FOLD_ROUND, K_ROUND2, K_TAIL };
struct Launch { int kind; int64_t size; uint64_t r0, r1; int first; const Coins* coins; };
template <int NT, bool SIMPLE>
int launch_t(const Problem& pb, const Launch& l, const Sink& sk, cudaStream_t st) {
    switch (l.kind) {
        case K_ROUND: k_round<NT, SIMPLE, false><<<grid_for(l.size / 2, MAX_GRID), BLOCK, 0, st>>>(pb.tb, pb.tm, l.size, 0, sk); break;
        case K_FOLD_ROUND: k_round<NT, SIMPLE, true><<<grid_for(l.size / 4, MAX_GRID), BLOCK, 0, st>>>(pb.tb, pb.tm, l.size, l.r0, sk); break;
        case K_ROUND2: k_round2<NT, SIMPLE><<<grid_for(l.size / 4, MAX_GRID / 2), BLOCK, 0, st>>>(pb.tb, pb.tm, l.size, l.r0, l.r1, l.first, sk); break;
        default: {
            const int smem = NT * (int)l.size * 8;
            if (smem > 40 * 1024)
                VI_CUDA(cudaFuncSetAttribute(k_tail<NT, SIMPLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, NT * (8 << TAIL_LOG)));
            k_tail<NT, SIMPLE><<<1, TAIL_BLOCK, smem, st>>>(pb.tb, pb.tm, (int)l.size, *l.coins, l.first, sk);
        }
    }
    return vi::check_launch("sumcheck");
}
int launch(const Problem& pb, const Launch& l, const Sink& sk, cudaStream_t st) {
    vi::ProfScope prof(vi::PROF_SUMCHECK, st);
    if (pb.simple) {
        switch (pb.nt) {
            case 1: return launch_t<1, true>(pb, l, sk, st);
            case 2: return launch_t<2, true>(pb, l, sk, st);
            case 3: return launch_t<3, true>(pb, l, sk, st);
            case 4: return launch_t<4, true>(pb, l, sk, st);
        }
    }
    switch (pb.nt) {
#define VI_CASE(x) case x: return launch_t<x, false>(pb, l, sk, st);
        VI_CASE(1) VI_CASE(2) VI_CASE(3) VI_CASE(4) VI_CASE(5) VI_CASE(6) VI_CASE(7) VI_CASE(8)
#undef VI_CASE
    }
    return vi::fail(VI_ERR_ARG, "sumcheck: table count");
}

// Round polynomial from its sums: coefficients c[0..deg], samples out[0..deg].  row: values at 0, 1, infinity, -1, 2;
// with a polynomial before it the value at 1 is claim - row[0].
uint64_t hadd(uint64_t a, uint64_t b) { return vgl::add_c(a, b); }
uint64_t hsub(uint64_t a, uint64_t b) { return vgl::sub_c(a, b); }
void round_poly(const volatile uint64_t* row, int deg, bool first, uint64_t claim, uint64_t* c, uint64_t* out) {
    const uint64_t P = vgl::P, inv2 = (P + 1) / 2, inv3 = 12297829379609722881ull;        // 3 * inv3 = 2p + 1
    auto word = [&](int i) { const uint64_t v = row[i]; return v >= P ? v - P : v; };
    const uint64_t g0 = word(0), g1 = first ? word(1) : hsub(claim, g0);
    for (int i = 0; i <= 4; ++i) c[i] = 0;
    c[0] = g0;
    if (deg == 1) c[1] = hsub(g1, g0);
    else if (deg == 2) { c[2] = word(2); c[1] = hsub(hsub(g1, g0), c[2]); }
    else {
        const uint64_t lead = word(2), gm = word(3);
        const uint64_t even = vgl::hmul(hadd(g1, gm), inv2), odd = vgl::hmul(hsub(g1, gm), inv2);   // c0+c2+c4, c1+c3
        c[2] = hsub(even, g0);
        c[3] = lead;
        if (deg == 4) {
            c[4] = lead;
            c[2] = hsub(c[2], lead);
            // (g(2) - c0 - 4 c2 - 16 c4) / 2 = c1 + 4 c3
            const uint64_t t = hsub(hsub(hsub(word(4), g0), vgl::hmul(4, c[2])), vgl::hmul(16, lead));
            c[3] = vgl::hmul(hsub(vgl::hmul(t, inv2), odd), inv3);
        }
        c[1] = hsub(odd, c[3]);
    }
    for (int x = 0; x <= deg; ++x) {
        uint64_t v = 0;
        for (int i = deg; i >= 0; --i) v = hadd(vgl::hmul(v, (uint64_t)x), c[i]);
        out[x] = v;
    }
}
uint64_t poly_at(const uint64_t* c, int deg, uint64_t r) {
    uint64_t v = 0;
    for (int i = deg; i >= 0; --i) v = hadd(vgl::hmul(v, r), c[i]);
    return v;
}

constexpr int64_t PARTIAL_BYTES = (int64_t)MAX_GRID * 2 * NPT * 8;

struct Session {
    Problem pb;
    int64_t size;
    uint64_t *work, *partials;
    Slot* slot;
    cudaStream_t st;
    bool own;                // the tables are copied by the first step and folded in place
    bool seen;
    bool failed;             // a launch may not have ended: the slot is not used again
    uint64_t c[NPT];
};

}  // namespace

namespace vi {
void release_sumcheck_slots() {
    std::lock_guard<std::mutex> lk(g_slot_mu);
    while (g_slots) {
        Slot* s = g_slots;
        g_slots = s->next;
        free_slot(s);
    }
}
}  // namespace vi

extern "C" int64_t vi_sumcheck_prove_work_bytes(int n_tables, int64_t size) {
    if (n_tables <= 0 || size <= 0) return 0;
    return PARTIAL_BYTES + (size > (int64_t(1) << TAIL_LOG) ? n_tables * (size / 4) * 8 : 0);
}

extern "C" int vi_sumcheck_prove(const uint64_t* const* tables, int n_tables, int64_t size, int n_terms, const uint64_t* coefs,
                                 const int32_t* nfac, const int32_t* fac, const uint64_t* coins, int n_rounds, void* work,
                                 int64_t work_bytes, uint64_t* samples_host, void* stream) {
    Problem pb;
    int rc = make_problem(pb, tables, n_tables, n_terms, coefs, nfac, fac);
    if (rc) return rc;
    VI_REQUIRE(n_rounds >= 0 && n_rounds <= MAX_ROUNDS && size == int64_t(1) << n_rounds, "sumcheck: size must be 2^n_rounds");
    if (n_rounds == 0) return VI_OK;
    VI_REQUIRE(coins && samples_host, "sumcheck: null pointer");
    for (int i = 0; i < n_rounds; ++i) VI_REQUIRE(coins[i] < vgl::P, "sumcheck: challenge not canonical");
    if (work == nullptr || work_bytes < vi_sumcheck_prove_work_bytes(n_tables, size))
        return vi::fail(VI_ERR_SCRATCH, "sumcheck: work buffer of at least %lld bytes required",
                        (long long)vi_sumcheck_prove_work_bytes(n_tables, size));
    cudaStream_t st = (cudaStream_t)stream;
    Slot* slot;
    rc = take_slot(&slot);
    if (rc) return rc;
    Sink sk{(uint64_t*)work, slot->ticket, nullptr, nullptr, nullptr, ++slot->stamp};
    uint64_t* buf = (uint64_t*)((char*)work + PARTIAL_BYTES);
    int rnd = 0;
    int64_t cur = size;
    while (cur > (int64_t(1) << TAIL_LOG) && !rc) {
        for (int k = 0; k < n_tables; ++k) pb.tb.out[k] = buf + k * (size / 4);
        sk.row0 = slot->dev + (size_t)rnd * ROW;
        sk.row1 = sk.row0 + ROW;
        rc = launch(pb, Launch{K_ROUND2, cur, coins[rnd], coins[rnd + 1], rnd == 0, nullptr}, sk, st);
        for (int k = 0; k < n_tables; ++k) pb.tb.in[k] = pb.tb.out[k];
        cur /= 4;
        rnd += 2;
    }
    if (!rc) {
        Coins tc{};
        for (int i = rnd; i < n_rounds; ++i) tc.c[i - rnd] = coins[i];
        sk.row0 = slot->dev + (size_t)rnd * ROW;
        sk.flag = slot->dev + (size_t)MAX_ROUNDS * ROW;
        rc = launch(pb, Launch{K_TAIL, cur, 0, 0, rnd == 0, &tc}, sk, st);
    }
    if (rc) {                      // earlier launches may still write the slot: it is not used again
        cudaStreamSynchronize(st);
        free_slot(slot);
        return rc;
    }
    rc = wait_stamp(slot, st);
    if (rc) return rc;
    uint64_t c[NPT], claim = 0;
    for (int i = 0; i < n_rounds; ++i) {
        round_poly(slot->host + (size_t)i * ROW, pb.tm.deg, i == 0, claim, c, samples_host + (size_t)i * ROW);
        claim = poly_at(c, pb.tm.deg, coins[i]);
    }
    give_slot(slot);
    return VI_OK;
}

extern "C" int64_t vi_sumcheck_session_work_bytes(int n_tables, int64_t size) {
    if (n_tables <= 0 || size <= 0) return 0;
    return PARTIAL_BYTES + n_tables * (size / 2) * 8;
}
extern "C" int64_t vi_sumcheck_session_work_bytes_own(int n_tables, int64_t size) {
    if (n_tables <= 0 || size <= 0) return 0;
    return PARTIAL_BYTES + n_tables * size * 8;
}

extern "C" int vi_sumcheck_open(const uint64_t* const* tables, int n_tables, int64_t size, int n_terms, const uint64_t* coefs,
                                const int32_t* nfac, const int32_t* fac, void* work, int64_t work_bytes, void* stream, void** session) {
    VI_REQUIRE(session != nullptr, "sumcheck: null pointer");
    VI_REQUIRE(vi::is_pow2(size) && size >= 2, "sumcheck: table size must be a power of two >= 2");
    if (work == nullptr || work_bytes < vi_sumcheck_session_work_bytes(n_tables, size))
        return vi::fail(VI_ERR_SCRATCH, "sumcheck: work buffer of at least %lld bytes required",
                        (long long)vi_sumcheck_session_work_bytes(n_tables, size));
    Session* s = new (std::nothrow) Session{};
    if (!s) return vi::fail(VI_ERR_CUDA, "sumcheck: out of host memory");
    int rc = make_problem(s->pb, tables, n_tables, n_terms, coefs, nfac, fac);
    if (!rc) rc = take_slot(&s->slot);
    if (rc) { delete s; return rc; }
    s->size = size;
    s->partials = (uint64_t*)work;
    s->work = (uint64_t*)((char*)work + PARTIAL_BYTES);
    s->own = work_bytes >= vi_sumcheck_session_work_bytes_own(n_tables, size);
    s->st = (cudaStream_t)stream;
    *session = s;
    return VI_OK;
}

extern "C" int vi_sumcheck_step(void* session, uint64_t r, uint64_t* samples_host) {
    VI_REQUIRE(session && samples_host, "sumcheck: null pointer");
    Session* s = (Session*)session;
    VI_REQUIRE(!s->seen || r < vgl::P, "sumcheck: challenge not canonical");
    VI_REQUIRE(!s->seen || s->size >= 4, "sumcheck: no round left");
    Slot* slot = s->slot;
    int dev;
    VI_CUDA(cudaGetDevice(&dev));
    VI_REQUIRE(dev == slot->device, "sumcheck: the session was opened on device %d, device %d is current", slot->device, dev);
    Sink sk{s->partials, slot->ticket, slot->dev, nullptr, slot->dev + (size_t)MAX_ROUNDS * ROW, ++slot->stamp};
    if (s->seen || s->own)      // from where the first launch that writes tables puts them, each stays in place
        for (int k = 0; k < s->pb.nt; ++k)
            if (!s->pb.tb.out[k]) s->pb.tb.out[k] = s->work + k * (s->own ? s->size : s->size / 2);
    int rc = launch(s->pb, Launch{s->seen ? K_FOLD_ROUND : K_ROUND, s->size, r, 0, 0, nullptr}, sk, s->st);
    if (!rc) rc = wait_stamp(slot, s->st);
    if (rc) { s->failed = true; return rc; }
    const int deg = s->pb.tm.deg;
    round_poly(slot->host, deg, !s->seen, s->seen ? poly_at(s->c, deg, r) : 0, s->c, samples_host);
    if (s->seen) s->size /= 2;
    if (s->seen || s->own)
        for (int k = 0; k < s->pb.nt; ++k) s->pb.tb.in[k] = s->pb.tb.out[k];
    s->seen = true;
    return VI_OK;
}

extern "C" int vi_sumcheck_close(void* session) {
    if (!session) return VI_OK;
    Session* s = (Session*)session;
    if (!s->failed) give_slot(s->slot);
    delete s;
    return VI_OK;
}
