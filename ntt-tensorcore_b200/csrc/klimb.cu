// klimb.cu -- the K-limb forward NTT (residues of K x 24-bit limbs in
// Montgomery form, the reference's DScalar<K> layout) behind
// nttb_klimb_forward.
//
// The transform is the radix-2 decimation-in-time network of the reference's
// host_ntt_naive (include/ntt_arbitrary.cuh:2651-2676) applied in the
// Montgomery domain: bit-reverse, then for stage s = 0..log_n-1 the butterfly
// (a[i], a[i + 2^s]) <- (u + t, u - t), t = a[i + 2^s] * tw[k * n / 2^(s+1)],
// k = i mod 2^s.  The network is reproduced stage for stage (not replaced by
// another DFT factorisation) because the reference's K = 2 field is not a
// field with the advertised root of unity, so only the network itself defines
// the result there.
//
// Execution: a transform that fits one tile is one launch.  Above, the first
// pass takes the bit reversal and the first h stages together: with the index
// split as (a, b, c), a the high and c the low h bits, the block of middle
// value b owns the 2^h x 2^h tiles of b and rev(b), which swap places, so that
// the pass runs in place without a workspace.  The other passes run r
// consecutive stages s0 .. s0 + r - 1 on tiles of 2^logC columns x 2^r elements,
// column (G, low) = { G 2^(s0+r) + j 2^s0 + low }, consecutive `low` values.
//
// A stage of a small transform is one butterfly per thread and at most one warp
// per scheduler (2^15 elements: 512 warps on 592 schedulers), so its time is that
// of one product.  Residues are therefore repacked in shared memory: K = 11 limbs
// of a modulus below 2^254 into eight 32-bit words (136 wide multiply-adds per
// product instead of 253, and no masking), K = 3 limbs of one below 2^64 into two.
// Montgomery radix and limb count differ by 2^8 there (2^264 against 2^256, 2^72
// against 2^64); a root is divided by 2^8 mod p as it is loaded.  Other moduli
// stay on the 24-bit limbs.
// Measured: one product, a warp alone on its scheduler, 832 cycles (544 of them the
// multiplier's); K = 11 at 2^15 63.6 -> 18.2 us, at 2^17 156 -> 47, at 2^18 305 -> 75;
// K = 3 at 2^15 26 -> 10 (the host), at 2^20 175 -> 68 (24-bit limbs, radix-2 sweeps of gathered
// roots behind a bit reversal of its own before).
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/ntt_b200.h"
#include "../../include/ntt_limb_arith.cuh"
#include "bounds.cuh"
#include "engines.hpp"
#include "klimb_plan.hpp"
#include "profiler.hpp"
#include "radix_host.cuh"

namespace nttb {
namespace {

#if NTTB_DEBUG_BOUNDS
__device__ uint32_t g_klimb_bounds;
// w < p, words from the lowest up
template <int W>
__device__ __forceinline__ bool below(const uint32_t* w, const uint32_t* p) {
    bool lt = false;
    for (int i = 0; i < W; i++) lt = w[i] != p[i] ? w[i] < p[i] : lt;
    return lt;
}
#endif

// ------------------------------------------------------------ residue forms
// Each form: W words per element in shared memory, load / store between them
// and the K limbs in memory, root() of a loaded twiddle, the butterfly, and
// finish() to the canonical value in [0, p).

// K limbs of 24 bits, as in memory: any odd modulus
template <int K_>
struct LimbForm {
    static constexpr int K = K_, W = K_;
    uint32_t p[W], np;
    __device__ __forceinline__ static void unpack(uint32_t* w, const uint32_t* l) {
#pragma unroll
        for (int k = 0; k < K; k++) w[k] = l[k];
    }
    __device__ __forceinline__ static void pack(uint32_t* l, const uint32_t* w) { unpack(l, w); }
    __device__ __forceinline__ void root(uint32_t* w, const uint32_t* l) const { unpack(w, l); }
    // ONE: the block is the whole launch.  Its one warp or so waits for each of the
    // modulus's limbs read from the parameters (K = 11 at 2^6 18.1 us a call), so they
    // are kept in registers (15.5); more warps hide that and lose 1 - 3 % by it.
    template <bool ONE>
    __device__ __forceinline__ void butterfly(uint32_t* u, uint32_t* v, const uint32_t* w) const {
        uint32_t x[W], d[W], q[W];
#pragma unroll
        for (int k = 0; k < K; k++) {
            if constexpr (ONE) asm("mov.u32 %0, %1;" : "=r"(q[k]) : "r"(p[k]));
            else q[k] = p[k];
        }
        nttb_limb::mont_mul<K>(x, v, w, q, np);
        nttb_limb::sub_mod<K>(d, u, x, q);
        nttb_limb::add_mod<K>(u, u, x, q);
        unpack(v, d);
    }
    __device__ __forceinline__ void finish(uint32_t* w) const {
        (void)NTTB_CHECK(g_klimb_bounds, kBoundsResidue, below<W>(w, p));
    }
};

// 24-bit limbs <-> 32-bit words (W words hold the value: its limbs above are 0)
template <int K, int W>
struct Words {
    __device__ __forceinline__ static void unpack(uint32_t* w, const uint32_t* l) {
#pragma unroll
        for (int i = 0; i < W; i++) {
            const int f = 32 * i / 24, sh = 32 * i % 24;  // word i starts at bit sh of limb f
            uint32_t v = (l[f] >> sh) | (l[f + 1] << (24 - sh));
            if (48 - sh < 32) v |= l[f + 2] << (48 - sh);
            w[i] = v;
        }
    }
    __device__ __forceinline__ static void pack(uint32_t* l, const uint32_t* w) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int f = 24 * k / 32, sh = 24 * k % 32;
            uint32_t v = f < W ? w[f] >> sh : 0u;
            if (sh > 8 && f + 1 < W) v |= w[f + 1] << (32 - sh);
            l[k] = v & nttb_limb::kMask;
        }
    }
};

// K = 11, p < 2^254: eight words, Montgomery radix 2^256
struct Form256 : Words<11, 8> {
    static constexpr int K = 11, W = 8;
    uint32_t p[W], p2[W], np;  // p, 2p, np = -p^-1 mod 2^32

    // w 2^-8 mod p: (w + m p) / 2^8, m = -w p^-1 mod 2^8, below p
    __device__ __forceinline__ void root(uint32_t* w, const uint32_t* l) const {
        unpack(w, l);
        const uint32_t m = (w[0] * np) & 255u;
        uint64_t c = 0;
        uint32_t lo = 0;
#pragma unroll
        for (int i = 0; i < W; i++) {
            c += (uint64_t)m * p[i] + w[i];
            if (i > 0) w[i - 1] = __funnelshift_r(lo, (uint32_t)c, 8);
            lo = (uint32_t)c;
            c >>= 32;
        }
        w[W - 1] = __funnelshift_r(lo, (uint32_t)c, 8);
    }

    // e[0..7] += (x0, x2, x4, x6) y, the carry out of word 7 into top
    __device__ __forceinline__ static void mad_even(uint32_t* e, uint32_t x0, uint32_t x2, uint32_t x4, uint32_t x6,
                                                    uint32_t y, uint32_t& top) {
        asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\tmadc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\tmadc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\tmadc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\tmadc.hi.cc.u32 %7, %12, %13, %7;\n\t"
            "addc.u32 %8, %8, 0;"
            : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(top)
            : "r"(x0), "r"(x2), "r"(x4), "r"(x6), "r"(y));
    }
    // o[0..7] += (x1, x3, x5, x7) y + carry of (e0 += in): in lies one word below o
    __device__ __forceinline__ static void mad_odd_in(uint32_t* o, uint32_t& e0, uint32_t in, uint32_t x1, uint32_t x3,
                                                      uint32_t x5, uint32_t x7, uint32_t y) {
        asm("add.cc.u32 %8, %8, %14;\n\t"
            "madc.lo.cc.u32 %0, %9, %13, %0;\n\tmadc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\tmadc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\tmadc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\tmadc.hi.u32 %7, %12, %13, %7;"
            : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(e0)
            : "r"(x1), "r"(x3), "r"(x5), "r"(x7), "r"(y), "r"(in));
    }
    // o[0..7] += (x1, x3, x5, x7) y
    __device__ __forceinline__ static void mad_odd(uint32_t* o, uint32_t x1, uint32_t x3, uint32_t x5, uint32_t x7,
                                                   uint32_t y) {
        asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\tmadc.hi.cc.u32 %1, %8, %12, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\tmadc.hi.cc.u32 %3, %9, %12, %3;\n\t"
            "madc.lo.cc.u32 %4, %10, %12, %4;\n\tmadc.hi.cc.u32 %5, %10, %12, %5;\n\t"
            "madc.lo.cc.u32 %6, %11, %12, %6;\n\tmadc.hi.u32 %7, %11, %12, %7;"
            : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7])
            : "r"(x1), "r"(x3), "r"(x5), "r"(x7), "r"(y));
    }

    // x = a b 2^-256 mod p in [0, 2p) for a < p, b < 2^256, by coarsely integrated
    // operand scanning (Koc, Acar, Kaliski, "Analyzing and comparing Montgomery
    // multiplication algorithms", IEEE Micro 1996).  The running sum is kept
    // as two columns of word pairs, e at word 0 and o at word 1: each product row is
    // two independent carry chains of four wide multiply-adds.  Per round
    // t += a b_i + m p, t / 2^32: the columns change roles and e[1] moves down to the
    // new e[0].  With t < 2p before a round, t + (a + p)(2^32 - 1) < 2^32 2p < 2^288:
    // o[7] does not overflow.
    __device__ __forceinline__ void mul(uint32_t* x, const uint32_t* a, const uint32_t* b) const {
        uint32_t e[8] = {0, 0, 0, 0, 0, 0, 0, 0}, o[8] = {0, 0, 0, 0, 0, 0, 0, 0}, in = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            mad_odd_in(o, e[0], in, a[1], a[3], a[5], a[7], b[i]);
            mad_even(e, a[0], a[2], a[4], a[6], b[i], o[7]);
            const uint32_t m = e[0] * np;
            mad_odd(o, p[1], p[3], p[5], p[7], m);
            mad_even(e, p[0], p[2], p[4], p[6], m, o[7]);
            in = e[1];
            uint32_t t[8];
#pragma unroll
            for (int j = 0; j < 8; j++) t[j] = o[j];
#pragma unroll
            for (int j = 0; j < 6; j++) o[j] = e[j + 2];
            o[6] = o[7] = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) e[j] = t[j];
        }
        // e + in + 2^32 o
        asm("add.cc.u32 %0, %0, %8;\n\taddc.cc.u32 %1, %1, %9;\n\taddc.cc.u32 %2, %2, %10;\n\t"
            "addc.cc.u32 %3, %3, %11;\n\taddc.cc.u32 %4, %4, %12;\n\taddc.cc.u32 %5, %5, %13;\n\t"
            "addc.cc.u32 %6, %6, %14;\n\taddc.u32 %7, %7, %15;"
            : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7])
            : "r"(in), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]));
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = e[i];
    }
    // r = a - b, 1 where it borrows
    __device__ __forceinline__ static uint32_t sub(uint32_t* r, const uint32_t* a, const uint32_t* b) {
        uint32_t br;
        asm("sub.cc.u32 %0, %9, %17;\n\tsubc.cc.u32 %1, %10, %18;\n\tsubc.cc.u32 %2, %11, %19;\n\t"
            "subc.cc.u32 %3, %12, %20;\n\tsubc.cc.u32 %4, %13, %21;\n\tsubc.cc.u32 %5, %14, %22;\n\t"
            "subc.cc.u32 %6, %15, %23;\n\tsubc.cc.u32 %7, %16, %24;\n\tsubc.u32 %8, 0, 0;"
            : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
              "=&r"(br)
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]),
              "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
        return br;
    }
    __device__ __forceinline__ static void add(uint32_t* r, const uint32_t* a, const uint32_t* b) {
        asm("add.cc.u32 %0, %8, %16;\n\taddc.cc.u32 %1, %9, %17;\n\taddc.cc.u32 %2, %10, %18;\n\t"
            "addc.cc.u32 %3, %11, %19;\n\taddc.cc.u32 %4, %12, %20;\n\taddc.cc.u32 %5, %13, %21;\n\t"
            "addc.cc.u32 %6, %14, %22;\n\taddc.u32 %7, %15, %23;"
            : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]),
              "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
    }
    // x = t where t < m, else t - m
    __device__ __forceinline__ static void reduce(uint32_t* x, const uint32_t* t, const uint32_t* m) {
        uint32_t d[8];
        const uint32_t borrow = sub(d, t, m);
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = borrow ? t[i] : d[i];
    }
    // Values between stages stay in [0, 4p): after the product one carry chain each.
    template <bool>
    __device__ __forceinline__ void butterfly(uint32_t* u, uint32_t* v, const uint32_t* w) const {
        uint32_t x[8], c[8], c2[8];
        reduce(c, u, p2);
        add(c2, c, p2);
        mul(x, w, v);
        add(u, c, x);
        sub(v, c2, x);
    }
    __device__ __forceinline__ void finish(uint32_t* w) const {
        reduce(w, w, p2);
        reduce(w, w, p);
        (void)NTTB_CHECK(g_klimb_bounds, kBoundsResidue, below<W>(w, p));
    }
};

// K = 3, p < 2^64: two words, Montgomery radix 2^64
struct Form64 : Words<3, 2> {
    static constexpr int K = 3, W = 2;
    uint64_t p, pinv;  // pinv = p^-1 mod 2^64

    __device__ __forceinline__ static uint64_t val(const uint32_t* w) { return w[0] | (uint64_t)w[1] << 32; }
    __device__ __forceinline__ static void put(uint32_t* w, uint64_t v) {
        w[0] = (uint32_t)v;
        w[1] = (uint32_t)(v >> 32);
    }
    __device__ __forceinline__ void root(uint32_t* w, const uint32_t* l) const {
        unpack(w, l);
        const uint64_t v = val(w), m = (0 - v * pinv) & 255u, lo = v + m * p;
        const uint64_t hi = __umul64hi(m, p) + (lo < v);
        put(w, (lo >> 8) | (hi << 56));
    }
    template <bool>
    __device__ __forceinline__ void butterfly(uint32_t* u, uint32_t* v, const uint32_t* w) const {
        const uint64_t a = val(v), b = val(w), c = val(u);
        const uint64_t hi = __umul64hi(a, b), q = __umul64hi(a * b * pinv, p);
        const uint64_t x = hi < q ? hi - q + p : hi - q;
        const uint64_t s = c + x;
        put(u, (s < c || s >= p) ? s - p : s);
        put(v, c < x ? c - x + p : c - x);
    }
    __device__ __forceinline__ void finish(uint32_t* w) const {
        (void)NTTB_CHECK(g_klimb_bounds, kBoundsResidue, val(w) < p);
    }
};

// ------------------------------------------------------------------- kernel
// Where a block's tile lies.  kWhole: the transform is one tile, its loads bit
// reversed.  kSwap: the tiles of middle values b and rev(b) (one tile where
// they agree), logC = h.  kStages: 2^logC columns of a group of 2^(s0 + r).
enum Where { kWhole, kSwap, kStages };

struct PassArgs {
    uint32_t* data;
    const uint32_t* tw;
    uint32_t log_n, s0, r, logC;
    bool vec_data, vec_tw;  // 16-byte accesses: aligned pointers, runs of whole 16 bytes
};

template <int B>
__device__ __forceinline__ void cp_async(uint32_t* dst, const uint32_t* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

template <class F, int WHERE, int MAXT>
__global__ void __launch_bounds__(MAXT) klimb_pass(const __grid_constant__ PassArgs g, const __grid_constant__ F f) {
    extern __shared__ __align__(16) uint32_t sm[];
    constexpr int K = F::K, W = F::W;
    const uint32_t log_n = g.log_n, r = g.r, tid = threadIdx.x;
    const uint32_t logC = WHERE == kStages ? g.logC : 0u, s0 = WHERE == kStages ? g.s0 : 0u;
    const uint32_t C = 1u << logC;
    uint32_t E = 1u << (r + logC);  // elements of the tile
    uint32_t low0 = 0, mid = 0, rmid = 0;
    size_t base = 0;
    if constexpr (WHERE == kSwap) {
        const uint32_t M = log_n - 2u * r;
        mid = blockIdx.x;
        rmid = M ? __brev(mid) >> (32u - M) : 0u;
        if (rmid < mid) return;
        E = (rmid == mid ? 1u : 2u) << (2u * r);
    } else if constexpr (WHERE == kStages) {
        const uint32_t chunks = (1u << s0) >> logC;  // column chunks per group
        low0 = (blockIdx.x % chunks) << logC;
        base = ((size_t)(blockIdx.x / chunks) << (s0 + r)) + low0;
    }
    // the tile between stages: word k of element e at k P + at(e); one spare word
    // after every 32 keeps the bit-reversed stores of the first stage off one bank
    const uint32_t P = E + (E >> 5);
    uint32_t* const roots = sm + E * K;
    uint32_t* const tile = roots + E * W;
#if NTTB_DEBUG_BOUNDS
    // every shared-memory index below is an element below E of one of the three arrays
    uint32_t dyn;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    if (!NTTB_CHECK(g_klimb_bounds, kBoundsShared, (E * (K + W) + P * W) * 4 <= dyn && E <= 2 * blockDim.x)) return;
#endif
    const size_t words = (size_t)K << log_n;  // of the data and of the table
    auto at = [](uint32_t e) { return e + (e >> 5); };
    auto sync = [] {
        if (blockDim.x <= 32) __syncwarp();
        else __syncthreads();
    };
    // element e of the tile in memory; `loading` gives where element `e` comes from
    auto place = [&](uint32_t e, bool loading) -> size_t {
        if constexpr (WHERE == kWhole) {
            return e;
        } else if constexpr (WHERE == kStages) {
            return base + ((size_t)(e >> logC) << s0) + (e & (C - 1));
        } else {
            const uint32_t mask = (1u << r) - 1, second = e >> (2u * r);
            const uint32_t m = (second != 0) == loading ? rmid : mid;  // tile 0 comes from mid and goes to rev(mid)
            return ((size_t)((e >> r) & mask) << (log_n - r)) + ((size_t)m << r) + (e & mask);
        }
    };
    // this thread's butterfly: pair number pi of column c
    const uint32_t c = tid & (C - 1), pi = tid >> logC;
    const bool busy = tid < E / 2;
    // The tile's roots, (2^t) C at stage t: gathered once, two per thread at most,
    // while the residues are on their way (a gather of 32 roots holds the load unit
    // for longer than a product takes).  16-byte loads where a root starts on such a
    // boundary (every fourth does); the words after the K-th belong to the next one.
    constexpr int RAW = K == 2 ? 2 : (K + 3) / 4 * 4;
    uint32_t raw[2][RAW];
    const uint32_t n_roots = ((1u << r) - 1) << logC;
    auto fetch_roots = [&] {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint32_t i = tid + q * blockDim.x, j1 = (i >> logC) + 1, t = 31 - __clz(j1);
            if (i >= n_roots) break;
            const uint32_t k = ((j1 - (1u << t)) << s0) + low0 + (i & (C - 1)), sh = log_n - s0 - t - 1;
            const size_t off = ((size_t)k << sh) * K;
            const bool wide = K > 2 && g.vec_tw && sh >= 2;
            if (!NTTB_CHECK(g_klimb_bounds, kBoundsGlobal, off + (wide ? RAW : K) <= words)) continue;
            const uint32_t* w = g.tw + off;
            if (wide) {
#pragma unroll
                for (int m = 0; m + 4 <= RAW; m += 4) {
                    const uint4* at = reinterpret_cast<const uint4*>(w + m);
                    const uint4 x = WHERE == kStages ? __ldg(at) : __ldcg(at);
                    raw[q][m] = x.x, raw[q][m + 1] = x.y, raw[q][m + 2] = x.z, raw[q][m + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int m = 0; m < K; m++) raw[q][m] = WHERE == kStages ? __ldg(w + m) : __ldcg(w + m);
            }
        }
    };
    // The table is older than the pass before this one, which waited for it; the
    // first pass of a transform has no such pass.  Its blocks may be older than the
    // table, so it reads past the read-only path, which asks for memory that does not
    // change while a grid is on the GPU.
    if constexpr (WHERE == kStages) fetch_roots();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (WHERE != kStages) fetch_roots();
    // Memory is read and written as runs of words (a warp's loads of one word of
    // 32 elements touch K lines each), by way of shared memory, where a stride of
    // K words is free of conflicts.
    if (g.vec_data) {
        for (uint32_t v = 4 * tid; v < E * K; v += 4 * blockDim.x) {
            const size_t i = place(v / K, true) * K + v % K;
            if (NTTB_CHECK(g_klimb_bounds, kBoundsGlobal, i + 4 <= words)) cp_async<16>(sm + v, g.data + i);
        }
    } else {
        for (uint32_t v = tid; v < E * K; v += blockDim.x) {
            const size_t i = place(v / K, true) * K + v % K;
            if (NTTB_CHECK(g_klimb_bounds, kBoundsGlobal, i < words)) cp_async<4>(sm + v, g.data + i);
        }
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const uint32_t i = tid + q * blockDim.x;
        if (i < n_roots) {
            uint32_t w[W];
            f.root(w, raw[q]);
#pragma unroll
            for (int k = 0; k < W; k++) roots[k * E + i] = w[k];
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    sync();
    for (uint32_t t = 0; t < r; t++) {
        const uint32_t half = 1u << t;
        if (busy) {
            uint32_t w[W], u[W], v[W], l[K];
            const uint32_t jlo = ((pi >> t) << (t + 1)) | (pi & (half - 1));
            uint32_t elo = (jlo << logC) + c, ehi = elo + (half << logC);
            if (t == 0) {  // from the loaded words: in bit-reversed order the pairs lie half a tile apart
                uint32_t from = elo, step = ehi - elo;
                if constexpr (WHERE != kStages) {
                    const uint32_t bits = WHERE == kWhole ? log_n : 2u * r, lo = tid & ((1u << (bits - 1)) - 1);
                    from = 2u * (tid - lo) + lo;
                    step = 1u << (bits - 1);
                    elo = 2u * (tid - lo) + (__brev(lo) >> (32u - bits));
                    ehi = elo + 1;
                }
#pragma unroll
                for (int k = 0; k < K; k++) l[k] = sm[from * K + k];
                F::unpack(u, l);
#pragma unroll
                for (int k = 0; k < K; k++) l[k] = sm[(from + step) * K + k];
                F::unpack(v, l);
            } else {
#pragma unroll
                for (int k = 0; k < W; k++) {
                    u[k] = tile[k * P + at(elo)];
                    v[k] = tile[k * P + at(ehi)];
                }
            }
            if (!NTTB_CHECK(g_klimb_bounds, kBoundsShared, elo < E && ehi < E)) elo = ehi = 0;
            const uint32_t* rt = roots + (((half - 1) + (pi & (half - 1))) << logC) + c;
            if (!NTTB_CHECK(g_klimb_bounds, kBoundsShared, rt < roots + E)) rt = roots;
#pragma unroll
            for (int k = 0; k < W; k++) w[k] = rt[k * E];
            f.template butterfly<WHERE == kWhole>(u, v, w);
            if (t + 1 < r) {
#pragma unroll
                for (int k = 0; k < W; k++) {
                    tile[k * P + at(elo)] = u[k];
                    tile[k * P + at(ehi)] = v[k];
                }
            } else {
                f.finish(u);
                F::pack(l, u);
#pragma unroll
                for (int k = 0; k < K; k++) sm[elo * K + k] = l[k];
                f.finish(v);
                F::pack(l, v);
#pragma unroll
                for (int k = 0; k < K; k++) sm[ehi * K + k] = l[k];
            }
        }
        sync();
    }
    if (g.vec_data) {
        for (uint32_t v = 4 * tid; v < E * K; v += 4 * blockDim.x) {
            const size_t i = place(v / K, false) * K + v % K;
            if (NTTB_CHECK(g_klimb_bounds, kBoundsGlobal, i + 4 <= words))
                *reinterpret_cast<uint4*>(g.data + i) = *reinterpret_cast<const uint4*>(sm + v);
        }
    } else {
        for (uint32_t v = tid; v < E * K; v += blockDim.x) {
            const size_t i = place(v / K, false) * K + v % K;
            if (NTTB_CHECK(g_klimb_bounds, kBoundsGlobal, i < words)) g.data[i] = sm[v];
        }
    }
}

// One butterfly per thread: `elements` / 2 threads.  A launch of up to four blocks an
// SM asks for the share of shared memory at which no more fit, so that blocks
// started early (behind a pass that is still draining) don't crowd some SMs.  us:
// K = 11 at 2^15 24.1 -> 18.4, K = 3 at 2^17 19.8 -> 15.3 (one block an SM); K = 11 at
// 2^17 67.8 -> 46.8, from 2^254 on 171 -> 133, K = 3 at 2^18 from 2^64 on 53.0 -> 40.0,
// K = 2 38.2 -> 26.7 (two to four).
template <class F, int WHERE>
int launch(const F& f, const PassArgs& g, uint32_t blocks, uint32_t elements, cudaStream_t s) {
    constexpr auto k = klimb_pass<F, WHERE, klimb_max_threads(F::K)>;
    rdx::kernel_smem<k, true>(kKlimbSmemMax);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(elements / 2);
    cfg.dynamicSmemBytes = klimb_smem_bytes(F::K, F::W, elements);
    if (blocks > 1) cfg.dynamicSmemBytes = rdx::spread_smem(blocks, cfg.dynamicSmemBytes, 1, 4);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ProfScope prof("klimb_pass", s);
    void* params[2] = {const_cast<PassArgs*>(&g), const_cast<F*>(&f)};
    return launch_rc(cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(k), params));
}

template <class F>
int klimb_forward(const F& f, uint32_t* d_data, const uint32_t* d_tw, uint32_t log_n, cudaStream_t s) {
    if (log_n == 0) return 0;  // the identity
    const uint32_t n = 1u << log_n;
    const KlimbPlan P = klimb_plan(F::K, log_n);
    const bool va = (reinterpret_cast<uintptr_t>(d_data) & 15) == 0, vt = (reinterpret_cast<uintptr_t>(d_tw) & 15) == 0;
    if (P.single_tile) return launch<F, kWhole>(f, {d_data, d_tw, log_n, 0, log_n, 0, va && log_n >= 2, vt}, 1, n, s);
    for (uint32_t i = 0; i < P.n_passes; i++) {
        const KlimbPass& ps = P.pass[i];
        const PassArgs g{d_data, d_tw, log_n, ps.s0, ps.r, ps.logC, va && (i == 0 || ps.logC >= 2), vt};
        const uint32_t elements = klimb_pass_elements(ps, i == 0);
        const int rc = i == 0 ? launch<F, kSwap>(f, g, n >> (2 * ps.r), elements, s)
                              : launch<F, kStages>(f, g, n / elements, elements, s);
        if (rc) return rc;
    }
    return 0;
}

template <int K>
int klimb_limbs(uint32_t* d_data, const uint32_t* d_tw, uint32_t log_n, const uint32_t* prime, uint32_t np,
                cudaStream_t s) {
    LimbForm<K> f;
    for (int k = 0; k < K; k++) f.p[k] = prime[k];
    f.np = np;
    return klimb_forward(f, d_data, d_tw, log_n, s);
}

int klimb3(uint32_t* d_data, const uint32_t* d_tw, uint32_t log_n, const uint32_t* prime, uint32_t np,
           cudaStream_t s) {
    if (prime[2] >> 16) return klimb_limbs<3>(d_data, d_tw, log_n, prime, np, s);  // p >= 2^64
    Form64 f;
    f.p = prime[0] | (uint64_t)prime[1] << 24 | (uint64_t)prime[2] << 48;
    f.pinv = f.p;  // inverse of an odd number mod 2^3; each step doubles the bits
    for (int i = 0; i < 5; i++) f.pinv *= 2u - f.p * f.pinv;
    return klimb_forward(f, d_data, d_tw, log_n, s);
}

int klimb11(uint32_t* d_data, const uint32_t* d_tw, uint32_t log_n, const uint32_t* prime, uint32_t np,
            cudaStream_t s) {
    if (prime[10] >> 14) return klimb_limbs<11>(d_data, d_tw, log_n, prime, np, s);  // p >= 2^254
    Form256 f;
    for (int i = 0; i < 8; i++) {
        const int l = 32 * i / 24, sh = 32 * i % 24;
        uint64_t v = prime[l] | (uint64_t)prime[l + 1] << 24;
        if (l + 2 < 11) v |= (uint64_t)prime[l + 2] << 48;
        f.p[i] = (uint32_t)(v >> sh);
        f.p2[i] = f.p[i] << 1 | (i > 0 ? f.p[i - 1] >> 31 : 0u);
    }
    f.np = f.p[0];
    for (int i = 0; i < 4; i++) f.np *= 2u - f.p[0] * f.np;
    f.np = 0u - f.np;
    return klimb_forward(f, d_data, d_tw, log_n, s);
}

}  // namespace

uint32_t klimb_bounds_errors(bool clear) {
    uint32_t v = 0;
#if NTTB_DEBUG_BOUNDS
    const uint32_t z = 0;
    cudaMemcpyFromSymbol(&v, g_klimb_bounds, sizeof v);
    if (clear) cudaMemcpyToSymbol(g_klimb_bounds, &z, sizeof z);
#else
    (void)clear;
#endif
    return v;
}

}  // namespace nttb

extern "C" {

NTTB_API int nttb_klimb_forward(uint32_t K, uint32_t* d_data, const uint32_t* d_tw, uint64_t n, uint32_t log_n,
                                const uint32_t* prime, uint32_t np, void* stream) {
    using nttb::fail;
    if (!d_data || !d_tw || !prime) return fail(NTTB_ERR_INVALID_ARG, "nttb_klimb_forward: null pointer");
    if (log_n > 24 || n != (1ull << log_n))
        return fail(NTTB_ERR_INVALID_ARG, "nttb_klimb_forward: n must be 2^log_n with log_n <= 24");
    if (K != 2 && K != 3 && K != 11)
        return fail(NTTB_ERR_UNSUPPORTED, "nttb_klimb_forward: K = %u (this build serves K = 2, 3, 11)", K);
    if ((prime[0] & 1u) == 0) return fail(NTTB_ERR_INVALID_ARG, "nttb_klimb_forward: even modulus");
    for (uint32_t k = 0; k < K; k++)
        if (prime[k] > nttb_limb::kMask) return fail(NTTB_ERR_INVALID_ARG, "nttb_klimb_forward: limb %u >= 2^24", k);
    if (np != nttb_limb::neg_inv24(prime[0]))
        return fail(NTTB_ERR_INVALID_ARG, "nttb_klimb_forward: np != -p^-1 mod 2^24");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = 0;
    switch (K) {
        case 2: rc = nttb::klimb_limbs<2>(d_data, d_tw, log_n, prime, np, s); break;
        case 3: rc = nttb::klimb3(d_data, d_tw, log_n, prime, np, s); break;
        default: rc = nttb::klimb11(d_data, d_tw, log_n, prime, np, s); break;
    }
    return rc ? fail(NTTB_ERR_CUDA, "nttb_klimb_forward: kernel launch failed") : NTTB_OK;
}

}  // extern "C"
