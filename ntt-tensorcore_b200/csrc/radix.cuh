// radix.cuh -- the register-radix NTT pass on CUDA cores: one kernel template
// for the single-pass transforms and for both passes of the two-pass ones.
//
// Network.  The forward transform runs the Cooley-Tukey butterflies of the
// ring splitting X^n -+ 1 (natural order in, bit-reversed positions): at
// stage s (m = 2^s blocks) block i multiplies by root^((n / 2m) (1 + 2 rev(i)))
// (negacyclic, root = psi) or root^((n / 2m) rev(i)) (cyclic, root = omega),
// so the twist and the four-step twiddles cost no products of their own.  The
// inverse is the same network backwards (Gentleman-Sande), n^-1 folded into
// its last stage.  Roots are Shoup pairs, tab[2^s + rev(i)]: natural order
// within a stage, so that neighbouring threads read neighbouring pairs.
//
// Two passes, n = N1 * N2, input index r N2 + c, output index k2 N1 + u:
//   forward  A: columns c of [N1][N2], stages 0 .. a-1 (the same roots for
//               every column), stored transposed: mid[c N1 + u];
//            B: columns u of [N2][N1], the remaining stages (roots of row u),
//               stored at the positions they were read from;
//   inverse  A: columns u of [N2][N1] (roots of row u), stored mid[u N2 + c];
//            B: columns c of [N1][N2] (the same roots for every column), in place.
// Pass B reads and writes one set of positions per tile, so `mid` may be the
// destination; pass A must not write over its source.
//
// Tile: V neighbouring columns of N = 2^LG elements, 2^LGE of them in the
// registers of a thread.  The stages run in register rounds of up to LGE
// stages; between rounds the tile is exchanged through shared memory, where
// element bit i has its own stride (Lay) chosen so that every round's loads
// and stores -- V columns x neighbouring positions, or 32 positions of one
// column -- fall into distinct banks without any address arithmetic per
// element.  A thread overwrites what it has read, so a round needs one barrier.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "arith.cuh"
#include "bounds.cuh"
#include "plan.hpp"

namespace nttb {
namespace rdx {

#if NTTB_DEBUG_BOUNDS
static __device__ uint32_t g_radix_bounds;  // one per file that includes this
#endif

struct Args {
    const void* src;
    void* dst;
    uint64_t poly_stride;  // words between consecutive polynomials
    uint32_t log_n;
    uint32_t polys;        // polynomials in all
    uint32_t polys_per_cta;
    uint32_t units;        // single pass: (polynomial, limb) rows
    uint32_t n_limbs;
};

__host__ __device__ constexpr uint32_t brv(uint32_t x, int bits) {
    uint32_t r = 0;
    for (int i = 0; i < bits; i++) r |= ((x >> i) & 1u) << (bits - 1 - i);
    return r;
}
__device__ __forceinline__ uint32_t brv_dev(uint32_t x, int bits) { return bits ? __brev(x) >> (32 - bits) : 0u; }

// Strides (in elements) of the LG position bits in shared memory; column v
// sits at offset v.  NB = log2 of the banks counted in elements (5 for 4-byte,
// 4 for 8-byte elements).  The NP bits next to either end, those that a warp's
// lanes enumerate, get distinct power-of-two residues mod 2^NB: first those
// above the V columns' own (lanes that run over columns, then positions), then
// the highest of the columns' (lanes that run over positions, then columns).
// Any order of one set does; the one taken keeps the padding below 13 % (a
// descending one took up to 50 %).
template <int LG, int LGV, int NB, int NP>
struct Lay {
    uint32_t s[LG > 0 ? LG : 1] = {};
    uint32_t words = 0;
    constexpr Lay() {
        uint32_t sum = (1u << LGV) - 1u;
        const uint32_t mod = 1u << NB;
        const int above = NB > LGV ? NB - LGV : 0;
        for (int i = 0; i < LG; i++) {
            const bool top = i >= LG / 2;
            const int pos = top ? LG - 1 - i : i;
            uint32_t st = sum + 1u;
            if (pos < NP) {
                const int bit = LGV == 0 && top && LG >= 2 * NB ? NB - 1 - pos : pos < above ? LGV + pos : NB - NP + pos - above;
                while ((st & (mod - 1u)) != (1u << bit)) st++;
            }
            s[i] = st;
            sum += st;
        }
        words = sum + 1u;
    }
};
template <class E>
constexpr int kBankBits = sizeof(E) == 8 ? 4 : 5;
// Lanes of the passes below: up to NB positions of one column.
template <class E, int LG, int LGV, int LGE>
constexpr int kLanePos = LGV == 0 || LG - LGE > kBankBits<E> ? kBankBits<E> : LG - LGE;

// Stages per round: the last takes LGE, the ones before it share the rest.
template <int LG, int LGE>
struct Rounds {
    int n = 0;
    int r[8] = {}, s0[8] = {};
    constexpr Rounds() {
        const int rest = LG - LGE, k = (rest + LGE - 1) / LGE;
        int done = 0;
        for (int i = 0; i < k; i++) {
            r[i] = (rest - done) / (k - i);
            s0[i] = done;
            done += r[i];
        }
        r[k] = LGE;
        s0[k] = rest;
        n = k + 1;
    }
};

template <class A>
struct PairOf;
template <>
struct PairOf<M32> { using type = uint2; };
template <>
struct PairOf<M64> { using type = ulonglong2; };

// min(x, x - q) on unsigned words: x - q when x >= q (x < 2q), one instruction.
__device__ __forceinline__ uint32_t sub_if(uint32_t x, uint32_t q) { return __viaddmin_u32(x, 0u - q, x); }

// Forward butterfly: M32 keeps values in [0, 2q) (q < 2^31), M64 in [0, 4q) (q < 2^62).
__device__ __forceinline__ void ct(const M32& ar, uint32_t& a, uint32_t& b, uint2 w) {
    const uint32_t u = sub_if(a, ar.q);
    const uint32_t t = sub_if(b * w.x - __umulhi(b, w.y) * ar.q, ar.q);
    a = u + t;
    b = u - t + ar.q;
}
__device__ __forceinline__ void ct(const M64& ar, uint64_t& a, uint64_t& b, ulonglong2 w) {
    const uint64_t u = ar.below2q(a);
    const uint64_t t = ar.mul_shoup_lazy(b, w.x, w.y);
    a = u + t;
    b = u - t + 2 * ar.q;
}
// Inverse butterfly: M32 keeps values in [0, q), M64 in [0, 2q).
__device__ __forceinline__ void gs(const M32& ar, uint32_t& a, uint32_t& b, uint2 w) {
    const uint32_t s = sub_if(a + b, ar.q), d = a - b + ar.q;
    a = s;
    b = sub_if(d * w.x - __umulhi(d, w.y) * ar.q, ar.q);
}
__device__ __forceinline__ void gs(const M64& ar, uint64_t& a, uint64_t& b, ulonglong2 w) {
    const uint64_t s = ar.below2q(a + b), d = a - b + 2 * ar.q;
    a = s;
    b = ar.mul_shoup_lazy(d, w.x, w.y);
}
// The inverse's last stage: both outputs times n^-1 (c = n^-1, w carries it too).
__device__ __forceinline__ void gs_scaled(const M32& ar, uint32_t& a, uint32_t& b, uint2 c, uint2 w) {
    const uint32_t s = a + b, d = a - b + ar.q;
    a = sub_if(s * c.x - __umulhi(s, c.y) * ar.q, ar.q);
    b = sub_if(d * w.x - __umulhi(d, w.y) * ar.q, ar.q);
}
__device__ __forceinline__ void gs_scaled(const M64& ar, uint64_t& a, uint64_t& b, ulonglong2 c, ulonglong2 w) {
    const uint64_t s = a + b, d = a - b + 2 * ar.q;
    a = ar.mul_shoup_lazy(s, c.x, c.y);
    b = ar.mul_shoup_lazy(d, w.x, w.y);
}
template <bool INV>
__device__ __forceinline__ uint32_t canon_out(const M32& ar, uint32_t x) { return INV ? x : sub_if(x, ar.q); }
template <bool INV>
__device__ __forceinline__ uint64_t canon_out(const M64& ar, uint64_t x) {
    return INV ? (x >= ar.q ? x - ar.q : x) : ar.canon4(x);
}

// Shoup pair from the constant tables; volatile, so that it is issued where it
// stands: a round's pairs are fetched before the barrier (or the wait for the
// previous grid) that its data waits for, when the data registers are free.
__device__ __forceinline__ uint2 ld_pair(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ ulonglong2 ld_pair(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

// Roots of round I: w[2^j - 1 + kt] for the round's stage j and block bits kt.
// `tw` points at tab + U (U the natural index of the thread's block at the
// round's first stage S): stage S + j, bits kt sit at 2^(S+j) + rev_j(kt) 2^S.
template <int LG, int LGE, int I, int S0, bool INV, int JJ = 0, class P>
__device__ __forceinline__ void round_roots(P (&w)[(1 << LGE) - 1], const P* tw) {
    constexpr Rounds<LG, LGE> R;
    constexpr int r = R.r[I], S = S0 + R.s0[I], j = INV ? r - 1 - JJ : JJ;
    if constexpr (!(INV && S + j == 0)) {  // the inverse's last stage multiplies by its scale
#pragma unroll
        for (uint32_t kt = 0; kt < (1u << j); kt++)
            w[(1u << j) - 1u + kt] = ld_pair(tw + ((size_t)1 << (S + j)) + ((size_t)brv(kt, j) << S));
    }
    if constexpr (JJ + 1 < r) round_roots<LG, LGE, I, S0, INV, JJ + 1>(w, tw);
}

// Stages of round I on the registers.  One instance per stage: as one loop nest
// the compiler kept the inverse's registers in local memory.
template <class A, int LG, int LGE, int I, int S0, bool INV, int JJ = 0, class E, class P>
__device__ __forceinline__ void round_stages(const A& ar, E (&x)[1 << LGE], const P (&w)[(1 << LGE) - 1], P c0, P c1) {
    constexpr Rounds<LG, LGE> R;
    constexpr int r = R.r[I], S = S0 + R.s0[I], xb = LGE - r;  // xb: extra held bits below the radix bits
    constexpr int j = INV ? r - 1 - JJ : JJ;
    constexpr uint32_t half = 1u << (r - 1 - j);
#pragma unroll
    for (uint32_t kt = 0; kt < (1u << j); kt++)
#pragma unroll
        for (uint32_t lo = 0; lo < half; lo++)
#pragma unroll
            for (uint32_t g = 0; g < (1u << xb); g++) {
                const uint32_t ia = (((kt << (r - j)) + lo) << xb) + g, ib = ia + (half << xb);
                if constexpr (INV && S + j == 0) gs_scaled(ar, x[ia], x[ib], c0, c1);
                else if constexpr (INV) gs(ar, x[ia], x[ib], w[(1u << j) - 1u + kt]);
                else ct(ar, x[ia], x[ib], w[(1u << j) - 1u + kt]);
            }
    if constexpr (JJ + 1 < r) round_stages<A, LG, LGE, I, S0, INV, JJ + 1>(ar, x, w, c0, c1);
}

// One round's place of a thread: its base offset in shared memory, and the
// natural index of its block within the pass.
template <class E, int LG, int LGV, int LGE, int I, int NP = kLanePos<E, LG, LGV, LGE>>
struct Place {
    static constexpr int NB = kBankBits<E>;
    static constexpr Rounds<LG, LGE> R{};
    static constexpr int s0 = R.s0[I], T = LG - s0, o = T - LGE;
    static constexpr bool last = I == R.n - 1;
    __device__ __forceinline__ static uint32_t base(uint32_t t) {
        constexpr Lay<LG, LGV, NB, NP> L;
        uint32_t a = 0;
#pragma unroll
        for (int b = 0; b < LG - LGE; b++) {
            // bits of t: low o bits are position bits 0 .. o-1, the others the
            // block (bit-reversed in the last round, whose t is the natural index)
            const int p = b < o ? b : last ? LG - 1 - (b - o) : T + (b - o);
            a += ((t >> b) & 1u) * L.s[p];
        }
        return a;
    }
    __device__ __forceinline__ static uint32_t natural(uint32_t t) {
        const uint32_t h = t >> o;
        return last ? h : brv_dev(h, s0);
    }
    static constexpr uint32_t reg(uint32_t e) {
        Lay<LG, LGV, NB, NP> L;
        uint32_t a = 0;
        for (int b = 0; b < LGE; b++) a += ((e >> b) & 1u) * L.s[o + b];
        return a;
    }
};

template <class Pl, bool ST, class E, int NE>
__device__ __forceinline__ void exchange(E* sm, E (&x)[NE]) {
#pragma unroll
    for (uint32_t e = 0; e < NE; e++) {
        if (ST) sm[Pl::reg(e)] = x[e];
        else x[e] = sm[Pl::reg(e)];
    }
}

template <int LG, int LGV, int LGE>
constexpr int kThreads = (1 << (LG + LGV - LGE)) > 128 ? (1 << (LG + LGV - LGE)) : 128;

// The rounds of one pass for a thread of a tile: where its registers sit before
// and after, the roots of a round (fetched ahead of the wait that the round's
// data needs), and the rounds.  TF: the first executed round's (else, TL, the
// last's) threads run over positions before columns, for contiguous columns in
// global memory.
template <class A, int LG, int LGV, int LGE, bool INV, int S0, bool TF, bool TL>
struct Pass {
    using E = typename A::elem;
    using P = typename PairOf<A>::type;
    static constexpr uint32_t N = 1u << LG, NE = 1u << LGE, V = 1u << LGV, NT = N >> LGE;
    static constexpr Rounds<LG, LGE> R{};
    static constexpr int NR = R.n;
    template <int K>
    static constexpr bool kT = (TF && K == 0) || (TL && K == NR - 1);
    template <int K>
    static constexpr int kI = INV ? NR - 1 - K : K;
    template <int K>
    using Pl = Place<E, LG, LGV, LGE, kI<K>>;
    // position t + (forward: e NT, natural; inverse: natural index t + rev(e) NT) of register e
    __device__ __forceinline__ static constexpr uint32_t in(uint32_t e) { return (INV ? brv(e, LGE) : e) * NT; }
    __device__ __forceinline__ static constexpr uint32_t out(uint32_t e) { return (INV ? e : brv(e, LGE)) * NT; }
    template <int K>
    __device__ __forceinline__ static uint32_t t() { return kT<K> ? threadIdx.x & (NT - 1u) : threadIdx.x >> LGV; }
    template <int K>
    __device__ __forceinline__ static uint32_t v() { return kT<K> ? threadIdx.x / NT : threadIdx.x & (V - 1u); }

    template <int K>
    __device__ __forceinline__ static void roots(P (&w)[NE - 1], const P* tab, uint32_t col0) {
        uint32_t block = (S0 > 0 ? col0 + v<K>() : 0u) + (Pl<K>::natural(t<K>()) << S0);
        // below the blocks of the round's first stage: then every index is below 2^(S0 + LG)
        if (!NTTB_CHECK(g_radix_bounds, kBoundsGlobal, block < (1u << (S0 + Pl<K>::s0)))) block = 0;
        round_roots<LG, LGE, kI<K>, S0, INV>(w, tab + block);
    }
    template <int K = 0>
    __device__ __forceinline__ static void run(const A& ar, E (&x)[NE], P (&w)[NE - 1], E* sm, const P* tab, uint32_t col0,
                                               P c0, P c1) {
        uint32_t at = NR > 1 ? Pl<K>::base(t<K>()) + v<K>() : 0u;
        if constexpr (NR > 1) {
            constexpr Lay<LG, LGV, kBankBits<E>, kLanePos<E, LG, LGV, LGE>> L;
            if (!NTTB_CHECK(g_radix_bounds, kBoundsShared, at + Pl<K>::reg(NE - 1u) < L.words)) at = 0;
        }
        E* base = sm + at;
        if constexpr (K > 0) exchange<Pl<K>, false>(base, x);
        round_stages<A, LG, LGE, kI<K>, S0, INV>(ar, x, w, c0, c1);
        if constexpr (K < NR - 1) {
            exchange<Pl<K>, true>(base, x);
            roots<K + 1>(w, tab, col0);
            __syncthreads();
            run<K + 1>(ar, x, w, sm, tab, col0, c0, c1);
        }
    }
};

// How a pass reads and writes its columns in global memory.
enum : int { kStrided = 0, kContOut = 1, kContIn = 2 };
// What it runs: the forward or the inverse stages, or the forward ones and then
// the inverse ones (a round trip's rows, which continue in registers).
enum : int { kFwd = 0, kInv = 1, kBoth = 2 };

// SINGLE (LGV = 0): rows of N = n elements, blockDim.y rows per CTA.
// S0: first stage of the pass; above 0 the roots depend on the column (row u).
// 2^LST: words between consecutive elements of a strided column.
// TSM: threads per SM that the registers are budgeted for.
template <class A, class S, class D, int LG, int LGV, int LGE, int DIR, int S0, int LST, int MODE, int TSM>
__global__ void __launch_bounds__(kThreads<LG, LGV, LGE>, TSM / kThreads<LG, LGV, LGE> > 0 ? TSM / kThreads<LG, LGV, LGE> : 1)
    radix_pass(const __grid_constant__ Args a, const LimbDev<A>* __restrict__ limbs) {
    using E = typename A::elem;
    using P = typename PairOf<A>::type;
    using First = Pass<A, LG, LGV, LGE, DIR == kInv, S0, MODE == kContIn, MODE == kContOut>;
    using Last = Pass<A, LG, LGV, LGE, DIR != kFwd, S0, MODE == kContIn, MODE == kContOut>;
    constexpr uint32_t NE = 1u << LGE, V = 1u << LGV;
    constexpr bool kSingle = LGV == 0;
    // the pass that leaves canonical residues
    constexpr bool kLast = DIR == kFwd ? MODE != kContOut : S0 == 0;
    // the pass that reads the caller's residues
    constexpr bool kFirst = kSingle || MODE == kContOut;
    constexpr bool kReduce = sizeof(S) == 8 && sizeof(E) == 4;
    extern __shared__ __align__(16) unsigned char rdx_smem[];
    constexpr Lay<LG, LGV, kBankBits<E>, kLanePos<E, LG, LGV, LGE>> L;
    E* sm = reinterpret_cast<E*>(rdx_smem) + (kSingle ? threadIdx.y * L.words : 0u);

    uint32_t limb, poly, col0 = 0, n_poly = 1;
    bool active = true;
    if (kSingle) {
        uint32_t unit = blockIdx.x * blockDim.y + threadIdx.y;
        active = unit < a.units;
        if (!active) unit = a.units - 1;
        limb = unit % a.n_limbs;
        poly = unit / a.n_limbs;
    } else {
        limb = blockIdx.y;
        poly = blockIdx.z * a.polys_per_cta;
        n_poly = min(a.polys_per_cta, a.polys - poly);
        col0 = blockIdx.x * V;
    }
    const LimbDev<A>& ld = limbs[limb];
    const A ar = ld.ar;
    const P* itab = reinterpret_cast<const P*>(ld.rt_inv);
    const P* tab = DIR == kInv ? itab : reinterpret_cast<const P*>(ld.rt);
    P c0{}, c1{}, one{}, w[NE - 1];
    if (DIR != kFwd && S0 == 0) {
        c0 = __ldg(reinterpret_cast<const P*>(ld.scale));
        c1 = __ldg(reinterpret_cast<const P*>(ld.scale) + 1);
    }
    if constexpr (kReduce) one = __ldg(tab + 1);  // cyclic tables: root^0 and floor(2^32 / q)
    const uint64_t off = (uint64_t)poly * a.poly_stride + ((uint64_t)limb << a.log_n);
    const S* src = reinterpret_cast<const S*>(a.src) + off;
    D* dst = reinterpret_cast<D*>(a.dst) + off;
    First::template roots<0>(w, tab, col0);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // words of either operand: no index reaches them (range checks)
    const uint64_t words = (uint64_t)a.polys * a.poly_stride;
    // register e's position is a thread's base plus a constant: the parts share no bit
    constexpr int LI = MODE == kContIn ? 0 : LST, LO = MODE == kContOut ? 0 : LST, NR = First::NR;
    for (uint32_t k = 0; k < n_poly; k++) {
        if (k) {
            First::template roots<0>(w, tab, col0);
            __syncthreads();  // the tile's last reads precede the next polynomial's stores
        }
        E x[NE];
        {
            const uint32_t t = First::template t<0>(), col = col0 + First::template v<0>();
            const S* p = src + (MODE == kContIn ? ((size_t)col << LG) + t : ((size_t)t << LST) + col);
#pragma unroll
            for (uint32_t e = 0; e < NE; e++) {
                const S* at = p + ((size_t)First::in(e) << LI);
                const bool ok = NTTB_CHECK(g_radix_bounds, kBoundsGlobal,
                                           (uint64_t)(at - reinterpret_cast<const S*>(a.src)) < words);
                const S y = ok ? __ldcg(at) : S(0);
                if constexpr (kFirst)
                    (void)NTTB_CHECK(g_radix_bounds, kBoundsInput, kReduce ? (uint64_t)y >> 32 == 0 : y < (S)ar.q);
                if constexpr (kReduce) {  // any word below 2^32: its residue
                    x[e] = sub_if((uint32_t)y - __umulhi((uint32_t)y, one.y) * ar.q, ar.q);
                } else {
                    x[e] = (E)y;
                }
            }
        }
        First::run(ar, x, w, sm, tab, col0, c0, c1);
        if constexpr (DIR == kBoth) {
            // the forward stages' last positions are the inverse's first, and a
            // thread overwrites the shared memory that it has read: no barrier
#pragma unroll
            for (uint32_t e = 0; e < NE; e++) x[e] = canon_out<false>(ar, x[e]);
            Last::template roots<0>(w, itab, col0);
            Last::run(ar, x, w, sm, itab, col0, c0, c1);
        }
        {
            const uint32_t t = Last::template t<NR - 1>(), col = col0 + Last::template v<NR - 1>();
            D* p = dst + (MODE == kContOut ? ((size_t)col << LG) + t : ((size_t)t << LST) + col);
#pragma unroll
            for (uint32_t e = 0; e < NE; e++) {
                const E y = kLast ? canon_out<(DIR != kFwd)>(ar, x[e]) : x[e];
                D* at = p + ((size_t)Last::out(e) << LO);
                if constexpr (kLast) (void)NTTB_CHECK(g_radix_bounds, kBoundsResidue, y < ar.q);
                if (active && NTTB_CHECK(g_radix_bounds, kBoundsGlobal,
                                         (uint64_t)(at - reinterpret_cast<D*>(a.dst)) < words))
                    *at = (D)y;
            }
        }
        src += a.poly_stride;
        dst += a.poly_stride;
    }
}

}  // namespace rdx
}  // namespace nttb
