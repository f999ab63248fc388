// batch_radix.cuh -- the batch queue's register-radix tiles and the
// persistent kernel that runs them (included by batch.cu).
//
// Every unit of 2^10 .. 2^20 residues runs tiles of 8192 residues on 512
// threads, 16 residues each, with the stages, exchanges and root order of
// radix.cuh:
//   2^10 .. 2^13: one tile holds 8192 / n whole rows (limbs);
//   2^14 .. 2^20: two passes of n / 8192 tiles (V = 8192 / N columns of the
//     pass's N points) through a workspace slot.  The slot is laid out in the
//     second pass's tiles -- block k holds its columns V k .. V k + V - 1, row
//     after row -- so that pass B reads one contiguous run of 32 KB per tile
//     and pass A writes runs of at least 32 bytes times the lanes that share a row.
// Roots.  Butterflies multiply by Shoup pairs (7.1 instructions, 12.4 per clock
// and SM when nothing else runs; Montgomery-form roots take 9.1 and reach 8.7).
// A pass whose roots are the same for every column reads pairs; a row pass and
// whole rows, which use one root per residue, read the pair's quotient ws =
// floor(w 2^32 / q) alone, 4 bytes, and make w = floor(ws q / 2^32) + 1 (ws q =
// w 2^32 - r with 0 < r < q).  Tables are per modulus, direction and twist, and
// one table serves its size and those below: root 2^s + i is zeta^(1 + 2 i), zeta of order
// 2^(s+2) (negacyclic), or zeta^i, zeta of order 2^(s+1) (cyclic).
//
// A seventeenth warp feeds the tiles: while the 512 threads run one, it claims
// the next ticket, copies the tile's record to shared memory, waits (bounded)
// for its dependencies and copies its roots and words into shared memory
// (cp.async), so that a tile starts on data that is there.  Words are copied 16 bytes at a time: a
// batch with a job off that alignment runs the other tiles.
#pragma once

constexpr uint32_t kRxLogTile = 13, kRxTile = 1u << kRxLogTile, kRxE = 4, kRxThreads = kRxTile >> kRxE;
constexpr uint32_t kRxCtas = 2;  // per SM
constexpr uint32_t kRxMinLog = 10, kRxMaxLog = 20;
constexpr uint32_t kRxFew = kRxTile >> kRxE;  // words of a tile's roots outside the last round
constexpr uint32_t rx_max(uint32_t a, uint32_t b) { return a > b ? a : b; }

__device__ __forceinline__ void rx_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kRxThreads) : "memory"); }

// The last round's roots (the stages with most of them) have their own
// hand-over: ready (the tile waits), and read (the feeding warp may refill them).
__device__ __forceinline__ void rx_roots_ready() { asm volatile("bar.sync 8, %0;" ::"n"(kRxThreads + 32) : "memory"); }
__device__ __forceinline__ void rx_roots_free() { asm volatile("bar.arrive 7, %0;" ::"n"(kRxThreads + 32) : "memory"); }
// The tile's threads have read the inbox: the feeding warp may refill it.
__device__ __forceinline__ void rx_inbox_free() { asm volatile("bar.arrive 6, %0;" ::"n"(kRxThreads + 32) : "memory"); }

// The root at index i (within the pass) of a thread whose block and column
// `box` points at: pairs, or quotients 2^LGV words apart.
template <int LGV>
__device__ __forceinline__ uint2 rx_root(const M32&, const uint2* box, uint32_t i) { return box[i]; }
template <int LGV>
__device__ __forceinline__ uint2 rx_root(const M32& ar, const uint32_t* box, uint32_t i) {
    const uint32_t ws = box[i << LGV];
    return make_uint2(__umulhi(ws, ar.q) + 1u, ws);
}

// Stages of round I from its J-th on (S0 > 0: none is the transform's first stage).
template <int LG, int LGV, int I, int S0, bool INV, int JJ = 0, class P>
__device__ __forceinline__ void rx_stages(const M32& ar, uint32_t (&x)[1 << kRxE], const P* box, uint2 c0, uint2 c1) {
    constexpr rdx::Rounds<LG, kRxE> R;
    constexpr int r = R.r[I], S = R.s0[I], xb = kRxE - r, j = INV ? r - 1 - JJ : JJ;
    constexpr uint32_t half = 1u << (r - 1 - j);
    constexpr bool scaled = INV && S0 + S + j == 0;
#pragma unroll
    for (uint32_t kt = 0; kt < (1u << j); kt++) {
        uint2 w = c1;
        if constexpr (!scaled) w = rx_root<LGV>(ar, box, (1u << (S + j)) + (rdx::brv(kt, j) << S));
#pragma unroll
        for (uint32_t lo = 0; lo < half; lo++)
#pragma unroll
            for (uint32_t g = 0; g < (1u << xb); g++) {
                const uint32_t ia = (((kt << (r - j)) + lo) << xb) + g, ib = ia + (half << xb);
                if constexpr (scaled) rdx::gs_scaled(ar, x[ia], x[ib], c0, w);
                else if constexpr (INV) rdx::gs(ar, x[ia], x[ib], w);
                else rdx::ct(ar, x[ia], x[ib], w);
            }
    }
    if constexpr (JJ + 1 < r) rx_stages<LG, LGV, I, S0, INV, JJ + 1>(ar, x, box, c0, c1);
}

// Position lanes of a tile's blocked store (rows: all five lane bits).
template <int LG, int LB>
constexpr int kRxTL = LB < LG - kRxE ? LB : LG - kRxE;
template <int LG, int LGV, int LB>
constexpr int kRxNP = LGV == 0 ? 5 : kRxTL<LG, LB> < 5 ? kRxTL<LG, LB> : 5;

// One tile.  LSI, LSO: log2 of the words between a column's elements in and
// out; LB >= 0: the output goes to the workspace in blocks of 2^LB (the second
// pass's columns); LBP: the LB that the placement is made for.  S0: the pass's
// first stage (above 0: a row pass).  In shared memory: `in`, element i of
// column v at (i << LGV) + v (uint64 words are read from `src` instead), and
// the roots: pairs, or (kQuot) quotients, root i of column v at (i << LGV) + v;
// `box` those of the last round (in the forward order), `few` the others.
// lim_in, lim_out: words from src (and pre) and from dst (range checks).
template <int LG, int LGV, bool INV, int S0, bool kQuot, int LSI, int LSO, int LB, int LBP, class S, class D>
__device__ __forceinline__ void rx_tile(const M32& ar, const uint32_t* in, const uint32_t* few,
                                        const uint32_t* box, const S* src, D* dst,
                                        const uint32_t* pre, uint2 one, uint2 c0, uint2 c1, uint32_t col0, uint32_t tid,
                                        uint32_t* sm, bool active, const uint32_t* drop, uint32_t lim_in,
                                        uint32_t lim_out) {
    using P = typename std::conditional<kQuot, uint32_t, uint2>::type;
    constexpr uint32_t NE = 1u << kRxE, V = 1u << LGV, NT = 1u << (LG - kRxE);
    constexpr rdx::Rounds<LG, kRxE> R;
    constexpr int NR = R.n;
    constexpr bool kBlock = LB >= 0;
    constexpr bool kInput = kBlock || LGV == 0;  // the pass that reads the caller's residues
    // the blocked store: positions below the block, then columns, then positions
    constexpr int TL = kRxTL<LG, LBP>;
    const uint32_t v_v = tid & (V - 1u), t_v = tid >> LGV;
    const uint32_t v_b = kBlock ? (tid >> TL) & (V - 1u) : v_v;
    const uint32_t t_b = kBlock ? (tid & ((1u << TL) - 1u)) | ((tid >> (TL + LGV)) << TL) : t_v;
    uint32_t x[NE];
    auto run = [&](auto self, auto step) -> void {
        constexpr int K = decltype(step)::value, I = INV ? NR - 1 - K : K;
        constexpr bool blk = kBlock && K == NR - 1;
        using Pl = rdx::Place<uint32_t, LG, LGV, kRxE, I, kRxNP<LG, LGV, LBP>>;
        const uint32_t t = blk ? t_b : t_v, v = blk ? v_b : v_v;
        uint32_t at0 = Pl::base(t) + v, block = Pl::natural(t);
        constexpr rdx::Lay<LG, LGV, 5, kRxNP<LG, LGV, LBP>> Y;
        if (!NTTB_CHECK(g_batch_bounds, kBoundsShared, at0 + Pl::reg(NE - 1u) < Y.words)) at0 = 0;
        // a block of the round's first stage: then every root's index is below 2^LG (box) or 2^LG / 16 (few)
        if (!NTTB_CHECK(g_batch_bounds, kBoundsShared, block < (1u << R.s0[I]) && v < V)) block = 0;
        uint32_t* base = sm + at0;
        const P* roots = reinterpret_cast<const P*>(I == NR - 1 ? box : few) + (kQuot ? (block << LGV) + v : block);
        if constexpr (K == 0) {
            // position t + rev(e) NT (inverse) or t + e NT: the parts share no bit, so
            // every address is a thread's base plus a constant
            const S* gsrc = src + (((size_t)t << LSI) + v);
            const uint32_t* isrc = in + ((t << LGV) + v);
#pragma unroll
            for (uint32_t e = 0; e < NE; e++) {
                const uint32_t ie = (INV ? rdx::brv(e, kRxE) : e) * NT;
                if constexpr (sizeof(S) == 8) {  // any word below 2^32: its residue
                    uint64_t w = 0;
                    if (NTTB_CHECK(g_batch_bounds, kBoundsGlobal, ((size_t)(t + ie) << LSI) + v < lim_in))
                        w = __ldcs(gsrc + ((size_t)ie << LSI));
                    (void)NTTB_CHECK(g_batch_bounds, kBoundsInput, w >> 32 == 0);
                    const uint32_t y = (uint32_t)w;
                    x[e] = rdx::sub_if(y - __umulhi(y, one.y) * ar.q, ar.q);
                } else {
                    x[e] = NTTB_CHECK(g_batch_bounds, kBoundsShared, ((t + ie) << LGV) + v < kRxTile) ? isrc[ie << LGV] : 0u;
                    if constexpr (kInput) (void)NTTB_CHECK(g_batch_bounds, kBoundsInput, !active || x[e] < ar.q);
                }
            }
            if constexpr (sizeof(S) != 8) rx_inbox_free();
            if (INV && pre) {  // a product's spectra; the scale carries the factor 2^32
                const uint32_t* p = pre + (((size_t)t << LSI) + v);
#pragma unroll
                for (uint32_t e = 0; e < NE; e++) {
                    const size_t i = (size_t)(rdx::brv(e, kRxE) * NT) << LSI;
                    if (!NTTB_CHECK(g_batch_bounds, kBoundsGlobal, ((size_t)t << LSI) + v + i < lim_in)) continue;
                    x[e] = rdx::sub_if(tca::mont_lazy(x[e], __ldcg(p + i), ar.q, ar.qinv), ar.q);
                }
            }
        } else {
            rdx::exchange<Pl, false>(base, x);
        }
        if constexpr (I == NR - 1) rx_roots_ready();
        rx_stages<LG, LGV, I, S0, INV>(ar, x, roots, c0, c1);
        if constexpr (I == NR - 1) rx_roots_free();
        if constexpr (K < NR - 1) {
            rdx::exchange<Pl, true>(base, x);
            rx_sync();
            // every load of the block has returned: drop its lines from the L2
            // (the slot's next owner rewrites them; otherwise they reach DRAM)
            if (K == 0 && drop && tid < kRxTile / 32)
                asm volatile("discard.global.L2 [%0], 128;" ::"l"(drop + 32u * tid) : "memory");
            self(self, std::integral_constant<int, K + 1>{});
        } else {
            if constexpr (kBlock) {
                const uint64_t keep = tc::l2_policy_evict_last();
                auto at = [](uint32_t i) { return ((size_t)(i >> LB) << (LSI + LB)) + (i & ((1u << LB) - 1u)); };
                const size_t p0 = at(t) + ((size_t)(col0 + v) << LB);
                D* p = dst + p0;
#pragma unroll
                for (uint32_t e = 0; e < NE; e++) {
                    const size_t i = at((INV ? e : rdx::brv(e, kRxE)) * NT);
                    if (NTTB_CHECK(g_batch_bounds, kBoundsWorkspace, p0 + i < lim_out)) st_keep(p + i, x[e], keep);
                }
            } else if (active) {
                const size_t p0 = ((size_t)t << LSO) + v;
                D* p = dst + p0;
#pragma unroll
                for (uint32_t e = 0; e < NE; e++) {
                    const size_t i = (size_t)((INV ? e : rdx::brv(e, kRxE)) * NT) << LSO;
                    const uint32_t y = rdx::canon_out<INV>(ar, x[e]);
                    (void)NTTB_CHECK(g_batch_bounds, kBoundsResidue, y < ar.q);
                    if (NTTB_CHECK(g_batch_bounds, kBoundsGlobal, p0 + i < lim_out)) __stcs(p + i, (D)y);
                }
            }
        }
    };
    run(run, std::integral_constant<int, 0>{});
}

// One pass of a two-pass unit of 2^L residues.
template <int L, bool INV, int PASS, bool W64>
__device__ __forceinline__ void rx_pass(const BUnit& u, uint32_t tile, uint32_t* sm, const uint32_t* in,
                                        const uint32_t* few) {
    constexpr int LA = (L + 1) / 2, LBB = L / 2;  // points of the uniform and of the row pass
    constexpr bool kRow = INV ? PASS == 0 : PASS == 1;
    constexpr int LG = kRow ? LBB : LA, LGV = kRxLogTile - LG, S0 = kRow ? LA : 0;
    constexpr int LC = kRow ? LA : LBB;                    // log2 of the pass's columns
    constexpr int LB = kRxLogTile - (kRow ? LA : LBB);     // the other pass's columns per tile
    using W = typename std::conditional<W64, uint64_t, uint32_t>::type;
    const M32 ar = u.ar;
    const uint32_t col0 = tile << LGV;
    const uint32_t* box = in + kRxTile;
    if constexpr (PASS == 0) {
        const W* src = static_cast<const W*>(u.in ? u.in : u.data) + col0;
        rx_tile<LG, LGV, INV, S0, kRow, LC, 0, LB, LB, W, uint32_t>(
            ar, in, few, box, src, u.ws, INV && u.pre_mul ? u.pre_mul + col0 : nullptr, u.one, u.scale[0], u.scale[1], col0,
            threadIdx.x, sm, true, nullptr, (1u << L) - col0, 1u << L);
    } else {
        const uint32_t* src = u.ws + (size_t)tile * kRxTile;
        rx_tile<LG, LGV, INV, S0, kRow, LGV, LC, -1, LB, uint32_t, W>(
            ar, in, few, box, src, reinterpret_cast<W*>(u.data) + col0, nullptr, u.one, u.scale[0], u.scale[1], col0, threadIdx.x,
            sm, true, src, 0, (1u << L) - col0);
    }
}

// Whole rows of 2^L residues, one limb each.
template <int L, bool INV>
__device__ __forceinline__ void rx_rows(const BArgs& a, const BUnit& u, uint32_t* sm, const uint32_t* in,
                                        const uint32_t* few) {
    constexpr uint32_t NT = 1u << (L - kRxE);
    constexpr rdx::Lay<L, 0, 5, 5> Y;
    const uint32_t tid = threadIdx.x & (NT - 1u);
    uint32_t row = threadIdx.x / NT;
    sm += row * Y.words;
    const bool active = row < u.rows;
    if (!active) row = u.rows - 1u;
    const RxModulus& M = a.rx[u.mod0 + row];
    const M32 ar = M.ar;
    uint2 c0 = make_uint2(0, 0), c1 = c0;
    if (INV) {
        const uint2* sc = M.scale[u.flags & UF_NEGA ? 1 : 0][u.pre_mul ? 1 : 0][L];
        c0 = __ldg(sc);
        c1 = __ldg(sc + 1);
    }
    uint32_t* x = u.data + ((size_t)row << L);
    rx_tile<L, 0, INV, 0, true, 0, 0, -1, 0, uint32_t, uint32_t>(
        ar, in + (row << L), few + (row << (L - kRxE)), in + kRxTile + (row << L), x, x, INV && u.pre_mul ? u.pre_mul + ((size_t)row << L) : nullptr,
        make_uint2(0, 0), c0, c1, 0, tid, sm, active, nullptr, 1u << L, 1u << L);
}

// What the tile threads do with a slot.
enum : uint32_t { kRxRun = 0, kRxStop = 1, kRxSkip = 2 };
struct RxSlot {
    BUnit u;
    uint32_t unit, pass, tile, stop;
};

// The feeding warp: `chunks` 16-byte pieces, 2^lgc <= 32 of them per row, rows
// `pitch` words apart, to shared memory past L1 (asynchronous).  A lane keeps
// its place in the row: one addition per copy, since this one warp shares the
// issue slots with the tiles' thirty-two.
__device__ __forceinline__ void rx_copy(const uint32_t* src, uint32_t lgc, size_t pitch, uint32_t chunks, uint32_t to,
                                        uint32_t lane) {
    const char* g = reinterpret_cast<const char*>(src + (size_t)(lane >> lgc) * pitch + 4 * (lane & ((1u << lgc) - 1u)));
    const size_t step = (pitch << (5 - lgc)) * 4;
    to += 16 * lane;
    uint32_t i = 0;
    for (; i + 256 <= chunks; i += 256) {
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 512 * k), "l"(g) : "memory");
            g += step;
        }
        to += 4096;
    }
    for (i += lane; i < chunks; i += 32) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(g) : "memory");
        g += step;
        to += 512;
    }
}

// The feeding warp's share of a tile: its 8192 words into the
// inbox: rows of 4 V bytes, or one contiguous run (second passes, whole rows).
__device__ __forceinline__ void rx_fetch(const BUnit& u, uint32_t pass, uint32_t tile, uint32_t inbox, uint32_t lane) {
    const uint32_t L = u.log_n;
    const uint32_t* src;
    uint32_t lgc = 5, chunks = kRxTile / 4;  // 16-byte pieces per row (log2), in all
    size_t pitch = 128;
    if (L <= kRxLogTile) {
        src = u.data;
        chunks = u.rows << (L - 2);
    } else if (pass) {
        src = u.ws + (size_t)tile * kRxTile;
    } else {
        const uint32_t la = (L + 1) / 2, lb = L / 2, lg = u.flags & UF_INV ? lb : la;
        lgc = kRxLogTile - lg - 2;
        pitch = (size_t)1 << (L - lg);
        src = static_cast<const uint32_t*>(u.in ? u.in : u.data) + ((size_t)tile << (kRxLogTile - lg));
    }
    // the last piece ends within the unit's words (or its slot) and the inbox
    const uint32_t* all = static_cast<const uint32_t*>(pass ? u.ws : u.in ? u.in : u.data);
    if (!NTTB_CHECK(g_batch_bounds, kBoundsGlobal,
                    (size_t)(src - all) + ((chunks >> lgc) - 1) * pitch + ((size_t)4 << lgc) <= ((size_t)u.rows << L)) ||
        !NTTB_CHECK(g_batch_bounds, kBoundsShared, chunks <= kRxTile / 4))
        return;
    rx_copy(src, lgc, pitch, chunks, inbox, lane);
}

// A tile's roots.  A row pass: columns V tile .. of the unit's quotients seen as
// [2^LG][2^LA] (entry (e << LA) + u is root e of row u); a uniform pass: its 2^LG
// pairs; whole rows: each row's 2^L quotients.  FEW: the entries below 1/16 (every
// round but the last); else all of them.
template <bool FEW>
__device__ __forceinline__ void rx_fetch_roots(const BArgs& a, const BUnit& u, uint32_t pass, uint32_t tile, uint32_t to,
                                               uint32_t lane) {
    const uint32_t L = u.log_n, la = (L + 1) / 2;
    constexpr int kF = FEW ? kRxE : 0;
    if (!u.lg1) {
        const uint32_t kind = (u.flags & UF_NEGA ? 2u : 0u) + (u.flags & UF_INV ? 1u : 0u);
        for (uint32_t r = 0; r < u.rows; r++)  // 4 quotients per piece
            rx_copy(a.rx[u.mod0 + r].quot[kind], 5, 128, 1u << (L - 2 - kF), to + ((4 * r) << (L - kF)), lane);
    } else if ((pass == 1) == !(u.flags & UF_INV)) {
        const uint32_t lgv = kRxLogTile - L / 2;
        rx_copy(u.quot + ((size_t)tile << lgv), lgv - 2, (size_t)1 << la, kRxTile >> (2 + kF), to, lane);
    } else {
        rx_copy(reinterpret_cast<const uint32_t*>(u.pairs), 5, 128, 1u << (la - 1 - kF), to, lane);  // 2 pairs per piece
    }
}

template <bool W64>
__device__ __forceinline__ void rx_dispatch(const BArgs& a, const RxSlot& s, uint32_t* sm, const uint32_t* in,
                                            const uint32_t* few, M32* s_ar) {
    const BUnit& u = s.u;
    const bool inv = u.flags & UF_INV;
#define NTTB_RX_TWO(l)                                                             \
    case l:                                                                        \
        if (s.pass == 0) {                                                         \
            if (inv) rx_pass<l, true, 0, W64>(u, s.tile, sm, in, few);                      \
            else rx_pass<l, false, 0, W64>(u, s.tile, sm, in, few);                         \
        } else {                                                                   \
            if (inv) rx_pass<l, true, 1, W64>(u, s.tile, sm, in, few);                      \
            else rx_pass<l, false, 1, W64>(u, s.tile, sm, in, few);                         \
        }                                                                          \
        return;
#define NTTB_RX_ROWS(l)                        \
    case l:                                    \
        if (inv) rx_rows<l, true>(a, u, sm, in, few); \
        else rx_rows<l, false>(a, u, sm, in, few); \
        return;
    if constexpr (W64) {
        switch (u.log_n) {
            NTTB_RX_TWO(17) NTTB_RX_TWO(18) NTTB_RX_TWO(19) NTTB_RX_TWO(20)
            default: return;
        }
    } else {
        if (!(u.flags & UF_RX)) {
            run_tile<kRxThreads, 3, true>(a, u, s.pass, s.tile, sm, s_ar);
            return;
        }
        switch (u.log_n) {
            NTTB_RX_ROWS(10) NTTB_RX_ROWS(11) NTTB_RX_ROWS(12) NTTB_RX_ROWS(13)
            NTTB_RX_TWO(14) NTTB_RX_TWO(15) NTTB_RX_TWO(16) NTTB_RX_TWO(17) NTTB_RX_TWO(18) NTTB_RX_TWO(19) NTTB_RX_TWO(20)
            default: return;
        }
    }
#undef NTTB_RX_TWO
#undef NTTB_RX_ROWS
}

// Two CTAs of 16 + 1 warps per SM.
template <bool W64>
__global__ void __launch_bounds__(kRxThreads + 32, kRxCtas) batch_queue_radix(const __grid_constant__ BArgs a) {
    extern __shared__ __align__(16) uint32_t rx_sm[];
    __shared__ __align__(16) RxSlot slot[2];
    __shared__ M32 s_ar[kMaxRows];
    static_assert(sizeof(BUnit) % 16 == 0 && sizeof(BUnit) / 16 <= 32, "one 16-byte piece per lane");
    uint32_t* inbox = rx_sm;                 // the next tile's words, 32 KB, and its last round's roots, 32 KB
    uint32_t* few = rx_sm + 2 * kRxTile;     // the other roots, 2 KB for each slot
    uint32_t* work = few + 2 * kRxFew;       // the running tile's exchanges
    // named barriers: 1 the tile's threads, 2 + s slot s filled, 4 + s slot s
    // free, 6 the inbox free (uint64 words are read by the tile itself), 7 the
    // last round's roots free, 8 filled
    if (threadIdx.x >= kRxThreads) {
        const uint32_t lane = threadIdx.x & 31u;
        bool inbox_used = false, roots_used = false;  // a tile that reads them precedes
        for (uint32_t k = 0;; k++) {
            const uint32_t s = k & 1u;
            if (k >= 2) asm volatile("bar.sync %0, %1;" ::"r"(4u + s), "n"(kRxThreads + 32) : "memory");
            uint32_t ticket = 0;
            if (lane == 0) ticket = atomicAdd(a.ctr, 1u);
            ticket = __shfl_sync(~0u, ticket, 0);
            uint32_t stop = ticket >= a.n_tiles ? kRxStop : kRxRun;
            bool rx = false;
            if (!stop) {
                const BTile tl = a.tiles[ticket];
#if NTTB_DEBUG_BOUNDS
                if (!tile_in_range(a, tl)) {  // recorded; the tile is passed over, and counted as done
                    stop = kRxSkip;
                    if (lane == 0) {
                        slot[s].unit = tl.unit;
                        slot[s].pass = tl.pass_tile >> 31;
                    }
                }
#endif
                if (!stop) {
                    if (lane < sizeof(BUnit) / 16)
                        reinterpret_cast<uint4*>(&slot[s].u)[lane] =
                            __ldg(reinterpret_cast<const uint4*>(a.units + tl.unit) + lane);
                    if (lane == 0) {
                        slot[s].unit = tl.unit;
                        slot[s].pass = tl.pass_tile >> 31;
                        slot[s].tile = tl.pass_tile & 0x7fffffffu;
                    }
                    __syncwarp();
                    const BUnit& u = slot[s].u;
                    const uint32_t pass = tl.pass_tile >> 31, tile = tl.pass_tile & 0x7fffffffu;
                    rx = u.flags & UF_RX;
                    if (rx) rx_fetch_roots<true>(a, u, pass, tile, tc::smem_u32(few + s * kRxFew), lane);
                    if (lane == 0 && !wait_deps(a, u, tl.unit, pass)) atomicOr(&g_batch_error, 1u);
                    __syncwarp();
                    if (rx && !(W64 && pass == 0)) {
                        if (inbox_used) asm volatile("bar.sync 6, %0;" ::"n"(kRxThreads + 32) : "memory");
                        inbox_used = true;
                        rx_fetch(u, pass, tile, tc::smem_u32(inbox), lane);
                    }
                    asm volatile("cp.async.wait_all;" ::: "memory");
                }
            }
            if (lane == 0) slot[s].stop = stop;
            __syncwarp();
            asm volatile("bar.arrive %0, %1;" ::"r"(2u + s), "n"(kRxThreads + 32) : "memory");
            if (stop == kRxStop) return;
            if (rx) {  // the roots of the running tile's last round are in use until then
                if (roots_used) asm volatile("bar.sync 7, %0;" ::"n"(kRxThreads + 32) : "memory");
                roots_used = true;
                rx_fetch_roots<false>(a, slot[s].u, slot[s].pass, slot[s].tile, tc::smem_u32(inbox + kRxTile), lane);
                asm volatile("cp.async.wait_all;" ::: "memory");
                asm volatile("bar.arrive 8, %0;" ::"n"(kRxThreads + 32) : "memory");
            }
        }
    }
    for (uint32_t k = 0;; k++) {
        const uint32_t s = k & 1u;
        asm volatile("bar.sync %0, %1;" ::"r"(2u + s), "n"(kRxThreads + 32) : "memory");
        if (slot[s].stop == kRxStop) return;
        bool signal = true;
#if NTTB_DEBUG_BOUNDS
        if (slot[s].stop == kRxSkip) signal = slot[s].unit < a.n_units;
        else
#endif
            rx_dispatch<W64>(a, slot[s], work, inbox, few + s * kRxFew, s_ar);
        rx_sync();
        if (threadIdx.x == 0 && signal) signal_done(a.ctr + 1 + 2 * slot[s].unit + slot[s].pass);
        asm volatile("bar.arrive %0, %1;" ::"r"(4u + s), "n"(kRxThreads + 32) : "memory");
    }
}

// Dynamic shared memory: the inbox, the roots and the largest exchange buffer.
template <int L, bool ROW>
constexpr uint32_t rx_two_words() {
    constexpr int LA = (L + 1) / 2, LG = ROW ? L / 2 : LA, LB = (int)kRxLogTile - (ROW ? LA : L / 2);
    return rdx::Lay<LG, (int)kRxLogTile - LG, 5, kRxNP<LG, (int)kRxLogTile - LG, LB>>().words;
}
template <int L>
constexpr uint32_t rx_two_words() { return rx_max(rx_two_words<L, false>(), rx_two_words<L, true>()); }
template <int L>
constexpr uint32_t rx_rows_words() { return (kRxTile >> L) * rdx::Lay<L, 0, 5, 5>().words; }
constexpr uint32_t kRxWork = rx_max(
    rx_max(rx_max(rx_two_words<14>(), rx_two_words<15>()), rx_max(rx_two_words<16>(), rx_two_words<17>())),
    rx_max(rx_max(rx_max(rx_two_words<18>(), rx_two_words<19>()), rx_two_words<20>()),
           rx_max(rx_max(rx_rows_words<10>(), rx_rows_words<11>()), rx_max(rx_rows_words<12>(), rx_rows_words<13>()))));
constexpr uint32_t kRxWords = 2 * kRxTile + 2 * kRxFew + kRxWork;
// units of other sizes run CUDA-core tiles of this many residues in the exchange buffer
constexpr uint32_t kRxCoreTile = 4096;
