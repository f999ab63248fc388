// klimb_plan.hpp -- the pass plan of the K-limb forward transform
// (csrc/klimb.cu), host-only so that it can be checked on the CPU.
//
// A transform of 2^log_n elements runs either as one tile in one launch (the
// bit reversal in its loads), or as a first pass that swaps tile pairs (the bit
// reversal and the first r stages, r bits at either end of the index), followed
// by passes of radix-2 DIT stages: pass i runs stages s0 .. s0 + r - 1 on tiles of
// 2^(r + logC) elements (2^logC columns of 2^r-element groups, logC <= s0), the
// stages spread evenly over as few passes as 8 stages each allow.
// The stage passes' tiles hold at most 2^log_emax elements and at most a thread per
// butterfly; log_emax shrinks while a pass would have fewer than kKlimbTargetCtas
// tiles (small transforms are bound by the latency of their stage chains, so more,
// shorter tiles win), but not below 2^6.  The swapping pass's blocks hold a pair of
// 2^r x 2^r tiles whatever log_emax is.
#pragma once

#include <cstdint>

namespace nttb {

struct KlimbPass {
    uint32_t s0, r, logC;
};

// Elements of a block, of which it has a thread for every two.
inline uint32_t klimb_pass_elements(const KlimbPass& p, bool first) { return first ? 2u << (2 * p.r) : 1u << (p.r + p.logC); }
// Threads that the kernel is built for.
constexpr uint32_t klimb_max_threads(uint32_t K) { return K <= 3 ? 512u : 256u; }
// Shared memory of a block whose elements have W words between stages: the limbs as
// in memory, the tile's roots, and the tile (a spare word after every 32).
constexpr uint64_t klimb_smem_bytes(uint32_t K, uint32_t W, uint64_t elements) {
    return (elements * (K + W) + (elements + elements / 32) * W) * 4;
}
// Shared memory that a block may ask for: more than the half of an SM's at which it
// has the SM to itself.  No block needs more.
constexpr uint64_t kKlimbSmemMax = 116 * 1024;

struct KlimbPlan {
    bool single_tile = false;  // one launch, bit reversal fused
    uint32_t log_emax = 0;     // largest tile of the stage passes
    uint32_t n_passes = 0;
    KlimbPass pass[24];
};

// 128 tiles of 128 threads are one warp per scheduler on most of the 148 SMs
constexpr uint32_t kKlimbTargetCtas = 128;

// K: limbs per element (2, 3 or 11); log_n <= 24
inline KlimbPlan klimb_plan(uint32_t K, uint32_t log_n) {
    KlimbPlan P;
    const uint32_t n = 1u << log_n;
    uint32_t log_emax = K <= 3 ? 12u : 10u;
    while (log_emax > 6 && (n >> log_emax) < kKlimbTargetCtas) log_emax--;
    P.log_emax = log_emax;
    // measured: K <= 3 up to 2^10, K = 11 up to 2^8 are fastest as one tile
    P.single_tile = log_n <= (K <= 3 ? 10u : 8u);
    if (P.single_tile) return P;
    // the swapping pass: pairs of 2^h x 2^h tiles, one butterfly per thread
    const uint32_t h = 4;
    P.pass[P.n_passes++] = {0, h, 0};
    // a thread per butterfly: tiles of at most 2^10 (K <= 3) or 2^9 elements
    const uint32_t log_tile = log_emax < (K <= 3 ? 10u : 9u) ? log_emax : (K <= 3 ? 10u : 9u);
    const uint32_t most = log_tile < 8 ? log_tile : 8u;
    uint32_t s0 = h;
    for (uint32_t left = (log_n - h + most - 1) / most; left > 0; left--) {
        const uint32_t r = (log_n - s0 + left - 1) / left;
        const uint32_t logC = log_tile - r < s0 ? log_tile - r : s0;
        P.pass[P.n_passes++] = {s0, r, logC};
        s0 += r;
    }
    return P;
}

}  // namespace nttb
