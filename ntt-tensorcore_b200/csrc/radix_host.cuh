// radix_host.cuh -- host side of the register-radix passes (radix.cuh): pass
// geometry, tile choice and launches, instantiated per residue type by the
// radix_*.cu files.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "plan.hpp"
#include "profiler.hpp"
#include "radix.cuh"

namespace nttb {
namespace rdx {

// Sizes served: one pass up to 2^kRadixSingleMax (a tile holds the whole row), two
// passes of 2^ceil(L/2) and 2^floor(L/2) points above.
constexpr uint32_t kThreadsMin = 128;  // rows are grouped into CTAs of at least this many threads

// Failed range checks of this file's passes (0 in the release build).
static inline uint32_t bounds_errors(bool clear) {
    uint32_t v = 0;
#if NTTB_DEBUG_BOUNDS
    const uint32_t z = 0;
    cudaMemcpyFromSymbol(&v, g_radix_bounds, sizeof v);
    if (clear) cudaMemcpyToSymbol(g_radix_bounds, &z, sizeof z);
#else
    (void)clear;
#endif
    return v;
}

// Shared-memory attributes of a kernel, set once per device: the dynamic size it
// may ask for and, with `carveout`, the largest shared-memory share of the SM, so that
// as many CTAs fit as it is built for (the roots that others read stay in L1, which
// that would take away: 33 x 2^17 25.6 -> 30.1 us).
template <auto K, bool carveout>
void kernel_smem(size_t smem) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return;
    cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (carveout)
        cudaFuncSetAttribute(K, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    done.fetch_or(bit, std::memory_order_release);
}

// Dynamic shared memory that keeps a grid of a few blocks an SM spread out.  With
// programmatic launches the blocks that start while the grid before drains crowd
// the SMs that happen to be free, and finish last.  Asking for a share of the SM's
// 228 KB such that only ceil(grid / 148) blocks fit prevents it.  us: 52 x 2^14
// round trip 14.2 -> 10.7, 33 x 2^15 forward 9.4 -> 7.5, 4 x 2^18 11.8 -> 9.3,
// 8 x 2^17 9.3 -> 8.4, 64-bit 18 x 2^15 12.1 -> 11.7, 4 x 2^17 12.7 -> 12.0.  Not below two blocks an SM,
// where the early start hides more than it costs (64-bit 1 x 2^18 8.5, spread 9.4);
// up to 4 for 32-bit words (beyond, L1 for the roots is worth more: 96 x 2^14 round
// trip 15.6, spread 16.1), 8 for 64-bit ones; from 3 for the round trip's middle
// pass, which reads two tables (18 x 2^15: 9.9, spread 12.1).  Two passes only: one
// launch by itself gains nothing.
inline size_t spread_smem(uint64_t grid, size_t smem, uint32_t least, uint32_t most) {
    const uint64_t per = (grid + 147) / 148;
    if (per < least || per > most) return smem;
    const size_t share = 228 * 1024 / (per + 1);
    return smem > share ? smem : share;
}
constexpr size_t kSpreadMax = 228 * 1024 / 3;

template <class K>
int launch(K kernel, const char* name, dim3 grid, dim3 block, size_t smem, const Args& a, const void* limbs,
           cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    // the next pass sets up (addresses, roots) while this one drains; it reads
    // no residue before this grid has completed (griddepcontrol.wait)
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ProfScope prof(name, s);
    void* params[2] = {const_cast<Args*>(&a), &limbs};
    return launch_rc(cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel), params));
}

template <class A, class S, int LG, int LGE, int DIR>
int launch_single(Args a, const LimbDev<A>* limbs, cudaStream_t s) {
    using E = typename A::elem;
    constexpr uint32_t NT = 1u << (LG - LGE);
    constexpr Lay<LG, 0, kBankBits<E>, kLanePos<E, LG, 0, LGE>> L;
    constexpr auto k = radix_pass<A, S, S, LG, 0, LGE, DIR, 0, 0, kStrided, 1024>;
    uint32_t rows = NT < kThreadsMin ? kThreadsMin / NT : 1u;
    while (rows > 1 && (a.units + rows - 1) / rows < 148) rows >>= 1;  // small calls spread over the SMs first
    const size_t smem = (size_t)rows * L.words * sizeof(E);
    if constexpr ((size_t)L.words * sizeof(E) > 48 * 1024) kernel_smem<k, true>((size_t)L.words * sizeof(E));
    return launch(k, "scalar_pass_row", dim3((a.units + rows - 1) / rows), dim3(NT, rows), smem, a, limbs, s);
}

template <class A, class S, class D, int LG, int LGV, int LGE, int DIR, int S0, int LST, int MODE>
int launch_pass(Args a, const LimbDev<A>* limbs, cudaStream_t s) {
    using E = typename A::elem;
    constexpr Lay<LG, LGV, kBankBits<E>, kLanePos<E, LG, LGV, LGE>> L;
    constexpr size_t tile_smem = (size_t)L.words * sizeof(E);
    constexpr uint32_t tiles = 1u << (LST - LGV);
    // a CTA keeps its columns' roots in L1 over several polynomials once the
    // launch has CTAs to spare
    const uint64_t ctas = (uint64_t)tiles * a.n_limbs * a.polys;
    uint32_t ppc = (uint32_t)(ctas / 4096);
    if (ppc < 1) ppc = 1;
    if (ppc > a.polys) ppc = a.polys;
    a.polys_per_cta = ppc;
    // A grid that leaves an SM few warps is bound by each thread's own latency and
    // runs faster with up to 128 registers a thread; larger ones are bound by L1 and
    // issue and want twice the warps.  The line lies at 1024 threads an SM, where the
    // larger variant is one full wave (the other one then runs up to two).  us
    // forward, 128 / 64 registers, by threads in units of the line: 0.35 52 x 2^14
    // 6.8 / 6.6; 0.54 80 x 2^14 9.1 / 9.8; 0.65 24 x 2^16 10.1 / 10.4; 1.3 24 x 2^17
    // 19.7 / 18.0; 2.0 36 x 2^17 27.8 / 23.4.  64-bit: 0.70 52 x 2^14 13.5 / 16.8; 0.97
    // 36 x 2^15 17.7 / 18.8; 2.6 3 x 2^20 73 / 62; nineteen of its 80 kernels, all
    // built for 1024 threads, spill 8 - 88 bytes.  Blocks of 512 threads, of which the 128 registers fit one
    // an SM, would rather change over at 0.5: 12 x 2^17 13.0 / 11.8, 2 x 2^20
    // 18.4 / 16.3, 64-bit 1 x 2^20 25.8 / 23.7.
    constexpr uint32_t threads = 1u << (LG + LGV - LGE);
    constexpr auto few = radix_pass<A, S, D, LG, LGV, LGE, DIR, S0, LST, MODE, 512>;
    constexpr auto many = radix_pass<A, S, D, LG, LGV, LGE, DIR, S0, LST, MODE, 1024>;
    const bool one_wave = ctas * threads <= 148u * 1024u;
    const uint32_t chunks = (a.polys + ppc - 1) / ppc;
    const size_t smem = spread_smem((uint64_t)tiles * a.n_limbs * chunks, tile_smem, DIR == kBoth ? 3 : 2, sizeof(E) == 8 ? 8 : 4);
    constexpr size_t most = tile_smem > kSpreadMax ? tile_smem : kSpreadMax;
    if (one_wave) kernel_smem<few, (tile_smem > 48 * 1024)>(most);
    else kernel_smem<many, (tile_smem > 48 * 1024)>(most);
    return launch(one_wave ? few : many, MODE == kContOut ? "scalar_pass_col" : DIR == kBoth ? "scalar_pass_mid" : "scalar_pass_col_b",
                  dim3(tiles, a.n_limbs, chunks), dim3(threads), smem, a, limbs, s);
}

// Columns per tile: a warp's loads touch 32 / V lines of 128 bytes, and at
// V = 8 the L1 data pipe was 75 % busy with them (192 x 2^16: 72 % at V = 8,
// 59 % at 16); 512 and 1024-point columns take half as many, which keeps two
// CTAs on an SM (8 x 2^20: 54.9 us at V = 8, 62.8 at 16; 1 x 2^20: 10.0, 14.7).
template <class A, class S, int L>
constexpr int kLogCols = sizeof(typename A::elem) == 8 ? 2 : sizeof(S) == 8 ? 3 : L <= 17 ? 4 : 3;

// Both passes of one size; S -> M -> S words (M: the workspace or destination).
template <class A, class S, class M, int L, int LGE>
int launch_two(Args a, void* mid, const LimbDev<A>* limbs, bool inverse, cudaStream_t s) {
    constexpr int LA = (L + 1) / 2, LB = L / 2, LGV = kLogCols<A, S, L>;
    void* dst = a.dst;
    a.dst = mid;
    int rc = inverse ? launch_pass<A, S, M, LB, LGV, LGE, kInv, LA, LA, kContOut>(a, limbs, s)
                     : launch_pass<A, S, M, LA, LGV, LGE, kFwd, 0, LB, kContOut>(a, limbs, s);
    if (rc) return rc;
    a.src = mid;
    a.dst = dst;
    return inverse ? launch_pass<A, M, S, LA, LGV, LGE, kInv, 0, LB, kStrided>(a, limbs, s)
                   : launch_pass<A, M, S, LB, LGV, LGE, kFwd, LA, LA, kStrided>(a, limbs, s);
}

// Forward then inverse of one size, in place through `mid`: the first pass, the
// rows' forward and inverse stages in one pass over `mid`, the last pass (which
// reads contiguous columns): three passes over memory instead of four.
template <class A, class S, int L, int LGE>
int launch_round_trip(Args a, void* mid, const LimbDev<A>* limbs, cudaStream_t s) {
    constexpr int LA = (L + 1) / 2, LB = L / 2, LGV = kLogCols<A, S, L>;
    void* data = a.dst;
    a.dst = mid;
    int rc = launch_pass<A, S, S, LA, LGV, LGE, kFwd, 0, LB, kContOut>(a, limbs, s);
    if (rc) return rc;
    a.src = mid;
    rc = launch_pass<A, S, S, LB, LGV, LGE, kBoth, LA, LA, kStrided>(a, limbs, s);
    if (rc) return rc;
    a.dst = data;
    return launch_pass<A, S, S, LA, LGV, LGE, kInv, 0, LB, kContIn>(a, limbs, s);
}

template <class A>
Args make_args(uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, uint32_t n_polys) {
    Args a{};
    a.src = src;
    a.dst = dst;
    a.poly_stride = (uint64_t)n_limbs << log_n;
    a.log_n = log_n;
    a.polys = n_polys;
    a.n_limbs = n_limbs;
    a.units = n_polys * n_limbs;
    return a;
}

// Runs one transform of n_polys x n_limbs rows; `mid` (two-pass sizes) holds
// the first pass in words of M.  Returns 1 when the size is not served.
template <class A, class S, class M, int LGE>
int transform(const LimbDev<A>* limbs, uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, void* mid,
              uint32_t n_polys, bool inverse, cudaStream_t s) {
    const Args a = make_args<A>(log_n, n_limbs, src, dst, n_polys);
#define NTTB_SINGLE(l) \
    case l: return inverse ? launch_single<A, S, l, LGE, kInv>(a, limbs, s) : launch_single<A, S, l, LGE, kFwd>(a, limbs, s);
#define NTTB_TWO(l) \
    case l: return launch_two<A, S, M, l, LGE>(a, mid, limbs, inverse, s);
    switch (log_n) {
        NTTB_SINGLE(5) NTTB_SINGLE(6) NTTB_SINGLE(7) NTTB_SINGLE(8) NTTB_SINGLE(9)
        NTTB_SINGLE(10) NTTB_SINGLE(11) NTTB_SINGLE(12)
        case 13:
            if constexpr (sizeof(typename A::elem) == 8) return launch_two<A, S, M, 13, LGE>(a, mid, limbs, inverse, s);
            else if (inverse) return launch_single<A, S, 13, LGE, kInv>(a, limbs, s);
            else return launch_single<A, S, 13, LGE, kFwd>(a, limbs, s);
        NTTB_TWO(14) NTTB_TWO(15) NTTB_TWO(16) NTTB_TWO(17) NTTB_TWO(18) NTTB_TWO(19) NTTB_TWO(20)
        default: return 1;
    }
#undef NTTB_SINGLE
#undef NTTB_TWO
}

}  // namespace rdx
}  // namespace nttb
