// engines.cu -- engine selection for 31-bit plans.
#include <cstdlib>
#include <cstring>

#include "../../include/ntt_b200.h"
#include "engines.hpp"

namespace nttb {

static int env_engine() {
    const char* e = std::getenv("NTT_B200_ENGINE");
    if (!e) return NTTB_ENGINE_AUTO;
    if (!std::strcmp(e, "scalar")) return NTTB_ENGINE_SCALAR;
    if (!std::strcmp(e, "dmma")) return NTTB_ENGINE_DMMA;
    if (!std::strcmp(e, "int8")) return NTTB_ENGINE_INT8;
    if (!std::strcmp(e, "tiles")) return NTTB_ENGINE_TILES;
    return NTTB_ENGINE_AUTO;
}

// The CUDA-core engine's register-radix passes (radix.cuh) are the fastest at
// every size (us, forward, the same buffers again and again, this engine / the
// other): 4 x 2^16 6.7 / 16.7 (INT8), 33 x 2^16 12.5 / 18.0 (INT8), 256 x 2^16 73 / 129
// (INT8), 33 x 2^17 22.8 / 61.9 (tensor tiles), 1 x 2^20 10.1 / 26.0 (queue).  Calls of
// 8 rows that take turns on four or more streams are bound by the host, where two
// launches cost 7 - 10 us and the INT8 kernel's one 4 - 6.  In place they stage their first pass
// in a workspace; calls for which it could not be had and the drop-in's and the
// host stream's calls, whose engines those entry points name, take the INT8
// cluster kernel at 2^16 from kInt8MinUnits (polynomial, limb) units on and the
// batch queue at 2^17 .. 2^20 once a call holds 2^20 residues (each prepared queue
// has a ring of its own).
constexpr uint64_t kInt8MinUnits = 8;
constexpr uint32_t kTilesMinLog = 17;
constexpr uint64_t kTilesMinResidues = 1ull << 20;

int auto_engine32(const Plan32& p, bool src_u64, uint64_t units, bool in_place) {
    if (!in_place && scalar_serves(p, units)) return NTTB_ENGINE_SCALAR;
    if (int8_serves(p, src_u64) && units >= kInt8MinUnits) return NTTB_ENGINE_INT8;
    if (tiles_serve(p) && p.log_n >= kTilesMinLog && (units << p.log_n) >= kTilesMinResidues) return NTTB_ENGINE_TILES;
    return NTTB_ENGINE_SCALAR;
}

bool auto_radix32(const Plan32& p, uint64_t units, int engine) {
    return engine == NTTB_ENGINE_AUTO && env_engine() == NTTB_ENGINE_AUTO && radix_serves(p.log_n) &&
           scalar_serves(p, units);
}

int run_transform32(Plan32& p, const void* src, void* dst, bool src_u64, uint32_t n_polys, bool inverse,
                    int engine, cudaStream_t s) {
    if (engine == NTTB_ENGINE_AUTO) engine = env_engine();
    const bool named = engine != NTTB_ENGINE_AUTO;
    if (!named) engine = auto_engine32(p, src_u64, (uint64_t)n_polys * p.n_limbs, src == dst);
    return run_engine32(p, src, dst, src_u64, n_polys, inverse, engine, named, s);
}

int run_engine32(Plan32& p, const void* src, void* dst, bool src_u64, uint32_t n_polys, bool inverse, int engine,
                 bool named, cudaStream_t s) {
    switch (engine) {
        case NTTB_ENGINE_SCALAR:
            return scalar_transform32(p, src, dst, src_u64, n_polys, inverse, s);
        case NTTB_ENGINE_INT8:
            return int8_transform32(p, src, dst, src_u64, n_polys, inverse, s);
        case NTTB_ENGINE_DMMA:
            return dmma_transform32(p, src, dst, src_u64, n_polys, inverse, s);
        case NTTB_ENGINE_TILES:
            return tiles_transform32(p, src, dst, src_u64, n_polys, inverse, named, s);
        default:
            return 1;
    }
}

void engines_release32(Plan32* p) {
    int8_release(p);
    dmma_release(p);
    tiles_release(p);
}

}  // namespace nttb
