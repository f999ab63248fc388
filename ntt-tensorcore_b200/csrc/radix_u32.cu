// radix_u32.cu -- register-radix passes (radix.cuh) over uint32 residues.
#include "radix_host.cuh"

namespace nttb {

int radix_u32(const LimbDev<M32>* limbs, uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, void* mid,
              uint32_t n_polys, bool inverse, cudaStream_t s) {
    return rdx::transform<M32, uint32_t, uint32_t, 4>(limbs, log_n, n_limbs, src, dst, mid, n_polys, inverse, s);
}

// Forward then inverse in place; two-pass sizes stage through `mid`.
int radix_round_trip_u32(const LimbDev<M32>* limbs, uint32_t log_n, uint32_t n_limbs, uint32_t* data, void* mid,
                         uint32_t n_polys, cudaStream_t s) {
    using namespace rdx;
    const Args a = make_args<M32>(log_n, n_limbs, data, data, n_polys);
#define NTTB_SINGLE(l) \
    case l: return launch_single<M32, uint32_t, l, 4, kBoth>(a, limbs, s);
#define NTTB_TWO(l) \
    case l: return launch_round_trip<M32, uint32_t, l, 4>(a, mid, limbs, s);
    switch (log_n) {
        NTTB_SINGLE(5) NTTB_SINGLE(6) NTTB_SINGLE(7) NTTB_SINGLE(8) NTTB_SINGLE(9)
        NTTB_SINGLE(10) NTTB_SINGLE(11) NTTB_SINGLE(12) NTTB_SINGLE(13)
        NTTB_TWO(14) NTTB_TWO(15) NTTB_TWO(16) NTTB_TWO(17) NTTB_TWO(18) NTTB_TWO(19) NTTB_TWO(20)
        default: return 1;
    }
#undef NTTB_SINGLE
#undef NTTB_TWO
}

uint32_t radix_u32_bounds_errors(bool clear) { return rdx::bounds_errors(clear); }

}  // namespace nttb
