// radix_q64.cu -- register-radix passes (radix.cuh) for moduli below 2^62.
#include "radix_host.cuh"

namespace nttb {

int radix_q64(const LimbDev<M64>* limbs, uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, void* mid,
              uint32_t n_polys, bool inverse, cudaStream_t s) {
    return rdx::transform<M64, uint64_t, uint64_t, 3>(limbs, log_n, n_limbs, src, dst, mid, n_polys, inverse, s);
}

uint32_t radix_q64_bounds_errors(bool clear) { return rdx::bounds_errors(clear); }

}  // namespace nttb
