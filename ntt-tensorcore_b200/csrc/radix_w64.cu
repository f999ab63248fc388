// radix_w64.cu -- register-radix passes (radix.cuh) over the drop-in API's
// uint64 words with a modulus below 2^31; the first pass stages uint32.
#include "radix_host.cuh"

namespace nttb {

int radix_w64(const LimbDev<M32>* limbs, uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, void* mid,
              uint32_t n_polys, bool inverse, cudaStream_t s) {
    return rdx::transform<M32, uint64_t, uint32_t, 4>(limbs, log_n, n_limbs, src, dst, mid, n_polys, inverse, s);
}

uint32_t radix_w64_bounds_errors(bool clear) { return rdx::bounds_errors(clear); }

}  // namespace nttb
