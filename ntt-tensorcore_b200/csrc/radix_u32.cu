// radix_u32.cu -- register-radix passes (radix.cuh) over uint32 residues.
#include "radix_host.cuh"

namespace nttb {

int radix_u32(const Plan32& p, const void* src, void* dst, void* mid, uint32_t n_polys, bool inverse, cudaStream_t s) {
    return rdx::transform<M32, uint32_t, uint32_t, 4>(p.d_limbs, p.log_n, p.n_limbs, src, dst, mid, n_polys, inverse, s);
}

}  // namespace nttb
