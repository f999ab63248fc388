// plan.cu -- host-side construction of per-modulus constants and device tables.
#include <cuda_runtime.h>

#include <cstring>
#include <type_traits>
#include <string>
#include <vector>

#include "plan.hpp"

namespace nttb {

// Smallest g >= 2 with g^((q-1)/p) != 1 for every p in {2,3,5,7} dividing
// q-1: the generator rule of include/modular_arith.cuh:130-147, kept
// identical so that omega (and hence every output) matches the reference.
uint64_t reference_generator(uint64_t q) {
    static const uint64_t small[4] = {2, 3, 5, 7};
    for (uint64_t g = 2; g < q; g++) {
        bool ok = true;
        for (uint64_t p : small)
            if ((q - 1) % p == 0 && h_powmod(g, (q - 1) / p, q) == 1) { ok = false; break; }
        if (ok) return g;
    }
    return 0;
}

static bool probably_prime(uint64_t q) {
    if (q < 2) return false;
    for (uint64_t p : {2ull, 3ull, 5ull, 7ull, 11ull, 13ull, 17ull, 19ull, 23ull, 29ull, 31ull, 37ull}) {
        if (q % p == 0) return q == p;
    }
    uint64_t d = q - 1;
    int r = 0;
    while ((d & 1) == 0) { d >>= 1; r++; }
    for (uint64_t a : {2ull, 3ull, 5ull, 7ull, 11ull, 13ull, 17ull, 19ull, 23ull, 29ull, 31ull, 37ull}) {
        uint64_t x = h_powmod(a, d, q);
        if (x == 1 || x == q - 1) continue;
        bool comp = true;
        for (int i = 1; i < r; i++) {
            x = h_mulmod(x, x, q);
            if (x == q - 1) { comp = false; break; }
        }
        if (comp) return false;
    }
    return true;
}

bool make_limb_host(uint64_t q, uint64_t n, bool need_psi, LimbHost* out, std::string* why) {
    if (q < 3 || (q & 1) == 0) { *why = "modulus must be an odd prime"; return false; }
    if (!probably_prime(q)) { *why = "modulus " + std::to_string(q) + " is not prime"; return false; }
    const uint64_t order = need_psi ? 2 * n : n;
    if ((q - 1) % order != 0) {
        *why = "modulus " + std::to_string(q) + " has no primitive " + std::to_string(order) + "-th root (q-1 not divisible)";
        return false;
    }
    LimbHost L;
    L.q = q;
    L.g = reference_generator(q);
    L.omega = h_powmod(L.g, (q - 1) / n, q);
    // The reference's generator test only screens {2,3,5,7}; require that the
    // resulting omega really has order n (it always does for the supported
    // primes because the p = 2 test makes g a non-residue).
    if (n > 1 && h_powmod(L.omega, n / 2, q) == 1) { *why = "omega is not a primitive n-th root"; return false; }
    L.omega_inv = h_invmod(L.omega, q);
    L.n_inv = h_invmod(n % q, q);
    if (need_psi) {
        L.psi = h_powmod(L.g, (q - 1) / (2 * n), q);
        L.psi_inv = h_invmod(L.psi, q);
    }
    *out = L;
    return true;
}

template <class E, class ToMont>
static void fill_powers(E* dst, uint64_t base, uint64_t start, uint64_t n, uint64_t q, ToMont tm) {
    uint64_t x = start % q;
    for (uint64_t e = 0; e < n; e++) {
        dst[e] = tm(x);
        x = h_mulmod(x, base, q);
    }
}

// Shoup pairs from Montgomery-form powers, on the device.  `pw` holds
// base^e R mod q, e < n.  Pair i = 2^s + k: base^((n / 2^(s+1)) (odd ? 1 + 2k :
// k)), or its inverse, which is base^(n - e) for a base of order n and its
// negative for one of order 2n (odd).  The plain root is a Montgomery product
// by 1; its quotient floor(w R / q) = (w R - r) / q, with r = w R mod q the
// table's own entry, is r * (-q^-1) mod R.
template <class A>
__global__ void shoup_pairs_kernel(typename A::elem* out, const typename A::elem* pw, uint32_t log_n, A ar, bool odd,
                                   bool inverse) {
    using E = typename A::elem;
    const uint32_t n = 1u << log_n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        E r = 0;
        if (i) {
            const uint32_t s = 31 - __clz(i), k = i - (1u << s), step = n >> (s + 1);
            const uint32_t e = odd ? step * (1 + 2 * k) : step * k;
            r = inverse && e ? pw[n - e] : pw[e];
            if (inverse && odd) r = ar.q - r;
        }
        out[2 * (size_t)i] = ar.mul(r, (E)1);
        out[2 * (size_t)i + 1] = r * ar.qinv;
    }
}

template <class A, class PlanT, class ToMont>
static int build_common(PlanT* p, uint32_t log_n, const uint64_t* moduli, uint32_t n_limbs, bool negacyclic,
                        uint64_t qmax, ToMont tm, std::string* why) {
    using E = typename A::elem;
    p->log_n = log_n;
    p->n = 1u << log_n;
    p->n_limbs = n_limbs;
    p->negacyclic = negacyclic;
    if constexpr (std::is_same<PlanT, Plan32>::value) {
        if (cudaGetDevice(&p->device) != cudaSuccess) p->device = -1;
    }
    const uint64_t n = p->n;
    if (n_limbs == 0) { *why = "no moduli"; return 1; }
    p->limbs.resize(n_limbs);
    for (uint32_t l = 0; l < n_limbs; l++) {
        if (moduli[l] >= qmax) { *why = "modulus " + std::to_string(moduli[l]) + " too large for this path"; return 1; }
        if (!make_limb_host(moduli[l], n, negacyclic, &p->limbs[l], why)) return 1;
    }
    // Powers in Montgomery form, uploaded: omega^e, omega^-e (, psi^e, n^-1
    // psi^-e); a negacyclic plan of a size that the register-radix passes serve
    // needs psi^e alone.  Behind them, made on the device, 2n words of Shoup
    // pairs per direction: of psi for such a plan, else of omega (one table for
    // the radix-2 and the register-radix passes).
    const bool radix = radix_serves(log_n), lean = negacyclic && radix;
    const uint32_t tables = lean ? 1 : negacyclic ? 4 : 2;
    const size_t per_limb = (size_t)(tables + 4) * n, up = (size_t)tables * n;
    std::vector<E> host(up), scale(4 * (size_t)n_limbs);
    std::vector<LimbDev<A>> devs(n_limbs);
    E *d_tables = nullptr, *d_scale = nullptr;
    if (cudaMalloc(&d_tables, per_limb * n_limbs * sizeof(E)) != cudaSuccess) { *why = "cudaMalloc failed"; return 4; }
    p->allocations.push_back(d_tables);
    if (cudaMalloc(&d_scale, scale.size() * sizeof(E)) != cudaSuccess) { *why = "cudaMalloc failed"; return 4; }
    p->allocations.push_back(d_scale);
    const unsigned grid = (unsigned)((n + 255) / 256 < 592 ? (n + 255) / 256 : 592);
    for (uint32_t l = 0; l < n_limbs; l++) {
        const LimbHost& L = p->limbs[l];
        const uint64_t q = L.q;
        E *h = host.data(), *d = d_tables + per_limb * l;
        auto mont = [&](uint64_t x) { return tm(x, q); };
        LimbDev<A> dv{};
        dv.ar.q = (E)q;
        if constexpr (sizeof(E) == 4) dv.ar.qinv = h_neg_inv32((uint32_t)q);
        else dv.ar.qinv = h_neg_inv64(q);
        dv.ninv_m = (E)tm(L.n_inv, q);
        E* pairs = d + up;
        if (lean) {
            fill_powers(h, L.psi, 1, n, q, mont);
            dv.psi = d;
        } else {
            fill_powers(h, L.omega, 1, n, q, mont);
            fill_powers(h + n, L.omega_inv, 1, n, q, mont);
            dv.tw = d;
            dv.tw_inv = d + n;
            if (negacyclic) {
                fill_powers(h + 2 * n, L.psi, 1, n, q, mont);
                fill_powers(h + 3 * n, L.psi_inv, L.n_inv, n, q, mont);
                dv.psi = d + 2 * n;
                dv.psi_inv = d + 3 * n;
            }
        }
        if (cudaMemcpy(d, h, up * sizeof(E), cudaMemcpyHostToDevice) != cudaSuccess) { *why = "cudaMemcpy failed"; return 3; }
        // pair 0 is unused: the radix-2 levels start at pair 1 (radix-2 root of length 2)
        for (int inv = 0; inv < 2; inv++) {
            E* t = pairs + (size_t)inv * 2 * n;
            shoup_pairs_kernel<A><<<grid, 256>>>(t, lean ? dv.psi : dv.tw, log_n, dv.ar, lean, inv != 0);
            (inv ? dv.rt_inv : dv.rt) = t;
            if (!lean) (inv ? dv.tw_inv_sh : dv.tw_sh) = t + 2;
        }
        // n^-1 and n^-1 W, W = the inverse's one root of stage 0 (psi^-(n/2) or 1)
        const uint64_t w0 = lean ? h_mulmod(L.n_inv, h_powmod(L.psi_inv, n / 2, q), q) : L.n_inv;
        const uint64_t sc[2] = {L.n_inv, w0};
        for (int i = 0; i < 2; i++) {
            scale[4 * l + 2 * i] = (E)sc[i];
            scale[4 * l + 2 * i + 1] = (E)((((unsigned __int128)sc[i]) << (8 * sizeof(E))) / q);
        }
        dv.scale = d_scale + 4 * l;
        devs[l] = dv;
    }
    if (cudaMemcpy(d_scale, scale.data(), scale.size() * sizeof(E), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaStreamSynchronize(0) != cudaSuccess) {
        *why = "table set-up failed";
        return 3;
    }
    LimbDev<A>* d_limbs = nullptr;
    if (cudaMalloc(&d_limbs, devs.size() * sizeof(LimbDev<A>)) != cudaSuccess) { *why = "cudaMalloc failed"; return 4; }
    p->allocations.push_back(d_limbs);
    if (cudaMemcpy(d_limbs, devs.data(), devs.size() * sizeof(LimbDev<A>), cudaMemcpyHostToDevice) != cudaSuccess) {
        *why = "cudaMemcpy failed";
        return 3;
    }
    p->d_limbs = d_limbs;
    return 0;
}

int build_plan32(Plan32* p, uint32_t log_n, const uint64_t* moduli, uint32_t n_limbs, bool negacyclic,
                 std::string* why) {
    return build_common<M32>(p, log_n, moduli, n_limbs, negacyclic, 1ull << 31,
                             [](uint64_t x, uint64_t q) { return h_to_mont32(x, q); }, why);
}

int build_plan64(Plan64* p, uint32_t log_n, const uint64_t* moduli, uint32_t n_limbs, bool negacyclic,
                 std::string* why) {
    return build_common<M64>(p, log_n, moduli, n_limbs, negacyclic, 1ull << 62,
                             [](uint64_t x, uint64_t q) { return h_to_mont64(x, q); }, why);
}

void* plan_workspace(void** ws, size_t* ws_bytes, size_t bytes) {
    if (*ws_bytes >= bytes) return *ws;
    if (*ws) cudaFree(*ws);
    *ws = nullptr;
    *ws_bytes = 0;
    if (cudaMalloc(ws, bytes) != cudaSuccess) {
        *ws = nullptr;
        return nullptr;
    }
    *ws_bytes = bytes;
    return *ws;
}

static cudaMemPool_t plan_pool(PlanPool& pp) {  // pp.mu held
    if (pp.tried) return pp.pool;
    pp.tried = true;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    if (cudaGetDevice(&props.location.id) != cudaSuccess || cudaMemPoolCreate(&pp.pool, &props) != cudaSuccess) {
        cudaGetLastError();
        pp.pool = nullptr;
        return nullptr;
    }
    pp.device = props.location.id;
    // what one call frees, the next takes; the pool goes with the plan
    uint64_t keep = 2 * PlanPool::kHeldMax;
    int off = 0;            // streams never wait for one another for memory
    cudaMemPoolSetAttribute(pp.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolSetAttribute(pp.pool, cudaMemPoolReuseAllowInternalDependencies, &off);
    return pp.pool;
}

namespace {
struct GraphRef {
    std::shared_ptr<GraphWorkspaces> all;
    GraphWorkspaces::Buf* buf;
};
void CUDART_CB drop_graph_ref(void* p) {  // no CUDA calls here
    GraphRef* r = static_cast<GraphRef*>(p);
    {
        std::lock_guard<std::mutex> lock(r->all->mu);
        r->buf->held = false;
    }
    delete r;
}
}  // namespace

// A workspace of the graph that `s` is being captured into: calls captured on one
// stream of one capture run one after the other and share it.  The stream's handle
// stands for it, which does not change hands during a capture (the per-thread
// handle is one of several streams; cudaStreamGetId invalidates a capture).
static GraphWorkspaces::Buf* graph_workspace(const std::shared_ptr<GraphWorkspaces>& all, size_t bytes,
                                             unsigned long long capture, cudaGraph_t graph, cudaStream_t stream) {
    GraphWorkspaces::Buf* b = nullptr;
    {
        std::lock_guard<std::mutex> lock(all->mu);
        for (GraphWorkspaces::Buf& t : all->bufs) {
            if (t.bytes < bytes) continue;
            if (t.held && t.capture == capture && t.stream == stream && stream != cudaStreamPerThread) return &t;
            if (!t.held && (!b || t.bytes < b->bytes)) b = &t;
        }
        if (b) {
            b->held = true;
            b->capture = capture;
            b->stream = stream;
        }
    }
    if (!b) {
        // no capture depends on the allocation: it may be made in the middle of one
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* ptr = nullptr;
        const cudaError_t e = cudaMalloc(&ptr, bytes);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) return nullptr;
        std::lock_guard<std::mutex> lock(all->mu);
        all->bufs.emplace_back();
        b = &all->bufs.back();
        b->ptr = ptr;
        b->bytes = bytes;
        b->held = true;
        b->capture = capture;
        b->stream = stream;
    }
    GraphRef* ref = new GraphRef{all, b};
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, ref, drop_graph_ref, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        drop_graph_ref(ref);
        return nullptr;
    }
    if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaUserObjectRelease(obj, 1);
        return nullptr;
    }
    return b;
}

StreamWorkspace::StreamWorkspace(PlanPool& pp, size_t bytes, cudaStream_t s) : stream_(s) {
    unsigned long long id = 0, capture = 0;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo(s, &status, &capture, &graph) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (status != cudaStreamCaptureStatusNone) {
        GraphWorkspaces::Buf* b = nullptr;
        if (status == cudaStreamCaptureStatusActive) {
            std::lock_guard<std::mutex> lock(pp.mu);
            b = graph_workspace(pp.graphs, bytes, capture, graph, s);
        }
        if (b) {
            lock_ = std::unique_lock<std::mutex>(b->mu);
            ptr = b->ptr;
        } else {
            cudaGetLastError();
        }
        return;
    }
    if (cudaStreamGetId(s, &id) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    PlanPool::Slot* slot = nullptr;
    {
        std::lock_guard<std::mutex> lock(pp.mu);
        if (!plan_pool(pp)) return;
        for (int i = 0; i < pp.used && !slot; i++)
            if (pp.slot[i].stream == id) slot = &pp.slot[i];
        if (!slot && pp.used < PlanPool::kSlots && pp.held + bytes <= PlanPool::kHeldMax) {
            slot = &pp.slot[pp.used++];
            slot->stream = id;
        }
    }
    if (slot) {
        lock_ = std::unique_lock<std::mutex>(slot->mu);
        if (slot->bytes >= bytes) {
            ptr = slot->ptr;
            return;
        }
        bool fits;
        {
            std::lock_guard<std::mutex> lock(pp.mu);
            fits = pp.held - slot->bytes + bytes <= PlanPool::kHeldMax;
            if (fits) pp.held += bytes - slot->bytes;
        }
        if (fits) {
            if (slot->ptr) cudaFreeAsync(slot->ptr, s);  // behind the stream's earlier calls
            slot->ptr = nullptr;
            slot->bytes = 0;
            if (cudaMallocFromPoolAsync(&slot->ptr, bytes, pp.pool, s) == cudaSuccess) {
                ptr = slot->ptr;
                slot->bytes = bytes;
            } else {
                cudaGetLastError();
                slot->ptr = nullptr;
                std::lock_guard<std::mutex> lock(pp.mu);
                pp.held -= bytes;
            }
            return;
        }
        lock_.unlock();
    }
    if (cudaMallocFromPoolAsync(&ptr, bytes, pp.pool, s) == cudaSuccess) {
        per_call_ = true;
    } else {
        cudaGetLastError();
        ptr = nullptr;
    }
}

StreamWorkspace::~StreamWorkspace() {
    if (per_call_) cudaFreeAsync(ptr, stream_);
}

static void free_pool(PlanPool& pp) {
    std::vector<void*> captured;  // freed without the lock, which graphs' callbacks take
    {
        std::lock_guard<std::mutex> lock(pp.graphs->mu);
        for (GraphWorkspaces::Buf& b : pp.graphs->bufs) {
            captured.push_back(b.ptr);
            b.ptr = nullptr;
            b.bytes = 0;
        }
    }
    for (void* p : captured) cudaFree(p);
    if (!pp.pool) return;  // no call has staged anything outside a capture
    // cudaFree of stream-ordered memory does not wait for the calls that still use
    // it, as that of cudaMalloc's does: wait for them here.  Where the device cannot
    // be waited for, the memory stays allocated.
    int dev = pp.device;
    cudaGetDevice(&dev);
    if (dev != pp.device) cudaSetDevice(pp.device);
    if (cudaDeviceSynchronize() == cudaSuccess) {
        for (PlanPool::Slot& t : pp.slot)
            if (t.ptr) cudaFree(t.ptr);
        cudaMemPoolDestroy(pp.pool);  // its memory goes once the last free has been reached
    } else {
        cudaGetLastError();
    }
    if (dev != pp.device) cudaSetDevice(dev);
    for (PlanPool::Slot& t : pp.slot) {
        t.stream = 0;
        t.ptr = nullptr;
        t.bytes = 0;
    }
    pp.used = 0;
    pp.held = 0;
    pp.pool = nullptr;
    pp.tried = false;
}

void free_plan32(Plan32* p) {
    free_pool(p->pool);
    if (p->ws) cudaFree(p->ws);
    p->ws = nullptr;
    p->ws_bytes = 0;
    for (void* a : p->allocations) cudaFree(a);
    p->allocations.clear();
    p->d_limbs = nullptr;
}

void free_plan64(Plan64* p) {
    free_pool(p->pool);
    if (p->ws) cudaFree(p->ws);
    p->ws = nullptr;
    p->ws_bytes = 0;
    for (void* a : p->allocations) cudaFree(a);
    p->allocations.clear();
    p->d_limbs = nullptr;
}

}  // namespace nttb
