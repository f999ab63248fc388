// plan.hpp -- host-side plan structures shared by the engines and the C-ABI.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <list>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "arith.cuh"

namespace nttb {

// Per-limb constants handed to the kernels (one array entry per limb).
template <class A>
struct LimbDev {
    A ar;                              // modulus + Montgomery constant
    typename A::elem ninv_m;           // n^-1 * R mod q
    typename A::elem pad_;
    const typename A::elem* tw;        // omega^e * R,   e < n
    const typename A::elem* tw_inv;    // omega^-e * R,  e < n
    const typename A::elem* psi;       // psi^e * R,     e < n (negacyclic only)
    const typename A::elem* psi_inv;   // n^-1 psi^-e R, e < n (negacyclic only)
    // Shoup pairs of the radix-2 butterflies, level by level: the roots of
    // length L = 2^l sit at pairs 2^(l-1) - 1 .. 2^l - 2 (k < L/2), each pair
    // root_L^k (plain form) and floor(root_L^k * 2^bits / q) (bits = 32 or 64),
    // so a pass of length L reads one contiguous run
    const typename A::elem* tw_sh;
    const typename A::elem* tw_inv_sh;
    // Shoup pairs of the register-radix passes (radix.cuh), stage by stage: pair
    // 2^s + i = root^((n / 2^(s+1)) (1 + 2 i)) (root = psi, negacyclic) or
    // root^((n / 2^(s+1)) i) (root = omega, cyclic), i < 2^s; the inverse's
    // roots in rt_inv; scale = the pairs of n^-1 and of n^-1 rt_inv[1]
    const typename A::elem* rt;
    const typename A::elem* rt_inv;
    const typename A::elem* scale;
};

// Host view of one modulus at one transform size.
struct LimbHost {
    uint64_t q = 0, g = 0, omega = 0, omega_inv = 0, psi = 0, psi_inv = 0, n_inv = 0;
};

// Fills LimbHost with the generator rule of the reference
// (include/modular_arith.cuh:130-151) plus psi = g^((q-1)/2n).
bool make_limb_host(uint64_t q, uint64_t n, bool need_psi, LimbHost* out, std::string* why);

// Transform direction / twist flags.
enum : uint32_t {
    F_PRE_PSI = 1u,       // multiply input element n by psi^n           (negacyclic forward)
    F_PRE_TW = 2u,        // multiply input (row a, col b) by root^(a*b)  (four-step inverse)
    F_POST_TW = 4u,       // multiply output (row d, col b) by root^(d*b) (four-step pass 1)
    F_POST_SCALE = 8u,    // multiply output by n^-1                      (cyclic inverse)
    F_POST_PSI_INV = 16u, // multiply output element n by n^-1 psi^-n    (negacyclic inverse)
    F_STORE_T = 32u,      // MODE_COL: store output (row k, col b) at b*N1 + k (transposed)
};

// Pass geometries of the scalar engine.
enum PassMode : int {
    MODE_COL = 0,          // vectors = columns of [N1 x N2]; out in place (row k, col b)
    MODE_ROW_NAT = 1,      // vectors = rows d; out X[d + N1*k] (natural order), or with F_STORE_T
                           // row by row at d*len + k (F_POST_TW: times root^(k*d))
    MODE_GATHER_T = 2,     // vectors = chunks of the N1 x N2 -> N2 x N1 transpose; out in place
    MODE_ROW_SCATTER_T = 3 // vectors = contiguous chunks; out through the transpose back
};

struct PassArgs {
    const void* src;
    void* dst;
    uint64_t poly_stride;  // elements between consecutive polynomials
    uint32_t n, log_n;
    uint32_t n1, n2;       // matrix view of one transform
    uint32_t len, log_len; // DFT length of this pass
    uint32_t vec_per_tile;
    uint32_t n_limbs;
    uint32_t flags;
    int inverse;
};

// Workspaces of captured calls.  A graph holds its own until it and what was
// instantiated from it are gone; then the next capture may take them.  The plan
// frees them, and the graphs' references may outlive it.
struct GraphWorkspaces {
    struct Buf {
        void* ptr = nullptr;
        size_t bytes = 0;
        unsigned long long capture = 0;  // the calls that share it: one stream of one capture
        cudaStream_t stream = nullptr;
        bool held = false;
        std::mutex mu;  // held by the call that is being captured
    };
    std::mutex mu;
    std::list<Buf> bufs;
};

// The pool behind a plan's stream-ordered workspaces (StreamWorkspace), and the
// workspaces that its first kSlots streams keep, kHeldMax bytes in all.
struct PlanPool {
    static constexpr int kSlots = 32;
    static constexpr size_t kHeldMax = 512u << 20;
    struct Slot {
        unsigned long long stream = 0;  // cudaStreamGetId: never reused
        void* ptr = nullptr;
        size_t bytes = 0;
        std::mutex mu;  // guards ptr and bytes; held by the call that uses them
    };
    cudaMemPool_t pool = nullptr;
    int device = -1;
    bool tried = false;
    Slot slot[kSlots];
    int used = 0;     // slots that have a stream
    size_t held = 0;  // bytes of all slots
    std::mutex mu;    // guards what is above but the slots' own memory
    std::shared_ptr<GraphWorkspaces> graphs = std::make_shared<GraphWorkspaces>();
};

// A u32-residue plan (q < 2^31 for every limb).
struct Plan32 {
    uint32_t log_n = 0, n = 0, n_limbs = 0;
    bool negacyclic = false;
    std::vector<LimbHost> limbs;
    LimbDev<M32>* d_limbs = nullptr;  // device array, n_limbs entries
    std::vector<void*> allocations;   // device memory owned by the plan
    void* engine_data[4] = {nullptr, nullptr, nullptr, nullptr};  // per-engine host-side caches
    std::mutex engine_mu;             // guards the lazy construction of engine_data
    void* ws = nullptr;               // plan_workspace's buffer
    size_t ws_bytes = 0;
    PlanPool pool;                    // stream-ordered workspaces (StreamWorkspace)
    int device = -1;                  // the CUDA device holding d_limbs and the tables
};

// A u64-residue plan (q < 2^62).
struct Plan64 {
    uint32_t log_n = 0, n = 0, n_limbs = 0;
    bool negacyclic = false;
    std::vector<LimbHost> limbs;
    LimbDev<M64>* d_limbs = nullptr;
    std::vector<void*> allocations;
    void* ws = nullptr;
    size_t ws_bytes = 0;
    PlanPool pool;
    void* engine_data = nullptr;  // the INT8 wide engine's constants (tc_wide.cu)
    std::mutex engine_mu;         // guards their lazy construction
};

// Status of the kernel launch just made: 0, or 2 after keeping its CUDA
// error for the C-ABI's message (cudaGetLastError clears a launch error, so
// the caller could not read it again).
int launch_rc();
// The same for a launch call that returned `e` itself (cudaLaunchKernelEx).
int launch_rc(cudaError_t e);
// C-ABI status of an engine's return code: 0 -> cudaGetLastError's status,
// 1 -> NTTB_ERR_UNSUPPORTED ("<what>: shape not served"), 2 or more ->
// NTTB_ERR_CUDA with the error kept by launch_rc (or the current one).
int engine_status(int rc, const char* what);

// A workspace for the call that constructs it, until the call has enqueued its
// launches: stream-ordered memory from a pool that the plan owns.  The first
// kSlots streams that use a plan keep theirs, as far as kHeldMax goes (an allocation
// and a free cost a call 2 us on the host, 10 where streams take turns: in place
// 8 x 2^16 on ten streams 6 -> 17 us a call); it is locked meanwhile, so that threads
// on one stream enqueue one after the other.  Further calls allocate their own.  So
// calls on several streams or threads never share one.  The pool keeps twice
// kHeldMax until the plan is destroyed, and gives back the rest.
// While the stream is being captured it is a buffer that the graph holds
// (GraphWorkspaces), so that a captured call needs no earlier one and replays race
// neither with other graphs nor with calls outside.  ptr: null on failure.
class StreamWorkspace {
public:
    StreamWorkspace(PlanPool& pool, size_t bytes, cudaStream_t s);
    ~StreamWorkspace();
    StreamWorkspace(const StreamWorkspace&) = delete;
    void* ptr = nullptr;

private:
    std::unique_lock<std::mutex> lock_;
    cudaStream_t stream_;
    bool per_call_ = false;
};
// scalar_transform32's and scalar_transform64's status when the workspace could not be had.
constexpr int kNoWorkspace = 3;

// Returns a device workspace of at least `bytes`, growing the plan's buffer
// (the DMMA and the INT8 wide engine stage their first pass there).  Calls
// that share a plan must be ordered on one stream while they use it.
void* plan_workspace(void** ws, size_t* ws_bytes, size_t bytes);

int build_plan32(Plan32* p, uint32_t log_n, const uint64_t* moduli, uint32_t n_limbs, bool negacyclic,
                 std::string* why);
int build_plan64(Plan64* p, uint32_t log_n, const uint64_t* moduli, uint32_t n_limbs, bool negacyclic,
                 std::string* why);
void free_plan32(Plan32* p);
void free_plan64(Plan64* p);

// Scalar engine entry points (scalar_engine.cu).  Storage is u32 or u64
// words; data layout is [poly][limb][n].
int scalar_transform32(Plan32& p, const void* src, void* dst, bool src_u64, uint32_t n_polys, bool inverse,
                       cudaStream_t s);
// Whether a call of `units` (polynomial, limb) rows is within its grid limits.
inline bool scalar_serves(const Plan32& p, uint64_t units) { return p.n_limbs <= 65535 && units / p.n_limbs <= 65535; }
int scalar_transform64(Plan64& p, const void* src, void* dst, uint32_t n_polys, bool inverse, cudaStream_t s);
// Forward then inverse in place (kNoWorkspace: as above; 1: size not served).
int scalar_round_trip32(Plan32& p, uint32_t* data, uint32_t n_polys, cudaStream_t s);
// In-place uint32 transform staging its first pass in a caller-supplied buffer
// `ws` (n_polys * n_limbs * n words); allocates nothing.
int scalar_transform32_ws(const Plan32& p, uint32_t* data, void* ws, uint32_t n_polys, bool inverse,
                          cudaStream_t s);
// Bytes of `ws` that scalar_transform32_ws stages in for n_polys polynomials
// (0 when the shape runs as one pass and stages nothing).
size_t scalar_transform32_ws_bytes(const Plan32& p, uint32_t n_polys);

// Register-radix passes on CUDA cores (radix.cuh): sizes 2^5 .. 2^20, n_polys x
// n_limbs rows under the moduli `limbs`.  Sizes above 2^13 (2^12: 64-bit) run two passes through
// `mid`, n_polys * n_limbs * n words (uint32 for the 31-bit moduli, uint64 for the
// wide ones): the destination, if the source is another buffer and the words have
// its size, or a workspace.
constexpr uint32_t kRadixMinLog = 5, kRadixMaxLog = 20;
// Largest size of one launch.  64-bit rows of 2^13 fill an SM with one block of 1024
// threads and five rounds of barriers: two passes take 9.5 us for up to 40 rows and
// 114 for 1200, one launch 14.5 and 133 (at 148 rows, one wave, 16.4 and 15.1).
constexpr uint32_t kRadixSingleMax = 13, kRadixSingleMax64 = 12;
inline bool radix_serves(uint32_t log_n) { return log_n >= kRadixMinLog && log_n <= kRadixMaxLog; }
int radix_u32(const LimbDev<M32>* limbs, uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, void* mid,
              uint32_t n_polys, bool inverse, cudaStream_t s);
int radix_round_trip_u32(const LimbDev<M32>* limbs, uint32_t log_n, uint32_t n_limbs, uint32_t* data, void* mid,
                         uint32_t n_polys, cudaStream_t s);
int radix_w64(const LimbDev<M32>* limbs, uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, void* mid,
              uint32_t n_polys, bool inverse, cudaStream_t s);
int radix_q64(const LimbDev<M64>* limbs, uint32_t log_n, uint32_t n_limbs, const void* src, void* dst, void* mid,
              uint32_t n_polys, bool inverse, cudaStream_t s);

// Rows that a call stages at a time: 2^25 words, or one row where that is larger.
// Longer calls run their rows in groups of that, one after the other, so that what a
// plan holds for a stream does not grow with the call.  A group pays for its last
// waves and shares roots among fewer polynomials; us in place at 2^24 / 2^25 words /
// one group: 64 x 24 x 2^16 448 / 425 / 385, 8 x 30 x 2^18 347 / 328 / 304, round
// trip 16 x 24 x 2^16 198 / 187 / 187, 64-bit 20 x 2^20 378 / 362 / 364.
constexpr uint64_t kStagedWordsMax = 1ull << 25;
struct RowGroups {
    uint32_t polys, limbs;  // per group; limbs < the plan's: groups lie within one polynomial
};
inline RowGroups row_groups(uint32_t log_n, uint32_t n_limbs, uint32_t n_polys) {
    const uint64_t most = kStagedWordsMax >> log_n > 0 ? kStagedWordsMax >> log_n : 1;
    // groups of even size: the last one is not a remainder of a few rows
    auto even = [](uint64_t total, uint64_t per) {
        const uint64_t k = (total + per - 1) / per;
        return (uint32_t)((total + k - 1) / k);
    };
    if (n_limbs <= most) return {even(n_polys, most / n_limbs), n_limbs};
    return {1, even(n_limbs, most)};
}

// INT8 tensor-core engine for the wide plans (tc_wide.cu): n = 2^20, cyclic,
// moduli below 2^62 on byte planes of uint64 words.  Returns 1 when the plan
// is not served; src may equal dst (the plan workspace holds the first pass).
bool wide_tc_serves(const Plan64& p);
int wide_tc_transform64(Plan64& p, const void* src, void* dst, uint32_t n_polys, bool inverse, cudaStream_t s);
void wide_tc_release(Plan64* p);
uint32_t wide_device_errors(bool clear);
uint32_t wide_bounds_errors(bool clear);

// INT8 tensor-core engine (tc_int8.cu).
bool int8_serves(const Plan32& p, bool src_u64);
int int8_transform32(Plan32& p, const void* src, void* dst, bool src_u64, uint32_t n_polys, bool inverse,
                     cudaStream_t s);
void int8_release(Plan32* p);
uint32_t int8_device_errors(bool clear);
// Failed range checks of the NTT_DEBUG_BOUNDS build (bounds.cuh bits; 0 in the
// release build), per kernel file.
uint32_t int8_bounds_errors(bool clear);
// The INT8 cluster kernel's phase counters (NTT_PHASE_PROFILE build; zeros otherwise).
void int8_phase_profile(uint64_t* out16, bool clear);
uint32_t dmma_bounds_errors(bool clear);
uint32_t batch_bounds_errors(bool clear);
uint32_t radix_u32_bounds_errors(bool clear);
uint32_t radix_w64_bounds_errors(bool clear);
uint32_t radix_q64_bounds_errors(bool clear);
uint32_t klimb_bounds_errors(bool clear);
// Forward then inverse, in place, in one persistent launch.
int int8_forward_inverse32(Plan32& p, uint32_t* data, uint32_t n_polys, cudaStream_t s);

// Uneven-batch queue kernel (batch.cu): its bounded-wait error bits.
uint32_t batch_device_errors(bool clear);

// TMA tile mover (tma_move.cu).  Each returns 0 on launch, 1 when the shape
// or alignment is not served (the caller uses the plain kernels), 2 on a CUDA error.
int tma_transpose_u64(uint64_t* dst, const uint64_t* src, uint64_t rows, uint64_t cols, cudaStream_t stream);
int tma_transpose_square_inplace_u64(uint64_t* d, uint64_t n, cudaStream_t stream);
int tma_bit_reverse_u64(uint64_t* d, int log_n, cudaStream_t stream);
uint32_t tma_move_device_errors(bool clear);

// FP64 DMMA tensor-core engine (tc_dmma.cu).
bool dmma_serves(const Plan32& p, bool src_u64);
int dmma_transform32(Plan32& p, const void* src, void* dst, bool src_u64, uint32_t n_polys, bool inverse,
                     cudaStream_t s);
void dmma_release(Plan32* p);
int scalar_four_step32(const Plan32& p, uint64_t* data, uint64_t* scratch, bool inverse, cudaStream_t s);
// Transform of one uint64-word polynomial in the pre-transposed layout for
// n = M^2 (in place, staged in `mid`, n words); 1 when the plan is not served.
int scalar_pretransposed32(const Plan32& p, uint64_t* data, uint64_t* mid, bool inverse, cudaStream_t s);

}  // namespace nttb
