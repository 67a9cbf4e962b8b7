// State lifecycle, host<->device transfers and FP64 reductions.
//
// Reference: src/states/mod.rs (State, normalize, probabilities,
// inner_product_parallel, measure*) and src/optimization/observable.rs
// (PauliTerm::expectation, PauliObservable::expectation).

#include <algorithm>
#include <cstdarg>
#include <map>
#include <mutex>
#include <queue>
#include <type_traits>

#include "lq_internal.h"
#include "reduce.cuh"

namespace lq {

static thread_local std::string g_last_error;
static uint64_t g_alloc_limit = 0;
static std::mutex g_alloc_mu;
static uint64_t g_alloc_in_use = 0;
static int64_t g_handles = 0;  // live states

int set_error(int code, const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

void clear_error() { g_last_error.clear(); }

KeepError::KeepError() : text_(g_last_error) {}
KeepError::~KeepError() {
    if (on_) g_last_error = std::move(text_);
}

size_t alloc_room() {
    std::lock_guard<std::mutex> lk(g_alloc_mu);
    if (!g_alloc_limit) return (size_t)-1;
    return g_alloc_limit > g_alloc_in_use ? (size_t)(g_alloc_limit - g_alloc_in_use) : 0;
}

int check_state(const lq_state *s) {
    if (!s) return set_error(LQ_ERR_INVALID_ARG, "null state handle");
    if (!s->d) return set_error(LQ_ERR_INVALID_ARG, "state handle has no device buffer");
    return LQ_OK;
}

int check_qubit(const lq_state *s, int q) {
    if (q < 0 || q >= s->n)
        return set_error(LQ_ERR_QUBIT_INDEX, "Invalid qubit index: %d (must be < %d)", q, s->n);
    return LQ_OK;
}

int ensure_prog(lq_state *s, size_t bytes) {
    s->prog_valid = false;  // the caller is about to write the buffer
    if (s->prog_cap >= bytes) return LQ_OK;
    if (s->d_prog) {
        LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
        LQ_CUDA_TRY(cudaFree(s->d_prog));
        s->d_prog = nullptr;
        s->prog_cap = 0;
    }
    size_t cap = std::max<size_t>(bytes, 1 << 16);
    LQ_CUDA_TRY(device_malloc(&s->d_prog, cap));
    s->prog_cap = cap;
    return LQ_OK;
}

// ---------------------------------------------------------------------------
// Workspaces above kOwnWork, shared by all handles: a call takes one that its own stream used
// last or whose last use is over, else a new one, else (at most kPoolBytes are there, of at
// most kKeptWork each) the one unused for longest, and its stream waits for the last use;
// where none is large enough, the ones unused for longest make room.
// They stay until the last handle is destroyed or an allocation fails.  (Kept with each
// handle they were a second copy of every 20- to 22-qubit state that had once been damped or
// sampled; allocated afresh they cost a call 0.4 to 20 ms.)
// ---------------------------------------------------------------------------
constexpr size_t kPoolBytes = 256ull << 20;

struct Workspace {
    int device;
    void *p;
    size_t bytes;
    cudaEvent_t used;  // recorded after the last use, on
    cudaStream_t stream;
    bool idle;         // its last use is known to be over
};

static std::mutex g_pool_mu;
static size_t g_pool_bytes = 0;  // of the workspaces of at most kKeptWork, those in use too
// The free ones, in order of their last use (never destroyed: the driver may be gone by then).
static std::vector<Workspace> &pool() {
    static auto *v = new std::vector<Workspace>();
    return *v;
}

static void drop_workspace(const Workspace &w) {
    cudaFree(w.p);  // (waits for its users)
    cudaEventDestroy(w.used);
}

static void free_pool() {
    std::vector<Workspace> all;
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        all.swap(pool());
        for (const Workspace &w : all) g_pool_bytes -= w.bytes;
    }
    for (const Workspace &w : all) drop_workspace(w);
}

static void free_spares(size_t keep);

cudaError_t device_malloc_bytes(void **p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    free_spares(0);
    free_pool();
    e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

int Work::take(size_t bytes) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    LQ_CUDA_TRY(cudaStreamIsCapturing(s_->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) {  // a graph that outlives the call: its own memory
        LQ_CUDA_TRY(cudaMallocAsync(&p_, bytes, s_->stream));
        kind_ = kCaptured;
        return LQ_OK;
    }
    if (bytes <= kOwnWork) {
        if (s_->work_cap < bytes) {
            if (s_->d_work) {
                LQ_CUDA_TRY(cudaStreamSynchronize(s_->stream));
                LQ_CUDA_TRY(cudaFree(s_->d_work));
                s_->d_work = nullptr;
                s_->work_cap = 0;
            }
            LQ_CUDA_TRY(device_malloc(&s_->d_work, bytes));
            s_->work_cap = bytes;
        }
        p_ = s_->d_work;
        return LQ_OK;
    }
    kind_ = kPooled;
    bool wait = false;
    std::vector<Workspace> drop;
    if (bytes <= kKeptWork) {
        // (in steps of an eighth of the power of two below, so that calls of about the same
        // size share)
        size_t step = kOwnWork;
        while (step * 16 <= bytes) step *= 2;
        bytes = (bytes + step - 1) / step * step;
        std::lock_guard<std::mutex> lk(g_pool_mu);
        auto &v = pool();
        auto fits = [&](const Workspace &w) { return w.device == s_->device && w.bytes >= bytes; };
        auto own = [&](const Workspace &w) { return fits(w) && w.stream == s_->stream; };
        auto idle = [&](const Workspace &w) {
            if (!fits(w) || w.idle) return fits(w);
            const bool over = cudaEventQuery(w.used) == cudaSuccess;
            if (!over) cudaGetLastError();
            return over;
        };
        auto at = std::find_if(v.begin(), v.end(), own);
        if (at == v.end()) at = std::find_if(v.begin(), v.end(), idle);
        if (at == v.end() && g_pool_bytes + bytes > kPoolBytes) {
            at = std::find_if(v.begin(), v.end(), fits);
            wait = true;  // (none that fits is idle)
        }
        while (at == v.end() && !v.empty() && g_pool_bytes + bytes > kPoolBytes) {
            drop.push_back(v.front());  // too small ones make room
            g_pool_bytes -= v.front().bytes;
            v.erase(v.begin());
            at = v.end();
        }
        if (at != v.end()) {
            p_ = at->p;
            bytes_ = at->bytes;
            used_ = at->used;
            v.erase(at);
        } else {
            g_pool_bytes += bytes;
        }
    }
    for (const Workspace &w : drop) drop_workspace(w);
    if (p_) {
        if (wait) LQ_CUDA_TRY(cudaStreamWaitEvent(s_->stream, used_, 0));
        return LQ_OK;
    }
    bytes_ = bytes;
    LQ_CUDA_TRY(cudaEventCreateWithFlags(&used_, cudaEventDisableTiming));
    LQ_CUDA_TRY(device_malloc(&p_, bytes));
    return LQ_OK;
}

Work::~Work() {
    if (kind_ == kCaptured) cudaFreeAsync(p_, s_->stream);
    if (kind_ != kPooled) return;
    const bool counted = bytes_ > 0 && bytes_ <= kKeptWork;
    if (p_ && counted && (idle_ || cudaEventRecord(used_, s_->stream) == cudaSuccess)) {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        if (g_pool_bytes <= kPoolBytes) {
            pool().push_back(Workspace{s_->device, p_, bytes_, used_, s_->stream, idle_});
            return;
        }
    }
    if (p_) cudaStreamSynchronize(s_->stream);
    if (p_) cudaFree(p_);
    if (used_) cudaEventDestroy(used_);
    if (counted) {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        g_pool_bytes -= bytes_;
    }
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// Waits, with the given bound, on an mbarrier phase that never completes (the
// barrier expects one arrival and gets none; no copy targets it), then raises
// the timeout flag: the same give-up path as the pipeline waits of the fused
// and tensor-core passes, exercised without any copy in flight.
__global__ void k_wait_probe(unsigned *__restrict__ flag, unsigned polls) {
    __shared__ __align__(8) uint64_t bar;
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(&bar);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    uint32_t done = 0;
    for (unsigned it = 0; it < polls && !done; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(0u)
            : "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && !done) atomicOr(flag, kFlagTimeout);
}

template <class A>
__device__ __forceinline__ double2 load_amp(const A *v, uint64_t i);
template <>
__device__ __forceinline__ double2 load_amp<double2>(const double2 *v, uint64_t i) {
    return v[i];
}
template <>
__device__ __forceinline__ double2 load_amp<float2>(const float2 *v, uint64_t i) {
    float2 a = v[i];
    return make_double2(a.x, a.y);
}

template <class A>
__global__ void k_norm_partial(const A *__restrict__ v, uint64_t N, double *partials) {
    __shared__ double sh[32];
    double acc[1] = {0.0};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double2 a = load_amp(v, i);
        acc[0] += a.x * a.x + a.y * a.y;
    }
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

template <class A>
__global__ void k_inner_partial(const A *__restrict__ a, const A *__restrict__ b, uint64_t N,
                                double *partials) {
    __shared__ double sh[64];
    double acc[2] = {0.0, 0.0};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double2 x = load_amp(a, i), y = load_amp(b, i);
        // conj(x) * y
        acc[0] += x.x * y.x + x.y * y.y;
        acc[1] += x.x * y.y - x.y * y.x;
    }
    block_sum<2>(acc, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = acc[0];
        partials[2 * blockIdx.x + 1] = acc[1];
    }
}

// Sum nparts partials of NC components in a fixed order (deterministic).
template <int NC>
__global__ void k_final_sum(const double *partials, int nparts, double *out) {
    __shared__ double sh[32 * NC];
    double acc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = 0.0;
    for (int p = threadIdx.x; p < nparts; p += blockDim.x)
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] += partials[p * NC + c];
    block_sum<NC>(acc, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int c = 0; c < NC; ++c) out[c] = acc[c];
}

// v *= sqrt(target / current) (both squared norms, FP64, on the device).
template <class A>
__global__ void k_scale_to_norm(A *__restrict__ v, uint64_t N, const double *target_sq,
                                const double *current_sq) {
    if (!(*current_sq > 0.0) || !(*target_sq > 0.0)) return;
    const double f = sqrt(*target_sq / *current_sq);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        A a = v[i];
        a.x = (decltype(a.x))(a.x * f);
        a.y = (decltype(a.y))(a.y * f);
        v[i] = a;
    }
}

template <class A>
__global__ void k_set_basis(A *__restrict__ v, uint64_t N, uint64_t idx) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        A a;
        a.x = i == idx ? 1 : 0;
        a.y = 0;
        v[i] = a;
    }
}

template <class A>
__global__ void k_set_const(A *__restrict__ v, uint64_t N, double re) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        A a;
        a.x = re;
        a.y = 0;
        v[i] = a;
    }
}

// |a> (x) |b>: out[i * Nb + j] = a[i] * b[j] (src/states/mod.rs:298-314).
template <class A>
__global__ void k_kron(A *__restrict__ out, const A *__restrict__ a, const A *__restrict__ b,
                       int nb, uint64_t N) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < N;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const A x = a[k >> nb], y = b[k & ((1ull << nb) - 1)];
        A o;
        o.x = x.x * y.x - x.y * y.y;
        o.y = x.x * y.y + x.y * y.x;
        out[k] = o;
    }
}

__global__ void k_c128_to_c64(const double2 *__restrict__ src, float2 *__restrict__ dst,
                              uint64_t N) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double2 a = src[i];
        dst[i] = make_float2((float)a.x, (float)a.y);
    }
}

template <class A>
__global__ void k_probs(const A *__restrict__ v, double *__restrict__ p, uint64_t N) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double2 a = load_amp(v, i);
        p[i] = a.x * a.x + a.y * a.y;
    }
}

// Pauli-sum expectation for one group of terms sharing the same X mask.
// For every basis index i the group contributes
//     Re W_i * alpha(i) + Im W_i * beta(i),   W_i = conj(psi_i) psi_{i^x},
// with alpha(i) = sum_t c_t a_t s_t(i), beta(i) = sum_t c_t b_t s_t(i),
// s_t(i) = (-1)^popcount(i & z_t) and (a_t, b_t) the real/imag selectors of
// Re(Y^ny z) = a Re z + b Im z.  When x != 0 each unordered pair (i, i^x) is
// visited once (the i with the top bit of x clear) and adds both orientations.
struct TermCoef {
    uint64_t z;
    double ca;  // c_t * a_t
    double cb;  // c_t * b_t
};

template <class A>
__global__ void k_pauli_group(const A *__restrict__ v, int n, uint64_t xmask,
                              const TermCoef *__restrict__ tc, int nt, double *partials) {
    extern __shared__ TermCoef s_tc[];
    __shared__ double sh[32];
    for (int t = threadIdx.x; t < nt; t += blockDim.x) s_tc[t] = tc[t];
    __syncthreads();
    double acc[1] = {0.0};
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    // The grid-stride loops take kU steps at a time with every load issued
    // first (kU amplitudes, or kU pairs, in flight per thread); each thread
    // still adds its steps in the same order.
    constexpr int kU = 4;
    if (xmask == 0) {
        const uint64_t N = 1ull << n;
        auto add = [&](uint64_t i, double2 a) {
            double alpha = 0.0;
            for (int t = 0; t < nt; ++t) {
                const double s = (__popcll(i & s_tc[t].z) & 1) ? -1.0 : 1.0;
                alpha += s * s_tc[t].ca;
            }
            acc[0] += (a.x * a.x + a.y * a.y) * alpha;
        };
        uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
        for (; i + (kU - 1) * stride < N; i += kU * stride) {
            double2 a[kU];
#pragma unroll
            for (int k = 0; k < kU; ++k) a[k] = load_amp(v, i + k * stride);
#pragma unroll
            for (int k = 0; k < kU; ++k) add(i + k * stride, a[k]);
        }
        for (; i < N; i += stride) add(i, load_amp(v, i));
    } else {
        const int hb = 63 - __clzll(xmask);
        const uint64_t npairs = 1ull << (n - 1);
        const uint64_t lo_mask = (1ull << hb) - 1;
        auto pair_index = [&](uint64_t p) { return ((p & ~lo_mask) << 1) | (p & lo_mask); };
        auto add = [&](uint64_t i, double2 a, double2 b) {
            // W_i = conj(a) b ; W_j = conj(W_i), j = i ^ xmask.  The j-side sums
            // follow from the i side: a term's Z sign at j is its sign at i times
            // (-1)^ny, and ca = 0 for odd ny, cb = 0 for even ny, so
            // al_j = al_i and be_j = -be_i.
            const double wr = a.x * b.x + a.y * b.y;
            const double wi = a.x * b.y - a.y * b.x;
            double al_i = 0.0, be_i = 0.0;
            for (int t = 0; t < nt; ++t) {
                const double si = (__popcll(i & s_tc[t].z) & 1) ? -1.0 : 1.0;
                al_i += si * s_tc[t].ca;
                be_i += si * s_tc[t].cb;
            }
            acc[0] += 2.0 * (wr * al_i + wi * be_i);
        };
        uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
        for (; p + (kU - 1) * stride < npairs; p += kU * stride) {
            double2 a[kU], b[kU];
#pragma unroll
            for (int k = 0; k < kU; ++k) {
                const uint64_t i = pair_index(p + k * stride);
                a[k] = load_amp(v, i);
                b[k] = load_amp(v, i ^ xmask);
            }
#pragma unroll
            for (int k = 0; k < kU; ++k) add(pair_index(p + k * stride), a[k], b[k]);
        }
        for (; p < npairs; p += stride) {
            const uint64_t i = pair_index(p);
            add(i, load_amp(v, i), load_amp(v, i ^ xmask));
        }
    }
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

// Terms without X bits (one group, X mask 0), for states of 12 or more qubits,
// launched with 256 threads.  A block takes 4096-amplitude chunks; thread tid
// handles the 16 indices i = chunk | k << 8 | tid, k = 0..15.  A term's sign
// (-1)^popcount(i & z) is the sign of the bits the thread keeps fixed (chunk
// and tid) times (-1)^popcount(k & p), p = bits 8-11 of z.  The terms arrive
// sorted by p (pbeg[p] .. pbeg[p+1]), so each thread folds all of them into 16
// coefficients C[p], and one 16-point Walsh-Hadamard transform of C gives the
// sum of signed coefficients for all 16 k: a few operations per amplitude
// instead of a popcount and a select per term per amplitude.
template <class A>
__global__ void __launch_bounds__(256, 2)
    k_pauli_zfold(const A *__restrict__ v, int n, const TermCoef *__restrict__ tc, int nt,
                  const int *__restrict__ pbeg, double *partials) {
    extern __shared__ TermCoef s_tc[];
    __shared__ double sh[32];
    __shared__ int s_pbeg[17];
    for (int t = threadIdx.x; t < nt; t += blockDim.x) s_tc[t] = tc[t];
    if (threadIdx.x < 17) s_pbeg[threadIdx.x] = pbeg[threadIdx.x];
    __syncthreads();
    double acc[1] = {0.0};
    const uint64_t nchunks = 1ull << (n - 12);
    for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const uint64_t fixed = (c << 12) | (uint64_t)threadIdx.x;
        double pr[16];  // |a|^2 of the 16 amplitudes
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const double2 a = load_amp(v, fixed | ((uint64_t)k << 8));
            pr[k] = a.x * a.x + a.y * a.y;
        }
        double C[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            double cq = 0.0;
            for (int t = s_pbeg[q]; t < s_pbeg[q + 1]; ++t)
                cq += (__popcll(fixed & s_tc[t].z) & 1) ? -s_tc[t].ca : s_tc[t].ca;
            C[q] = cq;
        }
#pragma unroll
        for (int hs = 1; hs < 16; hs <<= 1) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                if (q & hs) continue;
                const double x = C[q], y = C[q | hs];
                C[q] = x + y;
                C[q | hs] = x - y;
            }
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) acc[0] += pr[k] * C[k];
    }
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

// ---------------------------------------------------------------------------
// Pauli sums by windows.  A tile is the 2^T amplitudes of the index bits [0,4) and
// [h, h+T-4), held in shared memory as complex128; every group whose X bits lie in
// that window is evaluated from it, so the state is read once per window instead of
// once per X mask (a 24-qubit chain: 3 reads instead of 24), and a state of at most
// 2^12 amplitudes needs one launch for the whole sum.
//
// Reading the tile once per group would make shared memory the bound (two 16-byte loads
// for 2-4 FP64 instructions: 0.90 ms for that chain).  So the groups are taken in
// rounds: a round has four vectors v_0..v_3 (tile-local X masks, in reduced echelon
// form), a thread holds the 16 amplitudes l0 + span(v), and every group whose mask lies
// in that span is formed from registers.  A chain's X, XX and YY terms need a round for
// every three bits; arbitrary masks need one for every four of them.  All index work is
// linear over XOR: a term's sign splits into the bits outside the window (the tile), the
// thread's and the element's, of which the last is a mask made on the host.
// ---------------------------------------------------------------------------
constexpr int kWinT = 12, kWinMinT = 9;
constexpr int kWinStage = 8192;  // bytes of rounds, groups and terms staged at a time
constexpr size_t kWinSplit = 16; // terms of a round that are not worth sharing out

struct WinTerm {
    uint64_t z;      // Z bits outside the window
    double c;
    uint32_t lz;     // Z bits in the window, tile-local
    uint32_t mask;   // bit k: the sign at pair k of the group; without X: the parities of
                     // lz with the four vectors (by which these terms arrive sorted)
    uint32_t odd;    // an odd number of Y
    uint32_t pad;
};

struct WinGroup {
    int32_t d;       // its X mask as a sum of vectors, 1..15
    int32_t odd;     // some term has an odd number of Y
    int32_t term, nterms;
};

struct WinRound {
    uint32_t vec[4];   // places of the vectors
    uint32_t lane[8];  // tile bit of each thread-index bit
    int32_t group, ngroups;
    int32_t zterm, nz;  // terms without X
};

struct WinChunk {  // one stage: rounds, then groups, then terms
    int32_t offset, bytes;  // in the program
    int32_t nrounds, groups, terms;  // the latter two: byte offsets in the stage
};

struct WinDesc {
    int32_t h, chunk, nchunks;
    int32_t work;  // first work index of the window
};
static_assert(sizeof(WinTerm) % 16 == 0 && sizeof(WinGroup) % 16 == 0 && sizeof(WinRound) % 16 == 0,
              "staged in 16 bytes");

// Byte offset of a tile index: any three bits of different residues mod 3 spread eight
// threads over the eight 16-byte bank groups.
__host__ __device__ __forceinline__ uint32_t win_place(uint32_t l) {
    return (l ^ (((l >> 3) ^ (l >> 6) ^ (l >> 9)) & 7u)) << 4;
}
__device__ __forceinline__ double win_sign(double x, uint32_t neg) {  // bit 0 counts
    return __hiloint2double(__double2hiint(x) ^ (int)(neg << 31), __double2loint(x));
}
// Pair k of the group of mask d: element k with a zero inserted at d's top bit, and that
// element plus d.
__host__ __device__ constexpr int win_pair(int k, int d) {
    const int hb = d >= 8 ? 3 : d >= 4 ? 2 : d >= 2 ? 1 : 0;
    return ((k >> hb) << (hb + 1)) | (k & ((1 << hb) - 1));
}
// W = conj(a) b of the 8 pairs; the pair's other orientation doubles it (k_pauli_group).
template <int D>
__device__ __forceinline__ void win_pairs(const double2 (&a)[16], bool odd, double (&wr)[8],
                                          double (&wi)[8]) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double2 x = a[win_pair(k, D)], y = a[win_pair(k, D) ^ D];
        wr[k] = fma(x.x, y.x, x.y * y.y);
    }
    if (odd)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const double2 x = a[win_pair(k, D)], y = a[win_pair(k, D) ^ D];
            wi[k] = fma(x.x, y.y, -(x.y * y.x));
        }
}

template <class A>
__global__ void __launch_bounds__(256, 2)
    k_pauli_windows(const A *__restrict__ v, int n, int T, const WinDesc *__restrict__ wins,
                    int nwins, const WinChunk *__restrict__ chunks,
                    const unsigned char *__restrict__ program, int nwork,
                    double *__restrict__ partials) {
    extern __shared__ __align__(16) unsigned char win_smem[];
    __shared__ double sh[32];
    unsigned char *stage = win_smem + ((size_t)16 << T);
    const uint32_t tid = threadIdx.x;
    const uint64_t N = 1ull << n;
    uint32_t on[8];  // all ones where the thread-index bit is set
#pragma unroll
    for (int j = 0; j < 8; ++j) on[j] = 0u - ((tid >> j) & 1u);
    double acc[1] = {0.0};
    int held = -1, wi = 0;  // chunk in the stage; window
    for (int w = (int)blockIdx.x; w < nwork; w += (int)gridDim.x) {
        while (wi + 1 < nwins && wins[wi + 1].work <= w) ++wi;
        const WinDesc win = wins[wi];
        const int tile = w - win.work, h = win.h;
        const uint64_t c2 = n > T ? (uint64_t)(tile & ((1 << (h - 4)) - 1)) : 0;
        const uint64_t c4 = n > T ? (uint64_t)(tile >> (h - 4)) : 0;
        const uint64_t tb = (c2 << 4) | (c4 << (h + T - 4));
        __syncthreads();  // the previous tile has been read
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const uint32_t l = tid | (uint32_t)k << (T - 4);
            const uint64_t i = tb | (uint64_t)(l & 15u) | ((uint64_t)(l >> 4) << h);
            *(double2 *)(win_smem + win_place(l)) = i < N ? load_amp(v, i) : make_double2(0.0, 0.0);
        }
        for (int ci = win.chunk; ci < win.chunk + win.nchunks; ++ci) {
            const WinChunk ch = chunks[ci];
            if (held != ci) {
                if (ci != win.chunk) __syncthreads();  // the previous chunk has been read
                for (int o = (int)tid * 16; o < ch.bytes; o += (int)blockDim.x * 16)
                    *(double2 *)(stage + o) = *(const double2 *)(program + ch.offset + o);
                held = ci;
            }
            __syncthreads();
            const WinGroup *groups = (const WinGroup *)(stage + ch.groups);
            const WinTerm *terms = (const WinTerm *)(stage + ch.terms);
            for (int r = 0; r < ch.nrounds; ++r) {
                const WinRound &rd = ((const WinRound *)stage)[r];
                uint32_t l0 = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) l0 |= rd.lane[j] & on[j];
                const uint32_t at = win_place(l0);
                const uint32_t E0 = rd.vec[0], E1 = rd.vec[1], E2 = rd.vec[2], E3 = rd.vec[3];
                auto amp = [&](int e) {
                    return *(const double2 *)(win_smem +
                                              (at ^ ((e & 1) ? E0 : 0u) ^ ((e & 2) ? E1 : 0u) ^
                                               ((e & 4) ? E2 : 0u) ^ ((e & 8) ? E3 : 0u)));
                };
                auto neg = [&](const WinTerm &tm) {
                    return (uint32_t)(__popcll(tb & tm.z) + __popc(l0 & tm.lz));
                };
                if (rd.nz) {
                    // the terms add up by their parities with the vectors, and a 16-point
                    // Walsh-Hadamard transform gives every element's coefficient
                    double c[16];
                    int t = rd.zterm;
                    const int t1 = t + rd.nz;
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        c[q] = 0.0;
                        for (; t < t1 && terms[t].mask == (uint32_t)q; ++t)
                            c[q] += win_sign(terms[t].c, neg(terms[t]));
                    }
#pragma unroll
                    for (int s = 1; s < 16; s <<= 1)
#pragma unroll
                        for (int q = 0; q < 16; ++q) {
                            if (q & s) continue;
                            const double x = c[q], y = c[q | s];
                            c[q] = x + y;
                            c[q | s] = x - y;
                        }
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const double2 a = amp(e);
                        acc[0] += (a.x * a.x + a.y * a.y) * c[e];
                    }
                }
                if (rd.ngroups == 0) continue;
                double2 a[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) a[e] = amp(e);
                for (int g = rd.group; g < rd.group + rd.ngroups; ++g) {
                    const WinGroup gr = groups[g];
                    const bool odd = gr.odd != 0;
                    double wr[8], wi_[8];
                    // (else every mask's products are taken out of the loop, into memory)
#pragma unroll
                    for (int e = 0; e < 16; ++e) asm volatile("" : "+d"(a[e].x), "+d"(a[e].y));
                    switch (gr.d) {
#define LQ_WIN(D) case D: win_pairs<D>(a, odd, wr, wi_); break;
                        LQ_WIN(1) LQ_WIN(2) LQ_WIN(3) LQ_WIN(4) LQ_WIN(5) LQ_WIN(6) LQ_WIN(7)
                        LQ_WIN(8) LQ_WIN(9) LQ_WIN(10) LQ_WIN(11) LQ_WIN(12) LQ_WIN(13) LQ_WIN(14)
                        default: win_pairs<15>(a, odd, wr, wi_); break;
#undef LQ_WIN
                    }
                    for (int t = gr.term; t < gr.term + gr.nterms; ++t) {
                        const WinTerm tm = terms[t];
                        double x = 0.0;  // a term counts the real or the imaginary parts
                        if (tm.odd) {
#pragma unroll
                            for (int k = 0; k < 8; ++k) x += win_sign(wi_[k], tm.mask >> k);
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k) x += win_sign(wr[k], tm.mask >> k);
                        }
                        acc[0] += 2.0 * win_sign(tm.c * x, neg(tm));
                    }
                }
            }
        }
    }
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// ---------------------------------------------------------------------------
// Cumulative distribution for sampling: a deterministic three-phase FP64
// inclusive scan with a fixed summation order (so a CPU restatement reproduces
// every value bit for bit).  A chunk is 1024 values = 256 threads x 4:
//   s_j    = running sum of the thread's 4 values (left to right);
//   incl_t = Kogge-Stone inclusive scan of the threads' s_3 inside each warp
//            (shuffle offsets 1, 2, 4, 8, 16);
//   W_w    = exclusive running sum of the 8 warp totals (one thread, in order);
//   cdf    = (W_w + incl_{t-1}) + s_j   (incl_{-1} = 0 at lane 0),
// and the chunk total is the chunk's last cdf value.  Chunk totals are scanned
// the same way (recursively) and added as base + value to every later chunk.
// ---------------------------------------------------------------------------
constexpr int kScanChunk = 1024;

// |a|^2 with no contraction, and plain doubles (the totals of a lower level).
__device__ __forceinline__ double scan_value(double2 a) {
    return __dadd_rn(__dmul_rn(a.x, a.x), __dmul_rn(a.y, a.y));
}
__device__ __forceinline__ double scan_value(float2 a) {
    return scan_value(make_double2(a.x, a.y));
}
__device__ __forceinline__ double scan_value(double x) { return x; }

// The scan of one chunk (256 threads): v[j] of value base + j, base = 4 * thread
// within the chunk.  W: 8 doubles of shared memory.
template <class V>
__device__ __forceinline__ void scan_chunk(const V *__restrict__ in, uint64_t base, uint64_t N,
                                           double *W, double (&v)[4]) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const double x = base + j < N ? scan_value(in[base + j]) : 0.0;
        s[j] = j == 0 ? x : __dadd_rn(s[j - 1], x);
    }
    double incl = s[3];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl = __dadd_rn(y, incl);
    }
    double excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = 0.0;
    if (lane == 31) W[warp] = incl;  // warp total
    __syncthreads();
    if (t == 0) {
        double run = 0.0;
        for (int w = 0; w < 8; ++w) {
            const double tot = W[w];
            W[w] = run;
            run = __dadd_rn(run, tot);
        }
    }
    __syncthreads();
    const double off = __dadd_rn(W[warp], excl);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __dadd_rn(off, s[j]);
}

// Chunk scans of in (amplitudes, or totals of a lower level) into out, if given, and
// the chunk totals.
template <class V>
__global__ void __launch_bounds__(256) k_scan_chunks(const V *__restrict__ in,
                                                     double *__restrict__ out,
                                                     double *__restrict__ chunk_total,
                                                     uint64_t N) {
    __shared__ double W[8];
    const uint64_t base = (uint64_t)blockIdx.x * kScanChunk + 4u * threadIdx.x;
    double v[4];
    scan_chunk(in, base, N, W, v);
    if (out) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (base + j < N) out[base + j] = v[j];
    }
    if (threadIdx.x == 255) chunk_total[blockIdx.x] = v[3];
}

__global__ void k_scan_add_base(double *__restrict__ cdf, const double *__restrict__ incl_total,
                                uint64_t N) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x + kScanChunk; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t c = i / kScanChunk;
        cdf[i] = __dadd_rn(incl_total[c - 1], cdf[i]);
    }
}

__device__ __forceinline__ double shot_uniform(uint64_t seed, uint64_t s, double total) {
    const uint64_t r = splitmix64(seed ^ splitmix64(s));
    return (double)(r >> 11) * (1.0 / 9007199254740992.0) * total;
}

// cdf(i) = scanned total of the chunks before i's + i's value in its chunk's scan: the
// sum that a sweep adding the bases would store, formed at the values the search probes.
__device__ __forceinline__ double chunk_base(const double *__restrict__ incl_total, uint64_t c,
                                             double local) {
    return c ? __dadd_rn(incl_total[c - 1], local) : local;
}

__global__ void k_sample(const double *__restrict__ local, const double *__restrict__ incl_total,
                         uint64_t N, uint64_t nshots, uint64_t seed, uint64_t *__restrict__ out) {
    auto cdf = [&](uint64_t i) { return chunk_base(incl_total, i / kScanChunk, local[i]); };
    const double total = cdf(N - 1);
    for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < nshots;
         s += (uint64_t)gridDim.x * blockDim.x) {
        const double u = shot_uniform(seed, s, total);
        // first index with cdf > u
        uint64_t lo = 0, hi = N - 1;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (cdf(mid) > u) hi = mid;
            else lo = mid + 1;
        }
        out[s] = lo;
    }
}

// The same search without the stored scan (N a power of two of at least two chunks):
// every probe above a chunk's width falls on a chunk's last value, which is its total;
// the chunk it ends in is scanned again.  One block per shot.
template <class A>
__global__ void __launch_bounds__(256)
    k_sample_rescan(const A *__restrict__ v, const double *__restrict__ chunk_total,
                    const double *__restrict__ incl_total, uint64_t N, uint64_t nshots,
                    uint64_t seed, uint64_t *__restrict__ out) {
    __shared__ double W[8];
    __shared__ double s_v[kScanChunk];
    __shared__ uint64_t s_chunk;
    const uint64_t nc = N / kScanChunk;
    const double total = chunk_base(incl_total, nc - 1, chunk_total[nc - 1]);
    for (uint64_t s = blockIdx.x; s < nshots; s += gridDim.x) {
        const double u = shot_uniform(seed, s, total);
        if (threadIdx.x == 0) {
            uint64_t lo = 0, hi = nc - 1;
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (chunk_base(incl_total, mid, chunk_total[mid]) > u) hi = mid;
                else lo = mid + 1;
            }
            s_chunk = lo;
        }
        __syncthreads();
        const uint64_t c = s_chunk;
        double x[4];
        scan_chunk(v, c * kScanChunk + 4u * threadIdx.x, N, W, x);
#pragma unroll
        for (int j = 0; j < 4; ++j) s_v[4 * threadIdx.x + j] = x[j];
        __syncthreads();
        if (threadIdx.x == 0) {
            uint64_t lo = 0, hi = kScanChunk - 1;
            while (lo < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (chunk_base(incl_total, c, s_v[mid]) > u) hi = mid;
                else lo = mid + 1;
            }
            out[s] = c * kScanChunk + lo;
        }
    }
}

static int grid_for(uint64_t N, int threads) {
    uint64_t g = (N + threads - 1) / threads;
    const uint64_t cap = 148ull * 64;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

static int norm_sqr_device(const lq_state *s, double *d_out) {
    const uint64_t N = 1ull << s->n;
    const int th = 256, g = red_grid(N, th);
    prof_begin(s->stream, kProfReduce);
    if (s->dtype == LQ_C128)
        k_norm_partial<<<g, th, 0, s->stream>>>((const double2 *)s->d, N, s->d_red);
    else
        k_norm_partial<<<g, th, 0, s->stream>>>((const float2 *)s->d, N, s->d_red);
    k_final_sum<1><<<1, 256, 0, s->stream>>>(s->d_red, g, d_out);
    prof_end(s->stream, kProfReduce);
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

int normalize_impl(lq_state *s) {
    const uint64_t N = 1ull << s->n;
    const int g = red_grid(N, 256);
    prof_begin(s->stream, kProfReduce);
    if (s->dtype == LQ_C128)
        k_norm_partial<<<g, 256, 0, s->stream>>>((const double2 *)s->d, N, s->d_red);
    else
        k_norm_partial<<<g, 256, 0, s->stream>>>((const float2 *)s->d, N, s->d_red);
    prof_end(s->stream, kProfReduce);
    LQ_CUDA_TRY(cudaGetLastError());
    return scale_by_partials(s, nullptr, g);
}

int scale_by_partials(lq_state *s, const void *src, int nparts) {
    const uint64_t N = 1ull << s->n;
    if (s->dtype == LQ_C128)
        k_scale_by_partials<<<red_grid(N, 256), 256, 0, s->stream>>>(
            (double2 *)s->d, (const double2 *)src, N, s->d_red, nparts);
    else
        k_scale_by_partials<<<red_grid(N, 256), 256, 0, s->stream>>>(
            (float2 *)s->d, (const float2 *)src, N, s->d_red, nparts);
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

// FP64 norm bookkeeping of the precision form: remember the squared norm now,
// and later scale the state back to it (two slots at the end of the reduction
// scratch, clear of the partial sums and of normalize's slot).
int norm_snapshot(lq_state *s) {
    double *d_in = s->d_red + kRedBlocks * 2 * kMaxTermsPerPass - 2;
    return norm_sqr_device(s, d_in);
}

int norm_restore(lq_state *s) {
    double *d_in = s->d_red + kRedBlocks * 2 * kMaxTermsPerPass - 2;
    double *d_now = s->d_red + kRedBlocks * 2 * kMaxTermsPerPass - 3;
    LQ_TRY(norm_sqr_device(s, d_now));
    const uint64_t N = 1ull << s->n;
    if (s->dtype == LQ_C128)
        k_scale_to_norm<<<grid_for(N, 256), 256, 0, s->stream>>>((double2 *)s->d, N, d_in, d_now);
    else
        k_scale_to_norm<<<grid_for(N, 256), 256, 0, s->stream>>>((float2 *)s->d, N, d_in, d_now);
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

int expectation_impl(const lq_state *s, const lq_pauli_term *terms, int nterms, int yconv,
                     double *out, double *per_term) {
    const int n = s->n;
    for (int t = 0; t < nterms; ++t) {
        const uint64_t lim = n == 64 ? ~0ull : ((1ull << n) - 1);
        if ((terms[t].xmask & ~lim) || (terms[t].zmask & ~lim))
            return set_error(LQ_ERR_QUBIT_INDEX, "Pauli term %d acts on a qubit >= %d", t, n);
        const int ny = __builtin_popcountll(terms[t].xmask & terms[t].zmask);
        if (terms[t].ny != ny)
            return set_error(LQ_ERR_INVALID_ARG,
                             "Pauli term %d: ny=%d but xmask&zmask has %d bits", t, terms[t].ny, ny);
    }
    // Re(Y^ny z) selectors: Y = +i (reference convention) or -i (textbook).
    auto selectors = [&](int ny, double &a, double &b) {
        int k = ny & 3;
        if (yconv == LQ_Y_TEXTBOOK) k = (4 - k) & 3;
        // Re(i^k (x + i y)): k=0: x ; 1: -y ; 2: -x ; 3: y
        a = k == 0 ? 1.0 : k == 2 ? -1.0 : 0.0;
        b = k == 1 ? -1.0 : k == 3 ? 1.0 : 0.0;
    };
    // Group terms by X mask (one pass over the state per group), or one group
    // per term when per-term values are requested.
    std::vector<std::pair<uint64_t, std::vector<int>>> groups;
    if (per_term) {
        for (int t = 0; t < nterms; ++t) groups.push_back({terms[t].xmask, {t}});
    } else {
        std::map<uint64_t, size_t> idx;
        for (int t = 0; t < nterms; ++t) {
            auto it = idx.find(terms[t].xmask);
            if (it == idx.end()) {
                idx[terms[t].xmask] = groups.size();
                groups.push_back({terms[t].xmask, {t}});
            } else {
                groups[it->second].second.push_back(t);
            }
        }
    }
    for (const auto &gr : groups)
        if (gr.second.size() > (size_t)kMaxGroupTerms)
            return set_error(LQ_ERR_UNSUPPORTED,
                             "%zu Pauli terms share one X mask; at most %d per X mask "
                             "(split the observable)",
                             gr.second.size(), kMaxGroupTerms);
    const uint64_t N = 1ull << n;
    const int th = 256;
    const int g = red_grid(std::max<uint64_t>(N / 2, 1), th);
    // Windows: the fewest that hold every group's X bits (each is a sweep).  A group's X
    // bits above bit 3 need h in [hi - m + 1, lo]; points stabbing every such interval,
    // chosen greedily by right end, are a minimum set.  Groups with none go to the first
    // window, and groups too wide for any keep a sweep of their own.
    // Tile bits: the whole state up to 2^12 amplitudes (zeros above it below 2^9), else at
    // least 2^7 tiles down to 2^10 amplitudes each, so that smaller states still fill the
    // chip.
    const int T = n <= kWinT ? std::max(n, kWinMinT) : std::max(10, std::min(kWinT, n - 7));
    const int m = T - 4;
    struct Need {
        int a, b;
        size_t group;
    };
    std::vector<Need> needs;
    std::vector<size_t> anywhere, sweeps;
    for (size_t gi = 0; gi < groups.size(); ++gi) {
        const uint64_t up = groups[gi].first & ~0xFull;
        if (per_term) {
            sweeps.push_back(gi);
        } else if (!up) {
            anywhere.push_back(gi);
        } else {
            const int lo = __builtin_ctzll(up), hi = 63 - __builtin_clzll(up);
            const int a = std::max(4, hi - m + 1), b = std::min(lo, std::max(4, n - m));
            if (a <= b) needs.push_back(Need{a, b, gi});
            else sweeps.push_back(gi);
        }
    }
    std::stable_sort(needs.begin(), needs.end(),
                     [](const Need &x, const Need &y) { return x.b < y.b; });
    std::vector<std::pair<int, std::vector<size_t>>> wsets;
    for (const Need &q : needs) {
        if (wsets.empty() || wsets.back().first < q.a) wsets.push_back({q.b, {}});
        wsets.back().second.push_back(q.group);
    }
    // A window reads the state at 0.74 of the copy peak, a sweep at the peak (28 qubits, one
    // term: 0.89 and 0.60 ms; of complex64 a sweep is half of that).  So a window for one
    // group of few terms, or two of complex64, is sweeps instead where the state is large
    // enough for that to count more than the launches (20 qubits, two windows of a group
    // each: 38 us, two sweeps 46), and a sum of terms without X alone is one folded sweep, as
    // far as that goes (n >= 12).  A single group that fits a window (alone, or beside others
    // that fit none) is a sweep unless its many terms on a large state count more than the
    // window's longer start: 8 qubits 25-29 us for 20 terms and 60 for 1000 (a window 35-38
    // and 71-96), 20 qubits 40 us for 20 terms (44), but 67 for 100 (52-60), 24 qubits 153 for
    // 20 (130); 18 qubits, ten random terms of which one fits 94 us (106).
    constexpr int kSweepQubits = 22;
    constexpr size_t kSweepTerms = 4;
    const bool only = needs.size() + anywhere.size() == 1;
    auto few = [&](const std::vector<size_t> &gs) {
        const size_t most = !only ? kSweepTerms
                            : n < 19 ? (size_t)kMaxGroupTerms
                                     : std::max<size_t>(kSweepTerms, 64 >> std::min(n - 19, 6));
        bool ok = (n >= kSweepQubits || only) && gs.size() <= (s->dtype == LQ_C64 ? 2 : 1);
        for (size_t gi : gs) ok = ok && groups[gi].second.size() <= most;
        return ok;
    };
    auto to_sweeps = [&](std::vector<size_t> &gs) {
        sweeps.insert(sweeps.end(), gs.begin(), gs.end());
        gs.clear();
    };
    for (auto &ws : wsets)
        if (few(ws.second)) to_sweeps(ws.second);
    wsets.erase(std::remove_if(wsets.begin(), wsets.end(),
                               [](const auto &ws) { return ws.second.empty(); }),
                wsets.end());
    if (wsets.empty() && (few(anywhere) || (anywhere.size() == 1 && n >= 12 &&
                                            groups[anywhere[0]].first == 0)))
        to_sweeps(anywhere);
    int pbeg[17] = {0};  // k_pauli_zfold: its terms sorted by bits 8-11 of the Z mask
    int zfold = -1;
    for (size_t k = 0; k < sweeps.size() && !per_term && n >= 12; ++k) {
        if (groups[sweeps[k]].first != 0) continue;
        zfold = (int)k;
        auto pat = [&](int t) { return (int)((terms[t].zmask >> 8) & 15); };
        std::vector<int> &ts = groups[sweeps[k]].second;
        std::stable_sort(ts.begin(), ts.end(), [&](int x, int y) { return pat(x) < pat(y); });
        for (int t : ts)
            for (int q = pat(t) + 1; q <= 16; ++q) ++pbeg[q];
    }
    if (wsets.empty() && !anywhere.empty()) wsets.push_back({4, {}});
    if (!wsets.empty())
        wsets[0].second.insert(wsets[0].second.end(), anywhere.begin(), anywhere.end());
    auto coef_of = [&](int t) {
        double a, b;
        selectors(terms[t].ny, a, b);
        return TermCoef{terms[t].zmask, terms[t].coefficient * a, terms[t].coefficient * b};
    };
    std::vector<WinDesc> wins;
    std::vector<WinChunk> chunks;
    std::vector<unsigned char> program;
    const int tiles = 1 << std::max(n - T, 0);
    int nwork = 0;
    for (const auto &ws : wsets) {
        const int h = ws.first;
        const uint64_t inside = 15ull | ((1ull << m) - 1) << h;
        auto local = [&](uint64_t mask) {
            return (uint32_t)(mask & 15u) | (uint32_t)((mask >> h) & ((1ull << m) - 1)) << 4;
        };
        auto parity = [](uint32_t x) { return (uint32_t)__builtin_parity(x); };
        // rounds: in order of their masks, a group joins if it lies in the span of the
        // vectors or there are fewer than four
        struct Round {
            uint32_t vec[4];
            int piv[4], rank = 0;
            std::vector<size_t> groups;
        };
        std::vector<Round> rounds;
        std::vector<size_t> left = ws.second;
        std::stable_sort(left.begin(), left.end(), [&](size_t x, size_t y) {
            return local(groups[x].first) < local(groups[y].first);
        });
        while (!left.empty()) {
            Round r;
            std::vector<size_t> later;
            for (size_t gi : left) {
                uint32_t x = local(groups[gi].first);
                for (int k = 0; k < r.rank; ++k)
                    if ((x >> r.piv[k]) & 1u) x ^= r.vec[k];
                if (x && r.rank == 4) {
                    later.push_back(gi);
                    continue;
                }
                if (x) {
                    const int p = 31 - __builtin_clz(x);
                    for (int k = 0; k < r.rank; ++k)
                        if ((r.vec[k] >> p) & 1u) r.vec[k] ^= x;
                    r.vec[r.rank] = x;
                    r.piv[r.rank++] = p;
                }
                r.groups.push_back(gi);
            }
            for (int p = T - 1; r.rank < 4; --p) {
                bool used = false;
                for (int k = 0; k < r.rank; ++k) used |= r.piv[k] == p;
                if (used) continue;
                for (int k = 0; k < r.rank; ++k)
                    if ((r.vec[k] >> p) & 1u) r.vec[k] ^= 1u << p;
                r.vec[r.rank] = 1u << p;
                r.piv[r.rank++] = p;
            }
            rounds.push_back(std::move(r));
            left.swap(later);
        }
        // every round's program: its terms without X first, then the groups
        struct Entry {
            bool z;
            WinGroup wg;
            std::vector<WinTerm> terms;
        };
        struct RoundTerms {
            WinRound hd;
            std::vector<Entry> entries;
            size_t nterms;
        };
        std::vector<RoundTerms> prog;
        prog.reserve(rounds.size());
        size_t all_terms = 0;
        for (const Round &r : rounds) {
            RoundTerms rt{};
            rt.entries.reserve(r.groups.size());
            uint32_t pivots = 0;
            for (int k = 0; k < 4; ++k) {
                rt.hd.vec[k] = win_place(r.vec[k]);
                pivots |= 1u << r.piv[k];
            }
            // thread bits: first three whose places lie in different banks
            std::vector<int> lanes;
            for (int turn = 0; turn < 2; ++turn)
                for (int p = 0, seen = 0; p < T; ++p) {
                    if (pivots >> p & 1u) continue;
                    const bool first = !(seen >> (p % 3) & 1);
                    seen |= 1 << (p % 3);
                    if (first == (turn == 0)) lanes.push_back(p);
                }
            for (size_t j = 0; j < lanes.size(); ++j) rt.hd.lane[j] = 1u << lanes[j];
            for (int zturn = 1; zturn >= 0; --zturn)
                for (size_t gi : r.groups) {
                    const uint32_t lx = local(groups[gi].first);
                    if ((lx == 0) != (zturn == 1)) continue;
                    Entry en{lx == 0, WinGroup{}, {}};
                    for (int k = 0; k < 4; ++k) en.wg.d |= (int)((lx >> r.piv[k]) & 1u) << k;
                    // the pairs (or, without X, the vector itself) whose sign bit j turns
                    uint32_t turns[4];
                    for (int j = 0; j < 4; ++j) {
                        turns[j] = lx == 0 ? 1u << j : 0u;
                        for (int k = 0; lx != 0 && k < 8; ++k)
                            turns[j] |= (uint32_t)((win_pair(k, en.wg.d) >> j) & 1) << k;
                    }
                    en.terms.reserve(groups[gi].second.size());
                    for (int t : groups[gi].second) {
                        const TermCoef c = coef_of(t);
                        const uint32_t odd = terms[t].ny & 1;
                        WinTerm wt{c.z & ~inside, odd ? c.cb : c.ca, local(c.z), 0, odd, 0};
                        for (int j = 0; j < 4; ++j)
                            wt.mask ^= turns[j] & (0u - parity(wt.lz & r.vec[j]));
                        en.wg.odd |= (int)odd;
                        en.terms.push_back(wt);
                    }
                    if (lx == 0)
                        std::stable_sort(en.terms.begin(), en.terms.end(),
                                         [](const WinTerm &x, const WinTerm &y) { return x.mask < y.mask; });
                    rt.nterms += en.terms.size();
                    rt.entries.push_back(std::move(en));
                }
            all_terms += rt.nterms;
            prog.push_back(std::move(rt));
        }
        // Few tiles: the rounds are shared out among more blocks, and so are the terms of a
        // round that has more than its share.  (A block takes 0.16 us for each term of a round,
        // one after the other: 16 masks of 400 terms on 12 qubits 1010 us in two rounds' blocks,
        // 260 so.)
        const size_t share = (size_t)std::max(1, 2 * 148 / (tiles * (int)wsets.size()));
        const size_t most = share == 1 ? all_terms : std::max<size_t>(kWinSplit, (all_terms + share - 1) / share);
        struct Slice {
            size_t entry, begin, end;
        };
        std::vector<Slice> slices;
        struct Job {
            size_t round, nterms, slice, end, part;
        };
        std::vector<Job> jobs;
        for (size_t ri = 0; ri < prog.size(); ++ri) {
            auto next = [&] { jobs.push_back(Job{ri, 0, slices.size(), slices.size(), 0}); };
            next();
            for (size_t ei = 0; ei < prog[ri].entries.size(); ++ei)
                for (size_t b = 0, n_e = prog[ri].entries[ei].terms.size(); b < n_e;) {
                    if (jobs.back().nterms == most) next();
                    const size_t e = std::min(n_e, b + most - jobs.back().nterms);
                    slices.push_back(Slice{ei, b, e});
                    jobs.back().end = slices.size();
                    jobs.back().nterms += e - b;
                    b = e;
                }
        }
        const size_t parts = std::min(jobs.size(), share);
        if (parts > 1) {
            // the largest first, each to the part with the fewest terms so far
            std::stable_sort(jobs.begin(), jobs.end(),
                             [](const Job &x, const Job &y) { return x.nterms > y.nterms; });
            using Load = std::pair<size_t, size_t>;  // terms, part
            std::priority_queue<Load, std::vector<Load>, std::greater<Load>> loads;
            for (size_t k = 0; k < parts; ++k) loads.push({0, k});
            for (Job &j : jobs) {
                const Load l = loads.top();
                loads.pop();
                j.part = l.second;
                loads.push({l.first + j.nterms + 1, l.second});
            }
            std::stable_sort(jobs.begin(), jobs.end(),
                             [](const Job &x, const Job &y) { return x.part < y.part; });
        }
        std::vector<WinRound> cr;
        std::vector<WinGroup> cg;
        std::vector<WinTerm> ct;
        size_t ji = 0;
        for (size_t part = 0; part < parts; ++part) {
            WinDesc wd{h, (int)chunks.size(), 0, nwork};
            nwork += tiles;
            auto bytes = [&] {
                return cr.size() * sizeof(WinRound) + cg.size() * sizeof(WinGroup) +
                       ct.size() * sizeof(WinTerm);
            };
            auto close = [&] {
                if (cr.empty()) return;
                WinChunk c{(int)program.size(), (int)bytes(), (int)cr.size(),
                           (int)(cr.size() * sizeof(WinRound)),
                           (int)(cr.size() * sizeof(WinRound) + cg.size() * sizeof(WinGroup))};
                program.resize(program.size() + bytes());
                unsigned char *to = program.data() + c.offset;
                memcpy(to, cr.data(), c.groups);
                if (!cg.empty()) memcpy(to + c.groups, cg.data(), c.terms - c.groups);
                memcpy(to + c.terms, ct.data(), c.bytes - c.terms);
                chunks.push_back(c);
                cr.clear(), cg.clear(), ct.clear();
            };
            for (; ji < jobs.size() && jobs[ji].part == part; ++ji) {
                const Job *job = &jobs[ji];
                auto open = [&](size_t more) {
                    if (!cr.empty() && bytes() + more > (size_t)kWinStage) close();
                    WinRound hd = prog[job->round].hd;
                    hd.group = (int)cg.size(), hd.ngroups = 0;
                    hd.zterm = (int)ct.size(), hd.nz = 0;
                    cr.push_back(hd);
                };
                // (a piece of a group must fit a stage of its own)
                constexpr size_t piece = (kWinStage - sizeof(WinRound) - sizeof(WinGroup)) / sizeof(WinTerm);
                bool opened = false;
                for (size_t si = job->slice; si < job->end; ++si) {
                    const Slice &sl = slices[si];
                    const Entry &en = prog[job->round].entries[sl.entry];
                    for (size_t b = sl.begin; b < sl.end; b += piece) {
                        const size_t e = std::min(sl.end, b + piece);
                        const size_t need = (e - b) * sizeof(WinTerm) + sizeof(WinGroup);
                        if (!opened || bytes() + need > (size_t)kWinStage)
                            open(need + sizeof(WinRound)), opened = true;
                        WinRound &rd = cr.back();
                        if (en.z) {
                            rd.zterm = (int)ct.size();
                            rd.nz = (int)(e - b);
                        } else {
                            WinGroup wg = en.wg;
                            wg.term = (int)ct.size();
                            wg.nterms = (int)(e - b);
                            cg.push_back(wg);
                            ++rd.ngroups;
                        }
                        ct.insert(ct.end(), en.terms.begin() + b, en.terms.begin() + e);
                    }
                }
            }
            close();
            wd.nchunks = (int)chunks.size() - wd.chunk;
            wins.push_back(wd);
        }
    }
    // Host-side packed coefficients of the sweeps, uploaded with the windows' once per
    // call, and the results: the windows' sum, then one per sweep.
    std::vector<int> offs;
    std::vector<TermCoef> packed;
    for (size_t gi : sweeps) {
        offs.push_back((int)packed.size());
        for (int t : groups[gi].second) packed.push_back(coef_of(t));
    }
    lq_state *ms = const_cast<lq_state *>(s);
    auto al = [](size_t x) { return (x + 15) / 16 * 16; };
    const size_t o_win = al(packed.size() * sizeof(TermCoef));
    const size_t o_chk = o_win + al(wins.size() * sizeof(WinDesc));
    const size_t o_pgm = o_chk + al(chunks.size() * sizeof(WinChunk));
    const size_t o_beg = o_pgm + al(program.size());
    const size_t o_res = o_beg + (zfold >= 0 ? al(sizeof(pbeg)) : 0);
    const size_t nres = sweeps.size() + (wins.empty() ? 0 : 1);
    LQ_TRY(ensure_prog(ms, o_res + al(nres * sizeof(double)) + 256));
    char *dp = (char *)ms->d_prog;
    const TermCoef *d_tc = (const TermCoef *)dp;
    double *d_res = (double *)(dp + o_res);
    {
        std::vector<char> up(o_res, 0);
        auto put = [&](size_t o, const auto &x) {
            if (!x.empty()) memcpy(up.data() + o, x.data(), x.size() * sizeof(x[0]));
        };
        put(0, packed);
        put(o_win, wins);
        put(o_chk, chunks);
        put(o_pgm, program);
        if (zfold >= 0) memcpy(up.data() + o_beg, pbeg, sizeof(pbeg));
        LQ_CUDA_TRY(cudaMemcpyAsync(dp, up.data(), o_res, cudaMemcpyHostToDevice, s->stream));
    }
    prof_begin(s->stream, kProfReduce);
    size_t ri = 0;
    if (!wins.empty()) {
        const int blocks = std::min(nwork, 2 * 148);
        const size_t shm = ((size_t)16 << T) + kWinStage;
        auto run = [&](auto *v) -> cudaError_t {
            using A = std::remove_const_t<std::remove_pointer_t<decltype(v)>>;
            const cudaError_t e =
                cudaFuncSetAttribute(k_pauli_windows<A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (16 << kWinT) + kWinStage);
            if (e != cudaSuccess) return e;
            k_pauli_windows<A><<<blocks, 1 << m, shm, s->stream>>>(
                v, n, T, (const WinDesc *)(dp + o_win), (int)wins.size(),
                (const WinChunk *)(dp + o_chk), (const unsigned char *)(dp + o_pgm), nwork,
                ms->d_red);
            return cudaGetLastError();
        };
        LQ_CUDA_TRY(s->dtype == LQ_C128 ? run((const double2 *)s->d) : run((const float2 *)s->d));
        k_final_sum<1><<<1, 256, 0, s->stream>>>(s->d_red, blocks, d_res + ri++);
    }
    for (size_t k = 0; k < sweeps.size(); ++k) {
        const auto &gr = groups[sweeps[k]];
        const int nt = (int)gr.second.size();
        const size_t shm = nt * sizeof(TermCoef);
        if ((int)k == zfold && s->dtype == LQ_C128)
            k_pauli_zfold<<<g, th, shm, s->stream>>>((const double2 *)s->d, n, d_tc + offs[k], nt,
                                                     (const int *)(dp + o_beg), s->d_red);
        else if ((int)k == zfold)
            k_pauli_zfold<<<g, th, shm, s->stream>>>((const float2 *)s->d, n, d_tc + offs[k], nt,
                                                     (const int *)(dp + o_beg), s->d_red);
        else if (s->dtype == LQ_C128)
            k_pauli_group<<<g, th, shm, s->stream>>>((const double2 *)s->d, n, gr.first,
                                                     d_tc + offs[k], nt, s->d_red);
        else
            k_pauli_group<<<g, th, shm, s->stream>>>((const float2 *)s->d, n, gr.first,
                                                     d_tc + offs[k], nt, s->d_red);
        k_final_sum<1><<<1, 256, 0, s->stream>>>(s->d_red, g, d_res + ri++);
    }
    prof_end(s->stream, kProfReduce);
    LQ_CUDA_TRY(cudaGetLastError());
    std::vector<double> res(nres);
    if (nres)
        LQ_CUDA_TRY(cudaMemcpyAsync(res.data(), d_res, nres * sizeof(double),
                                    cudaMemcpyDeviceToHost, s->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    double sum = 0.0;
    for (size_t k = 0; k < nres; ++k) {
        sum += res[k];
        // (with per-term values every term is a sweep of its own, in order)
        if (per_term) per_term[groups[sweeps[k]].second[0]] = res[k];
    }
    *out = sum;
    return LQ_OK;
}

// ---------------------------------------------------------------------------
// Pauli-sum expectation that allocates nothing (lq_expectation_pauli_static).
//
// Its scratch -- the per-block partial sums, the per-group results and the
// packed term coefficients -- lives in one file-scope device array of fixed
// size instead of memory obtained from cudaMalloc.  Host code cannot hand the
// array's name to a kernel (on the host that name is only a stand-in, not a
// device address), so the device address is fetched once per device with
// cudaGetSymbolAddress and cached.
// ---------------------------------------------------------------------------
constexpr int kStaticMaxTerms = 1024;
constexpr size_t kStaticPartialBytes = sizeof(double) * kRedBlocks;
constexpr size_t kStaticResultBytes = sizeof(double) * kStaticMaxTerms;
constexpr size_t kStaticCoefBytes = sizeof(TermCoef) * kStaticMaxTerms;
constexpr size_t kStaticScratchBytes = 64 * 1024;
static_assert(kStaticPartialBytes + kStaticResultBytes + kStaticCoefBytes <= kStaticScratchBytes,
              "static scratch too small");

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

static int static_scratch_address(unsigned char **out) {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static unsigned char *addr[kMaxDevices] = {};
    int dev = 0;
    LQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return set_error(LQ_ERR_UNSUPPORTED, "device %d", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            return set_error(LQ_ERR_CUDA, "cudaGetSymbolAddress(static scratch): %s",
                             cudaGetErrorString(e));
        addr[dev] = (unsigned char *)p;
    }
    *out = addr[dev];
    return LQ_OK;
}

}  // namespace lq

using namespace lq;

namespace lq {

// ---------------------------------------------------------------------------
// Spare resources of small handles.  Creating and destroying a handle costs 52 + 64 us
// for its stream, and up to some milliseconds for its buffers when no other allocation
// keeps the driver's memory block mapped: a gradient of a 4-qubit circuit, which makes a
// handle of its own, took 2.6 ms, nearly all of it there (0.075 ms now).  So a destroyed handle of
// at most 1 MiB leaves its stream, scratch and buffers to the next one on its device.  All of
// them are used on the handle's own stream, which its destruction waits for; a wait for the
// whole device would break a graph capture on any other stream.  Only the amplitudes may be
// known elsewhere (lq_state::lent): they are then given back by cudaFree, which waits for
// their readers.  At most four sets of at most 4 MiB are kept; a failed allocation
// (device_malloc) frees them.
// ---------------------------------------------------------------------------
constexpr size_t kSpares = 4, kSpareBytes = 1 << 20;

struct Spare {
    int device;
    size_t bytes;  // of d
    void *d, *d_prog, *d_work;
    size_t prog_cap, work_cap;
    double *d_red;
    unsigned *d_flag;
    cudaStream_t stream;
};

static std::mutex g_spare_mu;
static std::vector<Spare> &spares() {  // (never destroyed: the driver may be gone by then)
    static auto *v = new std::vector<Spare>();
    return *v;
}

// s's amplitudes may be read on other streams from now on.
static void lend(const lq_state *s) { const_cast<lq_state *>(s)->lent = true; }

static void free_resources(lq_state *s) {
    if (s->d) cudaFree(s->d);
    if (s->d_red) cudaFree(s->d_red);
    if (s->d_flag) cudaFree(s->d_flag);
    if (s->d_prog) cudaFree(s->d_prog);
    if (s->d_work) cudaFree(s->d_work);
    if (s->stream) cudaStreamDestroy(s->stream);
}

static void move_spare(lq_state *s, const Spare &x) {
    s->d = x.d;
    s->d_red = x.d_red;
    s->d_flag = x.d_flag;
    s->d_prog = x.d_prog;
    s->prog_cap = x.prog_cap;
    s->d_work = x.d_work;
    s->work_cap = x.work_cap;
    s->stream = x.stream;
}

static void free_spares(size_t keep) {
    std::lock_guard<std::mutex> lk(g_spare_mu);
    while (spares().size() > keep) {
        lq_state t;
        move_spare(&t, spares().back());
        spares().pop_back();
        free_resources(&t);
    }
}

// A spare for s (its device), with a buffer of its size if there is one.
static bool take_spare(lq_state *s) {
    if (s->bytes > kSpareBytes) return false;
    Spare x;
    {
        std::lock_guard<std::mutex> lk(g_spare_mu);
        auto &v = spares();
        size_t best = v.size();
        for (size_t k = 0; k < v.size(); ++k)
            if (v[k].device == s->device && (best == v.size() || v[k].bytes == s->bytes)) best = k;
        if (best == v.size()) return false;
        x = v[best];
        v.erase(v.begin() + best);
    }
    move_spare(s, x);
    if (x.bytes != s->bytes) {
        if (s->d) cudaFree(s->d);
        s->d = nullptr;
    }
    return true;
}

// The caller has waited for s's stream.
static bool give_spare(lq_state *s) {
    if (s->bytes > kSpareBytes || !s->d || !s->d_red || !s->d_flag || !s->stream) return false;
    auto room = [] { return spares().size() < kSpares; };
    {
        std::lock_guard<std::mutex> lk(g_spare_mu);
        if (!room()) return false;
    }
    auto trim = [](void *&p, size_t &cap) {
        if (p && cap > kSpareBytes) {
            cudaFree(p);
            p = nullptr;
            cap = 0;
        }
    };
    trim(s->d_prog, s->prog_cap);
    trim(s->d_work, s->work_cap);
    if (s->lent) {
        cudaFree(s->d);
        s->d = nullptr;
    }
    std::lock_guard<std::mutex> lk(g_spare_mu);
    if (!room()) return false;
    spares().push_back(Spare{s->device, s->d ? s->bytes : 0, s->d, s->d_prog, s->d_work,
                             s->prog_cap, s->work_cap, s->d_red, s->d_flag, s->stream});
    return true;
}

}  // namespace lq

extern "C" {

int lq_expectation_pauli_static(const void *d_amplitudes, int num_qubits, int dtype,
                                const lq_pauli_term *terms, int nterms, int y_convention,
                                void *stream, double *out) {
    clear_error();
    if (!d_amplitudes || !out || (nterms > 0 && !terms) || nterms < 0)
        return set_error(LQ_ERR_INVALID_ARG, "null pointer or negative term count");
    if (num_qubits < 1 || num_qubits > 36)
        return set_error(LQ_ERR_STATE_DIMENSION, "num_qubits %d outside 1..36", num_qubits);
    if (dtype != LQ_C128 && dtype != LQ_C64)
        return set_error(LQ_ERR_INVALID_ARG, "unknown dtype %d", dtype);
    if (y_convention != LQ_Y_REFERENCE && y_convention != LQ_Y_TEXTBOOK)
        return set_error(LQ_ERR_INVALID_ARG, "unknown Y convention %d", y_convention);
    if (nterms > kStaticMaxTerms)
        return set_error(LQ_ERR_UNSUPPORTED,
                         "%d Pauli terms exceed the fixed scratch of this entry point "
                         "(at most %d terms; use lq_expectation_pauli)",
                         nterms, kStaticMaxTerms);
    if (nterms == 0) {
        *out = 0.0;
        return LQ_OK;
    }
    const int n = num_qubits;
    const uint64_t lim = n == 64 ? ~0ull : ((1ull << n) - 1);
    for (int t = 0; t < nterms; ++t) {
        if ((terms[t].xmask & ~lim) || (terms[t].zmask & ~lim))
            return set_error(LQ_ERR_QUBIT_INDEX, "Pauli term %d acts on a qubit >= %d", t, n);
        if (terms[t].ny != __builtin_popcountll(terms[t].xmask & terms[t].zmask))
            return set_error(LQ_ERR_INVALID_ARG, "Pauli term %d: ny does not match its masks", t);
    }
    // host-stack copies and a stream wait cannot be captured into a graph
    {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        LQ_CUDA_TRY(cudaStreamIsCapturing((cudaStream_t)stream, &cs));
        if (cs != cudaStreamCaptureStatusNone)
            return set_error(LQ_ERR_UNSUPPORTED,
                             "lq_expectation_pauli_static cannot run on a capturing stream");
    }
    // The scratch array is per device: the amplitudes must be on the current one.
    {
        cudaPointerAttributes pa{};
        int dev = 0;
        LQ_CUDA_TRY(cudaGetDevice(&dev));
        if (cudaPointerGetAttributes(&pa, d_amplitudes) != cudaSuccess) {
            cudaGetLastError();
            return set_error(LQ_ERR_INVALID_ARG, "d_amplitudes is not a CUDA pointer");
        }
        if (pa.type != cudaMemoryTypeDevice && pa.type != cudaMemoryTypeManaged)
            return set_error(LQ_ERR_INVALID_ARG, "d_amplitudes is not device memory");
        if (pa.device != dev)
            return set_error(LQ_ERR_INVALID_ARG,
                             "d_amplitudes is on device %d, the current device is %d", pa.device,
                             dev);
    }
    unsigned char *scratch = nullptr;
    LQ_TRY(static_scratch_address(&scratch));
    double *d_partials = (double *)scratch;
    double *d_results = (double *)(scratch + kStaticPartialBytes);
    TermCoef *d_coef = (TermCoef *)(scratch + kStaticPartialBytes + kStaticResultBytes);
    cudaStream_t st = (cudaStream_t)stream;

    // Group the terms by X mask with fixed-size host arrays (no heap).
    int order[kStaticMaxTerms], gbegin[kStaticMaxTerms + 1];
    uint64_t gx[kStaticMaxTerms];
    bool used[kStaticMaxTerms] = {};
    int ng = 0, k = 0;
    for (int t = 0; t < nterms; ++t) {
        if (used[t]) continue;
        gx[ng] = terms[t].xmask;
        gbegin[ng] = k;
        for (int u = t; u < nterms; ++u)
            if (!used[u] && terms[u].xmask == gx[ng]) {
                used[u] = true;
                order[k++] = u;
            }
        ++ng;
    }
    gbegin[ng] = k;
    TermCoef packed[kStaticMaxTerms];  // host stack: 24 KiB
    for (int i = 0; i < nterms; ++i) {
        const lq_pauli_term &pt = terms[order[i]];
        int q = pt.ny & 3;
        if (y_convention == LQ_Y_TEXTBOOK) q = (4 - q) & 3;
        const double a = q == 0 ? 1.0 : q == 2 ? -1.0 : 0.0;
        const double b = q == 1 ? -1.0 : q == 3 ? 1.0 : 0.0;
        packed[i] = TermCoef{pt.zmask, pt.coefficient * a, pt.coefficient * b};
    }
    LQ_CUDA_TRY(cudaMemcpyAsync(d_coef, packed, sizeof(TermCoef) * nterms,
                                cudaMemcpyHostToDevice, st));
    const uint64_t N = 1ull << n;
    const int th = 256;
    const int g = red_grid(std::max<uint64_t>(N / 2, 1), th);
    for (int gi = 0; gi < ng; ++gi) {
        const int nt = gbegin[gi + 1] - gbegin[gi];
        const size_t shm = nt * sizeof(TermCoef);
        if (dtype == LQ_C128)
            k_pauli_group<<<g, th, shm, st>>>((const double2 *)d_amplitudes, n, gx[gi],
                                              d_coef + gbegin[gi], nt, d_partials);
        else
            k_pauli_group<<<g, th, shm, st>>>((const float2 *)d_amplitudes, n, gx[gi],
                                              d_coef + gbegin[gi], nt, d_partials);
        k_final_sum<1><<<1, 256, 0, st>>>(d_partials, g, d_results + gi);
    }
    LQ_CUDA_TRY(cudaGetLastError());
    double res[kStaticMaxTerms];  // host stack: 8 KiB
    LQ_CUDA_TRY(cudaMemcpyAsync(res, d_results, sizeof(double) * ng, cudaMemcpyDeviceToHost, st));
    LQ_CUDA_TRY(cudaStreamSynchronize(st));
    double sum = 0.0;
    for (int gi = 0; gi < ng; ++gi) sum += res[gi];
    *out = sum;
    return LQ_OK;
}

const char *lq_last_error(void) { return g_last_error.c_str(); }

int lq_version(void) { return 1 * 10000 + 0 * 100 + 0; }

int lq_device_count(int *count) {
    if (!count) return set_error(LQ_ERR_INVALID_ARG, "null count");
    int c = 0;
    cudaError_t e = cudaGetDeviceCount(&c);
    if (e != cudaSuccess) {
        *count = 0;
        cudaGetLastError();
        return set_error(LQ_ERR_CUDA, "cudaGetDeviceCount: %s", cudaGetErrorString(e));
    }
    *count = c;
    return LQ_OK;
}

int lq_set_device(int device) {
    LQ_CUDA_TRY(cudaSetDevice(device));
    return LQ_OK;
}

int lq_set_alloc_limit(uint64_t bytes) {
    std::lock_guard<std::mutex> lk(g_alloc_mu);
    g_alloc_limit = bytes;
    return LQ_OK;
}

int lq_state_create(int num_qubits, int dtype, lq_state **out) {
    clear_error();
    if (!out) return set_error(LQ_ERR_INVALID_ARG, "null output pointer");
    *out = nullptr;
    if (dtype != LQ_C128 && dtype != LQ_C64)
        return set_error(LQ_ERR_INVALID_ARG, "unknown dtype %d", dtype);
    if (num_qubits < 1 || num_qubits > 36)
        return set_error(LQ_ERR_STATE_DIMENSION,
                         "Invalid state dimension: 2^%d (supported 1..36 qubits)", num_qubits);
    const size_t bytes = (size_t)amp_bytes(dtype) << num_qubits;
    {
        std::lock_guard<std::mutex> lk(g_alloc_mu);
        if (g_alloc_limit && g_alloc_in_use + bytes > g_alloc_limit)
            return set_error(LQ_ERR_OOM,
                             "state of %zu bytes exceeds the allocation limit (%llu in use, "
                             "limit %llu)",
                             bytes, (unsigned long long)g_alloc_in_use,
                             (unsigned long long)g_alloc_limit);
    }
    lq_state *s = new lq_state();
    s->n = num_qubits;
    s->dtype = dtype;
    s->bytes = bytes;
    cudaGetDevice(&s->device);
    cudaError_t e = cudaSuccess;
    if (!take_spare(s)) {
        e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
        if (e == cudaSuccess)
            e = device_malloc(&s->d_red, sizeof(double) * kRedBlocks * 2 * kMaxTermsPerPass);
        if (e == cudaSuccess) e = device_malloc(&s->d_flag, sizeof(unsigned) * 4);
    }
    if (e == cudaSuccess && !s->d) e = device_malloc(&s->d, bytes);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->d_flag, 0, sizeof(unsigned) * 4, s->stream);
    if (e != cudaSuccess) {
        const int code = e == cudaErrorMemoryAllocation ? LQ_ERR_OOM : LQ_ERR_CUDA;
        free_resources(s);
        delete s;
        cudaGetLastError();
        return set_error(code, "creating a %d-qubit state: %s", num_qubits, cudaGetErrorString(e));
    }
    {
        std::lock_guard<std::mutex> lk(g_alloc_mu);
        g_alloc_in_use += bytes;
        ++g_handles;
    }
    *out = s;
    int rc = lq_state_set_basis(s, 0);
    if (rc != LQ_OK) {
        lq_state_destroy(s);
        *out = nullptr;
        return rc;
    }
    return LQ_OK;
}

int lq_state_destroy(lq_state *s) {
    if (!s) return LQ_OK;
    // (a stream that cannot be waited for is not handed on)
    const bool idle = s->stream && cudaStreamSynchronize(s->stream) == cudaSuccess;
    bool last;
    {
        std::lock_guard<std::mutex> lk(g_alloc_mu);
        g_alloc_in_use -= s->bytes;
        last = --g_handles == 0;
    }
    free_plan_cache(s);
    if (!idle || !give_spare(s)) free_resources(s);
    delete s;
    if (last) free_pool();
    return LQ_OK;
}

int lq_state_num_qubits(const lq_state *s, int *out) {
    LQ_TRY(check_state(s));
    if (!out) return set_error(LQ_ERR_INVALID_ARG, "null output");
    *out = s->n;
    return LQ_OK;
}

int lq_state_dtype(const lq_state *s, int *out) {
    LQ_TRY(check_state(s));
    if (!out) return set_error(LQ_ERR_INVALID_ARG, "null output");
    *out = s->dtype;
    return LQ_OK;
}

int lq_state_set_basis(lq_state *s, uint64_t index) {
    LQ_TRY(check_state(s));
    const uint64_t N = 1ull << s->n;
    if (index >= N)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "basis index %llu >= 2^%d",
                         (unsigned long long)index, s->n);
    if (s->dtype == LQ_C128)
        k_set_basis<<<grid_for(N, 256), 256, 0, s->stream>>>((double2 *)s->d, N, index);
    else
        k_set_basis<<<grid_for(N, 256), 256, 0, s->stream>>>((float2 *)s->d, N, index);
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

int lq_state_set_plus(lq_state *s) {
    LQ_TRY(check_state(s));
    const uint64_t N = 1ull << s->n;
    const double norm = 1.0 / std::sqrt((double)N);  // plus_state: 1/sqrt(size)
    if (s->dtype == LQ_C128)
        k_set_const<<<grid_for(N, 256), 256, 0, s->stream>>>((double2 *)s->d, N, norm);
    else
        k_set_const<<<grid_for(N, 256), 256, 0, s->stream>>>((float2 *)s->d, N, norm);
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

int lq_state_upload(lq_state *s, const double *host, size_t num_amplitudes) {
    LQ_TRY(check_state(s));
    if (!host) return set_error(LQ_ERR_INVALID_ARG, "null host buffer");
    const uint64_t N = 1ull << s->n;
    if (num_amplitudes != N)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected %llu, got %zu",
                         (unsigned long long)N, num_amplitudes);
    if (s->dtype == LQ_C128) {
        LQ_CUDA_TRY(cudaMemcpyAsync(s->d, host, N * 16, cudaMemcpyHostToDevice, s->stream));
    } else {
        // Stage in chunks through a temporary complex128 buffer.
        const uint64_t chunk = std::min<uint64_t>(N, 1ull << 24);
        double2 *tmp = nullptr;
        LQ_CUDA_TRY(cudaMallocAsync(&tmp, chunk * 16, s->stream));
        for (uint64_t o = 0; o < N; o += chunk) {
            const uint64_t c = std::min(chunk, N - o);
            LQ_CUDA_TRY(cudaMemcpyAsync(tmp, host + 2 * o, c * 16, cudaMemcpyHostToDevice,
                                        s->stream));
            k_c128_to_c64<<<grid_for(c, 256), 256, 0, s->stream>>>(tmp, (float2 *)s->d + o, c);
        }
        LQ_CUDA_TRY(cudaFreeAsync(tmp, s->stream));
    }
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return LQ_OK;
}

int lq_state_download(const lq_state *s, double *host, size_t num_amplitudes) {
    LQ_TRY(check_state(s));
    if (!host) return set_error(LQ_ERR_INVALID_ARG, "null host buffer");
    const uint64_t N = 1ull << s->n;
    if (num_amplitudes != N)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected %llu, got %zu",
                         (unsigned long long)N, num_amplitudes);
    if (s->dtype == LQ_C128) {
        LQ_CUDA_TRY(cudaMemcpyAsync(host, s->d, N * 16, cudaMemcpyDeviceToHost, s->stream));
        LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    } else {
        std::vector<float> tmp(2 * N);
        LQ_CUDA_TRY(cudaMemcpyAsync(tmp.data(), s->d, N * 8, cudaMemcpyDeviceToHost, s->stream));
        LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
        for (uint64_t i = 0; i < 2 * N; ++i) host[i] = tmp[i];
    }
    return LQ_OK;
}

int lq_state_upload_c64(lq_state *s, const float *host, size_t num_amplitudes) {
    LQ_TRY(check_state(s));
    if (s->dtype != LQ_C64) return set_error(LQ_ERR_UNSUPPORTED, "state is not complex64");
    if (!host) return set_error(LQ_ERR_INVALID_ARG, "null host buffer");
    const uint64_t N = 1ull << s->n;
    if (num_amplitudes != N)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected %llu, got %zu",
                         (unsigned long long)N, num_amplitudes);
    LQ_CUDA_TRY(cudaMemcpyAsync(s->d, host, N * 8, cudaMemcpyHostToDevice, s->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return LQ_OK;
}

int lq_state_download_c64(const lq_state *s, float *host, size_t num_amplitudes) {
    LQ_TRY(check_state(s));
    if (s->dtype != LQ_C64) return set_error(LQ_ERR_UNSUPPORTED, "state is not complex64");
    if (!host) return set_error(LQ_ERR_INVALID_ARG, "null host buffer");
    const uint64_t N = 1ull << s->n;
    if (num_amplitudes != N)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected %llu, got %zu",
                         (unsigned long long)N, num_amplitudes);
    LQ_CUDA_TRY(cudaMemcpyAsync(host, s->d, N * 8, cudaMemcpyDeviceToHost, s->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return LQ_OK;
}

int lq_state_copy(lq_state *dst, const lq_state *src) {
    LQ_TRY(check_state(dst));
    LQ_TRY(check_state(src));
    if (dst->n != src->n || dst->dtype != src->dtype)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected 2^%d, got 2^%d",
                         dst->n, src->n);
    LQ_CUDA_TRY(cudaStreamSynchronize(src->stream));
    lend(src);
    LQ_CUDA_TRY(cudaMemcpyAsync(dst->d, src->d, dst->bytes, cudaMemcpyDeviceToDevice, dst->stream));
    return LQ_OK;
}

int lq_state_tensor_product(lq_state *out, const lq_state *a, const lq_state *b) {
    LQ_TRY(check_state(out));
    LQ_TRY(check_state(a));
    LQ_TRY(check_state(b));
    if (out->n != a->n + b->n)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected 2^%d, got 2^%d",
                         a->n + b->n, out->n);
    if (out->dtype != a->dtype || a->dtype != b->dtype)
        return set_error(LQ_ERR_UNSUPPORTED, "mixed dtypes");
    LQ_CUDA_TRY(cudaStreamSynchronize(a->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(b->stream));
    lend(a);
    lend(b);
    const uint64_t N = 1ull << out->n;
    if (out->dtype == LQ_C128)
        k_kron<<<grid_for(N, 256), 256, 0, out->stream>>>(
            (double2 *)out->d, (const double2 *)a->d, (const double2 *)b->d, b->n, N);
    else
        k_kron<<<grid_for(N, 256), 256, 0, out->stream>>>(
            (float2 *)out->d, (const float2 *)a->d, (const float2 *)b->d, b->n, N);
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

int lq_state_synchronize(lq_state *s) {
    LQ_TRY(check_state(s));
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    unsigned flags = 0;
    LQ_CUDA_TRY(cudaMemcpy(&flags, s->d_flag, sizeof(unsigned), cudaMemcpyDeviceToHost));
    if (flags & kFlagTimeout) {
        cudaMemset(s->d_flag, 0, sizeof(unsigned));
        return set_error(LQ_ERR_TIMEOUT, "a bounded device wait ran out");
    }
    return LQ_OK;
}

int lq_check_wait_timeout(lq_state *s, unsigned polls) {
    LQ_TRY(check_state(s));
    if (polls < 1 || polls > (1u << 20))
        return set_error(LQ_ERR_INVALID_ARG, "polls must be 1..1048576 (got %u)", polls);
    k_wait_probe<<<1, 32, 0, s->stream>>>(s->d_flag, polls);
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

int lq_state_device_ptr(lq_state *s, void **dptr) {
    LQ_TRY(check_state(s));
    if (!dptr) return set_error(LQ_ERR_INVALID_ARG, "null output");
    lend(s);
    *dptr = s->d;
    return LQ_OK;
}

int lq_state_stream(lq_state *s, void **stream) {
    LQ_TRY(check_state(s));
    if (!stream) return set_error(LQ_ERR_INVALID_ARG, "null output");
    *stream = (void *)s->stream;
    return LQ_OK;
}

int lq_norm_sqr(const lq_state *s, double *out) {
    LQ_TRY(check_state(s));
    if (!out) return set_error(LQ_ERR_INVALID_ARG, "null output");
    lq_state *ms = const_cast<lq_state *>(s);
    double *d_out = ms->d_red + kRedBlocks * 2 * kMaxTermsPerPass - 2;
    LQ_TRY(norm_sqr_device(s, d_out));
    LQ_CUDA_TRY(cudaMemcpyAsync(ms->h_red, d_out, sizeof(double), cudaMemcpyDeviceToHost,
                                s->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    *out = ms->h_red[0];
    return LQ_OK;
}

int lq_normalize(lq_state *s) {
    LQ_TRY(check_state(s));
    return normalize_impl(s);
}

int lq_probabilities(const lq_state *s, double *host, size_t len) {
    LQ_TRY(check_state(s));
    if (!host) return set_error(LQ_ERR_INVALID_ARG, "null host buffer");
    const uint64_t N = 1ull << s->n;
    if (len != N)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected %llu, got %zu",
                         (unsigned long long)N, len);
    const uint64_t chunk = std::min<uint64_t>(N, 1ull << 24);
    double *tmp = nullptr;
    LQ_CUDA_TRY(cudaMallocAsync(&tmp, chunk * 8, s->stream));
    for (uint64_t o = 0; o < N; o += chunk) {
        const uint64_t c = std::min(chunk, N - o);
        if (s->dtype == LQ_C128)
            k_probs<<<grid_for(c, 256), 256, 0, s->stream>>>((const double2 *)s->d + o, tmp, c);
        else
            k_probs<<<grid_for(c, 256), 256, 0, s->stream>>>((const float2 *)s->d + o, tmp, c);
        LQ_CUDA_TRY(cudaMemcpyAsync(host + o, tmp, c * 8, cudaMemcpyDeviceToHost, s->stream));
    }
    LQ_CUDA_TRY(cudaFreeAsync(tmp, s->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return LQ_OK;
}

int lq_probability(const lq_state *s, uint64_t basis, double *out) {
    LQ_TRY(check_state(s));
    if (!out) return set_error(LQ_ERR_INVALID_ARG, "null output");
    if (basis >= (1ull << s->n)) {
        *out = 0.0;  // State::probability returns 0.0 out of range
        return LQ_OK;
    }
    double a[2];
    if (s->dtype == LQ_C128) {
        LQ_CUDA_TRY(cudaMemcpyAsync(a, (const double2 *)s->d + basis, 16, cudaMemcpyDeviceToHost,
                                    s->stream));
        LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    } else {
        float f[2];
        LQ_CUDA_TRY(cudaMemcpyAsync(f, (const float2 *)s->d + basis, 8, cudaMemcpyDeviceToHost,
                                    s->stream));
        LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
        a[0] = f[0];
        a[1] = f[1];
    }
    *out = a[0] * a[0] + a[1] * a[1];
    return LQ_OK;
}

int lq_inner_product(const lq_state *a, const lq_state *b, double out[2]) {
    LQ_TRY(check_state(a));
    LQ_TRY(check_state(b));
    if (!out) return set_error(LQ_ERR_INVALID_ARG, "null output");
    if (a->n != b->n)
        return set_error(LQ_ERR_DIMENSION_MISMATCH, "Dimension mismatch: expected %llu, got %llu",
                         (unsigned long long)(1ull << a->n), (unsigned long long)(1ull << b->n));
    if (a->dtype != b->dtype) return set_error(LQ_ERR_UNSUPPORTED, "mixed dtypes");
    LQ_CUDA_TRY(cudaStreamSynchronize(b->stream));
    lq_state *ma = const_cast<lq_state *>(a);
    const uint64_t N = 1ull << a->n;
    const int th = 256, g = red_grid(N, th);
    double *d_out = ma->d_red + kRedBlocks * 2 * kMaxTermsPerPass - 4;
    prof_begin(a->stream, kProfReduce);
    if (a->dtype == LQ_C128)
        k_inner_partial<<<g, th, 0, a->stream>>>((const double2 *)a->d, (const double2 *)b->d, N,
                                                 ma->d_red);
    else
        k_inner_partial<<<g, th, 0, a->stream>>>((const float2 *)a->d, (const float2 *)b->d, N,
                                                 ma->d_red);
    k_final_sum<2><<<1, 256, 0, a->stream>>>(ma->d_red, g, d_out);
    prof_end(a->stream, kProfReduce);
    LQ_CUDA_TRY(cudaGetLastError());
    LQ_CUDA_TRY(cudaMemcpyAsync(ma->h_red, d_out, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                                a->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(a->stream));
    out[0] = ma->h_red[0];
    out[1] = ma->h_red[1];
    return LQ_OK;
}

// Inclusive scan of in[0..N) into out (the fixed-order scan above); tot holds
// the chunk totals of every level (ceil(N/1024) + ceil(N/2^20) + ... doubles).
static int scan_inclusive(const double *in, double *out, double *tot, uint64_t N,
                          cudaStream_t st) {
    const uint64_t nc = (N + kScanChunk - 1) / kScanChunk;
    if (nc > 0x7fffffffull) return set_error(LQ_ERR_UNSUPPORTED, "scan too long");
    k_scan_chunks<<<(unsigned)nc, 256, 0, st>>>(in, out, tot, N);
    LQ_CUDA_TRY(cudaGetLastError());
    if (nc > 1) {
        double *incl = tot + nc;  // scanned chunk totals, in place after the totals
        LQ_TRY(scan_inclusive(tot, incl, incl + nc, nc, st));
        k_scan_add_base<<<grid_for(N, 256), 256, 0, st>>>(out, incl, N);
        LQ_CUDA_TRY(cudaGetLastError());
    }
    return LQ_OK;
}

static uint64_t scan_scratch(uint64_t N) {  // doubles needed by scan_inclusive's tot
    uint64_t need = 0;
    for (uint64_t n = N; n > 1;) {
        const uint64_t nc = (n + kScanChunk - 1) / kScanChunk;
        need += 2 * nc;
        n = nc;
    }
    return need + 2;
}

}  // extern "C"

// The amplitudes' scan: chunk scans (kept or not), their totals, the totals scanned.
template <class A>
static int measure_shots_t(lq_state *s, const A *v, uint64_t n_shots, uint64_t seed,
                           uint64_t *host_out) {
    const uint64_t N = 1ull << s->n, nc = (N + kScanChunk - 1) / kScanChunk;
    if (nc > 0x7fffffffull) return set_error(LQ_ERR_UNSUPPORTED, "scan too long");
    cudaStream_t st = s->stream;
    // The chunk scans are kept where they fit a workspace that stays, or where so many
    // shots come that one chunk each would cost more.  Above that a call would allocate
    // half the state's size for some probes (mapping 64 MB fresh and returning it takes
    // 0.4 to 20 ms); a chunk scanned again costs a shot about 6 ns of the whole GPU.
    // (23 qubits, 4096 shots: 86 us with the scans kept, 84 scanned again, 100 shots 84 and 60,
    // 20000 shots 94 and 174; 24 qubits, 1000 shots 780 us allocated, 82 scanned again; 131072
    // shots 880 and 840, 262144 = N / 64 940 and 1590.)
    const bool keep = N * 8 <= kKeptWork / 2 || n_shots > N / 64;
    const uint64_t scratch = scan_scratch(N);
    const uint64_t need = ((keep ? N : 0) + scratch + n_shots) * 8;
    Work work(s);
    LQ_TRY(work.take(need));
    double *tot = (double *)work.get(), *local = keep ? tot + scratch + n_shots : nullptr;
    uint64_t *d_out = (uint64_t *)(tot + scratch);
    double *incl = tot + nc;
    k_scan_chunks<<<(unsigned)nc, 256, 0, st>>>(v, local, tot, N);
    LQ_CUDA_TRY(cudaGetLastError());
    if (nc > 1) LQ_TRY(scan_inclusive(tot, incl, incl + nc, nc, st));
    if (keep)
        k_sample<<<grid_for(n_shots, 256), 256, 0, st>>>(local, incl, N, n_shots, seed, d_out);
    else
        k_sample_rescan<<<(unsigned)std::min<uint64_t>(n_shots, 148 * 8), 256, 0, st>>>(
            v, tot, incl, N, n_shots, seed, d_out);
    LQ_CUDA_TRY(cudaGetLastError());
    LQ_CUDA_TRY(cudaMemcpyAsync(host_out, d_out, n_shots * 8, cudaMemcpyDeviceToHost, st));
    LQ_CUDA_TRY(cudaStreamSynchronize(st));
    work.waited();
    return LQ_OK;
}

extern "C" {

int lq_measure_shots(const lq_state *s, uint64_t n_shots, uint64_t seed, uint64_t *host_out) {
    LQ_TRY(check_state(s));
    if (!host_out && n_shots) return set_error(LQ_ERR_INVALID_ARG, "null output");
    if (n_shots == 0) return LQ_OK;
    lq_state *ms = const_cast<lq_state *>(s);  // (its workspace)
    if (s->dtype == LQ_C128)
        return measure_shots_t(ms, (const double2 *)s->d, n_shots, seed, host_out);
    return measure_shots_t(ms, (const float2 *)s->d, n_shots, seed, host_out);
}

int lq_expectation_pauli(const lq_state *s, const lq_pauli_term *terms, int nterms,
                         int y_convention, double *out, double *per_term) {
    LQ_TRY(check_state(s));
    if (!out) return set_error(LQ_ERR_INVALID_ARG, "null output");
    if (nterms < 0 || (nterms > 0 && !terms))
        return set_error(LQ_ERR_INVALID_ARG, "bad term list");
    if (y_convention != LQ_Y_REFERENCE && y_convention != LQ_Y_TEXTBOOK)
        return set_error(LQ_ERR_INVALID_ARG, "unknown Y convention %d", y_convention);
    if (nterms == 0) {
        *out = 0.0;
        return LQ_OK;
    }
    return expectation_impl(s, terms, nterms, y_convention, out, per_term);
}

}  // extern "C"
