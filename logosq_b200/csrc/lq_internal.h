// Internal declarations shared by the translation units of liblogosq_b200.so.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/logosq_b200.h"

namespace lq {

// ---------------------------------------------------------------------------
// Errors: every C entry point returns a status and records a message in a
// thread-local buffer read by lq_last_error().
// ---------------------------------------------------------------------------
int set_error(int code, const char *fmt, ...);
void clear_error();

// Puts the calling thread's last error text back at its end, unless released: around an
// attempt whose failure the call makes up for.
class KeepError {
public:
    KeepError();
    ~KeepError();
    KeepError(const KeepError &) = delete;
    void release() { on_ = false; }

private:
    std::string text_;
    bool on_ = true;
};

#define LQ_CUDA_TRY(expr)                                                             \
    do {                                                                              \
        cudaError_t _e = (expr);                                                      \
        if (_e != cudaSuccess) {                                                      \
            return ::lq::set_error(_e == cudaErrorMemoryAllocation ? LQ_ERR_OOM        \
                                                                   : LQ_ERR_CUDA,      \
                                   "%s failed: %s (%s:%d)", #expr,                    \
                                   cudaGetErrorString(_e), __FILE__, __LINE__);       \
        }                                                                             \
    } while (0)

#define LQ_TRY(expr)                 \
    do {                             \
        int _rc = (expr);            \
        if (_rc != LQ_OK) return _rc; \
    } while (0)

// ---------------------------------------------------------------------------
// Device-side complex helpers (complex128 as double2, complex64 as float2).
// ---------------------------------------------------------------------------
struct Mat2 {  // 2x2 complex, row-major
    double2 m00, m01, m10, m11;
};

struct Phases4 {  // up to 4 complex phases
    double2 p[4];
};

// Reduction scratch sizes (per state handle).
constexpr int kRedBlocks = 148 * 8;   // partial slots of a two-stage reduction
constexpr int kMaxTermsPerPass = 32;  // Pauli terms accumulated per sweep
// Terms of one X mask in a Pauli sweep: they sit in its dynamic shared memory (24
// bytes each, 48 KB per block without an opt-in); larger groups are refused.
constexpr int kMaxGroupTerms = 2000;

// Flag word written by kernels that wait (bounded) on a barrier.
constexpr unsigned kFlagTimeout = 1u;

}  // namespace lq

// The opaque handle of the C ABI.
struct lq_state {
    int n = 0;
    int dtype = LQ_C128;
    int device = 0;
    void *d = nullptr;        // 2^n amplitudes
    size_t bytes = 0;
    bool lent = false;        // work on other streams may read d (its pointer was given out, ...)
    cudaStream_t stream = nullptr;
    double *d_red = nullptr;  // kRedBlocks * 2 * kMaxTermsPerPass doubles
    // Host mirror of the final reduction results.  Plain memory: page-locking 512
    // bytes took 2.4 ms of every handle's creation and 0.4 ms of its destruction.
    double h_red[4] = {0.0, 0.0, 0.0, 0.0};
    unsigned *d_flag = nullptr;  // timeout / error flags of waiting kernels
    // Per-handle device buffer for gate programs of fused passes.
    void *d_prog = nullptr;
    size_t prog_cap = 0;
    // Workspace of at most kOwnWork bytes for calls that need temporary arrays (Work).
    void *d_work = nullptr;
    size_t work_cap = 0;
    // Statistics of the last circuit call.
    int last_launches = 0;
    int last_passes = 0;
    // The fused program now in d_prog and its launch list, kept so that the same
    // circuit submitted again skips planning and the upload (fused.cu).  Any
    // other writer of d_prog goes through ensure_prog, which clears prog_valid.
    void *plan_cache = nullptr;
    bool prog_valid = false;
};

namespace lq {

inline size_t amp_bytes(int dtype) { return dtype == LQ_C64 ? 8 : 16; }

int check_state(const lq_state *s);
int check_qubit(const lq_state *s, int q);
int ensure_prog(lq_state *s, size_t bytes);
// Bytes of amplitudes that may still be allocated under lq_set_alloc_limit.
size_t alloc_room();

// gates.cu
int apply_gate_c128(lq_state *s, const lq_gate *g, const double *theta, int ntheta,
                    int *launches);
int apply_gate_c64(lq_state *s, const lq_gate *g, const double *theta, int ntheta,
                   int *launches);
int gate_num_qubits(int kind);
int validate_gate(const lq_gate *g, int n, int ntheta);
double gate_angle(const lq_gate *g, int k, const double *theta);
// Dense matrix (2^k x 2^k complex, row-major, qubit list order: q[0] high bit)
// of a gate as the reference applies it.  Returns k (number of qubits).
int gate_matrix(const lq_gate *g, const double *theta, double *m /* 2*64 doubles */);
// Classification used by the planner and the per-gate dispatcher.
enum GateClass { kClassGeneral = 0, kClassDiagonal = 1, kClassPermutation = 2 };
int gate_class(int kind);

// cudaMalloc; if it fails for lack of memory, again after what is kept for later calls
// (workspaces, spare resources of small handles) has been given back.
cudaError_t device_malloc_bytes(void **p, size_t bytes);
template <class T>
cudaError_t device_malloc(T **p, size_t bytes) {
    return device_malloc_bytes((void **)p, bytes);
}

// Temporary device memory for one call on s's stream, given back at the end of its scope.  Up
// to kOwnWork bytes stay with the handle (one call at a time: the stream orders their use), up
// to kKeptWork with a pool for all handles; more is allocated and returned each time.
constexpr size_t kOwnWork = 1ull << 20, kKeptWork = 128ull << 20;
class Work {
public:
    explicit Work(lq_state *s) : s_(s) {}
    ~Work();
    Work(const Work &) = delete;
    int take(size_t bytes);  // once
    void *get() const { return p_; }
    void waited() { idle_ = true; }  // the caller has waited for its last use

private:
    enum Kind { kOwn, kPooled, kCaptured };
    lq_state *s_;
    void *p_ = nullptr;
    size_t bytes_ = 0;
    cudaEvent_t used_ = nullptr;
    Kind kind_ = kOwn;
    bool idle_ = false;
};

// api_state.cu
int normalize_impl(lq_state *s);
// The state, or src in its place, divided by the norm whose squared partial sums are
// in s->d_red[0 .. nparts).
int scale_by_partials(lq_state *s, const void *src, int nparts);
// Record the state's FP64 squared norm; later rescale the state to it.
int norm_snapshot(lq_state *s);
int norm_restore(lq_state *s);
int expectation_impl(const lq_state *s, const lq_pauli_term *terms, int nterms, int yconv,
                     double *out, double *per_term);

// profile.cu: optional CUDA-event timing of launches, by kernel class.
enum ProfClass { kProfFused = 0, kProfGate = 1, kProfReduce = 2, kProfBatch = 3, kProfTc = 4,
                 kProfClasses = 5 };
bool prof_enabled();
// Record an event pair around a launch: call prof_begin before, prof_end after.
void prof_begin(cudaStream_t st, int cls);
void prof_end(cudaStream_t st, int cls);

// fused.cu
void free_plan_cache(lq_state *s);
int apply_circuit_impl(lq_state *s, const lq_gate *ops, int nops, const double *theta,
                       int ntheta, int mode);
int apply_block_impl(lq_state *s, int k, const int *qubits, const double *m);

}  // namespace lq
