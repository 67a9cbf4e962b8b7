// Noise models of the reference (NoiseModel::apply, src/noise/mod.rs) on the
// device, with the reference's semantics:
//   * noise addresses index bit `qubit` (1 << qubit), unlike the gates, which
//     address bit n-1-qubit (src/noise/mod.rs:337-380);
//   * the Y error is the reference's YGate (-Y): new[bit 0] = i old[bit 1],
//     new[bit 1] = -i old[bit 0] (src/noise/mod.rs:350-368);
//   * amplitude damping sums K0 psi + K1 psi over every target qubit into one
//     fresh vector and then normalises (src/noise/mod.rs:108-146);
//   * phase damping rewrites the vector per target qubit, so only the last
//     target's damping survives, then normalises (src/noise/mod.rs:173-210).
// The Pauli errors reuse the per-gate kernels (a permutation, the -Y op, a one-bit
// diagonal).  Each damping model is two kernels: the map with the squared norm's
// partial sums, and the division by that norm.
#include <cmath>
#include <vector>

#include "gate_ops.h"
#include "reduce.cuh"

namespace lq {

// Amplitude damping: out = sum over the target bits of (K0 + K1) psi, K0 + K1 =
// [[1, sg], [0, s1]] on the bit, and the squared norm's partial sums.  Every target in
// one pass (amplitude i takes psi[i | bit] of its clear target bits, through the
// caches), where a sweep per target read psi twice and rewrote out each time: at 15
// qubits 46 ms for 58 applications of all 15 targets became 0.9 ms, most of the former
// in allocating and freeing the scratch vector and in 17 launches per application.
struct DampSpec {
    int count;
    int bit[36];
    double times[36];  // how often the bit is listed
    double sg, s1;
};

__global__ void __launch_bounds__(256)
    k_damp_norm(const double2 *__restrict__ psi, double2 *__restrict__ out, uint64_t N,
                const __grid_constant__ DampSpec d, double *__restrict__ partials) {
    __shared__ double sh[32];
    double acc[1] = {0.0};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double2 a = psi[i];
        double own = 0.0;
        double2 o = make_double2(0.0, 0.0);
        for (int k = 0; k < d.count; ++k) {
            const uint64_t bit = 1ull << d.bit[k];
            const double t = d.times[k];
            if (i & bit) {
                own += t * d.s1;
            } else {
                const double2 b = psi[i | bit];
                own += t;
                o.x = fma(t, b.x, o.x);
                o.y = fma(t, b.y, o.y);
            }
        }
        o.x = fma(own, a.x, d.sg * o.x);
        o.y = fma(own, a.y, d.sg * o.y);
        out[i] = o;
        acc[0] += o.x * o.x + o.y * o.y;
    }
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

// One target, in place: a thread takes both amplitudes of a pair, so no second vector is
// needed.  (Through one, 22 qubits, of which L2 holds a state but not two, took 80 us against
// 61 so, 26 qubits 900 against 770.)
__global__ void __launch_bounds__(256)
    k_damp_pair_norm(double2 *__restrict__ psi, uint64_t pairs, int bit, double times, double sg,
                     double s1, double *__restrict__ partials) {
    __shared__ double sh[32];
    double acc[1] = {0.0};
    const uint64_t low = (1ull << bit) - 1;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < pairs;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = (k & ~low) << 1 | (k & low), j = i | 1ull << bit;
        const double2 a = psi[i], b = psi[j];
        const double2 p = make_double2(times * fma(sg, b.x, a.x), times * fma(sg, b.y, a.y));
        const double2 q = make_double2(times * (s1 * b.x), times * (s1 * b.y));
        psi[i] = p;
        psi[j] = q;
        acc[0] += p.x * p.x + p.y * p.y + (q.x * q.x + q.y * q.y);
    }
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

// Phase damping in place: amplitudes with the bit set times f, and the squared norm's
// partial sums.
__global__ void __launch_bounds__(256)
    k_phase_norm(double2 *__restrict__ psi, uint64_t N, uint64_t bit, double f,
                 double *__restrict__ partials) {
    __shared__ double sh[32];
    double acc[1] = {0.0};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        double2 a = psi[i];
        if (i & bit) {
            a.x *= f;
            a.y *= f;
            psi[i] = a;
        }
        acc[0] += a.x * a.x + a.y * a.y;
    }
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
}

static int noise_targets(const lq_state *s, const int *qubits, int nqubits, std::vector<int> &out) {
    out.clear();
    if (!qubits) {  // None: every qubit (src/noise/mod.rs:66-69)
        for (int q = 0; q < s->n; ++q) out.push_back(q);
        return LQ_OK;
    }
    if (nqubits < 1) return set_error(LQ_ERR_INVALID_ARG, "empty target qubit list");
    for (int k = 0; k < nqubits; ++k) {
        LQ_TRY(check_qubit(s, qubits[k]));
        out.push_back(qubits[k]);
    }
    return LQ_OK;
}

static int noise_state(const lq_state *s) {
    LQ_TRY(check_state(s));
    if (s->dtype != LQ_C128)
        return set_error(LQ_ERR_UNSUPPORTED, "noise models run on complex128 states");
    return LQ_OK;
}

}  // namespace lq

using namespace lq;

extern "C" {

int lq_noise_pauli(lq_state *s, int qubit, int pauli) {
    LQ_TRY(noise_state(s));
    LQ_TRY(check_qubit(s, qubit));
    if (pauli < 1 || pauli > 3) return set_error(LQ_ERR_INVALID_ARG, "pauli must be 1 (X), 2 (Y) or 3 (Z)");
    lq_gate g;
    memset(&g, 0, sizeof(g));
    g.kind = pauli == 1 ? LQ_GATE_X : pauli == 2 ? LQ_GATE_Y : LQ_GATE_Z;
    g.q[0] = s->n - 1 - qubit;  // gate qubit whose basis bit is `qubit`
    g.q[1] = g.q[2] = -1;
    g.param[0] = g.param[1] = g.param[2] = -1;
    GateOp op;
    LQ_TRY(make_gate_op(&g, nullptr, s->n, &op));
    return launch_gate_op(s, op);
}

int lq_noise_amplitude_damping(lq_state *s, double gamma, const int *qubits, int nqubits) {
    LQ_TRY(noise_state(s));
    if (!(gamma >= 0.0 && gamma <= 1.0))
        return set_error(LQ_ERR_INVALID_ARG, "error probability must lie in [0, 1]");
    std::vector<int> tq;
    LQ_TRY(noise_targets(s, qubits, nqubits, tq));
    const double sg = std::sqrt(gamma), s1 = std::sqrt(1.0 - gamma);
    const uint64_t N = 1ull << s->n;
    DampSpec d{};
    d.sg = sg;
    d.s1 = s1;
    for (int b : tq) {
        int k = 0;
        while (k < d.count && d.bit[k] != b) ++k;
        if (k == d.count) d.bit[d.count++] = b;
        d.times[k] += 1.0;
    }
    if (d.count == 1) {
        const int grid = red_grid(N / 2, 256);
        prof_begin(s->stream, kProfGate);
        k_damp_pair_norm<<<grid, 256, 0, s->stream>>>((double2 *)s->d, N / 2, d.bit[0],
                                                     d.times[0], sg, s1, s->d_red);
        prof_end(s->stream, kProfGate);
        LQ_CUDA_TRY(cudaGetLastError());
        return scale_by_partials(s, nullptr, grid);
    }
    Work work(s);
    LQ_TRY(work.take(N * sizeof(double2)));
    void *out = work.get();
    const int grid = red_grid(N, 256);
    prof_begin(s->stream, kProfGate);
    k_damp_norm<<<grid, 256, 0, s->stream>>>((const double2 *)s->d, (double2 *)out, N, d,
                                            s->d_red);
    prof_end(s->stream, kProfGate);
    LQ_CUDA_TRY(cudaGetLastError());
    return scale_by_partials(s, out, grid);
}

int lq_noise_phase_damping(lq_state *s, double lambda, const int *qubits, int nqubits) {
    LQ_TRY(noise_state(s));
    if (!(lambda >= 0.0 && lambda <= 1.0))
        return set_error(LQ_ERR_INVALID_ARG, "error probability must lie in [0, 1]");
    std::vector<int> tq;
    LQ_TRY(noise_targets(s, qubits, nqubits, tq));
    // each target rewrites the vector: the last one survives
    const uint64_t N = 1ull << s->n;
    const int grid = red_grid(N, 256);
    prof_begin(s->stream, kProfGate);
    k_phase_norm<<<grid, 256, 0, s->stream>>>((double2 *)s->d, N, 1ull << tq.back(),
                                             std::sqrt(1.0 - lambda), s->d_red);
    prof_end(s->stream, kProfGate);
    LQ_CUDA_TRY(cudaGetLastError());
    return scale_by_partials(s, nullptr, grid);
}

}  // extern "C"
