// Variational calls on one state: the VQE objective (src/optimization/vqe.rs:63-67),
// ParameterShift::compute_gradient (src/optimization/gradient.rs:44-78) and
// FiniteDifference::compute_gradient (src/optimization/gradient.rs:96-125).
//
// An energy is one Circuit::execute from |0...0> (fused passes) followed by one
// Pauli-sum reduction.  A parameter-shift gradient is one reverse sweep over the
// circuit where that gives the same values (adjoint.cu); otherwise every shifted
// circuit is simulated, as the reference does.
#include <cmath>
#include <map>

#include "adjoint.h"
#include "lq_internal.h"

namespace lq {

static int check_variational(lq_state *work, const lq_gate *ops, int nops, const double *theta,
                             int nparams, const lq_pauli_term *terms, int nterms, int yconv) {
    LQ_TRY(check_state(work));
    if (nops < 0 || (nops > 0 && !ops)) return set_error(LQ_ERR_INVALID_ARG, "bad op list");
    if (nparams < 0 || (nparams > 0 && !theta))
        return set_error(LQ_ERR_INVALID_ARG, "bad parameter vector");
    if (nterms < 0 || (nterms > 0 && !terms)) return set_error(LQ_ERR_INVALID_ARG, "bad terms");
    if (yconv != LQ_Y_REFERENCE && yconv != LQ_Y_TEXTBOOK)
        return set_error(LQ_ERR_INVALID_ARG, "unknown Y convention %d", yconv);
    for (int i = 0; i < nops; ++i) LQ_TRY(validate_gate(&ops[i], work->n, nparams));
    return LQ_OK;
}

static int energy_at(lq_state *work, const lq_gate *ops, int nops, const double *theta,
                     int nparams, const lq_pauli_term *terms, int nterms, int yconv, double *e) {
    LQ_TRY(lq_state_set_basis(work, 0));
    LQ_TRY(apply_circuit_impl(work, ops, nops, theta, nparams, LQ_EXEC_FUSED));
    if (nterms == 0) {
        *e = 0.0;
        return LQ_OK;
    }
    return expectation_impl(work, terms, nterms, yconv, e, nullptr);
}

// Whether the observable is one that every energy of the gradient would accept
// (otherwise the shifted circuits report the error).
static bool plain_terms(const lq_pauli_term *terms, int nterms, int n) {
    const uint64_t lim = (1ull << n) - 1;
    std::map<uint64_t, int> per_mask;
    for (int t = 0; t < nterms; ++t) {
        if ((terms[t].xmask & ~lim) || (terms[t].zmask & ~lim)) return false;
        if (terms[t].ny != __builtin_popcountll(terms[t].xmask & terms[t].zmask)) return false;
        if (++per_mask[terms[t].xmask] > kMaxGroupTerms) return false;
    }
    return true;
}

// The gradient by a reverse sweep; *done stays false where the shifted circuits
// have to run (adj_plan declines, or its second state cannot be allocated).
static int sweep_gradient(lq_state *work, const lq_gate *ops, int nops, const double *theta,
                          int nparams, const lq_pauli_term *terms, int nterms, int yconv,
                          double shift, double *grad, bool *done) {
    *done = false;
    if (nparams == 0 || work->dtype != LQ_C128 || !std::isfinite(shift)) return LQ_OK;
    for (int i = 0; i < nparams; ++i)
        if (!std::isfinite(theta[i])) return LQ_OK;
    if (!plain_terms(terms, nterms, work->n)) return LQ_OK;
    KeepError keep;  // (where the shifted circuits run, the sweep's reason is no error)
    const auto plan = adj_plan({AdjSpec{work->n, ops, nops, nparams, terms, nterms, yconv}}, 11,
                               (size_t)-1);
    if (!plan) return LQ_OK;
    const int rc = adj_upload(*plan, work, work->stream);
    if (rc == LQ_ERR_OOM) return LQ_OK;
    keep.release();
    LQ_TRY(rc);
    std::vector<double> up(theta, theta + nparams), out(nparams + 1);
    up.push_back(shift);
    LQ_TRY(adj_enqueue(*plan, work->stream, up.data(), out.data()));
    LQ_CUDA_TRY(cudaStreamSynchronize(work->stream));
    std::copy(out.begin() + 1, out.end(), grad);
    *done = true;
    return LQ_OK;
}

}  // namespace lq

using namespace lq;

extern "C" {

int lq_ansatz_energy(lq_state *work, const lq_gate *ops, int nops, const double *theta,
                     int nparams, const lq_pauli_term *terms, int nterms, int y_convention,
                     double *energy) {
    LQ_TRY(check_variational(work, ops, nops, theta, nparams, terms, nterms, y_convention));
    if (!energy) return set_error(LQ_ERR_INVALID_ARG, "null output");
    return energy_at(work, ops, nops, theta, nparams, terms, nterms, y_convention, energy);
}

int lq_parameter_shift(lq_state *work, const lq_gate *ops, int nops, const double *theta,
                       int nparams, const lq_pauli_term *terms, int nterms, int y_convention,
                       double shift, double *grad) {
    LQ_TRY(check_variational(work, ops, nops, theta, nparams, terms, nterms, y_convention));
    if (nparams > 0 && !grad) return set_error(LQ_ERR_INVALID_ARG, "null gradient output");
    bool done;
    LQ_TRY(sweep_gradient(work, ops, nops, theta, nparams, terms, nterms, y_convention, shift,
                          grad, &done));
    if (done) return LQ_OK;
    std::vector<double> p(theta, theta + nparams);
    for (int i = 0; i < nparams; ++i) {
        double ep, em;
        p[i] = theta[i] + shift;
        LQ_TRY(energy_at(work, ops, nops, p.data(), nparams, terms, nterms, y_convention, &ep));
        p[i] = theta[i] - shift;
        LQ_TRY(energy_at(work, ops, nops, p.data(), nparams, terms, nterms, y_convention, &em));
        p[i] = theta[i];
        grad[i] = (ep - em) / 2.0;
    }
    return LQ_OK;
}

int lq_finite_difference(lq_state *work, const lq_gate *ops, int nops, const double *theta,
                         int nparams, const lq_pauli_term *terms, int nterms, int y_convention,
                         double epsilon, double *grad) {
    LQ_TRY(check_variational(work, ops, nops, theta, nparams, terms, nterms, y_convention));
    if (nparams > 0 && !grad) return set_error(LQ_ERR_INVALID_ARG, "null gradient output");
    std::vector<double> p(theta, theta + nparams);
    double fx;
    LQ_TRY(energy_at(work, ops, nops, theta, nparams, terms, nterms, y_convention, &fx));
    for (int i = 0; i < nparams; ++i) {
        double fp;
        p[i] = theta[i] + epsilon;
        LQ_TRY(energy_at(work, ops, nops, p.data(), nparams, terms, nterms, y_convention, &fp));
        p[i] = theta[i];
        grad[i] = (fp - fx) / epsilon;
    }
    return LQ_OK;
}

}  // extern "C"
