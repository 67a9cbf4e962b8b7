// Parameter-shift gradients by one reverse sweep (adjoint.cu), used by the plain
// path (variational.cu) and the batched engine (batch.cu).
#pragma once

#include <memory>
#include <vector>

#include "fused_plan.h"
#include "fused_round.cuh"

namespace lq {

struct AdjSpec {  // one circuit and its observable
    int n;
    const lq_gate *ops;
    int nops;
    int nparams;
    const lq_pauli_term *terms;
    int nterms;
    int yconv;
};

class AdjProgram;

// Plan the gradients of `specs`; tile_bits is the tile width of states larger than
// 2^12 amplitudes, budget_bytes the device memory that the states of one wave may
// take.  Returns nullptr when some circuit has no reverse sweep with the same
// results (see adjoint.cu); host work only.
std::shared_ptr<AdjProgram> adj_plan(const std::vector<AdjSpec> &specs, int tile_bits,
                                     size_t budget_bytes);
// Device buffers and program upload.  With a work state the program sits in its
// program buffer and psi in its amplitudes (one circuit); LQ_ERR_OOM leaves
// nothing allocated.
int adj_upload(AdjProgram &p, lq_state *work, cudaStream_t st);
// Queue one evaluation on st: all parameters, then the shift, go up; the energies
// (of circuit adj_order()[k] at k), then the gradients, come down to `out`.
int adj_enqueue(AdjProgram &p, cudaStream_t st, const double *theta_and_shift, double *out);
const std::vector<int> &adj_order(const AdjProgram &p);

}  // namespace lq
