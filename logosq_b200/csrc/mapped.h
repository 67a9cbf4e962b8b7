// Fused circuits as mapped rounds (mapped.cu).
#pragma once

#include <vector>

#include "gate_ops.h"

namespace lq {

struct MapLaunch {   // one pass over the state
    int h;           // its window: index bits [0,4) and [h, h+T-4)
    int nrounds;
    int ntabs;
    size_t offset;   // of its program in the blob
    size_t bytes;
};

struct MapStep {     // a pass, or a gate that fits no window (its own sweep)
    bool fused;
    MapLaunch pass;
    GateOp gate;
};

struct MapProgram {
    int T = 0;
    int rounds = 0;
    std::vector<MapStep> steps;
    std::vector<unsigned char> blob;
};

// Plan gops (canonical ops in order, none renormalising) for n qubits and tile bits
// T.  False when some gate has no mapped form or, unless `always`, the op records are the
// faster engine for such a circuit; host work only.
bool map_plan(const std::vector<GateOp> &gops, int n, int T, MapProgram &out, bool always = false);
// Launch one pass of the program (its blob stays on the host).
int map_launch(lq_state *s, int T, const MapLaunch &pass, const unsigned char *blob);

}  // namespace lq
