// Parameter-shift gradients (ParameterShift::compute_gradient,
// src/optimization/gradient.rs:44-78) by one reverse sweep per circuit.
//
// A parameter that turns one rotation exp(-i a/2 P), a = scale * theta + offset, P a
// Pauli matrix, enters the energy as E = A + B cos a + C sin a, so the rule's value
//     (E(theta + s) - E(theta - s)) / 2 = sin(scale * s) * dE/da        for every s,
// and dE/da = Im <lambda| P |psi> with psi the state after the rotation and lambda
// the observable times the final state, both carried back to that gate.  So
// instead of 2P circuits there is one circuit forward, one application of the
// Pauli sum, and one sweep back over the pair (psi, lambda) that undoes each gate
// on both and takes the inner products on the way: 3 circuits' worth of gate work
// for any number of parameters.  (256 chains of 12-16 qubits, 28 160 parameters:
// 181 ms as shifted circuits with shared prefixes.)
//
// The sweep takes a circuit when every parameter turns at most one angle of an
// RX, RY, RZ, PHASE or U3 gate, every other gate is unitary, and all numbers are
// finite.  Any other circuit (a parameter used twice, CRX, CPHASE, RXX, a
// non-unitary matrix, a gate that fits no window) keeps the shifted circuits.
//
// Rounds.  (psi, lambda) is one state with a selector bit above the tile: a tile
// holds 2^T amplitudes of each in shared memory, and a register round gives every
// thread the 16 amplitudes that differ in three tile bits and the selector (going
// forward: in four tile bits of psi alone).  A round undoes one run of single-qubit
// gates on each of its bits, straight-line code in place.  All rotations of a run
// share one 2x2 and one set of sums (S_x, S_y, S_z) = Im <lambda| (X, Y, Z) |psi> taken just
// before the run is undone; a parameter's derivative is the combination of the three
// with its axis turned by the run's later gates, computed with the 2x2s on the device.
//
// Gates that permute basis states linearly (CNOT, X, SWAP) move no data: the tile
// keeps a map logical index -> shared-memory place, linear over XOR, and such a gate
// only changes the map's vectors, which the planner knows (a control outside the
// window adds a vector where that bit of the tile's index is 1).  Rounds address
// through the map and the store writes logical order back.  The first form of this
// kernel ran each gate as an op of the ping-pong rounds (fused_round.cuh): of its
// 2570 instructions per warp and round 690 were FP64, the rest register moves at the
// op switch's joins, selects of the CNOTs and the op dispatch.
//
// States of up to 2^12 amplitudes: one CTA does everything in shared memory
// (k_adj_small).  Larger ones: one launch per pass over the tiles of all circuits
// (k_adj_pass), three 128-thread CTAs per SM.
#include "adjoint.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace lq {

constexpr int kAdjSmallMax = 12;   // largest state kept in one CTA's shared memory
constexpr int kAdjMinN = 5;        // smaller circuits are planned as 5 qubits (upper bits 0)
constexpr int kAdjSmallThreads = 256;
constexpr int kAdjThreads = 128;
constexpr int kRoundSlots = 3;     // gradient runs of one round
constexpr int kHChunk = 2048;      // amplitudes of one block of k_adj_h
constexpr int kHStage = 12288;     // bytes of a Pauli sum that its blocks keep in shared memory
constexpr int kStageBytes = 4096;  // program bytes of one chunk (two are staged)

enum RoundType {
    RT_RUN = 0,   // nrun runs of single-qubit gates, on register bits 0 .. nrun-1
    RT_DIAG = 1,  // diagonal gates
    RT_CTRL = 2,  // controlled 2x2 or X on register bit 0
    RT_M2 = 3     // 4x4 on register bits 0 (high) and 1
};

constexpr int kMaxCst = 8;  // outside bits that a pass's map may depend on

struct AdjRound {
    int32_t type, nrun;
    int32_t data;           // offset of its coefficients (doubles) in the program's data
    int32_t ndiag;
    uint32_t reg[4];        // byte offsets of the register bits (swizzled tile)
    uint32_t base;          // byte offset of logical index 0
    int32_t nlane;
    int32_t slots;          // the pass's first gradient slot of this round << 8 | mask of runs
                            // that have one
    int32_t ncst;
    uint32_t lane[12];      // byte offset << 4 | tile position of the thread-index bits
    uint32_t cst_vec[kMaxCst];
    int32_t cst_bit[kMaxCst];
    uint64_t gpos[4];       // index masks of the register bits
};
static_assert(sizeof(AdjRound) % 16 == 0, "rounds are staged in 16-byte pieces");

struct AdjMap {  // logical tile index -> byte offset in the swizzled tile
    uint32_t vec[kMaxT];
    uint32_t base;
    int32_t ncst;
    uint32_t cst_vec[kMaxCst];
    int32_t cst_bit[kMaxCst];
};

struct AdjDiagOp {  // amplitude *= ph[pattern] where the index bits fix are all 1
    uint64_t fix;
    int32_t pb0, pb1, npat, pad;
    double pad2;
    double ph[8];
};
static_assert(sizeof(AdjDiagOp) == 12 * sizeof(double), "whole 16-byte pieces");

struct AdjCtrlOp {
    uint64_t gmask;      // index bits outside the registers that must be 1
    int32_t cm, is_x;    // register bits that must be 1
    double pad[2];
    double m[8];
};
static_assert(sizeof(AdjCtrlOp) == 12 * sizeof(double), "whole 16-byte pieces");

enum AtomKind { AT_CONST = 0, AT_RX = 1, AT_RY = 2, AT_RZ = 3 };

struct AdjAtom {  // one factor of a run of single-qubit gates, in time order
    int32_t kind, param;  // param: index into the call's parameters (-1: fixed angle)
    double scale, off;
    int64_t cmat;         // AT_CONST: offset of its 2x2 in the static coefficients
};

struct AdjRun {
    int32_t atom_begin, atom_end;
    int64_t coef_f, coef_b;  // where the 2x2 and its inverse go
    int64_t part;            // its partial sums, [3][ntiles]; -1: no parameter in it
    int32_t ntiles, pad;
};

// Consecutive rounds whose program (round records and data, each contiguous) is
// staged into shared memory together.
struct AdjChunk {
    int32_t round_begin, nrounds;
    int32_t data_begin, ndata;
};

struct AdjInst {
    int32_t n, T;
    int32_t f_chunk, f_nchunks;  // small circuits: chunks forward and back
    int32_t b_chunk, b_nchunks;
    int32_t group_begin, ngroups;
    int64_t off;                 // first amplitude in the wave's buffers (large circuits)
    int64_t epart;               // energy partials
    int32_t neparts, pad;
    int64_t part;                // small circuits: partial sums
    int32_t map;                 // small circuits: layout of the final state
    int32_t term_begin, nterms, pad2;
};

struct AdjPass {
    int32_t inst, h;
    int32_t chunk_begin, nchunks;
    int32_t tile_begin, ntiles;  // its blocks in the launch
    int64_t part;                // partial sums of its gradient runs
    int32_t map, pad;            // layout after its last round
};

struct AdjGroup {  // Pauli terms sharing an X mask
    uint32_t x;
    int32_t term_begin, nterms;
    uint32_t vx;       // small circuits: x through the final state's layout
    int32_t odd;       // some term has an odd number of Y (an imaginary element)
    int32_t flat;      // no term has a Z bit among bits 8-10
};
static_assert(sizeof(AdjGroup) == 24, "staged in 8-byte pieces");

struct AdjTerm {  // matrix element (-1)^popcount(i & z) (ca - i cb) between i and i ^ x
    double ca, cb;
    uint32_t z;       // (circuits of at most 32 qubits)
    uint8_t p;        // bits 8-10 of z: terms without X are sorted by it
    uint8_t flips;    // bit k: parity of k & p, the sign between i and i + 256 k
    uint16_t pad;
};
static_assert(sizeof(AdjTerm) == 24, "staged in 8-byte pieces");

// ---------------------------------------------------------------------------
// Device: coefficients of every run from the parameters
// ---------------------------------------------------------------------------
struct M22 {
    double2 a, b, c, d;  // [[a, b], [c, d]]
};

__device__ __forceinline__ M22 m22_mul(const M22 &x, const M22 &y) {
    M22 r;
    r.a = cmad2(x.a, y.a, x.b, y.c);
    r.b = cmad2(x.a, y.b, x.b, y.d);
    r.c = cmad2(x.c, y.a, x.d, y.c);
    r.d = cmad2(x.c, y.b, x.d, y.d);
    return r;
}

__global__ void __launch_bounds__(128)
    k_adj_coef(const AdjRun *__restrict__ runs, int nruns, const AdjAtom *__restrict__ atoms,
               const double *__restrict__ theta, double *__restrict__ coef,
               double *__restrict__ wts) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nruns) return;
    const AdjRun run = runs[r];
    M22 V;  // product of the gates after the current one
    V.a = V.d = make_double2(1.0, 0.0);
    V.b = V.c = make_double2(0.0, 0.0);
    for (int k = run.atom_end - 1; k >= run.atom_begin; --k) {
        const AdjAtom at = atoms[k];
        M22 g;
        if (at.kind == AT_CONST) {
            const double *m = coef + at.cmat;
            g.a = make_double2(m[0], m[1]);
            g.b = make_double2(m[2], m[3]);
            g.c = make_double2(m[4], m[5]);
            g.d = make_double2(m[6], m[7]);
        } else {
            double ang = at.off;
            if (at.param >= 0) ang = theta[at.param] * at.scale + at.off;
            double s, c;
            sincos(ang / 2.0, &s, &c);
            if (at.kind == AT_RX) {
                g.a = g.d = make_double2(c, 0.0);
                g.b = g.c = make_double2(0.0, -s);
            } else if (at.kind == AT_RY) {
                g.a = g.d = make_double2(c, 0.0);
                g.b = make_double2(-s, 0.0);
                g.c = make_double2(s, 0.0);
            } else {
                g.a = make_double2(c, -s);
                g.d = make_double2(c, s);
                g.b = g.c = make_double2(0.0, 0.0);
            }
            if (at.param >= 0) {
                // the axis turned by the later gates: V P V^dagger = x X + y Y + z Z
                M22 p, vd;
                p.a = p.b = p.c = p.d = make_double2(0.0, 0.0);
                if (at.kind == AT_RX) {
                    p.b = p.c = make_double2(1.0, 0.0);
                } else if (at.kind == AT_RY) {
                    p.b = make_double2(0.0, -1.0);
                    p.c = make_double2(0.0, 1.0);
                } else {
                    p.a = make_double2(1.0, 0.0);
                    p.d = make_double2(-1.0, 0.0);
                }
                vd.a = make_double2(V.a.x, -V.a.y);
                vd.b = make_double2(V.c.x, -V.c.y);
                vd.c = make_double2(V.b.x, -V.b.y);
                vd.d = make_double2(V.d.x, -V.d.y);
                const M22 m = m22_mul(m22_mul(V, p), vd);
                wts[3 * (int64_t)k] = m.c.x;
                wts[3 * (int64_t)k + 1] = m.c.y;
                wts[3 * (int64_t)k + 2] = m.a.x;
            }
        }
        V = m22_mul(V, g);
    }
    double *f = coef + run.coef_f, *b = coef + run.coef_b;
    f[0] = V.a.x, f[1] = V.a.y, f[2] = V.b.x, f[3] = V.b.y;
    f[4] = V.c.x, f[5] = V.c.y, f[6] = V.d.x, f[7] = V.d.y;
    b[0] = V.a.x, b[1] = -V.a.y, b[2] = V.c.x, b[3] = -V.c.y;
    b[4] = V.b.x, b[5] = -V.b.y, b[6] = V.d.x, b[7] = -V.d.y;
}

// ---------------------------------------------------------------------------
// Device: register rounds
// ---------------------------------------------------------------------------
template <int K>
__device__ __forceinline__ void m1_inplace(double2 (&v)[16], const double *__restrict__ c) {
    const double2 m00 = *(const double2 *)c, m01 = *(const double2 *)(c + 2);
    const double2 m10 = *(const double2 *)(c + 4), m11 = *(const double2 *)(c + 6);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        if (e & (1 << K)) continue;
        const double2 x0 = v[e], x1 = v[e | (1 << K)];
        v[e] = cmad2(m00, x0, m01, x1);
        v[e | (1 << K)] = cmad2(m10, x0, m11, x1);
    }
}

// Sums of one gradient run over this thread's amplitudes: register elements 0-7 are
// psi, 8-15 lambda.
template <int K>
__device__ __forceinline__ void grad3(const double2 (&s)[16], double &sx, double &sy, double &sz) {
    sx = sy = sz = 0.0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        if (e & (1 << K)) continue;
        const double2 a = s[e], b = s[e | (1 << K)];
        const double2 p = s[8 | e], q = s[8 | e | (1 << K)];
        sz = fma(p.x, a.y, fma(-p.y, a.x, fma(-q.x, b.y, fma(q.y, b.x, sz))));
        sx = fma(p.x, b.y, fma(-p.y, b.x, fma(q.x, a.y, fma(-q.y, a.x, sx))));
        sy = fma(q.x, a.x, fma(q.y, a.y, fma(-p.x, b.x, fma(-p.y, b.y, sy))));
    }
}

struct GradOut {
    double *part;      // shared: [slot][3][warps]
    unsigned mask;     // the warp's threads that hold amplitudes
    int half;          // half their number (0: one)
    bool add;          // a thread's second set of amplitudes
};

__device__ __forceinline__ void grad_emit(const GradOut &go, int nwarps, int slot, double sx,
                                          double sy, double sz) {
    for (int o = go.half; o > 0; o >>= 1) {
        sx += __shfl_down_sync(go.mask, sx, o);
        sy += __shfl_down_sync(go.mask, sy, o);
        sz += __shfl_down_sync(go.mask, sz, o);
    }
    if ((threadIdx.x & 31) == 0) {
        double *p = go.part + slot * 3 * nwarps + (threadIdx.x >> 5);
        if (go.add) {
            p[0] += sx, p[nwarps] += sy, p[2 * nwarps] += sz;
        } else {
            p[0] = sx, p[nwarps] = sy, p[2 * nwarps] = sz;
        }
    }
}

// One round for register set `v` (of 2^(T-4) forward, 2^(T-3) back) of the tile.
template <bool BWD, int NW>
__device__ __forceinline__ void adj_round(uint32_t tile_a, const AdjRound &rd,
                                          const double *__restrict__ data, uint64_t tile_base,
                                          int h, int v, const GradOut &go) {
    uint32_t sb = rd.base;
    int tbase = 0;
    for (int j = 0; j < rd.nlane; ++j) {
        const uint32_t on = 0u - ((uint32_t)(v >> j) & 1u), w = rd.lane[j];
        sb ^= (w >> 4) & on;
        tbase |= (int)((1u << (w & 15u)) & on);
    }
    for (int j = 0; j < rd.ncst; ++j)
        sb ^= rd.cst_vec[j] & (0u - (uint32_t)((tile_base >> rd.cst_bit[j]) & 1ull));
    const uint32_t E0 = rd.reg[0], E1 = rd.reg[1], E2 = rd.reg[2], E3 = rd.reg[3];
    auto addr_of = [&](int e) {
        const uint32_t x = ((e & 1) ? E0 : 0u) ^ ((e & 2) ? E1 : 0u) ^ ((e & 4) ? E2 : 0u) ^
                           ((e & 8) ? E3 : 0u);
        return tile_a + (sb ^ x);
    };
    double2 a[16];
    auto load = [&]() {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                         : "=d"(a[e].x), "=d"(a[e].y)
                         : "r"(addr_of(e)));
    };
    auto store = [&](const double2 (&x)[16]) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr_of(e)), "d"(x[e].x),
                         "d"(x[e].y)
                         : "memory");
    };
    const double *c = data + rd.data;
    if (rd.type == RT_RUN) {
        // Load, runs and store in each branch: no register is live across the joins.
#define LQ_RUN(K)                                                \
    {                                                            \
        if constexpr (BWD) {                                     \
            double sx, sy, sz;                                   \
            grad3<K>(a, sx, sy, sz);                             \
            grad_emit(go, NW, K, sx, sy, sz);                    \
        }                                                        \
        m1_inplace<K>(a, c + 8 * K);                             \
    }
        if (rd.nrun == 3) {
            load();
            LQ_RUN(0) LQ_RUN(1) LQ_RUN(2)
            store(a);
        } else if (rd.nrun == 2) {
            load();
            LQ_RUN(0) LQ_RUN(1)
            store(a);
        } else if (rd.nrun == 1) {
            load();
            LQ_RUN(0)
            store(a);
        } else if constexpr (!BWD) {
            load();
            LQ_RUN(0) LQ_RUN(1) LQ_RUN(2) LQ_RUN(3)
            store(a);
        }
#undef LQ_RUN
        return;
    }
    const uint64_t gbase = tile_base | (uint64_t)(tbase & 15) | ((uint64_t)(tbase >> 4) << h);
    load();
    if (rd.type == RT_DIAG) {
        for (int k = 0; k < rd.ndiag; ++k) {
            const AdjDiagOp &op = ((const AdjDiagOp *)c)[k];
            const uint64_t fm = op.fix;
            const uint64_t u0 = op.npat > 0 ? 1ull : 0ull, u1 = op.npat > 1 ? 1ull : 0ull;
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const uint64_t gi = gbase | ((e & 1) ? rd.gpos[0] : 0ull) |
                                    ((e & 2) ? rd.gpos[1] : 0ull) | ((e & 4) ? rd.gpos[2] : 0ull) |
                                    ((e & 8) ? rd.gpos[3] : 0ull);
                if ((gi & fm) != fm) continue;
                const int pat = (int)((gi >> op.pb0) & u0) | (int)((gi >> op.pb1) & u1) << 1;
                const double pr = op.ph[2 * pat], pi = op.ph[2 * pat + 1];
                a[e] = make_double2(fma(-a[e].y, pi, a[e].x * pr), fma(a[e].x, pi, a[e].y * pr));
            }
        }
        store(a);
    } else if (rd.type == RT_CTRL) {
        const AdjCtrlOp &op = *(const AdjCtrlOp *)c;
        if ((gbase & op.gmask) != op.gmask) return;
        double2 d[16];
        if (op.is_x) pp_x<0>(a, d, op.cm);
        else pp_m1<0>(a, d, op.m, op.cm);
        store(d);
    } else {
        double2 d[16];
        pp_m2<0, 1, false>(a, d, c);
        store(d);
    }
}

struct AdjProg {  // the device program
    const AdjRound *rounds;
    const double *data;
    const AdjChunk *chunks;
    const AdjMap *maps;
};

// Start the copy of one chunk's program into shared memory: round records, then data.
template <int NT>
__device__ __forceinline__ void adj_stage(uint32_t dst, const AdjChunk &ch, const AdjProg &pg) {
    auto copy = [&](const void *src, int bytes) {
        for (int o = (int)threadIdx.x * 16; o < bytes; o += NT * 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)o),
                         "l"((const char *)src + o)
                         : "memory");
        dst += (uint32_t)bytes;
    };
    copy(pg.rounds + ch.round_begin, ch.nrounds * (int)sizeof(AdjRound));
    copy(pg.data + ch.data_begin, ch.ndata * (int)sizeof(double));
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// All rounds of one pass on the tile, with the gradient runs' sums over the tile
// written to part[(slot * 3 + c) * ntiles + tile].
//
// The program comes from shared memory, staged chunk by chunk (the caller has
// started the first one): every circuit has its own, read by a few tiles only, so
// a record read where it is used would miss the first-level cache every time.
template <bool BWD, int NT>
__device__ __forceinline__ void adj_rounds(uint32_t tile_a, int T, int h, uint64_t tile_base,
                                           const AdjProg &pg, int chunk, int nchunks,
                                           unsigned char *stage, double *s_part,
                                           double *__restrict__ part, int ntiles, int tile) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x;
    const int nthr = 1 << (T - (BWD ? 3 : 4));
    GradOut go;
    go.mask = nthr >= 32 ? 0xffffffffu : (1u << nthr) - 1u;
    go.half = nthr >= 32 ? 16 : nthr >> 1;
    const int nw = nthr >= NT ? NW : nthr >= 32 ? nthr >> 5 : 1;  // warps that hold amplitudes
    int parity = 0;
    if (nchunks == 0) {  // permutations only: the map does it all
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
    for (int c = 0; c < nchunks; ++c) {
        const AdjChunk ch = pg.chunks[chunk + c];
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        unsigned char *cur = stage + (c & 1) * kStageBytes;
        if (c + 1 < nchunks)  // (that half was last read before the barrier above)
            adj_stage<NT>(smem_u32(stage + ((c + 1) & 1) * kStageBytes), pg.chunks[chunk + c + 1],
                          pg);
        const AdjRound *rounds = (const AdjRound *)cur;
        const double *data = (const double *)(rounds + ch.nrounds) - ch.data_begin;
        for (int r = 0; r < ch.nrounds; ++r) {
            const AdjRound &rd = rounds[r];
            go.part = s_part + parity * (kRoundSlots * 3 * NW);
            parity ^= 1;
            for (int v = tid; v < nthr; v += NT) {
                go.add = v != tid;
                adj_round<BWD, NW>(tile_a, rd, data, tile_base, h, v, go);
            }
            __syncthreads();
            if (BWD) {
                // (this half of s_part is written again two rounds on, past a barrier)
                // Runs with a parameter have the pass's next slots, in order.
                const int first = rd.slots >> 8;
                if (tid < 3 * kRoundSlots && (rd.slots >> (tid / 3) & 1)) {
                    const int slot = first + __popc(rd.slots & ((1 << (tid / 3)) - 1));
                    double sum = 0.0;
                    for (int w = 0; w < nw; ++w) sum += go.part[tid * NW + w];
                    part[(int64_t)(slot * 3 + tid % 3) * ntiles + tile] = sum;
                }
            }
        }
    }
}

__device__ __forceinline__ uint32_t map_base(const AdjMap &m, uint64_t tile_base) {
    uint32_t b = m.base;
    for (int j = 0; j < m.ncst; ++j)
        b ^= m.cst_vec[j] & (0u - (uint32_t)((tile_base >> m.cst_bit[j]) & 1ull));
    return b;
}

__device__ __forceinline__ uint32_t map_of(const AdjMap &m, uint32_t base, int l, int T) {
    for (int j = 0; j < T; ++j) base ^= m.vec[j] & (0u - ((uint32_t)(l >> j) & 1u));
    return base;
}

__device__ __forceinline__ double flip_sign(double x, uint32_t neg) {  // neg: bit 0 counts
    return __hiloint2double(__double2hiint(x) ^ (int)(neg << 31), __double2loint(x));
}

__device__ __forceinline__ void adj_sign_term(const AdjTerm &t, uint32_t i, double &al,
                                              double &be) {
    const uint32_t neg = (uint32_t)__popc(i & t.z);
    al += flip_sign(t.ca, neg);
    be += flip_sign(t.cb, neg);
}

// ---------------------------------------------------------------------------
// Small circuits: everything in one CTA
// ---------------------------------------------------------------------------
constexpr size_t adj_small_smem(int T) {
    return ((size_t)32 << T) + 1024 + 2 * kStageBytes +
           sizeof(double) * 2 * kRoundSlots * 3 * (kAdjSmallThreads / 32);
}

__global__ void __launch_bounds__(kAdjSmallThreads, 1)
    k_adj_small(const AdjInst *__restrict__ insts, AdjProg pg,
                const AdjGroup *__restrict__ groups, const AdjTerm *__restrict__ terms,
                double *__restrict__ part, double *__restrict__ epart) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t tile_a = smem_u32(base);
    const AdjInst in = insts[blockIdx.x];
    const int T = in.n, tid = threadIdx.x, N = 1 << T;
    unsigned char *stage = base + ((size_t)32 << T);
    double *s_part = (double *)(stage + 2 * kStageBytes);
    __shared__ double s_e[kAdjSmallThreads / 32];
    auto addr = [&](int l) { return tile_a + ((uint32_t)swz(l) << 4); };
    if (in.f_nchunks) adj_stage<kAdjSmallThreads>(smem_u32(stage), pg.chunks[in.f_chunk], pg);
    for (int l = tid; l < N; l += kAdjSmallThreads)
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr(l)), "d"(l == 0 ? 1.0 : 0.0),
                     "d"(0.0)
                     : "memory");
    __syncthreads();
    adj_rounds<false, kAdjSmallThreads>(tile_a, T, 4, 0ull, pg, in.f_chunk, in.f_nchunks, stage,
                                        s_part, nullptr, 1, 0);
    if (in.b_nchunks) adj_stage<kAdjSmallThreads>(smem_u32(stage), pg.chunks[in.b_chunk], pg);
    // lambda = H psi, and the energy; lambda takes psi's layout
    const AdjMap &mp = pg.maps[in.map];
    const uint32_t sel = (uint32_t)swz(N) << 4;
    double e = 0.0;
    for (int l = tid; l < N; l += kAdjSmallThreads) {
        const uint32_t at = map_of(mp, mp.base, l, T);
        double2 lam = make_double2(0.0, 0.0);
        for (int g = in.group_begin; g < in.group_begin + in.ngroups; ++g) {
            const AdjGroup gr = groups[g];
            double2 v;
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                         : "=d"(v.x), "=d"(v.y)
                         : "r"(tile_a + (at ^ gr.vx)));
            double al = 0.0, be = 0.0;
            for (int t = gr.term_begin; t < gr.term_begin + gr.nterms; ++t)
                adj_sign_term(terms[t], (uint32_t)l, al, be);
            lam.x += fma(al, v.x, be * v.y);
            lam.y += fma(al, v.y, -(be * v.x));
        }
        double2 a;
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a.x), "=d"(a.y) : "r"(tile_a + at));
        e += fma(a.x, lam.x, a.y * lam.y);
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(tile_a + (at ^ sel)), "d"(lam.x),
                     "d"(lam.y)
                     : "memory");
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if ((tid & 31) == 0) s_e[tid >> 5] = e;
    __syncthreads();
    if (tid == 0) {
        double sum = 0.0;
        for (int w = 0; w < kAdjSmallThreads / 32; ++w) sum += s_e[w];
        epart[in.epart] = sum;
    }
    adj_rounds<true, kAdjSmallThreads>(tile_a, T, 4, 0ull, pg, in.b_chunk, in.b_nchunks, stage,
                                       s_part, part + in.part, 1, 0);
}

// ---------------------------------------------------------------------------
// Large circuits: one launch per pass over the tiles of all circuits of a wave
// ---------------------------------------------------------------------------
static size_t adj_pass_smem(int T, bool bwd) {
    return ((size_t)(bwd ? 32 : 16) << T) + 1024 + 2 * kStageBytes +
           sizeof(double) * 2 * kRoundSlots * 3 * (kAdjThreads / 32);
}

template <bool BWD>
__global__ void __launch_bounds__(kAdjThreads, 3)
    k_adj_pass(const AdjInst *__restrict__ insts, const AdjPass *__restrict__ passes, int npasses,
               AdjProg pg, double2 *__restrict__ psi, double2 *__restrict__ lam, double *__restrict__ part, int T, int first) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t tile_a = smem_u32(base);
    unsigned char *stage = base + ((size_t)(BWD ? 32 : 16) << T);
    double *s_part = (double *)(stage + 2 * kStageBytes);
    const int tid = threadIdx.x;
    int lo = 0, hi = npasses - 1;  // the pass whose tiles hold this block
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (passes[mid].tile_begin <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const AdjPass ps = passes[lo];
    const int tile = (int)blockIdx.x - ps.tile_begin, h = ps.h;
    const int64_t off = insts[ps.inst].off;
    const uint64_t c2 = (uint64_t)(tile & ((1 << (h - 4)) - 1)), c4 = (uint64_t)(tile >> (h - 4));
    const uint64_t tb = (c2 << 4) | (c4 << (h + T - 4));
    auto global_of = [&](int l) { return tb | (uint64_t)(l & 15) | ((uint64_t)(l >> 4) << h); };
    const int N = 1 << T;
    if (ps.nchunks) adj_stage<kAdjThreads>(smem_u32(stage), pg.chunks[ps.chunk_begin], pg);
    if (!BWD && first) {  // |0...0>
        for (int l = tid; l < N; l += kAdjThreads)
            asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(tile_a + ((uint32_t)swz(l) << 4)),
                         "d"(global_of(l) == 0 ? 1.0 : 0.0), "d"(0.0)
                         : "memory");
    } else {
        for (int l = tid; l < N; l += kAdjThreads) {
            const uint64_t g = global_of(l);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             tile_a + ((uint32_t)swz(l) << 4)),
                         "l"(psi + off + g)
                         : "memory");
            if (BWD)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 tile_a + ((uint32_t)swz(l | N) << 4)),
                             "l"(lam + off + g)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // (adj_rounds waits for every copy and synchronises before its first round)
    adj_rounds<BWD, kAdjThreads>(tile_a, T, h, tb, pg, ps.chunk_begin, ps.nchunks, stage, s_part,
                                 part + ps.part, ps.ntiles, tile);
    if (BWD && first) return;  // the last pass back: nothing reads the states again
    const AdjMap &mp = pg.maps[ps.map];
    const uint32_t sel = (uint32_t)swz(N) << 4;
    // (thread-index bits once, the upper ones by the loop count)
    const uint32_t mb = map_of(mp, map_base(mp, tb), tid, 7);
    static_assert(kAdjThreads == 128, "seven thread-index bits");
    for (int k = 0; k < (N >> 7); ++k) {
        uint32_t at = mb;
        for (int j = 7; j < T; ++j) at ^= mp.vec[j] & (0u - ((uint32_t)(k >> (j - 7)) & 1u));
        const uint64_t g = global_of(tid + (k << 7));
        double2 v;
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                     : "=d"(v.x), "=d"(v.y)
                     : "r"(tile_a + at));
        psi[off + g] = v;
        if (BWD) {
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                         : "=d"(v.x), "=d"(v.y)
                         : "r"(tile_a + (at ^ sel)));
            lam[off + g] = v;
        }
    }
}

// lambda = H psi and the energy's partial sums, one block per kHChunk amplitudes.
// A thread takes the eight amplitudes i0 + 256 k: a term's sign at k is its sign at
// i0 times the parity of k and its bits 8-10, so the parity is taken once per term, a
// group without such bits has one coefficient for all eight, and the terms without X
// fold into one 8-point Walsh-Hadamard transform.  Only groups with an odd number of
// Y somewhere have an imaginary coefficient.  (6.3 M amplitudes of 13-16-qubit
// chains: 371 us, 950 instructions per amplitude, with a sign per term and amplitude.)
__global__ void __launch_bounds__(256, 2)
    k_adj_h(const AdjInst *__restrict__ insts, const int32_t *__restrict__ list, int count,
            const int64_t *__restrict__ chunk_begin, const AdjGroup *__restrict__ groups,
            const AdjTerm *__restrict__ terms, const double2 *__restrict__ psi,
            double2 *__restrict__ lam, double *__restrict__ epart) {
    __shared__ double s_e[8];
    __shared__ __align__(16) unsigned char s_h[kHStage];
    constexpr int kA = kHChunk / 256;
    static_assert(kA == 8, "the fold is over index bits 8 to 10");
    const int64_t blk = blockIdx.x;
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (chunk_begin[mid] <= blk) lo = mid;
        else hi = mid - 1;
    }
    const AdjInst in = insts[list[lo]];
    const int64_t chunk = blk - chunk_begin[lo];
    const double2 *v = psi + in.off;
    const uint32_t i0 = (uint32_t)chunk * kHChunk + threadIdx.x;
    double2 acc[kA], own[kA];
#pragma unroll
    for (int k = 0; k < kA; ++k) {
        acc[k] = make_double2(0.0, 0.0);
        own[k] = v[i0 + 256u * k];
    }
    const AdjGroup *gp = groups + in.group_begin;
    const AdjTerm *tp = terms + in.term_begin;
    const int gb = in.ngroups * (int)sizeof(AdjGroup), tb = in.nterms * (int)sizeof(AdjTerm);
    if (gb + tb <= kHStage) {
        for (int o = (int)threadIdx.x * 8; o < gb; o += 256 * 8)
            *(double *)(s_h + o) = *(const double *)((const char *)gp + o);
        for (int o = (int)threadIdx.x * 8; o < tb; o += 256 * 8)
            *(double *)(s_h + gb + o) = *(const double *)((const char *)tp + o);
        __syncthreads();
        gp = (const AdjGroup *)s_h;
        tp = (const AdjTerm *)(s_h + gb);
    }
    for (int g = 0; g < in.ngroups; ++g) {
        const AdjGroup gr = gp[g];
        const AdjTerm *t0 = tp + (gr.term_begin - in.term_begin);
        if (gr.x == 0) {
            double c[8];
            int t = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                c[q] = 0.0;
                for (; t < gr.nterms && t0[t].p == q; ++t)
                    c[q] += flip_sign(t0[t].ca, (uint32_t)__popc(i0 & t0[t].z));
            }
#pragma unroll
            for (int hs = 1; hs < 8; hs <<= 1)
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    if (q & hs) continue;
                    const double x = c[q], y = c[q | hs];
                    c[q] = x + y;
                    c[q | hs] = x - y;
                }
#pragma unroll
            for (int k = 0; k < kA; ++k) {
                acc[k].x = fma(c[k], own[k].x, acc[k].x);
                acc[k].y = fma(c[k], own[k].y, acc[k].y);
            }
            continue;
        }
        double2 x[kA];
#pragma unroll
        for (int k = 0; k < kA; ++k) x[k] = v[(i0 + 256u * k) ^ gr.x];
        if (gr.flat) {
            double al = 0.0, be = 0.0;
            for (int t = 0; t < gr.nterms; ++t) adj_sign_term(t0[t], i0, al, be);
#pragma unroll
            for (int k = 0; k < kA; ++k) {
                acc[k].x = fma(al, x[k].x, acc[k].x);
                acc[k].y = fma(al, x[k].y, acc[k].y);
            }
            if (gr.odd) {
#pragma unroll
                for (int k = 0; k < kA; ++k) {
                    acc[k].x = fma(be, x[k].y, acc[k].x);
                    acc[k].y = fma(-be, x[k].x, acc[k].y);
                }
            }
            continue;
        }
        for (int t = 0; t < gr.nterms; ++t) {
            const AdjTerm tm = t0[t];
            const uint32_t f = tm.flips ^ (0u - ((uint32_t)__popc(i0 & tm.z) & 1u));
#pragma unroll
            for (int k = 0; k < kA; ++k) {
                const double al = flip_sign(tm.ca, f >> k);
                acc[k].x = fma(al, x[k].x, acc[k].x);
                acc[k].y = fma(al, x[k].y, acc[k].y);
            }
            if (gr.odd) {
#pragma unroll
                for (int k = 0; k < kA; ++k) {
                    const double be = flip_sign(tm.cb, f >> k);
                    acc[k].x = fma(be, x[k].y, acc[k].x);
                    acc[k].y = fma(-be, x[k].x, acc[k].y);
                }
            }
        }
    }
    double e = 0.0;
#pragma unroll
    for (int k = 0; k < kA; ++k) {
        e += fma(own[k].x, acc[k].x, own[k].y * acc[k].y);
        lam[in.off + i0 + 256u * k] = acc[k];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) s_e[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int w = 0; w < 8; ++w) sum += s_e[w];
        epart[in.epart + chunk] = sum;
    }
}

// One warp per run (its sums over the tiles, then its parameters' gradients), then
// one per circuit (its energy); fixed summation order.
__global__ void __launch_bounds__(128)
    k_adj_final(const AdjRun *__restrict__ runs, int nruns, const AdjAtom *__restrict__ atoms,
                const double *__restrict__ wts, const double *__restrict__ part,
                const AdjInst *__restrict__ insts, int ninst, const double *__restrict__ epart,
                const double *__restrict__ shift, double *__restrict__ energy,
                double *__restrict__ grad) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w < nruns) {
        const AdjRun run = runs[w];
        if (run.part < 0) return;
        double s[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double x = 0.0;
            for (int t = lane; t < run.ntiles; t += 32)
                x += part[run.part + (int64_t)c * run.ntiles + t];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            s[c] = x;
        }
        for (int k = run.atom_begin + lane; k < run.atom_end; k += 32) {
            const AdjAtom at = atoms[k];
            if (at.param < 0) continue;
            const double *wt = wts + 3 * (int64_t)k;
            grad[at.param] =
                sin(at.scale * shift[0]) * (wt[0] * s[0] + wt[1] * s[1] + wt[2] * s[2]);
        }
    } else if (w < nruns + ninst) {
        const AdjInst in = insts[w - nruns];
        double x = 0.0;
        for (int t = lane; t < in.neparts; t += 32) x += epart[in.epart + t];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) energy[w - nruns] = x;
    }
}

// ---------------------------------------------------------------------------
// Host: planning
// ---------------------------------------------------------------------------
struct AdjWave {
    std::vector<std::pair<int, int>> f, b;  // per launch: [first, end) of its AdjPass records
    int h_begin = 0, h_count = 0;           // its circuits in the H list
    int64_t h_blocks = 0;
};

class AdjProgram {
public:
    int T = 0;
    int ninst = 0, nsmall = 0, nparams = 0;
    int small_T = kAdjMinN;
    std::vector<AdjInst> insts;      // large circuits after the small ones
    std::vector<int> order;          // insts[k] is the caller's circuit order[k]
    std::vector<AdjRound> rounds;
    std::vector<double> data;        // static part filled in; runs' entries written on the device
    std::vector<AdjMap> maps;
    std::vector<AdjAtom> atoms;
    std::vector<AdjRun> runs;
    std::vector<AdjGroup> groups;
    std::vector<AdjTerm> terms;
    std::vector<AdjPass> passes;
    std::vector<AdjChunk> chunks;
    std::vector<int32_t> h_list;
    std::vector<int64_t> h_chunk;
    std::vector<AdjWave> waves;
    int64_t npart = 0, nepart = 0, amps = 0;

    void *blob = nullptr;
    double2 *states = nullptr;
    size_t blob_bytes = 0;
    AdjInst *d_insts = nullptr;
    AdjRound *d_rounds = nullptr;
    AdjMap *d_maps = nullptr;
    double *d_data = nullptr, *d_wts = nullptr, *d_part = nullptr, *d_epart = nullptr;
    double *d_theta = nullptr, *d_out = nullptr;
    AdjAtom *d_atoms = nullptr;
    AdjRun *d_runs = nullptr;
    AdjGroup *d_groups = nullptr;
    AdjTerm *d_terms = nullptr;
    AdjPass *d_passes = nullptr;
    AdjChunk *d_chunks = nullptr;
    int32_t *d_hlist = nullptr;
    int64_t *d_hchunk = nullptr;
    double2 *psi = nullptr, *lam = nullptr;
    bool own_blob = false;
    // the small circuits run beside the large ones
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;

    ~AdjProgram() {
        if (fork) cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
        if (side) cudaStreamDestroy(side);
        if (own_blob) cudaFree(blob);
        if (states) cudaFree(states);
    }
};

// The inverse of a unitary op that is no run of single-qubit gates.
static GateOp inverse_op(const GateOp &g) {
    GateOp r = g;
    if (g.type == OP_M1 || g.type == OP_M2) {
        const int dim = g.type == OP_M1 ? 2 : 4;
        for (int i = 0; i < dim; ++i)
            for (int j = 0; j < dim; ++j) {
                r.m[2 * (i * dim + j)] = g.m[2 * (j * dim + i)];
                r.m[2 * (i * dim + j) + 1] = -g.m[2 * (j * dim + i) + 1];
            }
    } else if (g.type == OP_DIAG) {
        for (int k = 0; k < 8; ++k) r.m[2 * k + 1] = -g.m[2 * k + 1];
    }
    return r;
}

// The atoms of a single-qubit gate; false when it is none that the sweep takes.
static bool gate_atoms(const lq_gate &g, int param_base, const GateOp &op, AdjProgram &p,
                       std::vector<AdjAtom> &out) {
    auto atom = [&](int kind, int k) {
        AdjAtom a{};
        a.kind = kind;
        a.param = g.param[k] >= 0 ? param_base + g.param[k] : -1;
        a.scale = g.scale[k];
        a.off = g.angle[k];
        out.push_back(a);
        return std::isfinite(a.scale) && std::isfinite(a.off);
    };
    switch (g.kind) {
    case LQ_GATE_RX: return atom(AT_RX, 0);
    case LQ_GATE_RY: return atom(AT_RY, 0);
    case LQ_GATE_RZ:
    case LQ_GATE_PHASE: return atom(AT_RZ, 0);  // equal up to a phase of the state
    case LQ_GATE_U3: return atom(AT_RZ, 2) && atom(AT_RY, 0) && atom(AT_RZ, 1);
    default: break;
    }
    double m[8] = {0};
    if (op.type == OP_M1) {
        memcpy(m, op.m, sizeof(m));
    } else if (op.type == OP_PERM1) {
        m[2] = m[4] = 1.0;
    } else if (op.nfix == 1) {  // Z, S, T
        m[0] = 1.0, m[6] = op.m[0], m[7] = op.m[1];
    } else {
        return false;
    }
    if (!unitary_matrix(m, 2)) return false;
    AdjAtom a{};
    a.kind = AT_CONST;
    a.param = -1;
    a.cmat = (int64_t)p.data.size();
    p.data.insert(p.data.end(), m, m + 8);
    out.push_back(a);
    return true;
}

static int angles_of(int kind) {
    switch (kind) {
    case LQ_GATE_U3: return 3;
    case LQ_GATE_RX: case LQ_GATE_RY: case LQ_GATE_RZ: case LQ_GATE_PHASE:
    case LQ_GATE_CPHASE: case LQ_GATE_CRX: case LQ_GATE_CRY: case LQ_GATE_CRZ:
    case LQ_GATE_CPHASE_PARAM: case LQ_GATE_RXX: case LQ_GATE_RYY: case LQ_GATE_RZZ:
        return 1;
    default: return 0;
    }
}

// A tile's map while its pass is planned (places unswizzled).
struct PlanMap {
    uint32_t vec[kMaxT + 1];
    uint32_t base = 0;
    std::vector<std::pair<int, uint32_t>> cst;  // outside bit, vector
    explicit PlanMap(int T) {
        for (int b = 0; b <= T; ++b) vec[b] = 1u << b;
    }
};

static uint32_t place(uint32_t v) { return (uint32_t)swz((int)v) << 4; }

static bool linear_perm(const GateOp &g) {
    return g.type == OP_SWAP || (g.type == OP_PERM1 && g.nctrl <= 1);
}

// Plan and encode the rounds of one pass (its gates in order) into chunks.  op_run[i]
// is the run of op i (-1: a gate with static coefficients); slot_runs collects the
// pass's gradient runs; map is the layout before and after.
static void adj_encode_pass(const std::vector<int> &gates, const std::vector<GateOp> &gops,
                            const std::vector<int> &op_run, bool bwd, int T, int h, PlanMap &map,
                            AdjProgram &p, std::vector<int> &slot_runs) {
    const int maxr = bwd ? 3 : 4, m = T - 4;
    auto local = [&](int b) { return b < 4 ? b : b >= h && b < h + m ? 4 + (b - h) : -1; };
    AdjChunk ch{(int)p.rounds.size(), 0, (int)p.data.size(), 0};
    auto close_chunk = [&]() {
        ch.nrounds = (int)p.rounds.size() - ch.round_begin;
        ch.ndata = (int)p.data.size() - ch.data_begin;
        if (ch.nrounds) p.chunks.push_back(ch);
        ch = AdjChunk{(int)p.rounds.size(), 0, (int)p.data.size(), 0};
    };
    constexpr int kDiagsPerRound = 8;
    auto emit = [&](int type, std::vector<int> bits, const std::vector<int> &ops) {
        // the largest round: its record and kDiagsPerRound diagonal gates
        constexpr size_t kMost = sizeof(AdjRound) + kDiagsPerRound * sizeof(AdjDiagOp);
        static_assert(kMost <= kStageBytes, "a chunk holds any round");
        if ((p.rounds.size() - ch.round_begin) * sizeof(AdjRound) +
                (p.data.size() - ch.data_begin) * sizeof(double) + kMost > kStageBytes)
            close_chunk();
        AdjRound rd{};
        rd.type = type;
        rd.data = (int)p.data.size();
        // Register bits: the op's, then pads.  Eight consecutive threads should touch
        // eight 16-byte bank groups: pads are taken where the places' low bits (the
        // bank group) stay spanned by the bits left to the threads.
        std::vector<char> used(T, 0);
        for (int b : bits) used[b] = 1;
        auto bank = [&](int b) { return (uint32_t)swz((int)map.vec[b]) & 7u; };
        auto rank_without = [&](int skip) {
            uint32_t basis[3] = {0, 0, 0};
            int r = 0;
            for (int b = 0; b < T; ++b) {
                if (used[b] || b == skip) continue;
                uint32_t v = bank(b);
                for (int k = 2; k >= 0 && v; --k) {
                    if (!(v >> k & 1)) continue;
                    if (!basis[k]) {
                        basis[k] = v;
                        ++r;
                        break;
                    }
                    v ^= basis[k];
                }
            }
            return r;
        };
        while ((int)bits.size() < maxr) {
            int best = -1, best_rank = -1;
            for (int b = T - 1; b >= 0; --b) {
                if (used[b]) continue;
                const int r = rank_without(b);
                if (r > best_rank) best = b, best_rank = r;
            }
            used[best] = 1;
            bits.push_back(best);
        }
        for (int k = 0; k < 4; ++k) {
            const bool sel = k >= maxr;
            rd.reg[k] = place(sel ? 1u << T : map.vec[bits[k]]);
            rd.gpos[k] = sel ? 0ull : 1ull << global_pos(bits[k], h);
        }
        // thread-index bits: three that span the bank groups first
        std::vector<int> lanes, rest;
        uint32_t basis[3] = {0, 0, 0};
        for (int b = 0; b < T; ++b) {
            if (used[b]) continue;
            uint32_t v = bank(b);
            bool indep = false;
            for (int k = 2; k >= 0 && v; --k) {
                if (!(v >> k & 1)) continue;
                if (!basis[k]) {
                    basis[k] = v;
                    indep = true;
                    break;
                }
                v ^= basis[k];
            }
            (indep ? lanes : rest).push_back(b);
        }
        lanes.insert(lanes.end(), rest.begin(), rest.end());
        rd.nlane = (int)lanes.size();
        for (int j = 0; j < rd.nlane; ++j)
            rd.lane[j] = place(map.vec[lanes[j]]) << 4 | (uint32_t)lanes[j];
        rd.base = place(map.base);
        rd.ncst = (int)map.cst.size();
        for (int j = 0; j < rd.ncst; ++j) {
            rd.cst_bit[j] = map.cst[j].first;
            rd.cst_vec[j] = place(map.cst[j].second);
        }
        rd.slots = (int)slot_runs.size() << 8;
        auto put = [&](const void *src, size_t doubles) {
            const size_t o = p.data.size();
            p.data.resize(o + doubles, 0.0);
            if (src) memcpy(p.data.data() + o, src, doubles * sizeof(double));
        };
        for (size_t k = 0; k < ops.size(); ++k) {
            const GateOp &g = gops[ops[k]];
            if (type == RT_RUN) {
                const int run = op_run[ops[k]];
                (bwd ? p.runs[run].coef_b : p.runs[run].coef_f) = (int64_t)p.data.size();
                put(nullptr, 8);
                if (bwd && p.runs[run].ntiles > 0) {
                    rd.slots |= 1 << k;
                    slot_runs.push_back(run);
                }
            } else if (type == RT_DIAG) {
                AdjDiagOp d{};
                for (int q = 0; q < g.nfix; ++q) d.fix |= 1ull << g.fix[q];
                d.npat = g.npat;
                d.pb0 = g.npat > 0 ? g.pat[0] : 0;
                d.pb1 = g.npat > 1 ? g.pat[1] : 0;
                memcpy(d.ph, g.m, sizeof(d.ph));
                put(&d, sizeof(d) / sizeof(double));
            } else if (type == RT_CTRL) {
                AdjCtrlOp c{};
                c.is_x = g.type == OP_PERM1;
                for (int q = 0; q < g.nctrl; ++q) {
                    const int lb = local(g.ctrl[q]);
                    const auto it = std::find(bits.begin(), bits.end(), lb);
                    if (lb >= 0 && it != bits.end()) c.cm |= 1 << (int)(it - bits.begin());
                    else c.gmask |= 1ull << g.ctrl[q];
                }
                memcpy(c.m, g.m, sizeof(c.m));
                put(&c, sizeof(c) / sizeof(double));
            } else {
                put(g.m, 32);
            }
        }
        rd.nrun = type == RT_RUN ? (int)ops.size() : 0;
        rd.ndiag = type == RT_DIAG ? (int)ops.size() : 0;
        p.rounds.push_back(rd);
    };
    std::vector<int> left(gates);
    while (!left.empty()) {
        std::vector<int> next, runs, diags, other;
        std::vector<int> run_bits;
        uint64_t blk = 0;
        // permutations move into the map; the first free ops of each kind are found
        for (int i : left) {
            const GateOp &g = gops[i];
            const uint64_t b = op_bits(g);
            const bool free = (b & blk) == 0;
            if (free && linear_perm(g)) {
                if (g.type == OP_SWAP) {
                    std::swap(map.vec[local(g.b0)], map.vec[local(g.b1)]);
                    continue;
                }
                const uint32_t vt = map.vec[local(g.t)];
                if (g.nctrl == 0) {
                    map.base ^= vt;
                    continue;
                }
                const int lc = local(g.ctrl[0]);
                if (lc >= 0) {
                    map.vec[lc] ^= vt;
                    continue;
                }
                auto it = std::find_if(map.cst.begin(), map.cst.end(),
                                       [&](const auto &c) { return c.first == g.ctrl[0]; });
                if (it != map.cst.end()) {
                    it->second ^= vt;
                    continue;
                }
                if ((int)map.cst.size() < kMaxCst) {
                    map.cst.push_back({g.ctrl[0], vt});
                    continue;
                }
            }
            if (free) {
                if (op_run[i] >= 0) {
                    if ((int)runs.size() < maxr) {
                        runs.push_back(i);
                        run_bits.push_back(local(g.t));
                    }
                } else if (g.type == OP_DIAG) {
                    if ((int)diags.size() < kDiagsPerRound) diags.push_back(i);
                } else {
                    other.push_back(i);
                }
            }
            next.push_back(i);
            blk |= b;
        }
        left = std::move(next);
        auto done = [&](const std::vector<int> &ops) {
            for (int i : ops) left.erase(std::find(left.begin(), left.end(), i));
        };
        if (left.empty()) break;
        // full rounds of runs first; with fewer, diagonal gates may free more of them
        if ((int)runs.size() == maxr || (!runs.empty() && diags.empty())) {
            emit(RT_RUN, run_bits, runs);
            done(runs);
        } else if (!diags.empty()) {
            emit(RT_DIAG, {}, diags);
            done(diags);
        } else {
            const GateOp &g = gops[other[0]];
            if (g.type == OP_M2) emit(RT_M2, {local(g.b0), local(g.b1)}, {other[0]});
            else emit(RT_CTRL, {local(g.t)}, {other[0]});
            done({other[0]});
        }
    }
    close_chunk();
}

static int push_map(AdjProgram &p, const PlanMap &map, int T) {
    AdjMap am{};
    for (int b = 0; b < T; ++b) am.vec[b] = place(map.vec[b]);
    am.base = place(map.base);
    am.ncst = (int)map.cst.size();
    for (int j = 0; j < am.ncst; ++j) {
        am.cst_bit[j] = map.cst[j].first;
        am.cst_vec[j] = place(map.cst[j].second);
    }
    p.maps.push_back(am);
    return (int)p.maps.size() - 1;
}

static bool adj_plan_one(const AdjSpec &sp, int param_base, int T_large, AdjProgram &p,
                         AdjInst &in, std::vector<AdjPass> &fpass, std::vector<AdjPass> &bpass) {
    const int n = std::max(sp.n, kAdjMinN);
    const int T = n <= kAdjSmallMax ? n : std::min(T_large, n);
    in.n = n;
    in.T = T;
    if (n > 32) return false;  // tile and chunk counts are 32-bit
    // runs of single-qubit gates on one bit, and the gates between them
    std::vector<GateOp> gops;
    std::vector<int> op_run;
    std::vector<std::vector<AdjAtom>> run_atoms;
    std::vector<int> open(64, -1);
    std::vector<char> used(std::max(sp.nparams, 1), 0);
    std::vector<double> zeros(std::max(sp.nparams, 1), 0.0);
    for (int k = 0; k < sp.nops; ++k) {
        const lq_gate &g = sp.ops[k];
        bool bound = false;
        for (int a = 0; a < angles_of(g.kind); ++a)
            if (g.param[a] >= 0) {
                if (used[g.param[a]]) return false;
                used[g.param[a]] = 1;
                bound = true;
            } else if (!std::isfinite(g.angle[a])) {
                return false;
            }
        GateOp op;
        if (make_gate_op(&g, zeros.data(), sp.n, &op) != LQ_OK) return false;
        // a unitary gate leaves the norm 1, so its renormalisation changes nothing
        op.renorm = false;
        if (gate_num_qubits(g.kind) == 1) {
            std::vector<AdjAtom> at;
            if (!gate_atoms(g, param_base, op, p, at)) return false;
            const int bit = sp.n - 1 - g.q[0];
            if (open[bit] < 0) {
                GateOp m{};
                m.type = OP_M1;
                m.t = bit;
                open[bit] = (int)run_atoms.size();
                gops.push_back(m);
                op_run.push_back(open[bit]);
                run_atoms.push_back({});
            }
            auto &ra = run_atoms[open[bit]];
            ra.insert(ra.end(), at.begin(), at.end());
            continue;
        }
        if (bound) return false;
        if (op.type == OP_M1 && !unitary_matrix(op.m, 2)) return false;
        if (op.type == OP_M2 && !unitary_matrix(op.m, 4)) return false;
        const uint64_t bits = op_bits(op);
        for (int b = 0; b < 64; ++b)
            if ((bits >> b) & 1) open[b] = -1;
        gops.push_back(op);
        op_run.push_back(-1);
    }
    const int run0 = (int)p.runs.size();
    for (auto &ra : run_atoms) {
        AdjRun r{};
        r.atom_begin = (int32_t)p.atoms.size();
        bool any = false;
        for (auto &a : ra) any = any || a.param >= 0;
        p.atoms.insert(p.atoms.end(), ra.begin(), ra.end());
        r.atom_end = (int32_t)p.atoms.size();
        r.part = -1;
        r.ntiles = any ? 1 << (n - T) : 0;
        p.runs.push_back(r);
    }
    for (int &r : op_run)
        if (r >= 0) r += run0;
    std::vector<GateOp> back;
    std::vector<int> back_run;
    for (size_t k = gops.size(); k-- > 0;) {
        back.push_back(op_run[k] >= 0 ? gops[k] : inverse_op(gops[k]));
        back_run.push_back(op_run[k]);
    }
    // (a small circuit's sweep back starts from the layout its way forward ended in)
    PlanMap small_map(T);
    for (int dir = 0; dir < 2; ++dir) {
        const auto &go = dir ? back : gops;
        const auto &gr = dir ? back_run : op_run;
        for (const PlanStep &st : plan_windows(go, n, T)) {
            if (!st.fused) return false;
            AdjPass ap{};
            ap.h = st.pass.h;
            ap.chunk_begin = (int)p.chunks.size();
            ap.ntiles = 1 << (n - T);
            ap.part = p.npart;
            std::vector<int> slots;
            PlanMap own(T);
            PlanMap &map = n == T ? small_map : own;
            adj_encode_pass(st.pass.gates, go, gr, dir == 1, T, st.pass.h, map, p, slots);
            if (n != T) ap.map = push_map(p, map, T);
            ap.nchunks = (int)p.chunks.size() - ap.chunk_begin;
            for (int r : slots) {
                p.runs[r].part = p.npart;
                p.npart += 3ll * ap.ntiles;
            }
            (dir ? bpass : fpass).push_back(ap);
        }
        if (dir == 0 && n == T) in.map = push_map(p, small_map, T);
    }
    // the Pauli sum, by X mask in order of first appearance
    std::vector<char> taken(sp.nterms, 0);
    in.group_begin = (int)p.groups.size();
    in.term_begin = (int)p.terms.size();
    for (int t = 0; t < sp.nterms; ++t) {
        if (taken[t]) continue;
        AdjGroup gr{(uint32_t)sp.terms[t].xmask, (int)p.terms.size(), 0, 0, 0, 1};
        if (n == T)
            for (int b = 0; b < n; ++b)
                if (gr.x >> b & 1) gr.vx ^= p.maps[in.map].vec[b];
        for (int u = t; u < sp.nterms; ++u) {
            const lq_pauli_term &pt = sp.terms[u];
            if (taken[u] || pt.xmask != sp.terms[t].xmask) continue;
            if (!std::isfinite(pt.coefficient)) return false;
            taken[u] = 1;
            int k = pt.ny & 3;
            if (sp.yconv == LQ_Y_TEXTBOOK) k = (4 - k) & 3;
            const double a = k == 0 ? 1.0 : k == 2 ? -1.0 : 0.0;
            const double b = k == 1 ? -1.0 : k == 3 ? 1.0 : 0.0;
            AdjTerm tm{pt.coefficient * a, pt.coefficient * b, (uint32_t)pt.zmask, 0, 0, 0};
            tm.p = (uint8_t)((pt.zmask >> 8) & 7);
            for (int q = 0; q < 8; ++q)
                tm.flips |= (uint8_t)((__builtin_popcount(q & tm.p) & 1) << q);
            if (k & 1) gr.odd = 1;
            if (tm.p) gr.flat = 0;
            p.terms.push_back(tm);
            ++gr.nterms;
        }
        if (gr.x == 0)
            std::stable_sort(p.terms.begin() + gr.term_begin, p.terms.end(),
                             [](const AdjTerm &u, const AdjTerm &v) { return u.p < v.p; });
        p.groups.push_back(gr);
    }
    in.nterms = (int)p.terms.size() - in.term_begin;
    in.ngroups = (int)p.groups.size() - in.group_begin;
    return p.data.size() < (size_t)1 << 30;
}

std::shared_ptr<AdjProgram> adj_plan(const std::vector<AdjSpec> &specs, int tile_bits,
                                     size_t budget_bytes) {
    auto pp = std::make_shared<AdjProgram>();
    AdjProgram &p = *pp;
    p.T = tile_bits;
    p.ninst = (int)specs.size();
    std::vector<int> base(specs.size());
    for (size_t i = 0; i < specs.size(); ++i) {
        base[i] = p.nparams;
        p.nparams += specs[i].nparams;
    }
    // small circuits first, the largest of them first (their CTAs start in order)
    for (int i = 0; i < p.ninst; ++i) p.order.push_back(i);
    std::stable_sort(p.order.begin(), p.order.end(), [&](int x, int y) {
        const bool sx = specs[x].n <= kAdjSmallMax, sy = specs[y].n <= kAdjSmallMax;
        if (sx != sy) return sx;
        return specs[x].n > specs[y].n;
    });
    std::vector<std::vector<AdjPass>> fp(p.ninst), bp(p.ninst);
    for (int k = 0; k < p.ninst; ++k) {
        const AdjSpec &sp = specs[p.order[k]];
        AdjInst in{};
        in.part = p.npart;
        if (!adj_plan_one(sp, base[p.order[k]], tile_bits, p, in, fp[k], bp[k])) return nullptr;
        if (in.n <= kAdjSmallMax) {
            // one tile: all passes run in one go
            ++p.nsmall;
            p.small_T = std::max(p.small_T, in.n);
            if (fp[k].size() > 1 || bp[k].size() > 1) return nullptr;
            if (!fp[k].empty()) in.f_chunk = fp[k][0].chunk_begin, in.f_nchunks = fp[k][0].nchunks;
            if (!bp[k].empty()) in.b_chunk = bp[k][0].chunk_begin, in.b_nchunks = bp[k][0].nchunks;
            in.neparts = 1;
        } else {
            if (fp[k].empty()) return nullptr;  // no gate at all
            in.neparts = (int32_t)((1ll << in.n) / kHChunk);
        }
        in.epart = p.nepart;
        p.nepart += in.neparts;
        p.insts.push_back(in);
    }
    // waves of large circuits within the memory budget
    for (int k = p.nsmall; k < p.ninst;) {
        AdjWave w;
        int64_t amps = 0;
        int end = k;
        while (end < p.ninst) {
            const int64_t a = 1ll << p.insts[end].n;
            if (end > k && (size_t)(amps + a) * 2 * sizeof(double2) > budget_bytes) break;
            p.insts[end].off = amps;
            amps += a;
            ++end;
        }
        p.amps = std::max(p.amps, amps);
        for (int dir = 0; dir < 2; ++dir) {
            auto &src = dir ? bp : fp;
            size_t most = 0;
            for (int i = k; i < end; ++i) most = std::max(most, src[i].size());
            // back: line the passes up at the end, so that the last launch is every
            // circuit's last pass
            for (size_t l = 0; l < most; ++l) {
                const int first = (int)p.passes.size();
                int tiles = 0;
                for (int i = k; i < end; ++i) {
                    const size_t skip = dir ? most - src[i].size() : 0;
                    if (l < skip || l - skip >= src[i].size()) continue;
                    AdjPass ap = src[i][l - skip];
                    ap.inst = i;
                    ap.tile_begin = tiles;
                    tiles += ap.ntiles;
                    p.passes.push_back(ap);
                }
                (dir ? w.b : w.f).push_back({first, (int)p.passes.size()});
            }
        }
        w.h_begin = (int)p.h_list.size();
        w.h_count = end - k;
        for (int i = k; i < end; ++i) {
            p.h_list.push_back(i);
            p.h_chunk.push_back(w.h_blocks);
            w.h_blocks += p.insts[i].neparts;
        }
        p.waves.push_back(std::move(w));
        k = end;
    }
    return pp;
}

int adj_upload(AdjProgram &p, lq_state *work, cudaStream_t st) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (std::max<size_t>(bytes, 8) + 255) / 256 * 256;
        return o;
    };
    const size_t o_insts = take(p.insts.size() * sizeof(AdjInst));
    const size_t o_rounds = take(p.rounds.size() * sizeof(AdjRound));
    const size_t o_maps = take(p.maps.size() * sizeof(AdjMap));
    const size_t o_atoms = take(p.atoms.size() * sizeof(AdjAtom));
    const size_t o_runs = take(p.runs.size() * sizeof(AdjRun));
    const size_t o_groups = take(p.groups.size() * sizeof(AdjGroup));
    const size_t o_terms = take(p.terms.size() * sizeof(AdjTerm));
    const size_t o_passes = take(p.passes.size() * sizeof(AdjPass));
    const size_t o_chunks = take(p.chunks.size() * sizeof(AdjChunk));
    const size_t o_hlist = take(p.h_list.size() * sizeof(int32_t));
    const size_t o_hchunk = take(p.h_chunk.size() * sizeof(int64_t));
    const size_t o_data = take(p.data.size() * sizeof(double));
    const size_t upload = off;
    const size_t o_wts = take(p.atoms.size() * 3 * sizeof(double));
    const size_t o_part = take((size_t)p.npart * sizeof(double));
    const size_t o_epart = take((size_t)p.nepart * sizeof(double));
    const size_t o_theta = take(((size_t)p.nparams + 1) * sizeof(double));
    const size_t o_out = take(((size_t)p.ninst + p.nparams) * sizeof(double));
    // A plain call works in its handle's own program buffer and amplitudes.  (The partial sums
    // of a large state, 24 bytes per tile and run of gates, would stay there for the handle's
    // life, 0.3 GB after a gradient of 28 qubits and 84 runs: they are given back.)
    constexpr size_t kHandleProgram = 32ull << 20;
    cudaError_t e = cudaSuccess;
    const size_t copies = work ? 1 : 2;
    const size_t states = (size_t)p.amps * copies * sizeof(double2);
    if (states > alloc_room())
        return set_error(LQ_ERR_OOM, "%zu bytes of states exceed the allocation limit", states);
    if (states > 0) e = device_malloc(&p.states, states);
    if (e == cudaSuccess) {
        if (work && off <= kHandleProgram) {
            LQ_TRY(ensure_prog(work, off));
            p.blob = work->d_prog;
        } else {
            e = device_malloc(&p.blob, off);
            p.own_blob = e == cudaSuccess;
        }
    }
    if (e != cudaSuccess) {
        if (p.states) cudaFree(p.states);
        p.states = nullptr;
        cudaGetLastError();
        return set_error(e == cudaErrorMemoryAllocation ? LQ_ERR_OOM : LQ_ERR_CUDA, "%s",
                         cudaGetErrorString(e));
    }
    p.psi = work ? (double2 *)work->d : p.states;
    p.lam = work ? p.states : p.states + p.amps;
    std::vector<char> h(upload, 0);
    auto put = [&](size_t o, const auto &v) {
        if (!v.empty()) memcpy(h.data() + o, v.data(), v.size() * sizeof(v[0]));
    };
    put(o_insts, p.insts);
    put(o_rounds, p.rounds);
    put(o_maps, p.maps);
    put(o_atoms, p.atoms);
    put(o_runs, p.runs);
    put(o_groups, p.groups);
    put(o_terms, p.terms);
    put(o_passes, p.passes);
    put(o_chunks, p.chunks);
    put(o_hlist, p.h_list);
    put(o_hchunk, p.h_chunk);
    put(o_data, p.data);
    char *b = (char *)p.blob;
    p.d_insts = (AdjInst *)(b + o_insts);
    p.d_rounds = (AdjRound *)(b + o_rounds);
    p.d_maps = (AdjMap *)(b + o_maps);
    p.d_atoms = (AdjAtom *)(b + o_atoms);
    p.d_runs = (AdjRun *)(b + o_runs);
    p.d_groups = (AdjGroup *)(b + o_groups);
    p.d_terms = (AdjTerm *)(b + o_terms);
    p.d_passes = (AdjPass *)(b + o_passes);
    p.d_chunks = (AdjChunk *)(b + o_chunks);
    p.d_hlist = (int32_t *)(b + o_hlist);
    p.d_hchunk = (int64_t *)(b + o_hchunk);
    p.d_data = (double *)(b + o_data);
    p.d_wts = (double *)(b + o_wts);
    p.d_part = (double *)(b + o_part);
    p.d_epart = (double *)(b + o_epart);
    p.d_theta = (double *)(b + o_theta);
    p.d_out = (double *)(b + o_out);
    if (p.nsmall && p.nsmall < p.ninst) {
        LQ_CUDA_TRY(cudaStreamCreateWithFlags(&p.side, cudaStreamNonBlocking));
        LQ_CUDA_TRY(cudaEventCreateWithFlags(&p.fork, cudaEventDisableTiming));
        LQ_CUDA_TRY(cudaEventCreateWithFlags(&p.join, cudaEventDisableTiming));
    }
    LQ_CUDA_TRY(cudaMemcpyAsync(p.blob, h.data(), upload, cudaMemcpyHostToDevice, st));
    LQ_CUDA_TRY(cudaFuncSetAttribute(k_adj_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)adj_small_smem(kAdjSmallMax)));
    LQ_CUDA_TRY(cudaFuncSetAttribute(k_adj_pass<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)adj_pass_smem(kMaxT, false)));
    LQ_CUDA_TRY(cudaFuncSetAttribute(k_adj_pass<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)adj_pass_smem(kMaxT, true)));
    return LQ_OK;
}

const std::vector<int> &adj_order(const AdjProgram &p) { return p.order; }

int adj_enqueue(AdjProgram &p, cudaStream_t st, const double *theta_and_shift, double *out) {
    LQ_CUDA_TRY(cudaMemcpyAsync(p.d_theta, theta_and_shift, sizeof(double) * (p.nparams + 1),
                                cudaMemcpyHostToDevice, st));
    double *energy = p.d_out, *grad = p.d_out + p.ninst;
    // a parameter that no gate uses has gradient 0
    if (p.nparams) LQ_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(double) * p.nparams, st));
    const int nruns = (int)p.runs.size();
    const AdjProg pg{p.d_rounds, p.d_data, p.d_chunks, p.d_maps};
    if (nruns)
        k_adj_coef<<<(nruns + 127) / 128, 128, 0, st>>>(p.d_runs, nruns, p.d_atoms, p.d_theta,
                                                       p.d_data, p.d_wts);
    if (p.nsmall) {
        cudaStream_t sm = st;
        if (p.side) {
            sm = p.side;
            LQ_CUDA_TRY(cudaEventRecord(p.fork, st));
            LQ_CUDA_TRY(cudaStreamWaitEvent(sm, p.fork, 0));
        }
        k_adj_small<<<p.nsmall, kAdjSmallThreads, adj_small_smem(p.small_T), sm>>>(
            p.d_insts, pg, p.d_groups, p.d_terms, p.d_part, p.d_epart);
        if (p.side) LQ_CUDA_TRY(cudaEventRecord(p.join, sm));
    }
    double2 *psi = p.psi, *lam = p.lam;
    for (const AdjWave &w : p.waves) {
        for (size_t l = 0; l < w.f.size(); ++l) {
            const auto [a, b] = w.f[l];
            const AdjPass &last = p.passes[b - 1];
            k_adj_pass<false><<<last.tile_begin + last.ntiles, kAdjThreads,
                                adj_pass_smem(p.T, false), st>>>(
                p.d_insts, p.d_passes + a, b - a, pg, psi, lam, p.d_part, p.T, l == 0);
        }
        k_adj_h<<<(unsigned)w.h_blocks, 256, 0, st>>>(p.d_insts, p.d_hlist + w.h_begin, w.h_count,
                                                     p.d_hchunk + w.h_begin, p.d_groups, p.d_terms,
                                                     psi, lam, p.d_epart);
        for (size_t l = 0; l < w.b.size(); ++l) {
            const auto [a, b] = w.b[l];
            const AdjPass &last = p.passes[b - 1];
            k_adj_pass<true><<<last.tile_begin + last.ntiles, kAdjThreads, adj_pass_smem(p.T, true),
                               st>>>(p.d_insts, p.d_passes + a, b - a, pg, psi, lam, p.d_part, p.T,
                                     l + 1 == w.b.size());
        }
    }
    if (p.nsmall && p.side) LQ_CUDA_TRY(cudaStreamWaitEvent(st, p.join, 0));
    const int warps = nruns + p.ninst;
    k_adj_final<<<(warps + 3) / 4, 128, 0, st>>>(p.d_runs, nruns, p.d_atoms, p.d_wts, p.d_part,
                                                p.d_insts, p.ninst, p.d_epart,
                                                p.d_theta + p.nparams, energy, grad);
    LQ_CUDA_TRY(cudaGetLastError());
    LQ_CUDA_TRY(cudaMemcpyAsync(out, p.d_out, sizeof(double) * (p.ninst + p.nparams),
                                cudaMemcpyDeviceToHost, st));
    return LQ_OK;
}

}  // namespace lq
