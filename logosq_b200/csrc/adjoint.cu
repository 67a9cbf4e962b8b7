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
// holds 2^T amplitudes of each, and a register round picks three tile bits plus
// the selector (tile position T), so the ping-pong routines of fused_round.cuh
// apply a gate to both halves and a thread holds the matching amplitudes of both
// for the inner products.  All rotations of a run on one qubit share one 2x2 and one
// set of sums (S_x, S_y, S_z) = Im <lambda| (X, Y, Z) |psi> taken just before the
// run is undone; a parameter's derivative is the combination of the three with its
// axis turned by the run's later gates, computed with the 2x2s on the device.
//
// States of up to 2^12 amplitudes: one CTA does everything in shared memory
// (k_adj_small).  Larger ones: one launch per pass over the tiles of all circuits
// (k_adj_pass), three 128-thread CTAs per SM.
#include "adjoint.h"

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>

namespace lq {

constexpr int kAdjSmallMax = 12;   // largest state kept in one CTA's shared memory
constexpr int kAdjMinN = 5;        // smaller circuits are planned as 5 qubits (upper bits 0)
constexpr int kAdjSmallThreads = 256;
constexpr int kAdjThreads = 128;
constexpr int kRoundSlots = 8;     // gradient runs of one round
constexpr int kHChunk = 1024;      // amplitudes of one block of k_adj_h

enum AdjCode { AC_M1 = 0, AC_M1C = 4, AC_X = 8, AC_XC = 12, AC_DIAG = 16, AC_SWAP = 17,
               AC_M2 = 23, AC_GM1 = 64 };

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

struct AdjInst {
    int32_t n, T;
    int32_t f_round, f_nrounds;  // small circuits: rounds forward and back
    int32_t b_round, b_nrounds;
    int32_t group_begin, ngroups;
    int64_t off;                 // first amplitude in the wave's buffers (large circuits)
    int64_t epart;               // energy partials
    int32_t neparts, pad;
    int64_t part;                // small circuits: partial sums
};

struct AdjPass {
    int32_t inst, h;
    int32_t round_begin, nrounds;
    int32_t tile_begin, ntiles;  // its blocks in the launch
    int64_t part;                // partial sums of its gradient runs
};

struct AdjGroup {  // Pauli terms sharing an X mask
    uint64_t x;
    int32_t term_begin, nterms;
};

struct AdjTerm {  // matrix element (-1)^popcount(i & z) (ca - i cb) between i and i ^ x
    uint64_t z;
    double ca, cb;
};

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
        sz += fma(p.x, a.y, -(p.y * a.x)) - fma(q.x, b.y, -(q.y * b.x));
        sx += fma(p.x, b.y, -(p.y * b.x)) + fma(q.x, a.y, -(q.y * a.x));
        sy += fma(q.x, a.x, q.y * a.y) - fma(p.x, b.x, p.y * b.y);
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

template <bool BWD, int NWARPS>
__device__ __forceinline__ void adj_apply(const double2 (&s)[16], double2 (&d)[16],
                                          const PassOp &op, const double *__restrict__ c,
                                          uint64_t gbase, const uint64_t *__restrict__ gp,
                                          const GradOut &go) {
    int code = (gbase & op.gmask) == op.gmask ? op.code : -1;
    if (BWD && code >= AC_GM1) {
        code -= AC_GM1;
        double sx, sy, sz;
        if (code == 0) grad3<0>(s, sx, sy, sz);
        else if (code == 1) grad3<1>(s, sx, sy, sz);
        else grad3<2>(s, sx, sy, sz);
        grad_emit(go, NWARPS, op.bits, sx, sy, sz);
    }
    switch (code) {
    case AC_M1 + 0: pp_m1<0>(s, d, c, 0); break;
    case AC_M1 + 1: pp_m1<1>(s, d, c, 0); break;
    case AC_M1 + 2: pp_m1<2>(s, d, c, 0); break;
    case AC_M1 + 3: if constexpr (!BWD) pp_m1<3>(s, d, c, 0); break;
    case AC_M1C + 0: pp_m1<0>(s, d, c, op.cm); break;
    case AC_M1C + 1: pp_m1<1>(s, d, c, op.cm); break;
    case AC_M1C + 2: pp_m1<2>(s, d, c, op.cm); break;
    case AC_M1C + 3: if constexpr (!BWD) pp_m1<3>(s, d, c, op.cm); break;
    case AC_X + 0: pp_x<0>(s, d, 0); break;
    case AC_X + 1: pp_x<1>(s, d, 0); break;
    case AC_X + 2: pp_x<2>(s, d, 0); break;
    case AC_X + 3: if constexpr (!BWD) pp_x<3>(s, d, 0); break;
    case AC_XC + 0: pp_x<0>(s, d, op.cm); break;
    case AC_XC + 1: pp_x<1>(s, d, op.cm); break;
    case AC_XC + 2: pp_x<2>(s, d, op.cm); break;
    case AC_XC + 3: if constexpr (!BWD) pp_x<3>(s, d, op.cm); break;
    case AC_DIAG: pp_diag(s, d, op, c, gbase, gp); break;
    case AC_SWAP + 0: pp_swap<0, 1>(s, d); break;
    case AC_SWAP + 1: pp_swap<0, 2>(s, d); break;
    case AC_SWAP + 2: if constexpr (!BWD) pp_swap<0, 3>(s, d); break;
    case AC_SWAP + 3: pp_swap<1, 2>(s, d); break;
    case AC_SWAP + 4: if constexpr (!BWD) pp_swap<1, 3>(s, d); break;
    case AC_SWAP + 5: if constexpr (!BWD) pp_swap<2, 3>(s, d); break;
    case AC_M2 + 0: pp_m2<0, 1, false>(s, d, c); break;
    case AC_M2 + 1: pp_m2<0, 2, false>(s, d, c); break;
    case AC_M2 + 2: if constexpr (!BWD) pp_m2<0, 3, false>(s, d, c); break;
    case AC_M2 + 3: pp_m2<1, 2, false>(s, d, c); break;
    case AC_M2 + 4: if constexpr (!BWD) pp_m2<1, 3, false>(s, d, c); break;
    case AC_M2 + 5: if constexpr (!BWD) pp_m2<2, 3, false>(s, d, c); break;
    default:
#pragma unroll
        for (int e = 0; e < 16; ++e) d[e] = s[e];
        break;
    }
}

// One round for register set `v` (of 2^(T-4) forward, 2^(T-3) back) of the tile.
template <bool BWD, int NWARPS>
__device__ __forceinline__ void adj_round(uint32_t tile_a, const FusedRound &rd,
                                          const PassOp *__restrict__ ops,
                                          const double *__restrict__ coef, uint64_t tile_base,
                                          int h, int v, const GradOut &go) {
    int tbase = 0;
    for (int j = 0; j < rd.nlane; ++j) tbase |= ((v >> j) & 1) << rd.lane[j];
    const uint32_t sb = (uint32_t)swz(tbase) << 4;
    const uint64_t gbase = tile_base | (uint64_t)(tbase & 15) | ((uint64_t)(tbase >> 4) << h);
    const uint32_t E0 = (uint32_t)rd.eoff[1], E1 = (uint32_t)rd.eoff[2];
    const uint32_t E2 = (uint32_t)rd.eoff[4], E3 = (uint32_t)rd.eoff[8];
    auto addr_of = [&](int e) {
        const uint32_t x = ((e & 1) ? E0 : 0u) ^ ((e & 2) ? E1 : 0u) ^ ((e & 4) ? E2 : 0u) ^
                           ((e & 8) ? E3 : 0u);
        return tile_a + (sb ^ x);
    };
    double2 a[16], b[16];
#pragma unroll
    for (int e = 0; e < 16; ++e)
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                     : "=d"(a[e].x), "=d"(a[e].y)
                     : "r"(addr_of(e)));
    const int o1 = rd.op_end;
    int o = rd.op_begin;
    for (; o + 1 < o1; o += 2) {
        const PassOp p0 = ops[o];
        const PassOp p1 = ops[o + 1];
        adj_apply<BWD, NWARPS>(a, b, p0, coef + p0.coef, gbase, rd.gpos, go);
        adj_apply<BWD, NWARPS>(b, a, p1, coef + p1.coef, gbase, rd.gpos, go);
    }
    const bool odd = o < o1;
    if (odd) {
        const PassOp p0 = ops[o];
        adj_apply<BWD, NWARPS>(a, b, p0, coef + p0.coef, gbase, rd.gpos, go);
    }
    if (odd) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr_of(e)), "d"(b[e].x),
                         "d"(b[e].y)
                         : "memory");
    } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr_of(e)), "d"(a[e].x),
                         "d"(a[e].y)
                         : "memory");
    }
}

// All rounds of one pass on the tile, with the gradient runs' sums over the tile
// written to part[(slot * 3 + c) * ntiles + tile].  FusedRound::pad holds the
// round's first slot << 8 | its slot count.
template <bool BWD, int NT>
__device__ __forceinline__ void adj_rounds(uint32_t tile_a, int T, int h, uint64_t tile_base,
                                           const FusedRound *__restrict__ rounds, int nrounds,
                                           const PassOp *__restrict__ ops,
                                           const double *__restrict__ coef, double *s_part,
                                           double *__restrict__ part, int ntiles, int tile) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x;
    const int nthr = 1 << (T - (BWD ? 3 : 4));
    GradOut go;
    go.mask = nthr >= 32 ? 0xffffffffu : (1u << nthr) - 1u;
    go.half = nthr >= 32 ? 16 : nthr >> 1;
    const int nw = nthr >= NT ? NW : nthr >= 32 ? nthr >> 5 : 1;  // warps that hold amplitudes
    for (int r = 0; r < nrounds; ++r) {
        const FusedRound &rd = rounds[r];
        go.part = s_part + (r & 1) * (kRoundSlots * 3 * NW);
        for (int v = tid; v < nthr; v += NT) {
            go.add = v != tid;
            adj_round<BWD, NW>(tile_a, rd, ops, coef, tile_base, h, v, go);
        }
        __syncthreads();
        if (BWD) {
            // (this half of s_part is written again two rounds on, after the next barrier)
            const int cnt = (rd.pad & 0xff) * 3, first = (rd.pad >> 8) * 3;
            for (int k = tid; k < cnt; k += NT) {
                double sum = 0.0;
                for (int w = 0; w < nw; ++w) sum += go.part[k * NW + w];
                part[(int64_t)(first + k) * ntiles + tile] = sum;
            }
        }
    }
}

__device__ __forceinline__ void adj_sign_term(const AdjTerm &t, uint64_t i, double &al,
                                              double &be) {
    const bool neg = __popcll(i & t.z) & 1;
    al += neg ? -t.ca : t.ca;
    be += neg ? -t.cb : t.cb;
}

// ---------------------------------------------------------------------------
// Small circuits: everything in one CTA
// ---------------------------------------------------------------------------
constexpr size_t adj_small_smem(int T) {
    return ((size_t)32 << T) + 1024 + sizeof(double) * 2 * kRoundSlots * 3 * (kAdjSmallThreads / 32);
}

__global__ void __launch_bounds__(kAdjSmallThreads, 1)
    k_adj_small(const AdjInst *__restrict__ insts, const FusedRound *__restrict__ rounds,
                const PassOp *__restrict__ ops, const double *__restrict__ coef,
                const AdjGroup *__restrict__ groups, const AdjTerm *__restrict__ terms,
                double *__restrict__ part, double *__restrict__ epart) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t tile_a = smem_u32(base);
    const AdjInst in = insts[blockIdx.x];
    const int T = in.n, tid = threadIdx.x, N = 1 << T;
    double *s_part = (double *)(base + ((size_t)32 << T));
    __shared__ double s_e[kAdjSmallThreads / 32];
    auto addr = [&](int l) { return tile_a + ((uint32_t)swz(l) << 4); };
    for (int l = tid; l < N; l += kAdjSmallThreads)
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr(l)), "d"(l == 0 ? 1.0 : 0.0),
                     "d"(0.0)
                     : "memory");
    __syncthreads();
    adj_rounds<false, kAdjSmallThreads>(tile_a, T, 4, 0ull, rounds + in.f_round, in.f_nrounds, ops,
                                        coef, s_part, nullptr, 1, 0);
    // lambda = H psi, and the energy
    double e = 0.0;
    for (int l = tid; l < N; l += kAdjSmallThreads) {
        double2 lam = make_double2(0.0, 0.0);
        for (int g = in.group_begin; g < in.group_begin + in.ngroups; ++g) {
            const AdjGroup gr = groups[g];
            double2 v;
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                         : "=d"(v.x), "=d"(v.y)
                         : "r"(addr(l ^ (int)gr.x)));
            double al = 0.0, be = 0.0;
            for (int t = gr.term_begin; t < gr.term_begin + gr.nterms; ++t)
                adj_sign_term(terms[t], (uint64_t)l, al, be);
            lam.x += fma(al, v.x, be * v.y);
            lam.y += fma(al, v.y, -(be * v.x));
        }
        double2 a;
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a.x), "=d"(a.y) : "r"(addr(l)));
        e += fma(a.x, lam.x, a.y * lam.y);
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr(l | N)), "d"(lam.x), "d"(lam.y)
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
    adj_rounds<true, kAdjSmallThreads>(tile_a, T, 4, 0ull, rounds + in.b_round, in.b_nrounds, ops,
                                       coef, s_part, part + in.part, 1, 0);
}

// ---------------------------------------------------------------------------
// Large circuits: one launch per pass over the tiles of all circuits of a wave
// ---------------------------------------------------------------------------
static size_t adj_pass_smem(int T, bool bwd) {
    return ((size_t)(bwd ? 32 : 16) << T) + 1024 +
           sizeof(double) * 2 * kRoundSlots * 3 * (kAdjThreads / 32);
}

template <bool BWD>
__global__ void __launch_bounds__(kAdjThreads, 3)
    k_adj_pass(const AdjInst *__restrict__ insts, const AdjPass *__restrict__ passes, int npasses,
               const FusedRound *__restrict__ rounds, const PassOp *__restrict__ ops,
               const double *__restrict__ coef, double2 *__restrict__ psi,
               double2 *__restrict__ lam, double *__restrict__ part, int T, int first) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t tile_a = smem_u32(base);
    double *s_part = (double *)(base + ((size_t)(BWD ? 32 : 16) << T));
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
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    adj_rounds<BWD, kAdjThreads>(tile_a, T, h, tb, rounds + ps.round_begin, ps.nrounds, ops, coef,
                                 s_part, part + ps.part, ps.ntiles, tile);
    if (BWD && first) return;  // the last pass back: nothing reads the states again
    for (int l = tid; l < N; l += kAdjThreads) {
        const uint64_t g = global_of(l);
        double2 v;
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                     : "=d"(v.x), "=d"(v.y)
                     : "r"(tile_a + ((uint32_t)swz(l) << 4)));
        psi[off + g] = v;
        if (BWD) {
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
                         : "=d"(v.x), "=d"(v.y)
                         : "r"(tile_a + ((uint32_t)swz(l | N) << 4)));
            lam[off + g] = v;
        }
    }
}

// lambda = H psi and the energy's partial sums, one block per kHChunk amplitudes.
__global__ void __launch_bounds__(256)
    k_adj_h(const AdjInst *__restrict__ insts, const int32_t *__restrict__ list, int count,
            const int64_t *__restrict__ chunk_begin, const AdjGroup *__restrict__ groups,
            const AdjTerm *__restrict__ terms, const double2 *__restrict__ psi,
            double2 *__restrict__ lam, double *__restrict__ epart) {
    __shared__ double s_e[8];
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
    constexpr int kA = kHChunk / 256;
    const uint64_t i0 = (uint64_t)chunk * kHChunk + threadIdx.x;
    double2 acc[kA];
#pragma unroll
    for (int k = 0; k < kA; ++k) acc[k] = make_double2(0.0, 0.0);
    for (int g = in.group_begin; g < in.group_begin + in.ngroups; ++g) {
        const AdjGroup gr = groups[g];
        double2 x[kA];
        double al[kA], be[kA];
#pragma unroll
        for (int k = 0; k < kA; ++k) {
            x[k] = v[(i0 + 256u * k) ^ gr.x];
            al[k] = be[k] = 0.0;
        }
        for (int t = gr.term_begin; t < gr.term_begin + gr.nterms; ++t) {
            const AdjTerm tm = terms[t];
#pragma unroll
            for (int k = 0; k < kA; ++k) adj_sign_term(tm, i0 + 256u * k, al[k], be[k]);
        }
#pragma unroll
        for (int k = 0; k < kA; ++k) {
            acc[k].x += fma(al[k], x[k].x, be[k] * x[k].y);
            acc[k].y += fma(al[k], x[k].y, -(be[k] * x[k].x));
        }
    }
    double e = 0.0;
#pragma unroll
    for (int k = 0; k < kA; ++k) {
        const double2 a = v[i0 + 256u * k];
        e += fma(a.x, acc[k].x, a.y * acc[k].y);
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
    std::vector<FusedRound> rounds;
    std::vector<PassOp> ops;
    std::vector<double> coef;        // static part filled in; runs' entries written on the device
    std::vector<AdjAtom> atoms;
    std::vector<AdjRun> runs;
    std::vector<AdjGroup> groups;
    std::vector<AdjTerm> terms;
    std::vector<AdjPass> passes;
    std::vector<int32_t> h_list;
    std::vector<int64_t> h_chunk;
    std::vector<AdjWave> waves;
    int64_t npart = 0, nepart = 0, amps = 0;

    void *blob = nullptr;
    double2 *states = nullptr;
    size_t blob_bytes = 0;
    AdjInst *d_insts = nullptr;
    FusedRound *d_rounds = nullptr;
    PassOp *d_ops = nullptr;
    double *d_coef = nullptr, *d_wts = nullptr, *d_part = nullptr, *d_epart = nullptr;
    double *d_theta = nullptr, *d_out = nullptr;
    AdjAtom *d_atoms = nullptr;
    AdjRun *d_runs = nullptr;
    AdjGroup *d_groups = nullptr;
    AdjTerm *d_terms = nullptr;
    AdjPass *d_passes = nullptr;
    int32_t *d_hlist = nullptr;
    int64_t *d_hchunk = nullptr;
    double2 *psi = nullptr, *lam = nullptr;
    bool own_blob = false;

    ~AdjProgram() {
        if (own_blob) cudaFree(blob);
        if (states) cudaFree(states);
    }
};

using cd = std::complex<double>;

static bool unitary(const double *m, int dim) {
    for (int r = 0; r < dim; ++r)
        for (int c = 0; c < dim; ++c) {
            cd s = 0.0;
            for (int k = 0; k < dim; ++k)
                s += std::conj(cd(m[2 * (k * dim + r)], m[2 * (k * dim + r) + 1])) *
                     cd(m[2 * (k * dim + c)], m[2 * (k * dim + c) + 1]);
            if (!(std::abs(s - (r == c ? 1.0 : 0.0)) <= 1e-14)) return false;
        }
    return true;
}

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
    if (!unitary(m, 2)) return false;
    AdjAtom a{};
    a.kind = AT_CONST;
    a.param = -1;
    a.cmat = (int64_t)p.coef.size();
    p.coef.insert(p.coef.end(), m, m + 8);
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

// Encode the rounds of one planned pass.  op_run[i] is the run of planned op i
// (-1: a gate with static coefficients); slots counts the pass's gradient runs.
static void adj_encode_pass(const PlannedPass &ps, const std::vector<GateOp> &gops,
                            const std::vector<int> &op_run, bool bwd, int T, AdjProgram &p,
                            std::vector<int> &slot_runs) {
    for (const PlannedRound &rd : ps.rounds) {
        FusedRound fr{};
        fill_round(fr, rd.rpos, T, ps.h);
        auto open = [&]() {
            fr.op_begin = (int)p.ops.size();
            fr.pad = (int)slot_runs.size() << 8;
        };
        auto close = [&]() {
            fr.op_end = (int)p.ops.size();
            p.rounds.push_back(fr);
        };
        open();
        for (int k : rd.ops) {
            const int gi = ps.gates[k], run = op_run[gi];
            const bool slot = bwd && run >= 0 && p.runs[run].ntiles > 0;
            if (slot && (fr.pad & 0xff) == kRoundSlots) {  // same register bits, a new round
                close();
                open();
            }
            std::vector<FusedOp> one;
            std::vector<double> c;
            encode_op(gops[gi], ps.h, T - 4, rd.rpos, one, c);
            PassOp po = pass_op(one[0]);
            if (run >= 0) {
                po.coef = (int32_t)(bwd ? p.runs[run].coef_b : p.runs[run].coef_f);
                if (slot) {
                    po.code += AC_GM1;
                    po.bits = fr.pad & 0xff;
                    slot_runs.push_back(run);
                    ++fr.pad;
                }
            } else {
                po.coef = (int32_t)p.coef.size();
                p.coef.insert(p.coef.end(), c.begin(), c.end());
            }
            p.ops.push_back(po);
        }
        close();
    }
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
        if (op.type == OP_M1 && !unitary(op.m, 2)) return false;
        if (op.type == OP_M2 && !unitary(op.m, 4)) return false;
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
        r.coef_f = (int64_t)p.coef.size();
        r.coef_b = r.coef_f + 8;
        p.coef.resize(p.coef.size() + 16, 0.0);
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
    for (int dir = 0; dir < 2; ++dir) {
        const auto &go = dir ? back : gops;
        const auto &gr = dir ? back_run : op_run;
        for (const PlanStep &st : plan_circuit(go, n, T, dir ? 3 : 4)) {
            if (!st.fused) return false;
            AdjPass ap{};
            ap.h = st.pass.h;
            ap.round_begin = (int)p.rounds.size();
            ap.ntiles = 1 << (n - T);
            ap.part = p.npart;
            std::vector<int> slots;
            adj_encode_pass(st.pass, go, gr, dir == 1, T, p, slots);
            ap.nrounds = (int)p.rounds.size() - ap.round_begin;
            for (int r : slots) {
                p.runs[r].part = p.npart;
                p.npart += 3ll * ap.ntiles;
            }
            (dir ? bpass : fpass).push_back(ap);
        }
    }
    // the Pauli sum, by X mask in order of first appearance
    std::vector<char> taken(sp.nterms, 0);
    in.group_begin = (int)p.groups.size();
    for (int t = 0; t < sp.nterms; ++t) {
        if (taken[t]) continue;
        AdjGroup gr{sp.terms[t].xmask, (int)p.terms.size(), 0};
        for (int u = t; u < sp.nterms; ++u) {
            const lq_pauli_term &pt = sp.terms[u];
            if (taken[u] || pt.xmask != gr.x) continue;
            if (!std::isfinite(pt.coefficient)) return false;
            taken[u] = 1;
            int k = pt.ny & 3;
            if (sp.yconv == LQ_Y_TEXTBOOK) k = (4 - k) & 3;
            const double a = k == 0 ? 1.0 : k == 2 ? -1.0 : 0.0;
            const double b = k == 1 ? -1.0 : k == 3 ? 1.0 : 0.0;
            p.terms.push_back(AdjTerm{pt.zmask, pt.coefficient * a, pt.coefficient * b});
            ++gr.nterms;
        }
        p.groups.push_back(gr);
    }
    in.ngroups = (int)p.groups.size() - in.group_begin;
    return p.coef.size() < (size_t)1 << 30 && p.ops.size() < (size_t)1 << 30;
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
            if (!fp[k].empty()) in.f_round = fp[k][0].round_begin, in.f_nrounds = fp[k][0].nrounds;
            if (!bp[k].empty()) in.b_round = bp[k][0].round_begin, in.b_nrounds = bp[k][0].nrounds;
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
    const size_t o_rounds = take(p.rounds.size() * sizeof(FusedRound));
    const size_t o_ops = take(p.ops.size() * sizeof(PassOp));
    const size_t o_atoms = take(p.atoms.size() * sizeof(AdjAtom));
    const size_t o_runs = take(p.runs.size() * sizeof(AdjRun));
    const size_t o_groups = take(p.groups.size() * sizeof(AdjGroup));
    const size_t o_terms = take(p.terms.size() * sizeof(AdjTerm));
    const size_t o_passes = take(p.passes.size() * sizeof(AdjPass));
    const size_t o_hlist = take(p.h_list.size() * sizeof(int32_t));
    const size_t o_hchunk = take(p.h_chunk.size() * sizeof(int64_t));
    const size_t o_coef = take(p.coef.size() * sizeof(double));
    const size_t upload = off;
    const size_t o_wts = take(p.atoms.size() * 3 * sizeof(double));
    const size_t o_part = take((size_t)p.npart * sizeof(double));
    const size_t o_epart = take((size_t)p.nepart * sizeof(double));
    const size_t o_theta = take(((size_t)p.nparams + 1) * sizeof(double));
    const size_t o_out = take(((size_t)p.ninst + p.nparams) * sizeof(double));
    // A plain call works in its handle's own program buffer and amplitudes.
    cudaError_t e = cudaSuccess;
    const size_t copies = work ? 1 : 2;
    if (p.amps > 0) e = cudaMalloc(&p.states, (size_t)p.amps * copies * sizeof(double2));
    if (e == cudaSuccess) {
        if (work) {
            LQ_TRY(ensure_prog(work, off));
            p.blob = work->d_prog;
        } else {
            e = cudaMalloc(&p.blob, off);
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
    put(o_ops, p.ops);
    put(o_atoms, p.atoms);
    put(o_runs, p.runs);
    put(o_groups, p.groups);
    put(o_terms, p.terms);
    put(o_passes, p.passes);
    put(o_hlist, p.h_list);
    put(o_hchunk, p.h_chunk);
    put(o_coef, p.coef);
    char *b = (char *)p.blob;
    p.d_insts = (AdjInst *)(b + o_insts);
    p.d_rounds = (FusedRound *)(b + o_rounds);
    p.d_ops = (PassOp *)(b + o_ops);
    p.d_atoms = (AdjAtom *)(b + o_atoms);
    p.d_runs = (AdjRun *)(b + o_runs);
    p.d_groups = (AdjGroup *)(b + o_groups);
    p.d_terms = (AdjTerm *)(b + o_terms);
    p.d_passes = (AdjPass *)(b + o_passes);
    p.d_hlist = (int32_t *)(b + o_hlist);
    p.d_hchunk = (int64_t *)(b + o_hchunk);
    p.d_coef = (double *)(b + o_coef);
    p.d_wts = (double *)(b + o_wts);
    p.d_part = (double *)(b + o_part);
    p.d_epart = (double *)(b + o_epart);
    p.d_theta = (double *)(b + o_theta);
    p.d_out = (double *)(b + o_out);
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
    if (nruns)
        k_adj_coef<<<(nruns + 127) / 128, 128, 0, st>>>(p.d_runs, nruns, p.d_atoms, p.d_theta,
                                                       p.d_coef, p.d_wts);
    if (p.nsmall)
        k_adj_small<<<p.nsmall, kAdjSmallThreads, adj_small_smem(p.small_T), st>>>(
            p.d_insts, p.d_rounds, p.d_ops, p.d_coef, p.d_groups, p.d_terms, p.d_part, p.d_epart);
    double2 *psi = p.psi, *lam = p.lam;
    for (const AdjWave &w : p.waves) {
        for (size_t l = 0; l < w.f.size(); ++l) {
            const auto [a, b] = w.f[l];
            const AdjPass &last = p.passes[b - 1];
            k_adj_pass<false><<<last.tile_begin + last.ntiles, kAdjThreads,
                                adj_pass_smem(p.T, false), st>>>(
                p.d_insts, p.d_passes + a, b - a, p.d_rounds, p.d_ops, p.d_coef, psi, lam,
                p.d_part, p.T, l == 0);
        }
        k_adj_h<<<(unsigned)w.h_blocks, 256, 0, st>>>(p.d_insts, p.d_hlist + w.h_begin, w.h_count,
                                                     p.d_hchunk + w.h_begin, p.d_groups, p.d_terms,
                                                     psi, lam, p.d_epart);
        for (size_t l = 0; l < w.b.size(); ++l) {
            const auto [a, b] = w.b[l];
            const AdjPass &last = p.passes[b - 1];
            k_adj_pass<true><<<last.tile_begin + last.ntiles, kAdjThreads, adj_pass_smem(p.T, true),
                               st>>>(p.d_insts, p.d_passes + a, b - a, p.d_rounds, p.d_ops,
                                     p.d_coef, psi, lam, p.d_part, p.T, l + 1 == w.b.size());
        }
    }
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
