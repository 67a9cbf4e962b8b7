// Fused circuits (Circuit::execute, src/circuits/mod.rs:352-375) as mapped rounds.
//
// Every gate of a circuit is written with three kinds of step:
//   * permutations of basis states that are linear over XOR (CNOT, X, SWAP): they move
//     no data.  The tile keeps the map between logical indices and places, and such a
//     gate changes the map, on the host;
//   * diagonal factors z^f, f the parity of some index bits: they wait on the host and
//     are multiplied, merged into one table per register round, when a rotation
//     mixes amplitudes on which f differs;
//   * scaled real rotations [[1, -t], [t, 1]], |t| <= 1, one FMA per real component,
//     possibly with t chosen by a control parity.
// A 2x2 unitary is w diag(1, e^{i phi}) [[c, -s], [s, c]] diag(1, e^{i lambda}) (the Euler form of
// U3, src/gates/parameterized.rs:249-282) with the scale c factored out into a diagonal;
// where |s| > |c| it is the rotation by a quarter turn less, followed by X and a sign.
// A controlled 2x2, and RXX / RYY, rotate by one of two angles: CNOT(a, b) turns the
// blocks {00, 11} and {01, 10} of the latter into bit a with control bit b.
//
// A pass is one read and write of the state: a CTA takes the tile of 2^T amplitudes of
// index bits [0,4) and [h, h+T-4) and runs the pass's rounds.  In a round a thread holds 16
// amplitudes that differ along four vectors v_0..v_3 (a logical bit's place after CNOTs is
// a sum of place bits) and does, in straight-line code and in place, the tables and the
// rotation of each vector in turn.  Places at the end of a pass are not logical order in
// general; the store reads through the map.
//
// Bound: 28 qubits, 20 brickwork layers: 17 passes of 9.5 rounds at T = 11.  A round reads
// and writes the tile in shared memory, whose pipe is 72-80 % busy (39 of 62.5 ms), FP64
// 40-44 %, issue 53 %, with 16 warps per SM; HBM would take 22 ms.  More amplitudes per
// thread would need fewer rounds but halve the warps.
//
// Against the op-record rounds (fused_round.cuh: 94.8 ms), which remain for circuits
// without this form or with many controlled rotations (map_plan): those keep two arrays of
// 16 amplitudes per thread (168 registers, 12 warps per SM) and dispatch every op through a
// switch; FP64 was 52 % of the instructions, and each issue waited 2.5 cycles on table and
// record loads and 0.9 on instruction fetch.  Here the code of a round is some 6 KB, the
// amplitudes take 64 registers, and tables come from the constant bank.
#pragma nv_diag_suppress 20208  // (long double is the host planner's)
#include "mapped.h"

#include <algorithm>
#include <array>
#include <complex>
#include <cstring>
#include <map>

#include "fused_plan.h"

namespace lq {

// Host arithmetic of the planner: a factor is rounded to double once, in its table.  (In
// double the same gate's rounding came back at every repetition: ten Trotter steps of 11 qubits
// had an error of 2e-14, nearly all of it in the norm, against 1.5e-15 gate by gate.)
using real = long double;
using cd = std::complex<real>;

// Place of tile index i in shared memory, in 16-byte units: each 3-bit group above the
// lowest is added to it, so that any three tile bits of different residues mod 3 put
// eight threads on the eight bank groups.  Linear over XOR.  (The 128-byte swizzle of a
// tensor copy adds bits 3-5 only: rounds on four neighbouring low bits then had up to
// 70 % more shared-memory cycles.)
__host__ __device__ __forceinline__ int mswz(int i) {
    return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7);
}

constexpr int kMapMaxCst = 8;              // outside bits that a pass's map may depend on
// The program of a pass is a kernel parameter: in the constant bank, read with uniform
// addresses into uniform registers.  Through shared memory every factor of a table took a
// 16-byte load per thread, a third of all shared-memory cycles, which were 85 % busy; and
// each tile brought its copy of the program with it.
constexpr int kMapLine = 64;                // bytes
constexpr size_t kMapProgram = 16 * 1024;  // a pass ends when it has grown past this
constexpr size_t kMapLargest = 28 * 1024;  // the largest parameter

// Rotation along a register vector v by t where the rotated bit is 0 at the element with
// v's register bit clear, by -t where it is 1 there (the pair is then the other way
// round): the sign is the parity of the bit's functional at that element.
struct MapSlot {
    int32_t kind;        // 0: no rotation; 1: one t per thread; 2: t per element
    int32_t ntab, tab;   // the table before it (0 or 1)
    uint32_t word;       // kind 2: the control's parity over the 16 elements (t0 / t1)
    double t0, t1;       // (kind 1: the same)
    uint64_t mask;       // kind 2: the control's index bits at the thread's base
    uint64_t smask;      // the sign's index bits at the thread's base
    uint32_t sword;      // kind 2: the sign's parity over the elements
    uint32_t pad[3];
};

struct MapRound {
    uint32_t vec[4];     // byte offsets of the register vectors
    int32_t bases;       // some sign, table or control reads the thread's own index
    int32_t nslot;
    int32_t ntail, tail; // tables after the last rotation
    uint32_t lane[8];    // byte offsets of the thread-index bits (unused ones 0)
    uint32_t lane_bit[8];  // and their tile index bits
    uint32_t base;       // byte offset of logical tile index 0
    int32_t ncst;
    int32_t path;        // 0: any (map_any); 1-4: that many rotations of kind 1 after one table of
                         // kind 0 whose variant a whole warp shares; + 4: without the table
    int32_t signs;       // some rotation's sign differs between threads
    int32_t npre, pre;   // tables of any kind, before the rest
    int32_t pad[2];
    uint32_t cst_vec[kMapMaxCst];  // added where an outside index bit is 1
    int32_t cst_bit[kMapMaxCst];
    MapSlot slot[4];
};
static_assert(sizeof(MapRound) % 16 == 0, "staged in 16-byte pieces");

struct MapTable {
    int32_t kind;        // 0, 2: 16 factors per variant, which for 0 a warp shares;
                         // 1: two factors made by the thread
    int32_t data;        // offset in the program's data, in 16-byte units
    int32_t count;       // kinds 0, 2: variant bits; kind 1: items
    uint32_t word;       // kind 1: elements that take the second factor
    uint64_t m[4];       // kinds 0, 2: index bits whose parities at the base pick the variant
};

struct MapItem {         // kind 1: z into the first factor where the parity is 1, else the second
    uint64_t mask;
    double zr, zi;
    double pad;
};
static_assert(sizeof(MapTable) == 48 && sizeof(MapItem) == 32, "16-byte pieces");

constexpr int kMapVariant = 16;    // factors of one variant
constexpr int kMapParts = 3;     // thread parts of one table (2^kMapParts variants)

struct MapStore {        // logical tile index -> byte offset
    uint32_t vec[kMaxT];
    uint32_t base;
    int32_t ncst;
    uint32_t cst_vec[kMapMaxCst];
    int32_t cst_bit[kMapMaxCst];
    uint32_t pad[2];
};
static_assert(sizeof(MapStore) % 16 == 0, "staged in 16-byte pieces");

// ---------------------------------------------------------------------------
// Device
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t parity64(uint64_t x) { return (uint32_t)__popcll(x) & 1u; }

__device__ __forceinline__ double2 cmul2(double2 v, double2 p) {
    return make_double2(fma(-v.y, p.y, v.x * p.x), fma(v.x, p.y, v.y * p.x));
}

// gbase is the thread's basis index in the round (register bits 0).
__device__ __forceinline__ uint32_t map_variant(const MapTable &tb, uint64_t gbase) {
    uint32_t v = 0;
    for (int q = 0; q < tb.count; ++q) v |= parity64(gbase & tb.m[q]) << q;
    return v * kMapVariant;
}

__device__ __forceinline__ double neg_if(double x, uint32_t bit) {  // bit 0 counts
    return __hiloint2double(__double2hiint(x) ^ (int)(bit << 31), __double2loint(x));
}

template <int K>
__device__ __forceinline__ void map_rotate1(double2 (&a)[16], double t) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        if (e & (1 << K)) continue;
        const int f = e | (1 << K);
        const double2 x = a[e], y = a[f];
        a[e] = make_double2(fma(-t, y.x, x.x), fma(-t, y.y, x.y));
        a[f] = make_double2(fma(t, x.x, y.x), fma(t, x.y, y.y));
    }
}

template <int K>
__device__ __forceinline__ void map_rotate(double2 (&a)[16], const MapSlot &sl, uint64_t gbase) {
    const uint32_t sg = parity64(gbase & sl.smask);
    const uint32_t w = sl.word ^ (0u - parity64(gbase & sl.mask));
    const uint32_t sw = sl.sword ^ (0u - sg);
    const double t0 = sl.t0, t1 = sl.t1;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        if (e & (1 << K)) continue;
        const int f = e | (1 << K);
        const double t = neg_if((w >> e) & 1u ? t1 : t0, sw >> e);
        const double2 x = a[e], y = a[f];
        a[e] = make_double2(fma(-t, y.x, x.x), fma(-t, y.y, x.y));
        a[f] = make_double2(fma(t, x.x, y.x), fma(t, x.y, y.y));
    }
}

// The 16 places of a thread in a round: E_k are the register vectors' byte offsets.
struct MapPlaces {
    unsigned char *tile;
    uint32_t sb, E[4];
    __device__ __forceinline__ double2 *at(int e) const {
        return (double2 *)(tile + (sb ^ ((e & 1) ? E[0] : 0u) ^ ((e & 2) ? E[1] : 0u) ^
                                   ((e & 4) ? E[2] : 0u) ^ ((e & 8) ? E[3] : 0u)));
    }
};

// A table of any kind on the thread's places, one amplitude at a time.
__device__ __forceinline__ void map_table(const MapPlaces &pl, const MapTable &tb,
                                          const double2 *data, uint64_t gbase, uint64_t gwarp) {
    if (tb.kind == 0) {  // (uniform addresses)
        const double2 *p = data + tb.data + map_variant(tb, gwarp);
#pragma unroll
        for (int e = 0; e < 16; ++e) *pl.at(e) = cmul2(*pl.at(e), p[e]);
        return;
    }
    if (tb.kind == 2) {
        const double2 *p = data + tb.data + map_variant(tb, gbase);
#pragma unroll
        for (int e = 0; e < 16; ++e) *pl.at(e) = cmul2(*pl.at(e), p[e]);
        return;
    }
    double2 f0 = make_double2(1.0, 0.0), f1 = f0;
    const MapItem *it = (const MapItem *)(data + tb.data);
    for (int k = 0; k < tb.count; ++k) {
        const double2 z = make_double2(it[k].zr, it[k].zi);
        const bool on = parity64(gbase & it[k].mask);
        const double2 n = cmul2(on ? f0 : f1, z);
        f0 = on ? n : f0;
        f1 = on ? f1 : n;
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) *pl.at(e) = cmul2(*pl.at(e), (tb.word >> e) & 1u ? f1 : f0);
}

// The common round as one straight line, with its load and store: the amplitudes are
// in no register at a branch, where the compiler would move them (with the general
// path below for every round a quarter of the instructions were such moves).
template <int NS, bool TABLE>
__device__ __forceinline__ void map_line(const MapPlaces &pl, const MapRound &rd,
                                         const MapTable *tabs, const double2 *data,
                                         uint64_t gbase, uint64_t gwarp) {
    double t[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) t[k] = rd.slot[k].t0;
    if (rd.signs)
#pragma unroll
        for (int k = 0; k < NS; ++k) t[k] = neg_if(t[k], parity64(gbase & rd.slot[k].smask));
    const double2 *p = nullptr;
    if (TABLE) {
        const MapTable &tb = tabs[rd.slot[0].tab];
        p = data + tb.data + map_variant(tb, gwarp);
    }
    double2 a[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        a[e] = *pl.at(e);
        if (TABLE) a[e] = cmul2(a[e], p[e]);
    }
    map_rotate1<0>(a, t[0]);
    if (NS > 1) map_rotate1<1>(a, t[NS > 1 ? 1 : 0]);
    if (NS > 2) map_rotate1<2>(a, t[NS > 2 ? 2 : 0]);
    if (NS > 3) map_rotate1<3>(a, t[NS > 3 ? 3 : 0]);
#pragma unroll
    for (int e = 0; e < 16; ++e) *pl.at(e) = a[e];
}

// Any round with rotations: a table of kind 0 before the first (always) and each of the
// others (or none), and rotations of either kind.
__device__ __forceinline__ void map_any(const MapPlaces &pl, const MapRound &rd,
                                        const MapTable *tabs, const double2 *data,
                                        uint64_t gbase, uint64_t gwarp) {
    double2 a[16];
    auto factors = [&](const MapSlot &sl) {
        const MapTable &tb = tabs[sl.tab];
        return data + tb.data + map_variant(tb, gwarp);
    };
    {
        const double2 *p = factors(rd.slot[0]);
#pragma unroll
        for (int e = 0; e < 16; ++e) a[e] = cmul2(*pl.at(e), p[e]);
    }
    map_rotate<0>(a, rd.slot[0], gbase);
#define LQ_SLOT(K)                                                  \
    if (rd.slot[K].ntab) {                                          \
        const double2 *p = factors(rd.slot[K]);                     \
        _Pragma("unroll") for (int e = 0; e < 16; ++e) a[e] = cmul2(a[e], p[e]); \
    }                                                               \
    if (rd.slot[K].kind) map_rotate<K>(a, rd.slot[K], gbase);
    LQ_SLOT(1) LQ_SLOT(2) LQ_SLOT(3)
#undef LQ_SLOT
#pragma unroll
    for (int e = 0; e < 16; ++e) *pl.at(e) = a[e];
}

template <int BYTES>
struct MapParam {
    alignas(16) unsigned char b[BYTES];
};

// Blocks of 2^(T-4) threads, at most 256; 128 registers: 16 warps per SM at T = 11
// (four tiles of 32 KB).
template <int BYTES>
__global__ void __launch_bounds__(256, 2)
    k_mapped_pass(double2 *__restrict__ state, int T, int h, int nrounds, int ntabs,
                  int bytes, const __grid_constant__ MapParam<BYTES> param) {
    extern __shared__ __align__(16) unsigned char map_smem[];
    const int tid = threadIdx.x;
    // (the same for all threads of a warp, and known to be)
    const int warp = blockDim.x >= 32 ? __shfl_sync(0xffffffffu, tid >> 5, 0) : 0;
    const int tile = blockIdx.x;
    const uint64_t c2 = (uint64_t)(tile & ((1 << (h - 4)) - 1)), c4 = (uint64_t)(tile >> (h - 4));
    const uint64_t tile_base = (c2 << 4) | (c4 << (h + T - 4));
    // The tile: 16-byte copies, 512 consecutive bytes per warp.
    {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(map_smem);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int l = tid | k << (T - 4);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             dst + ((uint32_t)mswz(l) << 4)),
                         "l"(state + (tile_base | (uint64_t)(l & 15) | ((uint64_t)(l >> 4) << h)))
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        // meanwhile the program comes into the constant cache: a line per thread
        for (int o = tid * kMapLine; o < bytes; o += (int)blockDim.x * kMapLine) {
            const int x = *(const int *)(param.b + o);
            asm volatile("" ::"r"(x));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    const MapStore &st = *(const MapStore *)param.b;
    const MapRound *rounds = (const MapRound *)(param.b + sizeof(MapStore));
    const MapTable *tabs = (const MapTable *)(rounds + nrounds);
    const double2 *data = (const double2 *)(tabs + ntabs);
    uint32_t on[8];  // all ones where the thread-index bit is set
#pragma unroll
    for (int j = 0; j < 8; ++j) on[j] = 0u - ((uint32_t)((j < 5 ? tid : warp << 5) >> j) & 1u);
    for (int r = 0; r < nrounds; ++r) {
        const MapRound &rd = rounds[r];
        MapPlaces pl;
        pl.tile = map_smem;
        uint32_t base = rd.base;
        for (int j = 0; j < rd.ncst; ++j)
            base ^= rd.cst_vec[j] & (0u - (uint32_t)((tile_base >> rd.cst_bit[j]) & 1ull));
        // thread bits 5 and up are the warp's
        uint32_t wbase = 0;
#pragma unroll
        for (int j = 5; j < 8; ++j) {
            base ^= rd.lane[j] & on[j];
            wbase |= rd.lane_bit[j] & on[j];
        }
        pl.sb = base;
#pragma unroll
        for (int j = 0; j < 5; ++j) pl.sb ^= rd.lane[j] & on[j];
        const uint64_t gwarp = tile_base | (uint64_t)(wbase & 15u) | ((uint64_t)(wbase >> 4) << h);
        uint64_t gbase = gwarp;
        if (rd.bases) {
            uint32_t tbase = wbase;
#pragma unroll
            for (int j = 0; j < 5; ++j) tbase |= rd.lane_bit[j] & on[j];
            gbase = tile_base | (uint64_t)(tbase & 15u) | ((uint64_t)(tbase >> 4) << h);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) pl.E[k] = rd.vec[k];
        switch (rd.path) {
        case 1: map_line<1, true>(pl, rd, tabs, data, gbase, gwarp); break;
        case 2: map_line<2, true>(pl, rd, tabs, data, gbase, gwarp); break;
        case 3: map_line<3, true>(pl, rd, tabs, data, gbase, gwarp); break;
        case 4: map_line<4, true>(pl, rd, tabs, data, gbase, gwarp); break;
        case 5: map_line<1, false>(pl, rd, tabs, data, gbase, gwarp); break;
        case 6: map_line<2, false>(pl, rd, tabs, data, gbase, gwarp); break;
        case 7: map_line<3, false>(pl, rd, tabs, data, gbase, gwarp); break;
        case 8: map_line<4, false>(pl, rd, tabs, data, gbase, gwarp); break;
        default:
            for (int k = 0; k < rd.npre; ++k) map_table(pl, tabs[rd.pre + k], data, gbase, gwarp);
            if (rd.nslot) map_any(pl, rd, tabs, data, gbase, gwarp);
            break;
        }
        for (int k = 0; k < rd.ntail; ++k) map_table(pl, tabs[rd.tail + k], data, gbase, gwarp);
        __syncthreads();
    }
    // Back in logical order through the map.
    uint32_t mb = st.base;
    for (int j = 0; j < st.ncst; ++j)
        mb ^= st.cst_vec[j] & (0u - (uint32_t)((tile_base >> st.cst_bit[j]) & 1ull));
    for (int j = 0; j < T - 4; ++j) mb ^= st.vec[j] & (0u - (uint32_t)((tid >> j) & 1));
    const uint32_t F0 = st.vec[T - 4], F1 = st.vec[T - 3], F2 = st.vec[T - 2], F3 = st.vec[T - 1];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const uint32_t at = mb ^ ((k & 1) ? F0 : 0u) ^ ((k & 2) ? F1 : 0u) ^ ((k & 4) ? F2 : 0u) ^
                            ((k & 8) ? F3 : 0u);
        const int l = tid | k << (T - 4);
        state[tile_base | (uint64_t)(l & 15) | ((uint64_t)(l >> 4) << h)] =
            *(const double2 *)(map_smem + at);
    }
}

// ---------------------------------------------------------------------------
// Host: gates -> permutations, diagonals, rotations
// ---------------------------------------------------------------------------
enum MapOpKind { MO_PERM, MO_SWAP, MO_DIAG, MO_ROT };

// (Small: a circuit becomes some thousand of them, and with the whole GateOp of 360 bytes in
// each, copying them was a quarter of the planning.)
struct MapOp {
    int kind;
    // MO_PERM: X on t, controlled by c if >= 0.  MO_SWAP: b0 and b1.  MO_DIAG: factor
    // p[v1 << 1 | v0] of bits b1, b0 (b1 < 0: p[0], p[1] of b0 alone).  MO_ROT: bit t by t0, or
    // by t0 / t1 for control bit c = 0 / 1.
    int t = -1, c = -1, b0 = -1, b1 = -1;
    uint64_t bits = 0;   // index bits that it touches
    double t0 = 0.0, t1 = 0.0;
    cd p[4];
};

static uint64_t bit_of(int b) { return b >= 0 ? 1ull << b : 0ull; }

static MapOp map_perm_x(int t, int c) {
    MapOp o;
    o.kind = MO_PERM;
    o.t = t;
    o.c = c;
    o.bits = bit_of(t) | bit_of(c);
    return o;
}

static MapOp map_diag(int b1, int b0, const cd &p00, const cd &p01, const cd &p10, const cd &p11) {
    MapOp o;
    o.kind = MO_DIAG;
    o.b0 = b0;
    o.b1 = b1;
    o.bits = bit_of(b0) | bit_of(b1);
    o.p[0] = p00, o.p[1] = p01, o.p[2] = p10, o.p[3] = p11;
    return o;
}

// Arithmetic on finite numbers of ordinary size: std::complex's operators distinguish
// infinities and scale against overflow, in library calls that were a fifth of the planning.
static inline cd mul(const cd &a, const cd &b) {
    return cd(a.real() * b.real() - a.imag() * b.imag(), a.real() * b.imag() + a.imag() * b.real());
}
static inline real norm2(const cd &a) { return a.real() * a.real() + a.imag() * a.imag(); }
static inline real length(const cd &a) { return std::sqrt(norm2(a)); }
static inline cd inverse(const cd &a) {
    const real d = 1 / norm2(a);
    return cd(a.real() * d, -a.imag() * d);
}
static inline cd root(const cd &a) {  // the principal square root
    const real r = length(a), h = std::sqrt((r + std::abs(a.real())) / 2);
    if (h == 0) return cd(0.0);
    const real g = a.imag() / (2 * h);
    if (a.real() >= 0) return cd(h, g);
    return std::signbit(a.imag()) ? cd(-g, -h) : cd(g, h);
}

// The last few results of a function of four factors: within a circuit the same gates tend to
// come again (every bond of a Trotter step).
template <class R>
struct Recent {
    static constexpr int kKept = 4;
    cd key[kKept][4];
    R value[kKept];
    int used = 0, next = 0;
    const R *find(const cd u[4]) const {
        for (int k = 0; k < used; ++k)
            if (std::equal(u, u + 4, key[k])) return &value[k];
        return nullptr;
    }
    void put(const cd u[4], const R &r) {
        std::copy(u, u + 4, key[next]);
        value[next] = r;
        used = std::max(used, next + 1);
        next = (next + 1) % kKept;
    }
};

struct MapEuler {
    cd w, phi, lam;
    double t;
    real scale;  // after the quarter turn was taken out
    bool turned;
};

// u = w diag(1, phi) [X and sign if turned] scale [[1, -t], [t, 1]] diag(1, lam)
static bool map_euler(const cd u[4], MapEuler &e) {
    const real ra = length(u[0]), rb = length(u[1]), rc = length(u[2]), rd = length(u[3]);
    if (!(std::abs(ra * ra + rc * rc - 1.0) <= 1e-12 && std::abs(rb - rc) <= 1e-12 &&
          std::abs(ra - rd) <= 1e-12))
        return false;  // not unitary
    constexpr real tiny = 1e-150;
    e.w = ra > tiny ? u[0] / ra : cd(1.0, 0.0);
    if (rc > tiny && rb > tiny) {
        e.phi = mul(u[2] / rc, std::conj(e.w));
        e.lam = mul(-u[1] / rb, std::conj(e.w));
    } else {
        e.phi = 1.0;
        e.lam = rd > tiny ? mul(u[3] / rd, std::conj(e.w)) : cd(1.0, 0.0);
    }
    const cd r[4] = {e.w * ra, mul(-e.w * rc, e.lam), mul(e.w * rc, e.phi),
                     mul(mul(e.w * ra, e.phi), e.lam)};
    for (int k = 0; k < 4; ++k)
        if (!(length(r[k] - u[k]) <= 1e-14)) return false;
    // [[c, -s], [s, c]] with s > c is [[0, -1], [1, 0]] [[s, c], [-c, s]]
    e.turned = rc > ra;
    e.t = (double)(e.turned ? -ra / rc : rc / ra);
    // (of the rotation by the rounded t)
    e.scale = std::sqrt((ra * ra + rc * rc) / (1 + (real)e.t * e.t));
    return true;
}

// One 2x2 (A on bit t), or A / B for control bit c = 0 / 1.
static bool map_rotation(const cd A[4], const cd B[4], int t, int c, Recent<MapEuler> &recent,
                         std::vector<MapOp> &out) {
    auto euler = [&](const cd u[4], MapEuler &e) {
        if (const MapEuler *r = recent.find(u)) {
            e = *r;
            return true;
        }
        if (!map_euler(u, e)) return false;
        recent.put(u, e);
        return true;
    };
    MapEuler a, b;
    if (!euler(A, a)) return false;
    if (c < 0) b = a;
    else if (!euler(B, b)) return false;
    // factors of t = 0 / 1 under A and under B
    auto diag = [&](const cd &a0, const cd &a1, const cd &b0, const cd &b1) {
        if (c < 0) out.push_back(map_diag(-1, t, a0, a1, 0.0, 0.0));
        else out.push_back(map_diag(c, t, a0, a1, b0, b1));
    };
    diag(1.0, a.lam, 1.0, b.lam);
    if (a.t != 0.0 || b.t != 0.0) {
        MapOp o;
        o.kind = MO_ROT;
        o.t = t;
        o.c = a.t == b.t ? -1 : c;  // (RXX, RYY: the two differ in their diagonals only)
        o.bits = bit_of(t) | bit_of(o.c);
        o.t0 = a.t;
        o.t1 = b.t;
        out.push_back(o);
    }
    // the quarter turn: X on t (where it applies), then diag(-1, 1)
    if (c < 0) {
        if (a.turned) out.push_back(map_perm_x(t, -1));
    } else {
        if (a.turned) out.push_back(map_perm_x(t, -1));
        if (a.turned != b.turned) out.push_back(map_perm_x(t, c));
    }
    const cd wa = a.w * a.scale, wb = b.w * b.scale;
    diag(a.turned ? -wa : wa, mul(wa, a.phi), b.turned ? -wb : wb, mul(wb, b.phi));
    return true;
}

static cd coef(const double *m, int k) { return cd(m[2 * k], m[2 * k + 1]); }

// The 2x2 of an uncontrolled single-qubit op; diag: it is diagonal by construction.
static bool map_single(const GateOp &g, int &bit, cd u[4], bool &diag) {
    diag = false;
    if ((g.type == OP_M1 || g.type == OP_PERM1) && g.nctrl == 0) {
        bit = g.t;
        if (g.type == OP_M1)
            for (int k = 0; k < 4; ++k) u[k] = coef(g.m, k);
        else
            u[0] = 0.0, u[1] = 1.0, u[2] = 1.0, u[3] = 0.0;
        return true;
    }
    if (g.type == OP_DIAG && g.nfix + g.npat == 1) {
        diag = true;
        u[1] = u[2] = 0.0;
        if (g.npat) bit = g.pat[0], u[0] = coef(g.m, 0), u[3] = coef(g.m, 1);
        else bit = g.fix[0], u[0] = 1.0, u[3] = coef(g.m, 0);
        return true;
    }
    return false;
}

static bool unit(const cd &z) { return std::abs(length(z) - 1) <= 1e-12; }

// What the window planner sees: a gate or a run of single-qubit gates, with the map ops
// that it became.  (Planned op by op, a 2x2 with a quarter turn counted twice, and 60
// single-qubit gates on 24 qubits took five passes instead of three: 480 us, now 326.)
struct MapUnit {
    const GateOp *swap;  // the gate if it is a SWAP
    int begin, end;
};

// The circuit as map ops, and its passes; runs of single-qubit gates on a bit become one 2x2
// first.
static bool map_lower(const std::vector<GateOp> &gops, int n, int T, std::vector<MapOp> &out,
                      std::vector<MapUnit> &units, std::vector<PlanStep> &steps) {
    struct Run {
        int bit;
        cd u[4];
        bool diag, x;  // all diagonal; a lone X
    };
    struct Entry {
        int run;       // index into runs, or -1
        const GateOp *g;
    };
    std::vector<Run> runs;
    std::vector<Entry> list;
    int open[64];
    std::fill(open, open + 64, -1);
    runs.reserve(gops.size());
    list.reserve(gops.size());
    for (const GateOp &g : gops) {
        if (g.renorm) return false;
        int bit;
        cd u[4];
        bool diag;
        if (map_single(g, bit, u, diag)) {
            if (open[bit] >= 0) {
                Run &r = runs[open[bit]];
                const cd p[4] = {mul(u[0], r.u[0]) + mul(u[1], r.u[2]),
                                 mul(u[0], r.u[1]) + mul(u[1], r.u[3]),
                                 mul(u[2], r.u[0]) + mul(u[3], r.u[2]),
                                 mul(u[2], r.u[1]) + mul(u[3], r.u[3])};
                std::copy(p, p + 4, r.u);
                r.diag = r.diag && diag;
                r.x = false;
            } else {
                open[bit] = (int)runs.size();
                runs.push_back(Run{bit, {u[0], u[1], u[2], u[3]}, diag, g.type == OP_PERM1});
                list.push_back(Entry{open[bit], nullptr});
            }
            continue;
        }
        for (uint64_t bits = op_bits(g); bits; bits &= bits - 1) open[__builtin_ctzll(bits)] = -1;
        list.push_back(Entry{-1, &g});
    }
    units.reserve(list.size());
    std::vector<PlanGate> shapes;
    shapes.reserve(list.size());
    for (const Entry &en : list) {
        PlanGate p;
        if (en.run >= 0) {
            p.bits = bit_of(runs[en.run].bit);
            p.mixed = runs[en.run].diag ? 0 : p.bits;
        } else {
            p = plan_gate(*en.g);
        }
        shapes.push_back(p);
        units.push_back(MapUnit{en.run < 0 && en.g->type == OP_SWAP ? en.g : nullptr, 0, 0});
    }
    steps = plan_windows(shapes, n, T);
    // (a two-qubit rotation across windows would be three passes here, 983 us on 26 qubits
    // where its own sweep takes 317; seen before the gates are taken apart, which costs more
    // than the windows)
    for (const PlanStep &st : steps)
        if (!st.fused && !units[st.gate].swap) return false;
    Recent<MapEuler> recent;
    out.reserve(3 * list.size());
    for (size_t k = 0; k < list.size(); ++k) {
        const Entry &en = list[k];
        if (k > 0) units[k - 1].end = (int)out.size();
        units[k].begin = (int)out.size();
        if (en.run >= 0) {
            const Run &r = runs[en.run];
            if (r.x) {
                out.push_back(map_perm_x(r.bit, -1));
            } else if (r.diag) {
                if (!unit(r.u[0]) || !unit(r.u[3])) return false;
                out.push_back(map_diag(-1, r.bit, r.u[0], r.u[3], 0.0, 0.0));
            } else if (!map_rotation(r.u, r.u, r.bit, -1, recent, out)) {
                return false;
            }
            continue;
        }
        const GateOp &g = *en.g;
        switch (g.type) {
        case OP_PERM1:
            if (g.nctrl != 1) return false;
            out.push_back(map_perm_x(g.t, g.ctrl[0]));
            break;
        case OP_SWAP: {
            MapOp o;
            o.kind = MO_SWAP;
            o.b0 = g.b0;
            o.b1 = g.b1;
            o.bits = bit_of(g.b0) | bit_of(g.b1);
            out.push_back(o);
            break;
        }
        case OP_DIAG: {
            // two bits, in fix / pat positions
            if (g.nfix + g.npat != 2) return false;
            int bits[2], nb = 0;
            for (int k = 0; k < g.npat; ++k) bits[nb++] = g.pat[k];
            for (int k = 0; k < g.nfix; ++k) bits[nb++] = g.fix[k];
            cd p[4];
            for (int v = 0; v < 4; ++v) {  // v = bits[1] << 1 | bits[0]
                int pat = 0;
                bool on = true;
                for (int q = 0; q < 2; ++q) {
                    const int val = v >> q & 1;
                    if (q < g.npat) pat |= val << q;
                    else on = on && val;
                }
                p[v] = on ? coef(g.m, pat) : cd(1.0);
                if (!unit(p[v])) return false;
            }
            out.push_back(map_diag(bits[1], bits[0], p[0], p[1], p[2], p[3]));
            break;
        }
        case OP_M1: {
            if (g.nctrl != 1) return false;
            const cd id[4] = {1.0, 0.0, 0.0, 1.0};
            const cd u[4] = {coef(g.m, 0), coef(g.m, 1), coef(g.m, 2), coef(g.m, 3)};
            if (!map_rotation(id, u, g.t, g.ctrl[0], recent, out)) return false;
            break;
        }
        case OP_M2: {
            // blocks {00, 11} and {01, 10}; bit a = b0, control b = b1 after CNOT(a, b)
            for (int r = 0; r < 4; ++r)
                for (int c = 0; c < 4; ++c)
                    if ((__builtin_popcount(r ^ c) & 1) && coef(g.m, r * 4 + c) != cd(0.0))
                        return false;
            const cd A[4] = {coef(g.m, 0), coef(g.m, 3), coef(g.m, 12), coef(g.m, 15)};
            const cd B[4] = {coef(g.m, 5), coef(g.m, 6), coef(g.m, 9), coef(g.m, 10)};
            out.push_back(map_perm_x(g.b1, g.b0));
            if (!map_rotation(A, B, g.b0, g.b1, recent, out)) return false;
            out.push_back(map_perm_x(g.b1, g.b0));
            break;
        }
        default: return false;
        }
    }
    if (!units.empty()) units.back().end = (int)out.size();
    return true;
}

// ---------------------------------------------------------------------------
// Host: passes
// ---------------------------------------------------------------------------
static inline int par(uint64_t x) { return __builtin_parityll(x); }

// Waiting diagonal factors z^parity(mask & place), and one number for all amplitudes.
struct Waiting {
    struct Item {
        uint64_t mask;
        cd z;
        int slot;   // added after this many rotations of the round being planned
    };
    std::vector<Item> items;
    cd scalar = 1.0;
    bool twice = false;  // a mask may be there for two slots
    uint64_t seen[4] = {0, 0, 0, 0};  // hashes of the masks (of some that left, too)
    static unsigned hash(uint64_t mask) { return (unsigned)(mask * 0x9E3779B97F4A7C15ull >> 56); }
    bool see(uint64_t mask) {
        const unsigned k = hash(mask);
        const bool was = seen[k >> 6] >> (k & 63) & 1;
        seen[k >> 6] |= 1ull << (k & 63);
        return was;
    }
    void clear() {
        items.clear();
        std::fill(seen, seen + 4, 0);
        twice = false;
    }
    void add(uint64_t mask, const cd &z, int slot) {
        if (mask == 0 || z == cd(1.0)) return;
        if (see(mask))
            for (Item &i : items) {
                if (i.mask != mask) continue;
                if (i.slot == slot) {
                    i.z = mul(i.z, z);
                    return;
                }
                twice = true;
            }
        items.push_back(Item{mask, z, slot});
    }
    // z^(parity(mask) ^ flip)
    void add1(uint64_t mask, int flip, cd z, int slot) {
        if (flip) {
            scalar = mul(scalar, z);
            z = inverse(z);
        }
        add(mask, z, slot);
    }
};

class PassBuilder {
public:
    PassBuilder(int n, int T, Waiting &w) : n(n), T(T), m(T - 4), wait(w) {}

    void begin(int window) {
        h = window;
        for (int b = 0; b < T; ++b) place_of[b] = 1u << b;
        place_base = 0;
        place_cst.clear();
        rounds.clear();
        tabs.clear();
        data.clear();
        begin_round();
    }

    bool inside(int b) const { return b < 4 || (b >= h && b < h + m); }
    // Logical bit b as a functional of the index at the round's start.
    uint64_t functional(int b, int &fl) const {
        if (!inside(b)) {
            fl = 0;
            return 1ull << b;
        }
        fl = flip[local_pos(b, h)];
        return row[local_pos(b, h)];
    }

    // A permutation whose target lies in the window; false when the map is full.
    bool permute(const MapOp &o) {
        if (o.kind == MO_SWAP) {
            const int x = local_pos(o.b0, h), y = local_pos(o.b1, h);
            std::swap(vec[x], vec[y]);
            std::swap(row[x], row[y]);
            std::swap(flip[x], flip[y]);
            return true;
        }
        const int t = local_pos(o.t, h);
        if (o.c < 0) {
            base ^= vec[t];
            flip[t] ^= 1;
            return true;
        }
        const int c = o.c;
        if (inside(c)) {
            const int lc = local_pos(c, h);
            vec[lc] ^= vec[t];
            row[t] ^= row[lc];
            flip[t] ^= flip[lc];
            return true;
        }
        auto it = std::find_if(cst.begin(), cst.end(), [&](auto &x) { return x.first == c; });
        if (it == cst.end()) {
            int outside = (int)place_cst.size();
            for (auto &x : cst)
                outside += std::none_of(place_cst.begin(), place_cst.end(),
                                        [&](auto &y) { return y.first == x.first; });
            if (std::none_of(place_cst.begin(), place_cst.end(),
                             [&](auto &y) { return y.first == c; }) &&
                outside == kMapMaxCst)
                return false;
            cst.push_back({c, vec[t]});
        } else {
            it->second ^= vec[t];
        }
        row[t] ^= 1ull << c;
        return true;
    }

    void diagonal(const MapOp &o, int slot) {
        int f0, f1 = 0;
        const uint64_t m0 = functional(o.b0, f0);
        if (o.b1 < 0) {
            wait.scalar = mul(wait.scalar, o.p[0]);
            wait.add1(m0, f0, o.p[1] == o.p[0] ? cd(1.0) : mul(o.p[1], inverse(o.p[0])), slot);
            return;
        }
        // p[v1 v0] = p00 z1^v1 z0^v0 z2^(v1 ^ v0)
        const uint64_t m1 = functional(o.b1, f1);
        wait.scalar = mul(wait.scalar, o.p[0]);
        // (equal factors are compared as such, so that what is 1 is 1 to the bit and left out)
        if (o.p[1] == o.p[0] && o.p[2] == o.p[0] && o.p[3] == o.p[0]) return;
        Split z;
        if (const Split *r = splits.find(o.p)) {
            z = *r;
        } else {
            const cd i0 = inverse(o.p[0]);
            cd q[4];
            for (int k = 1; k < 4; ++k) q[k] = o.p[k] == o.p[0] ? cd(1.0) : mul(o.p[k], i0);
            if (q[1] == q[2]) {
                z.z0 = z.z1 = root(q[3]);
                z.z2 = z.z1 == cd(1.0) ? q[2] : mul(q[2], inverse(z.z1));
            } else {
                z.z1 = root(mul(mul(q[2], q[3]), inverse(q[1])));
                z.z2 = mul(q[2], inverse(z.z1));
                z.z0 = mul(q[1], inverse(z.z2));
            }
            splits.put(o.p, z);
        }
        wait.add1(m1, f1, z.z1, slot);
        wait.add1(m0, f0, z.z0, slot);
        wait.add1(m0 ^ m1, f0 ^ f1, z.z2, slot);
    }

    // A round of the given rotations in planning.
    struct Slot {
        uint32_t v;            // its vector in the tile, over the round's first indices
        double t0, t1;
        uint64_t ctrl;         // control functional (0: none)
        int cflip;
        uint64_t bit;          // the rotated bit's functional
        int bflip;
        std::vector<Waiting::Item> tables;
    };
    // (their tables keep their memory from round to round)
    struct Slots {
        Slot s[4];
        size_t n = 0;
        size_t size() const { return n; }
        bool empty() const { return n == 0; }
        Slot *begin() { return s; }
        Slot *end() { return s + n; }
        const Slot *begin() const { return s; }
        const Slot *end() const { return s + n; }
        Slot &operator[](size_t k) { return s[k]; }
        const Slot &operator[](size_t k) const { return s[k]; }
    };
    Slots slots;

    bool independent(uint32_t v) const {
        uint32_t basis[4];
        int nb = 0;
        auto reduce = [&](uint32_t x) {
            for (int k = 0; k < nb; ++k) x = std::min(x, x ^ basis[k]);
            return x;
        };
        for (const Slot &s : slots) {
            const uint32_t x = reduce(s.v);
            if (x) basis[nb++] = x;
        }
        return reduce(v) != 0;
    }

    uint64_t spread(uint32_t v) const {  // tile bits -> index bits
        return (uint64_t)(v & 15u) | (uint64_t)(v >> 4) << h;
    }

    // The slot before which a factor may stand: back from slot k past the rotations that
    // it commutes with, so that a round mostly has one table, before its first rotation.
    int earliest(const Waiting::Item &it, int k) const {
        int at = std::min(it.slot, k);
        while (at > 0 && !par(it.mask & spread(slots[at - 1].v))) --at;
        return at;
    }

    // Whether the round's rotations so far are plain and its factors one table's.
    bool line_so_far() const {
        uint64_t parts[kMapParts], rest = ~0ull;
        int np = 0;
        for (const Slot &s : slots) {
            if (s.ctrl || (&s != &slots[0] && !s.tables.empty())) return false;
            rest &= ~s.bit;
        }
        for (const auto &it : slots[0].tables) {
            const uint64_t p = it.mask & rest;
            if (!p || std::find(parts, parts + np, p) != parts + np) continue;
            if (np == kMapParts) return false;
            parts[np++] = p;
        }
        return true;
    }

    // Add the rotation to the round if its vector is free; the factors that it does
    // not commute with join the tables before it.
    bool rotate(const MapOp &o) {
        const uint32_t v = vec[local_pos(o.t, h)];
        if (slots.size() == 4 || !independent(v)) return false;
        const int k = (int)slots.n++;
        Slot &s = slots[k];
        s.v = v;
        s.t0 = o.t0;
        s.t1 = o.t1;
        s.ctrl = 0;
        s.cflip = 0;
        s.bit = functional(o.t, s.bflip);
        if (o.c >= 0) s.ctrl = functional(o.c, s.cflip);
        s.tables.clear();
        const uint64_t gv = spread(v);
        // A round that is one straight line so far stays one: a rotation that needs a
        // table of its own after the first rotation opens the next round.  (28-qubit
        // brickwork: 158 rounds with 159 tables instead of 150 with 203, 36 of them on
        // the general path.)
        if (k > 0 && o.c < 0 && line_so_far()) {
            for (const auto &it : wait.items) {
                if (par(it.mask & gv) && earliest(it, k) > 0) {
                    --slots.n;
                    return false;
                }
            }
        }
        size_t keep = 0;
        for (size_t q = 0; q < wait.items.size(); ++q) {
            const Waiting::Item &it = wait.items[q];
            if (par(it.mask & gv)) slots[earliest(it, k)].tables.push_back(it);
            else if (keep++ != q) wait.items[keep - 1] = it;
        }
        wait.items.resize(keep);
        return true;
    }

    int round_slots() const { return (int)slots.size(); }

    // Close the round; tail: also apply everything that waits, after the rotations.
    void close_round(bool tail) {
        if (slots.empty() && !(tail && (!wait.items.empty() || wait.scalar != cd(1.0)))) {
            begin_next();
            return;
        }
        // One round, or as many as their tables make of it
        size_t to = emit_round(tail);
        if (to < slots.size()) {
            const Slots all = slots;
            for (size_t at = 0;;) {
                slots.n = to - at;
                std::copy(all.begin() + at, all.begin() + to, slots.begin());
                const size_t stop = at + emit_round(tail && to == all.size());
                if (stop < to) {
                    to = stop;
                    continue;
                }
                if (to == all.size()) break;
                at = to;
                to = all.size();
            }
        }
        slots.n = 0;
        begin_next();
    }

    // The round of the slots; returns how many: fewer (and then nothing was done) where
    // the table before that rotation is not one that a warp shares.
    size_t emit_round(bool tail) {
        const size_t old_tabs = tabs.size(), old_data = data.size();
        const cd old_scalar = wait.scalar;
        MapRound rd{};
        // register vectors: the rotations', then tile bits that leave the threads' bits
        // on different banks
        uint32_t reg[4];
        uint32_t piv = 0;  // one pivot bit per vector: thread bases are 0 there
        {
            Reduced red;
            Ranks ranks;
            for (int b = 0; b < T; ++b) ranks.free(banks[b] = bank(b));
            int nreg = 0;
            for (const Slot &s : slots) add_pivot(red, ranks, piv, reg[nreg++] = s.v);
            while (nreg < 4) {
                int best = -1, best_rank = -1;
                for (int b = T - 1; b >= 0; --b) {
                    if (piv >> b & 1) continue;
                    // (bits that no rotated bit depends on keep the sign per thread)
                    int r = ranks.without(banks[b]);
                    for (const Slot &s : slots)
                        if (!par(s.bit & spread(1u << b))) r += 4;
                    if (r > best_rank) best = b, best_rank = r;
                }
                add_pivot(red, ranks, piv, reg[nreg++] = 1u << best);
            }
        }
        for (int k = 0; k < 4; ++k) rd.vec[k] = (uint32_t)mswz((int)place(reg[k])) << 4;
        // Thread-index bits: three that span the banks first; bits that the first table's
        // variant depends on last, from thread bit 5 up, where a warp shares them.
        const uint64_t off_base = spread(piv);
        uint64_t shared = 0;
        for (const Slot &s : slots)
            for (const auto &it : s.tables) shared |= it.mask & ~off_base;
        int lanes[kMaxT], rest[kMaxT], last[kMaxT], nlane = 0, nrest = 0, nlast = 0;
        uint32_t basis[3] = {0, 0, 0};
        for (int b = 0; b < T; ++b) {
            if (piv >> b & 1) continue;
            if (shared & spread(1u << b)) last[nlast++] = b;
            else if (bank_add(basis, banks[b])) lanes[nlane++] = b;
            else rest[nrest++] = b;
        }
        for (int k = 0; k < nrest; ++k) lanes[nlane++] = rest[k];
        if (nlane < 5) {  // too many: some are thread bits all the same
            for (int k = 0; k < nlast; ++k) {
                if (!bank_add(basis, banks[last[k]])) continue;
                std::copy_backward(lanes, lanes + nlane, lanes + nlane + 1);
                lanes[0] = last[k];
                ++nlane;
            }
            for (int k = 0; k < nlast; ++k)
                if (std::find(lanes, lanes + nlane, last[k]) == lanes + nlane)
                    lanes[nlane++] = last[k];
        } else {
            for (int k = 0; k < nlast; ++k) lanes[nlane++] = last[k];
        }
        for (int j = 0; j < nlane; ++j) {
            rd.lane[j] = (uint32_t)mswz((int)place_of[lanes[j]]) << 4;
            rd.lane_bit[j] = 1u << lanes[j];
        }
        rd.base = (uint32_t)mswz((int)place_base) << 4;
        rd.ncst = (int)place_cst.size();
        for (int j = 0; j < rd.ncst; ++j) {
            rd.cst_bit[j] = place_cst[j].first;
            rd.cst_vec[j] = (uint32_t)mswz((int)place_cst[j].second) << 4;
        }
        rd.nslot = (int)slots.size();
        // what a functional is over the elements, and at a thread's base
        uint64_t gp[4];
        for (int k = 0; k < 4; ++k) gp[k] = spread(reg[k]);
        auto elements = [&](uint64_t mask) {
            constexpr uint32_t on[4] = {0xAAAAu, 0xCCCCu, 0xF0F0u, 0xFF00u};  // elements with bit k
            uint32_t w = 0;
            for (int k = 0; k < 4; ++k) w ^= on[k] & (0u - (uint32_t)par(mask & gp[k]));
            return w;
        };
        auto thread_part = [&](uint64_t mask) { return mask & ~off_base; };
        auto tables = [&](const std::vector<Waiting::Item> &items, bool scalar, int &count,
                          int &first) {
            first = (int)tabs.size();
            count = 0;
            parts.clear();
            groups.clear();
            bool fixed = false;  // some item has no thread part
            for (const auto &it : items) {
                const uint64_t tp = thread_part(it.mask);
                int g = -1;
                if (tp) {
                    g = (int)(std::find(groups.begin(), groups.end(), tp) - groups.begin());
                    if (g == (int)groups.size()) groups.push_back(tp);
                }
                fixed = fixed || g < 0;
                parts.push_back(Part{g, elements(it.mask), it.z});
            }
            cd sc = scalar ? wait.scalar : cd(1.0);
            if (scalar) wait.scalar = 1.0;
            if (groups.size() > kMapParts) {
                // many thread parts: two factors made by the thread for each pattern over
                // the elements that has more than one item
                std::stable_sort(parts.begin(), parts.end(),
                                 [](const Part &x, const Part &y) { return x.group < y.group; });
                std::map<uint32_t, std::vector<MapItem>> by_word;
                for (const Part &p : parts)
                    if (p.group >= 0)
                        by_word[p.word].push_back(MapItem{groups[p.group], (double)p.z.real(),
                                                          (double)p.z.imag(), 0.0});
                for (auto &bw : by_word) {
                    if (bw.second.size() < 2 && bw.first != 0) continue;
                    MapTable tb{};
                    tb.kind = 1;
                    tb.data = (int)(data.size() / 2);
                    tb.count = (int)bw.second.size();
                    tb.word = bw.first;
                    const size_t o = data.size();
                    data.resize(o + bw.second.size() * sizeof(MapItem) / sizeof(double));
                    memcpy(data.data() + o, bw.second.data(), bw.second.size() * sizeof(MapItem));
                    tabs.push_back(tb);
                    ++count;
                    parts.erase(std::remove_if(parts.begin(), parts.end(),
                                               [&](const Part &p) {
                                                   return p.group >= 0 && p.word == bw.first;
                                               }),
                                parts.end());
                }
                // the groups that are left, in their order
                std::vector<uint64_t> kept;
                int last = -1;
                for (Part &p : parts) {
                    if (p.group < 0) continue;
                    if (p.group != last) {
                        last = p.group;
                        kept.push_back(groups[last]);
                    }
                    p.group = (int)kept.size() - 1;
                }
                groups.swap(kept);
            }
            // tables of up to kMapParts thread parts, the first with what depends on none
            int gi = 0;
            const int ng = (int)groups.size();
            bool first_table = true;
            while (gi < ng || (first_table && (fixed || sc != cd(1.0)))) {
                const int nv = std::min(kMapParts, ng - gi);
                MapTable tb{};
                tb.data = (int)(data.size() / 2);
                tb.count = nv;
                for (int q = 0; q < nv; ++q) tb.m[q] = groups[gi + q];
                // variants of no part first, then doubled with each part
                real fr[(1 << kMapParts) * kMapVariant], fi[(1 << kMapParts) * kMapVariant];
                auto times = [&](int k, const cd &z) {
                    const real x = fr[k], y = fi[k];
                    fr[k] = x * z.real() - y * z.imag();
                    fi[k] = x * z.imag() + y * z.real();
                };
                for (int e = 0; e < kMapVariant; ++e) {
                    fr[e] = first_table ? sc.real() : 1;
                    fi[e] = first_table ? sc.imag() : 0;
                }
                if (first_table && fixed)
                    for (const Part &p : parts)
                        for (int e = 0; p.group < 0 && e < kMapVariant; ++e)
                            if (p.word >> e & 1) times(e, p.z);
                for (int q = 0; q < nv; ++q) {
                    // a part's factors over the patterns of its items, then on the variants
                    // (elements where the pattern is 0 have them where the thread part is 1)
                    const int half = kMapVariant << q;
                    std::copy(fr, fr + half, fr + half);
                    std::copy(fi, fi + half, fi + half);
                    cd z[2][kMapVariant];  // 0: none
                    for (const Part &p : parts) {
                        if (p.group != gi + q) continue;
                        for (int e = 0; e < kMapVariant; ++e) {
                            cd &w = z[(p.word >> e & 1) ^ 1][e];
                            w = w == cd(0.0) ? p.z : mul(w, p.z);
                        }
                    }
                    for (int v = 0; v < 2; ++v)
                        for (int e = 0; e < kMapVariant; ++e)
                            if (z[v][e] != cd(0.0))
                                for (int k = 0; k < half; k += kMapVariant)
                                    times(v * half + k + e, z[v][e]);
                }
                const size_t o = data.size(), count_f = (size_t)kMapVariant << nv;
                data.resize(o + 2 * count_f);
                for (size_t k = 0; k < count_f; ++k) {
                    data[o + 2 * k] = (double)fr[k];
                    data[o + 2 * k + 1] = (double)fi[k];
                }
                tabs.push_back(tb);
                ++count;
                gi += nv;
                first_table = false;
            }
        };
        for (size_t k = 0; k < slots.size(); ++k) {
            const Slot &s = slots[k];
            MapSlot &d = rd.slot[k];
            const double sg = s.bflip ? -1.0 : 1.0;
            d.t0 = sg * s.t0;
            d.t1 = sg * s.t1;
            d.word = s.ctrl ? elements(s.ctrl) ^ (s.cflip ? 0xffffu : 0u) : 0u;
            d.mask = thread_part(s.ctrl);
            d.smask = thread_part(s.bit);
            d.sword = elements(s.bit);
            // (only elements with this register bit clear count)
            uint32_t lower = 0;
            for (int e = 0; e < 16; ++e)
                if (!(e >> k & 1)) lower |= 1u << e;
            d.kind = !s.ctrl && (d.sword & lower) == 0 ? 1 : 2;
            if (!s.ctrl) d.t1 = d.t0;
            // the waiting number joins a table that is there anyway, or has one made before
            // amplitudes that lack it could leave the range of doubles
            const real a = std::abs(wait.scalar);
            tables(s.tables, !s.tables.empty() || !(a > 1e-30 && a < 1e30), d.ntab, d.tab);
        }
        uint32_t in_warp = 0;  // tile bits that differ between threads of a warp
        for (int j = 0; j < std::min(nlane, 5); ++j) in_warp |= 1u << lanes[j];
        auto mark = [&](size_t from) {  // kinds 0 and 2
            for (size_t k = from; k < tabs.size(); ++k)
                for (int q = 0; q < tabs[k].count && tabs[k].kind == 0; ++q)
                    if (tabs[k].m[q] & spread(in_warp)) tabs[k].kind = 2;
        };
        mark(old_tabs);
        for (int k = 1; k < rd.nslot; ++k) {
            const MapSlot &d = rd.slot[k];
            if (d.ntab > 1 || (d.ntab && tabs[d.tab].kind != 0)) {
                tabs.resize(old_tabs);
                data.resize(old_data);
                wait.scalar = old_scalar;
                return k;
            }
        }
        bool line = rd.nslot > 0;
        for (int k = 0; k < rd.nslot; ++k) {
            const MapSlot &d = rd.slot[k];
            line = line && d.kind == 1 && d.ntab <= (k == 0 ? 1 : 0);
            if (d.ntab) line = line && tabs[d.tab].kind == 0;
        }
        if (!line && rd.nslot) {
            MapSlot &d = rd.slot[0];
            rd.pre = d.tab;
            rd.npre = d.ntab;
            if (d.ntab && tabs[d.tab + d.ntab - 1].kind == 0) {
                --rd.npre;
                d.tab += d.ntab - 1;
            } else {  // (the straight line wants one)
                d.tab = (int)tabs.size();
                MapTable tb{};
                tb.data = (int)(data.size() / 2);
                for (int e = 0; e < kMapVariant; ++e) data.push_back(1.0), data.push_back(0.0);
                tabs.push_back(tb);
            }
            d.ntab = 1;
        }
        if (tail) {
            tables(wait.items, true, rd.ntail, rd.tail);
            wait.clear();
            mark((size_t)rd.tail);
        }
        for (int k = 0; k < rd.nslot; ++k) rd.signs |= rd.slot[k].smask != 0;
        if (line) rd.path = rd.nslot + (rd.slot[0].ntab ? 0 : 4);
        rd.bases = !line || rd.signs || rd.ntail;
        rounds.push_back(rd);
        return slots.size();
    }

    size_t bytes() const {
        return sizeof(MapStore) + rounds.size() * sizeof(MapRound) +
               tabs.size() * sizeof(MapTable) + data.size() * sizeof(double);
    }

    // End of the pass: its launch.
    void finish(MapProgram &out) {
        MapStore st{};
        for (int b = 0; b < T; ++b) st.vec[b] = (uint32_t)mswz((int)place_of[b]) << 4;
        st.base = (uint32_t)mswz((int)place_base) << 4;
        st.ncst = (int)place_cst.size();
        for (int j = 0; j < st.ncst; ++j) {
            st.cst_bit[j] = place_cst[j].first;
            st.cst_vec[j] = (uint32_t)mswz((int)place_cst[j].second) << 4;
        }
        MapStep step{};
        step.fused = true;
        step.pass.h = h;
        step.pass.nrounds = (int)rounds.size();
        step.pass.ntabs = (int)tabs.size();
        step.pass.offset = out.blob.size();
        step.pass.bytes = bytes();
        out.blob.resize((out.blob.size() + step.pass.bytes + 255) / 256 * 256, 0);
        unsigned char *p = out.blob.data() + step.pass.offset;
        auto put = [&](const void *src, size_t k) {
            if (k) memcpy(p, src, k);
            p += k;
        };
        put(&st, sizeof(st));
        put(rounds.data(), rounds.size() * sizeof(MapRound));
        put(tabs.data(), tabs.size() * sizeof(MapTable));
        put(data.data(), data.size() * sizeof(double));
        out.steps.push_back(step);
        out.rounds += (int)rounds.size();
    }

private:
    void begin_round() {
        for (int b = 0; b < T; ++b) vec[b] = 1u << b, row[b] = 1ull << global_pos(b, h);
        std::fill(flip, flip + kMaxT, 0);
        base = 0;
        cst.clear();
    }

    uint32_t place(uint32_t v) const {  // of a vector over the round's first indices
        uint32_t p = 0;
        for (int b = 0; b < T; ++b)
            if (v >> b & 1) p ^= place_of[b];
        return p;
    }

    // The round's permutations join the map, and the waiting factors are written over
    // the indices that they leave.
    void begin_next() {
        // col[j]: what a mask's tile bit j becomes; bit 63 stands for a factor turned round
        constexpr uint64_t kTurn = 1ull << 63;
        uint64_t col[kMaxT];
        for (int j = 0; j < T; ++j) {
            uint64_t c = base >> j & 1 ? kTurn : 0;
            for (int b = 0; b < T; ++b)
                if (vec[b] >> j & 1) c |= 1ull << global_pos(b, h);
            for (auto &x : cst)
                if (x.second >> j & 1) c ^= 1ull << x.first;
            col[j] = c;
        }
        const uint64_t in = window_mask(h, m);
        const bool twice = wait.twice;
        later.swap(wait.items);
        wait.clear();
        for (const auto &it : later) {
            uint64_t mk = it.mask & ~in;
            for (uint64_t x = it.mask & in; x; x &= x - 1)
                mk ^= col[local_pos(__builtin_ctzll(x), h)];
            const bool turn = mk & kTurn;
            mk &= ~kTurn;
            // (the map is one to one: masks meet only if they did before)
            if (twice) {
                wait.add1(mk, turn, it.z, 0);
            } else if (it.z != cd(1.0)) {
                cd z = it.z;
                if (turn) {
                    wait.scalar = mul(wait.scalar, z);
                    z = inverse(z);
                }
                wait.see(mk);
                wait.items.push_back(Waiting::Item{mk, z, 0});
            }
        }
        uint32_t next[kMaxT];
        for (int b = 0; b < T; ++b) next[b] = place(vec[b]);
        place_base ^= place(base);
        for (auto &c : cst) {
            auto it = std::find_if(place_cst.begin(), place_cst.end(),
                                   [&](auto &x) { return x.first == c.first; });
            if (it == place_cst.end()) place_cst.push_back({c.first, place(c.second)});
            else it->second ^= place(c.second);
        }
        std::copy(next, next + T, place_of);
        begin_round();
    }

    uint32_t bank(int b) const { return (uint32_t)mswz((int)place_of[b]) & 7u; }

    static bool bank_add(uint32_t (&basis)[3], uint32_t v) {
        for (int k = 2; k >= 0 && v; --k) {
            if (!(v >> k & 1)) continue;
            if (!basis[k]) {
                basis[k] = v;
                return true;
            }
            v ^= basis[k];
        }
        return false;
    }
    // How many of the banks' three dimensions the bits not yet taken span.
    struct Ranks {
        int count[8] = {0}, present = 0;  // free bits by bank
        void free(uint32_t v) { present |= 1 << v, ++count[v]; }
        void take(uint32_t v) {
            if (--count[v] == 0) present &= ~(1 << v);
        }
        int without(uint32_t v) const { return rank(count[v] > 1 ? present : present & ~(1 << v)); }
        static int rank(int set) {  // of vectors 0-7
            static const auto table = [] {
                std::array<unsigned char, 256> t{};
                for (int s = 0; s < 256; ++s) {
                    uint32_t basis[3] = {0, 0, 0};
                    for (uint32_t v = 0; v < 8; ++v) t[s] += (s >> v & 1) && bank_add(basis, v);
                }
                return t;
            }();
            return table[set];
        }
    };
    // Gaussian elimination: a pivot bit for v that no earlier vector has, chosen so that
    // the bits left to the threads keep spanning the banks.
    struct Reduced {  // vectors and their pivots
        uint32_t v[4];
        int at[4], n = 0;
    };
    void add_pivot(Reduced &red, Ranks &ranks, uint32_t &piv, uint32_t v) const {
        for (int k = 0; k < red.n; ++k)
            if (v >> red.at[k] & 1) v ^= red.v[k];
        int best = -1, best_rank = -1;
        for (int b = T - 1; b >= 0; --b) {
            if (!(v >> b & 1)) continue;
            const int rk = ranks.without(banks[b]);
            if (rk > best_rank) best = b, best_rank = rk;
        }
        ranks.take(banks[best]);
        for (int k = 0; k < red.n; ++k)
            if (red.v[k] >> best & 1) red.v[k] ^= v;
        red.v[red.n] = v;
        red.at[red.n++] = best;
        piv |= 1u << best;
    }

    int n, T, m, h = 4;
    Waiting &wait;
    // the map at the round's start: places of the logical tile bits, of index 0, and of
    // outside bits
    uint32_t place_of[kMaxT];
    uint32_t banks[kMaxT];  // and their banks, while a round is written
    uint32_t place_base = 0;
    std::vector<std::pair<int, uint32_t>> place_cst;
    // the round's permutations so far, over the indices at its start: what each logical
    // bit's vector and functional have become
    uint32_t vec[kMaxT];
    uint64_t row[kMaxT];
    int flip[kMaxT];
    uint32_t base = 0;
    std::vector<std::pair<int, uint32_t>> cst;
    std::vector<Waiting::Item> later;  // begin_next's
    struct Split {                     // diagonal()'s factors of the bits and of their sum
        cd z0, z1, z2;
    };
    Recent<Split> splits;
    struct Part {                      // a table's factor: emit_round's
        int group;                     // its thread part, -1: none
        uint32_t word;                 // its pattern over the elements
        cd z;
    };
    std::vector<Part> parts;
    std::vector<uint64_t> groups;      // thread parts
    std::vector<MapRound> rounds;
    std::vector<MapTable> tabs;
    std::vector<double> data;
};

// (Its host time is in every call with new angles: ten Trotter steps of 19 qubits, 730 gates,
// 0.86 ms, 235 gates of 16-qubit brickwork 0.18; with GateOp records in every op, vectors per
// round and the complex library's operators 2.25 and 0.48, more than the rounds save there.)
bool map_plan(const std::vector<GateOp> &gops, int n, int T, MapProgram &out, bool always) {
    // A controlled rotation is a whole rotation and a table here, and one record there; RXX and
    // RYY are two such rotations in one.  Whether the rest of the circuit makes up for them
    // depends on the size (times of 60 to 200 gates submitted again, here against there).
    // Up to 10 qubits, a few dozen threads, next to none: controlled rotations a tenth of the
    // gates 85 us against 68, four Trotter steps, half of whose gates are RXX and RYY, 150
    // against 118 on 6 qubits and 228 against 231 on 10.  Up to 19 qubits a sixth of controlled
    // rotations (15 %, 16 qubits: 119 against 140; 20 % with new angles 325 against 293) and
    // half of RXX and RYY (Trotter steps of 11 to 19 qubits: 203 against 280, 340 against 395,
    // 481 against 638; 60 % with new angles 556 against 392).  Above, a fifth and any number (26
    // qubits: 40 CRX and CRY alone 4.55 ms against 3.76; 40 RXX and RYY alone 3.9 against 4.3).
    size_t controlled = 0, blocks = 0;
    for (const GateOp &g : gops) {
        controlled += g.type == OP_M1 && g.nctrl > 0;
        blocks += g.type == OP_M2;
    }
    if (!always &&
        (n <= 10  ? 12 * (controlled + blocks) > gops.size()
         : n < 20 ? 6 * controlled > gops.size() || 2 * (controlled + blocks) > gops.size()
                  : 5 * controlled > gops.size()))
        return false;
    std::vector<MapOp> ops;
    std::vector<MapUnit> units;
    std::vector<PlanStep> steps;
    if (!map_lower(gops, n, T, ops, units, steps)) return false;
    // the last pass takes what still waits (sweeps after it only move amplitudes)
    size_t last = steps.size();
    for (size_t si = 0; si < steps.size(); ++si)
        if (steps[si].fused) last = si;
    out.T = T;
    Waiting wait;
    PassBuilder pb(n, T, wait);
    for (size_t si = 0; si < steps.size(); ++si) {
        const PlanStep &st = steps[si];
        if (!st.fused) {
            // a SWAP across windows: its own sweep; what waits changes bits with it
            MapStep ms{};
            ms.fused = false;
            ms.gate = *units[st.gate].swap;
            out.steps.push_back(ms);
            for (auto &it : wait.items) {
                const uint64_t x = it.mask >> ms.gate.b0 & 1, y = it.mask >> ms.gate.b1 & 1;
                if (x != y) it.mask ^= 1ull << ms.gate.b0 | 1ull << ms.gate.b1;
                wait.see(it.mask);
            }
            continue;
        }
        std::vector<int> left;
        for (int u : st.pass.gates)
            for (int i = units[u].begin; i < units[u].end; ++i) left.push_back(i);
        bool closed = false;
        pb.begin(st.pass.h);
        while (!left.empty()) {
            size_t keep = 0;
            uint64_t blk = 0;
            for (int i : left) {
                const MapOp &o = ops[i];
                bool done = false;
                if (!(o.bits & blk)) {
                    if (o.kind == MO_PERM || o.kind == MO_SWAP) done = pb.permute(o);
                    else if (o.kind == MO_DIAG) pb.diagonal(o, pb.round_slots()), done = true;
                    else done = pb.rotate(o);
                }
                if (!done) {
                    left[keep++] = i;
                    blk |= o.bits;
                }
            }
            const bool stuck = keep == left.size();
            left.resize(keep);
            // (in its last round, if there is room)
            closed = left.empty() && si == last && pb.bytes() <= kMapProgram / 2;
            pb.close_round(closed);
            // a map or program that is full: the pass ends here and goes on as another
            // over the same window
            if (!left.empty() && (stuck || pb.bytes() > kMapProgram)) {
                pb.finish(out);
                pb.begin(st.pass.h);
            }
        }
        if (si == last && !closed) {
            if (pb.bytes() > kMapProgram) {
                pb.finish(out);
                pb.begin(st.pass.h);
            }
            pb.close_round(true);
        }
        pb.finish(out);
    }
    // (a number from sweeps alone)
    if (!wait.items.empty() || wait.scalar != cd(1.0)) {
        pb.begin(4);
        pb.close_round(true);
        pb.finish(out);
    }
    for (const MapStep &s : out.steps)
        if (s.fused && s.pass.bytes > kMapLargest) return false;
    return true;
}

// ---------------------------------------------------------------------------
// Host: launch
// ---------------------------------------------------------------------------
template <int BYTES>
static cudaError_t map_launch_t(lq_state *s, int T, const MapLaunch &ps,
                                const unsigned char *blob) {
    MapParam<BYTES> param;
    memcpy(param.b, blob + ps.offset, ps.bytes);
    const cudaError_t e = cudaFuncSetAttribute(
        k_mapped_pass<BYTES>, cudaFuncAttributeMaxDynamicSharedMemorySize, 16 << kMaxT);
    if (e != cudaSuccess) return e;
    k_mapped_pass<BYTES><<<1u << (s->n - T), 1u << (T - 4), (size_t)16 << T, s->stream>>>(
        (double2 *)s->d, T, ps.h, ps.nrounds, ps.ntabs, (int)ps.bytes, param);
    return cudaGetLastError();
}

int map_launch(lq_state *s, int T, const MapLaunch &ps, const unsigned char *blob) {
    prof_begin(s->stream, kProfFused);
    // (a launch copies its parameters: small programs take the small kernel)
    const cudaError_t e = ps.bytes <= 4096    ? map_launch_t<4096>(s, T, ps, blob)
                          : ps.bytes <= 12288 ? map_launch_t<12288>(s, T, ps, blob)
                                              : map_launch_t<(int)kMapLargest>(s, T, ps, blob);
    prof_end(s->stream, kProfFused);
    LQ_CUDA_TRY(e);
    return LQ_OK;
}

}  // namespace lq
