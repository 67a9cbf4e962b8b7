// Precision form: complex64 state, gates fused into 5-qubit blocks applied as
// complex 32x32 GEMMs on the 5th-generation tensor cores (tcgen05, TF32 inputs,
// FP32 accumulation in tensor memory) with the 3xTF32 split
//     X W ~= Xh Wh + Xh Wl + Xl Wh,   Xh = tf32(X), Xl = tf32(X - Xh).
//
// A pass owns a window of T = 12 index bits ([0,4) U [h, h+8), as the FP64
// fused passes) and applies its 5-qubit blocks to every 2^12-amplitude
// complex64 tile (32 KiB, TMA with 128-byte swizzle).  For a block on tile bits
// k0..k4 the tile is a 128 x 32 complex matrix X (rows: the other seven tile
// bits; columns: the block index).  Viewed as reals interleaved (re, im) it is
// X' (128 x 64) and the block is Y' = X' W' with the real 64 x 64 matrix
// W' = [[Re U^T, Im U^T], [-Im U^T, Re U^T]] interleaved the same way.
//
// GEMM row m is also tensor-memory lane m.  Two threads share a row, each with half of
// its columns: they split them into TF32 hi / lo parts and write them to tensor memory
// (tcgen05.st); one elected thread issues 3 x 8 tcgen05.mma (K = 8 each) with A read from
// tensor memory and B (W' hi / lo, prepared on the host in the swizzled K-major byte
// order) from shared memory, into a 128-lane x 64-column FP32 accumulator; the threads
// read it back with tcgen05.ld and scatter it into the tile.
//
// Bound: per SM a block of a tile takes some 860 cycles of the tensor pipe, 700 issue
// slots per scheduler and 1000 cycles of shared memory (the tile read and written, B read
// by the products); its chain split -> products -> read back is some 3000.  So tiles must
// overlap.  Tensor memory holds 512 columns, and a tile needs 128 for A from the split to
// the end of its products and 64 for D from their start to the read back: three groups of
// 256 threads, each with its tile and its A region, take turns on two D regions.  (Two A
// regions and three of D: 3 % slower.)  A CTA per SM is persistent.  One further warp moves tiles through five buffers, another brings
// the B images (32 KiB) for all groups into two slots, where up to two blocks stay for the
// whole pass.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <complex>
#include <cstring>
#include <mutex>

#include "fused_plan.h"

namespace lq {

constexpr int kTcT = 12;                  // tile bits
constexpr int kTcGroup = 256;             // two threads per GEMM row = TMEM lane
constexpr int kTcGroups = 3;
constexpr int kTcThreads = kTcGroups * kTcGroup + 64;  // and two warps that move tiles and B
constexpr int kTcBuffers = 5;              // tiles in shared memory (one more for one block)
constexpr int kTcSlots = 2;                // B images
constexpr uint32_t kTileBytes = 8u << kTcT;  // 32 KiB complex64 tile
constexpr uint32_t kBBytes = 64 * 64 * 4;    // 16 KiB per B part (hi / lo)
// shared memory: tiles, B images, barriers
constexpr uint32_t kTcSmem = kTcBuffers * kTileBytes + kTcSlots * 2 * kBBytes + 1024 + 256;
static_assert(kTcSmem + 1024 <= 227 * 1024, "one CTA per SM");
// tensor memory columns: the groups' A, hi [0,64) and lo [64,128), then two D regions (FP32
// accumulator), 64 each
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColA = 128, kColAl = 64, kColD = 384;

struct TcBlock {
    uint32_t row[7];    // byte offset in the tile of each row bit
    uint32_t col[5];    // and of each block index bit
    uint32_t pair;      // block bit 0 is tile bit 0: columns 2c, 2c+1 are 16 bytes
    uint32_t b_offset;  // of the block's 32 KiB B image (hi then lo), in bytes / 16
    uint32_t pad[2];
};
static_assert(sizeof(TcBlock) == 64, "read in four pieces");

static bool tc_restore_norm() {
    static const int v = [] {
        const char *e = getenv("LQ_TC_RENORM");
        return e ? atoi(e) : 1;
    }();
    return v != 0;
}

struct TcPass {
    int32_t h;
    int32_t block_begin, nblocks;
    int32_t pad;
};

__device__ __forceinline__ uint32_t tc_smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Byte offset of complex64 tile element l in the TMA 128-byte-swizzled tile: 128-byte rows
// hold 16 amplitudes (bits 0-3), 16-byte chunks hold 2; the row's number has tile bits
// 9-11 lowest, so that these are the ones that the swizzle adds to the chunk.  A block on
// neighbouring low bits then leaves its rows on different banks (with bits 4-6 there, a
// block on bits 0-4 or 1-5 had up to four-way conflicts).  Linear over XOR.
__host__ __device__ __forceinline__ uint32_t tile_off(uint32_t l) {
    const uint32_t row = (l >> 9) | (((l >> 4) & 31) << 3), chunk = (l & 15) >> 1;
    return row * 128 + ((chunk ^ (row & 7)) << 4) + ((l & 1) << 3);
}

// Round a finite FP32 value to TF32 (10 explicit mantissa bits), to nearest with
// ties away from zero: add half a unit of the last kept place (bit 12) to the
// IEEE bit pattern and clear the 13 dropped bits.  The pattern is
// sign-magnitude, so the same addition rounds negative values by magnitude, and
// a carry out of the mantissa steps into the next binade as rounding up should.
// Two integer operations instead of a conversion sequence that also handles
// NaN and infinity, which amplitudes (magnitude at most 1) never are.
__device__ __forceinline__ float to_tf32(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}

__device__ __forceinline__ uint64_t make_sdesc(uint32_t addr, uint32_t sbo_bytes) {
    // tcgen05 shared-memory descriptor: start address >> 4 [0,14), leading
    // byte offset (unused for swizzled K-major, 1) [16,30), stride byte offset
    // >> 4 [32,46), version 1 [46,48), layout SWIZZLE_128B (2) [61,64).
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < (1u << 24); ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Instruction descriptor: D f32, A/B tf32, both K-major, N = 64, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((64u >> 3) << 17) |
                            ((128u >> 4) << 24);

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, "
        "%10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
        "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
        "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])),
        "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
        "r"(__float_as_uint(v[15]))
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, "
        "%10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float4 lds4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(a)
                 : "memory");
    return v;
}
__device__ __forceinline__ float2 lds2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts4(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z),
                 "f"(w)
                 : "memory");
}
__device__ __forceinline__ void sts2(uint32_t a, float x, float y) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}

// Byte offset in the tile of the thread's column c (0..15 of its half), over XOR, from its
// row's first.
struct TcCols {
    uint32_t b[4];
    __device__ __forceinline__ uint32_t off(int c) const {
        return ((c & 1) ? b[0] : 0u) ^ ((c & 2) ? b[1] : 0u) ^ ((c & 4) ? b[2] : 0u) ^
               ((c & 8) ? b[3] : 0u);
    }
};

template <bool PAIR>
__device__ __forceinline__ void tc_read(uint32_t tile, uint32_t at, const TcCols &cols,
                                        float (&x)[32]) {
#pragma unroll
    for (int c = 0; c < 16; c += 2) {
        if (PAIR) {
            const float4 v = lds4(tile + (at ^ cols.off(c)));
            x[2 * c] = v.x, x[2 * c + 1] = v.y, x[2 * c + 2] = v.z, x[2 * c + 3] = v.w;
        } else {
            const float2 v = lds2(tile + (at ^ cols.off(c)));
            const float2 w = lds2(tile + (at ^ cols.off(c + 1)));
            x[2 * c] = v.x, x[2 * c + 1] = v.y, x[2 * c + 2] = w.x, x[2 * c + 3] = w.y;
        }
    }
}

__device__ __forceinline__ void tc_split(const float (&x)[32], uint32_t tm) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        float hi[16], lo[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            hi[u] = to_tf32(x[16 * q + u]);
            lo[u] = to_tf32(x[16 * q + u] - hi[u]);
        }
        tmem_st16(tm + q * 16, hi);
        tmem_st16(tm + kColAl + q * 16, lo);
    }
}

__device__ __forceinline__ bool tc_elect() {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r));
    return r != 0;
}

// The row's half from D, which is free for other products then (bar), into the tile.
template <bool PAIR>
__device__ __forceinline__ void tc_back(uint32_t tile, uint32_t at, const TcCols &cols,
                                        uint32_t tm, uint32_t bar) {
    float d[2][16];
#pragma unroll
    for (int q = 0; q < 2; ++q) tmem_ld16(tm + q * 16, d[q]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(d[q][i]));  // (read after the wait)
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (tc_elect()) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
            const uint32_t p = tile + (at ^ cols.off(q * 8 + c));
            if (PAIR) {
                sts4(p, d[q][2 * c], d[q][2 * c + 1], d[q][2 * c + 2], d[q][2 * c + 3]);
            } else {
                sts2(p, d[q][2 * c], d[q][2 * c + 1]);
                sts2(tile + (at ^ cols.off(q * 8 + c + 1)), d[q][2 * c + 2], d[q][2 * c + 3]);
            }
        }
}

// Whether any thread of the group says so: the same answer for all of them.
__device__ __forceinline__ bool tc_any(int g, bool x) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)x), "r"(1 + g), "n"(kTcGroup)
        : "memory");
    return r != 0;
}

// The CTA's tiles are blockIdx.x + q gridDim.x, q = 0, 1, ...; group q % 3 takes tile q in
// buffer q mod their number.  Step s = 3 j + g is the j-th block of group g in all its
// tiles; it uses D region s % 2, when that of step s - 2 was read.  A group without a tile in
// the last round goes through its steps without work.
// Every barrier is awaited, phase by phase, by the same threads: a phase's parity alone
// does not tell it from the one two before or after.  So there are two barriers per group
// and purpose, in turn: a group's next step, or tile, may be done before the last is seen.
// Waits are bounded; one that ran out is carried to the group's next barrier, where all its
// threads leave.  The others of the CTA then run into their own limits.
// The operands of the products are the same for the warp and known to be (shfl): else each
// took a loop over the warp's values, 83 cycles instead of the tensor pipe's 36.
__global__ void __launch_bounds__(kTcThreads, 1)
    k_tc_pass(const __grid_constant__ CUtensorMap tmap, int32_t h, int32_t ntiles,
              const TcBlock *__restrict__ blocks, int nblocks,
              const unsigned char *__restrict__ bimg, unsigned *__restrict__ flag) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t tiles = (tc_smem_u32(smem_raw) + 1023u) & ~1023u;
    // (slots from the end: a pass of one block has the other for a sixth tile)
    const uint32_t images = tiles + (kTcBuffers + kTcSlots - 1) * kTileBytes;  // B: hi, then lo
    const uint32_t bars = images + kTileBytes;
    const uint32_t bar_load = bars;                          // [2][group]: a tile is there
    const uint32_t bar_mma = bar_load + 16 * kTcGroups;      // [2][group]: products are done
    const uint32_t bar_read = bar_mma + 16 * kTcGroups;      // [2][group]: and D was read
    const uint32_t bar_done = bar_read + 16 * kTcGroups;     // [2][group]: a tile is finished
    const uint32_t bar_full = bar_done + 16 * kTcGroups;     // [slot]: the image is there
    const uint32_t bar_free = bar_full + 8 * kTcSlots;       // [slot]: all groups are done
    const int nbuf = nblocks == 1 ? kTcBuffers + 1 : kTcBuffers;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int32_t zero = 0;
    const bool resident = nblocks <= kTcSlots;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         tc_smem_u32(&tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        constexpr int all = 8 * kTcGroups + kTcSlots;
        for (int i = 0; i < all + kTcSlots; ++i) {
            const bool warps = i >= 4 * kTcGroups && i < 6 * kTcGroups;  // bar_read
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars + 8u * i),
                         "r"(i >= all ? kTcGroups : warps ? kTcGroup / 32 : 1)
                         : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    const int mine = (int)blockIdx.x < ntiles
                         ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;  // tiles
    const int rounds = (mine + kTcGroups - 1) / kTcGroups;
    // event k of group g (a tile or a step) on one of its two barriers
    auto of = [&](uint32_t bar, int g, int k) { return bar + 8u * (g + kTcGroups * (k & 1)); };
    auto seen = [&](uint32_t bar, int g, int k) {
        return tc_wait(of(bar, g, k), (uint32_t)(k >> 1) & 1u);
    };
    auto arrive = [&](uint32_t bar) {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
    };

    if (warp == kTcGroups * kTcGroup / 32) {
        // ---- the B images, in the order of use
        if ((tid & 31) == 0) {
            const int total = nblocks * (resident ? std::min(rounds, 1) : rounds);
            int slot = 0, use = 0, bi = 0, sent = 0;
            bool bad = false;
            for (; sent < total; ++sent) {
                if (use > 0 && !tc_wait(bar_free + 8u * slot, (uint32_t)(use - 1) & 1u)) {
                    bad = true;
                    break;
                }
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                 bar_full + 8u * slot),
                             "r"(2 * kBBytes)
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes"
                    " [%0], [%1], %2, [%3];" ::"r"(images - slot * 2 * kBBytes),
                    "l"((uint64_t)(bimg + ((uint64_t)blocks[bi].b_offset << 4))),
                    "r"(2 * kBBytes), "r"(bar_full + 8u * slot)
                    : "memory");
                if (++bi == nblocks) bi = 0;
                if (++slot == kTcSlots) slot = 0, ++use;
            }
            // the copies have landed before the CTA's memory is released
            for (int k = std::max(0, sent - kTcSlots); k < sent; ++k)
                bad |= !tc_wait(bar_full + 8u * (k % kTcSlots), (uint32_t)(k / kTcSlots) & 1u);
            if (bad) atomicOr(flag, kFlagTimeout);
        }
    } else if (warp == kTcGroups * kTcGroup / 32 + 1) {
        // ---- the tiles: a finished one is stored, and its buffer loaded again
        if ((tid & 31) == 0) {
            auto coords = [&](int q, int32_t &c1, int32_t &c3) {
                const int t = (int)blockIdx.x + q * (int)gridDim.x;
                c1 = t & ((1 << (h - 4)) - 1), c3 = t >> (h - 4);
            };
            bool bad = false;
            int asked = 0;
            for (int q = 0; q < mine + nbuf; ++q) {
                const uint32_t buf = tiles + (uint32_t)(q % nbuf) * kTileBytes;
                int32_t c1, c3;
                if (q >= nbuf && q - nbuf < mine) {
                    if (!seen(bar_done, (q - nbuf) % kTcGroups, (q - nbuf) / kTcGroups)) {
                        bad = true;
                        break;
                    }
                    coords(q - nbuf, c1, c3);
                    asm volatile(
                        "cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group"
                        " [%0, {%1, %1, %1, %2, %3}], [%4];" ::"l"((uint64_t)&tmap),
                        "r"(zero), "r"(c1), "r"(c3), "r"(buf)
                        : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                if (q < mine) {
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    const uint32_t bar = of(bar_load, q % kTcGroups, q / kTcGroups);
                    coords(q, c1, c3);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                                 "r"(kTileBytes)
                                 : "memory");
                    asm volatile(
                        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx"
                        "::bytes [%0], [%1, {%2, %2, %2, %3, %4}], [%5];" ::"r"(buf),
                        "l"((uint64_t)&tmap), "r"(zero), "r"(c1), "r"(c3), "r"(bar)
                        : "memory");
                    asked = q + 1;
                }
            }
            if (bad) {
                atomicOr(flag, kFlagTimeout);
                for (int q = std::max(0, asked - nbuf); q < asked; ++q)
                    seen(bar_load, q % kTcGroups, q / kTcGroups);
            }
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else {
        const int g = warp / (kTcGroup / 32), gtid = tid & (kTcGroup - 1);
        const int half = gtid >> 7, row = gtid & 127;
        const uint32_t lane = ((uint32_t)(row & ~31) << 16) + 32u * half;
        const uint32_t tm_a = tmem + kColA * g;
        // step s - 2: of the next group but one, a step earlier unless that is group 0
        const int before = (g + 1) % kTcGroups, later = g >= 2 ? 0 : 1;
        int slot = 0;
        uint32_t full_phase = 0;
        int step = 0;
        auto next_slot = [&] {
            if (++slot == (resident ? nblocks : kTcSlots)) slot = 0, full_phase ^= resident ? 0u : 1u;
        };
        bool bad = false;
        const uint4 *desc = (const uint4 *)blocks;
        for (int j = 0; j < rounds; ++j) {
            const int q = j * kTcGroups + g;
            if (q >= mine) {  // (the last round)
                if (gtid == 0)
                    for (int bi = 0; bi < nblocks; ++bi, ++step) {
                        if (step >= later && !seen(bar_read, before, step - later)) break;
                        if (!resident) {
                            if (!tc_wait(bar_full + 8u * slot, full_phase)) break;
                            arrive(bar_free + 8u * slot);
                            next_slot();
                        }
                        for (int w = 0; w < kTcGroup / 32; ++w) arrive(of(bar_read, g, step));
                    }
                break;
            }
            const uint32_t tile = tiles + (uint32_t)(q % nbuf) * kTileBytes;
            bad = !seen(bar_load, g, j);
            uint4 d0 = __ldg(desc), d1 = __ldg(desc + 1), d2 = __ldg(desc + 2), d3 = __ldg(desc + 3);
            for (int bi = 0; bi < nblocks; ++bi, ++step) {
                auto on = [&](int j) { return 0u - ((uint32_t)(row >> j) & 1u); };
                const uint32_t at = (d0.x & on(0)) ^ (d0.y & on(1)) ^ (d0.z & on(2)) ^
                                    (d0.w & on(3)) ^ (d1.x & on(4)) ^ (d1.y & on(5)) ^
                                    (d1.z & on(6)) ^ (half ? d2.w : 0u);
                const TcCols cols{{d1.w, d2.x, d2.y, d2.z}};
                const bool pair = d3.x != 0;
                const uint32_t tm_d = tmem + kColD + 64u * ((step + g) & 1);
                float x[32];
                if (pair) tc_read<true>(tile, at, cols, x);
                else tc_read<false>(tile, at, cols, x);
                __syncwarp();  // the .aligned instructions want the warp together
                tc_split(x, tm_a + lane);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(kTcGroup) : "memory");
                if (warp == g * (kTcGroup / 32)) {
                    bad |= !tc_wait(bar_full + 8u * slot, full_phase);
                    if (step >= later) bad |= !seen(bar_read, before, step - later);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t bh = images - slot * 2 * kBBytes;
                    const uint64_t d64 = make_sdesc(bh, 1024);
                    const uint32_t dl = __shfl_sync(0xffffffffu, (uint32_t)d64, 0);
                    const uint32_t dhi = __shfl_sync(0xffffffffu, (uint32_t)(d64 >> 32), 0);
                    const uint32_t td = __shfl_sync(0xffffffffu, tm_d, 0);
                    const uint32_t done = __shfl_sync(0xffffffffu, of(bar_mma, g, step), 0);
                    const uint32_t freed = __shfl_sync(0xffffffffu, bar_free + 8u * slot, 0);
                    if (!__any_sync(0xffffffffu, bad) && tc_elect()) {
#pragma unroll
                        for (int prod = 0; prod < 3; ++prod) {
                            // hi.Bhi + hi.Blo + lo.Bhi
                            const uint32_t acol = prod == 2 ? kColAl : 0u;
#pragma unroll
                            for (int kk = 0; kk < 8; ++kk) {
                                const uint32_t boff =
                                    (prod == 1 ? kBBytes : 0u) + (kk >> 2) * (64 * 128) + (kk & 3) * 32;
                                const uint64_t db = (uint64_t)dhi << 32 | (dl + (boff >> 4));
                                const uint32_t acc = (prod | kk) ? 1u : 0u;
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\t"
                                    "setp.ne.b32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::
                                        "r"(td),
                                    "r"(tm_a + acol + kk * 8), "l"(db), "r"(kIdesc), "r"(acc)
                                    : "memory");
                            }
                        }
                        asm volatile(
                            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 "
                            "[%0];" ::"r"(done)
                            : "memory");
                        if (!resident)
                            asm volatile(
                                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster"
                                ".b64 [%0];" ::"r"(freed)
                                : "memory");
                    }
                    __syncwarp();
                }
                // (the next block's descriptor, while the products run)
                const uint4 *dn = desc + 4 * (bi + 1 < nblocks ? bi + 1 : 0);
                d0 = __ldg(dn), d1 = __ldg(dn + 1), d2 = __ldg(dn + 2), d3 = __ldg(dn + 3);
                bad |= !seen(bar_mma, g, step);
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (pair) tc_back<true>(tile, at, cols, tm_d + lane, of(bar_read, g, step));
                else tc_back<false>(tile, at, cols, tm_d + lane, of(bar_read, g, step));
                if (bi + 1 == nblocks) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                bad = tc_any(g, bad);
                if (bad) break;
                next_slot();
            }
            if (bad) break;
            if (gtid == 0) arrive(of(bar_done, g, j));
        }
        if (bad && gtid == 0) {
            atomicOr(flag, kFlagTimeout);
            // let products in flight finish before the CTA's memory is released
            seen(bar_mma, g, step);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmemCols)
                     : "memory");
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 tc_encode() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

// complex64 tile map for the window [0,4) U [h, h+8):
//   dim0: 32 floats (16 amplitudes, bits 0-3), box 32 (128 B)
//   dim1: 2^3 (bits h+5..h+7), box 8
//   dim2: 2^5 (bits h..h+4), box 32
//   dim3: 2^(h-4) (bits 4..h-1), box 1
//   dim4: 2^(n-h-8) (bits h+8..), box 1
static int tc_tile_map(CUtensorMap *map, void *d, int n, int h) {
    auto enc = tc_encode();
    if (!enc) return set_error(LQ_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
    cuuint64_t dims[5] = {32, 8, 32, 1ull << (h - 4), 1ull << (n - h - 8)};
    cuuint64_t strides[4] = {8ull << (h + 5), 8ull << h, 128, 8ull << (h + 8)};
    cuuint32_t box[5] = {32, 8, 32, 1, 1};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, d, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return set_error(LQ_ERR_CUDA, "cuTensorMapEncodeTiled (complex64) failed (%d)", (int)r);
    return LQ_OK;
}

using cd = std::complex<double>;

// SM count of the current device (persistent grid: one CTA per SM).
static int tc_sm_count() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(sms, 1);
}

// Apply canonical op g (global index bits) to a 32-dim vector whose block bit j
// corresponds to global bit gbit[j].
static void small_apply(const GateOp &g, const int gbit[5], cd *v) {
    auto loc = [&](int b) {
        for (int j = 0; j < 5; ++j)
            if (gbit[j] == b) return j;
        return -1;
    };
    auto c = [&](int k) { return cd(g.m[2 * k], g.m[2 * k + 1]); };
    switch (g.type) {
    case OP_M1:
    case OP_PERM1: {
        const int t = loc(g.t);
        int cm = 0;
        for (int k = 0; k < g.nctrl; ++k) cm |= 1 << loc(g.ctrl[k]);
        for (int e = 0; e < 32; ++e) {
            if ((e >> t) & 1) continue;
            if ((e & cm) != cm) continue;
            const int f = e | (1 << t);
            const cd a0 = v[e], a1 = v[f];
            if (g.type == OP_PERM1) {
                v[e] = a1;
                v[f] = a0;
            } else {
                v[e] = c(0) * a0 + c(1) * a1;
                v[f] = c(2) * a0 + c(3) * a1;
            }
        }
        break;
    }
    case OP_DIAG: {
        int fm = 0;
        for (int k = 0; k < g.nfix; ++k) fm |= 1 << loc(g.fix[k]);
        for (int e = 0; e < 32; ++e) {
            if ((e & fm) != fm) continue;
            int pat = 0;
            for (int k = 0; k < g.npat; ++k) pat |= ((e >> loc(g.pat[k])) & 1) << k;
            v[e] *= c(pat);
        }
        break;
    }
    case OP_SWAP: {
        const int a = loc(g.b0), b = loc(g.b1);
        for (int e = 0; e < 32; ++e)
            if (((e >> a) & 1) && !((e >> b) & 1)) std::swap(v[e], v[e ^ (1 << a) ^ (1 << b)]);
        break;
    }
    case OP_M2: {
        const int a = loc(g.b0), b = loc(g.b1);
        for (int e = 0; e < 32; ++e) {
            if (((e >> a) & 1) || ((e >> b) & 1)) continue;
            const int idx[4] = {e, e | (1 << b), e | (1 << a), e | (1 << a) | (1 << b)};
            cd in[4], out[4];
            for (int r = 0; r < 4; ++r) in[r] = v[idx[r]];
            for (int r = 0; r < 4; ++r) {
                out[r] = 0;
                for (int q = 0; q < 4; ++q) out[r] += cd(g.m[(r * 4 + q) * 2], g.m[(r * 4 + q) * 2 + 1]) * in[q];
            }
            for (int r = 0; r < 4; ++r) v[idx[r]] = out[r];
        }
        break;
    }
    }
}

static inline float host_tf32(double x) {
    // round-to-nearest (ties away) to a 10-bit mantissa, as cvt.rna.tf32.f32
    float f = (float)x;
    uint32_t u;
    memcpy(&u, &f, 4);
    if ((u & 0x7f800000u) != 0x7f800000u) {
        u += 0x1000u;
        u &= 0xffffe000u;
    }
    memcpy(&f, &u, 4);
    return f;
}

// Swizzled byte image of B (N x K K-major, two K atoms of 64 rows x 128 B).
static void write_b_image(const double W[64][64], unsigned char *hi, unsigned char *lo) {
    for (int n = 0; n < 64; ++n)
        for (int k = 0; k < 64; ++k) {
            const int atom = k >> 5, kb = (k & 31) * 4;
            const size_t off = (size_t)atom * 64 * 128 + n * 128 + (((kb >> 4) ^ (n & 7)) << 4) +
                               (kb & 15);
            const double w = W[k][n];
            const float h = host_tf32(w);
            const float l = host_tf32(w - (double)h);
            memcpy(hi + off, &h, 4);
            memcpy(lo + off, &l, 4);
        }
}

struct TcPlan {
    std::vector<PlanStep> steps;  // fused steps reuse the window; blocks below
    std::vector<std::vector<std::vector<int>>> pass_blocks;  // per fused step: blocks of gates
    std::vector<std::vector<std::vector<int>>> block_bits;   // per step/block: 5 global bits
};

// Split each window pass into 5-bit blocks: greedy in order, a gate joins the
// open block when all its bits fit in <= 5 bits and no earlier skipped gate
// shares a bit.
static void tc_blocks(const std::vector<GateOp> &gops, const std::vector<int> &gates, int h,
                      int T, std::vector<std::vector<int>> &blocks,
                      std::vector<std::vector<int>> &bits) {
    const int P = (int)gates.size();
    std::vector<char> sched(P, 0);
    int left = P;
    while (left > 0) {
        uint64_t B = 0, blk = 0;
        std::vector<int> cur;
        for (int k = 0; k < P; ++k) {
            if (sched[k]) continue;
            const uint64_t gb = op_bits(gops[gates[k]]);
            if ((gb & blk) == 0 && __builtin_popcountll(B | gb) <= 5) {
                B |= gb;
                cur.push_back(gates[k]);
                sched[k] = 1;
                --left;
            } else {
                blk |= gb;
            }
        }
        std::vector<int> bv;
        for (int b = 0; b < 64; ++b)
            if (B >> b & 1) bv.push_back(b);
        // pad to five bits of the window
        const uint64_t W = window_mask(h, T - 4);
        for (int b = 0; b < 64 && bv.size() < 5; ++b)
            if ((W >> b & 1) && !(B >> b & 1)) bv.push_back(b);
        std::sort(bv.begin(), bv.end());
        blocks.push_back(cur);
        bits.push_back(bv);
    }
}

int apply_circuit_tc_impl(lq_state *s, const lq_gate *ops, int nops, const double *theta,
                          int ntheta, int *nblocks_out, int *npasses_out) {
    const int n = s->n;
    if (s->dtype != LQ_C64)
        return set_error(LQ_ERR_UNSUPPORTED, "the tensor-core path runs on complex64 states");
    if (n < kTcT) return set_error(LQ_ERR_UNSUPPORTED, "the tensor-core path needs >= 12 qubits");
    std::vector<GateOp> gops(nops);
    for (int i = 0; i < nops; ++i) {
        LQ_TRY(validate_gate(&ops[i], n, ntheta));
        LQ_TRY(make_gate_op(&ops[i], theta, n, &gops[i]));
        if (gops[i].renorm)
            return set_error(LQ_ERR_UNSUPPORTED, "renormalising gates are not fused on tensor cores");
    }
    // Windows: the FP64 planner with every gate required fully inside the window
    // (dense blocks cannot read controls outside it).
    std::vector<GateOp> planner_ops = gops;
    for (auto &g : planner_ops) {
        // make every bit a mixed bit for window selection: widen to a 4x4-like op
        if (g.type == OP_DIAG || g.nctrl > 0 || g.type == OP_PERM1) {
            GateOp w = g;
            w.type = OP_M2;
            const uint64_t b = op_bits(g);
            int bits[3], nb = 0;
            for (int k = 0; k < 64 && nb < 3; ++k)
                if (b >> k & 1) bits[nb++] = k;
            if (nb == 1) {
                w.type = OP_M1;
                w.t = bits[0];
                w.nctrl = 0;
            } else if (nb == 2) {
                w.b0 = bits[0];
                w.b1 = bits[1];
            } else {
                return set_error(LQ_ERR_UNSUPPORTED, "3-qubit gates are not fused on tensor cores");
            }
            w.nfix = w.npat = 0;
            g = w;
        }
    }
    std::vector<PlanStep> steps = plan_windows(planner_ops, n, kTcT);
    std::vector<TcBlock> blocks;
    std::vector<TcPass> passes;
    std::vector<unsigned char> bimg;
    std::vector<int> step_pass(steps.size(), -1);
    for (size_t si = 0; si < steps.size(); ++si) {
        const PlanStep &st = steps[si];
        if (!st.fused) continue;
        std::vector<std::vector<int>> bl, bb;
        tc_blocks(gops, st.pass.gates, st.pass.h, kTcT, bl, bb);
        TcPass tp{st.pass.h, (int)blocks.size(), (int)bl.size(), 0};
        for (size_t b = 0; b < bl.size(); ++b) {
            int gbit[5];
            for (int j = 0; j < 5; ++j) gbit[j] = bb[b][j];
            // A block on tile bit 0 takes it as its block bit 0: columns 2c and
            // 2c+1 are then the two halves of one 16-byte chunk, read and written
            // as a pair.  U is built in this bit order, so the order is free.
            for (int j = 1; j < 5; ++j)
                if (local_pos(gbit[j], st.pass.h) == 0) std::swap(gbit[0], gbit[j]);
            // block unitary U (32 x 32): column e = product of gates on basis e
            cd U[32][32];
            for (int e = 0; e < 32; ++e) {
                cd v[32] = {};
                v[e] = 1.0;
                for (int gi : bl[b]) small_apply(gops[gi], gbit, v);
                for (int r = 0; r < 32; ++r) U[r][e] = v[r];
            }
            double W[64][64];
            for (int r = 0; r < 32; ++r)
                for (int c = 0; c < 32; ++c) {
                    W[2 * c][2 * r] = U[r][c].real();
                    W[2 * c + 1][2 * r] = -U[r][c].imag();
                    W[2 * c][2 * r + 1] = U[r][c].imag();
                    W[2 * c + 1][2 * r + 1] = U[r][c].real();
                }
            TcBlock tb{};
            int k[5];
            for (int j = 0; j < 5; ++j) {
                k[j] = local_pos(gbit[j], st.pass.h);
                tb.col[j] = tile_off(1u << k[j]);
            }
            tb.pair = k[0] == 0;
            // Row bits: thread m's bit j goes to the tile bit order[j].  The row order
            // is free (each thread writes back the row it read), so the five lane
            // bits (j < 5) take tile bits whose 8-byte bank slots in the swizzled
            // tile are linearly independent: slot(l) = (l0, l1^l9, l2^l10, l3^l11).
            // Up to 16 distinct slots per warp access = the two-wavefront minimum.
            std::vector<int> free_bits;
            for (int l = 0; l < kTcT; ++l) {
                bool inb = false;
                for (int j = 0; j < 5; ++j) inb |= k[j] == l;
                if (!inb) free_bits.push_back(l);
            }
            auto slot_vec = [](int b) { return b < 4 ? 1u << b : b < 9 ? 0u : 1u << (b - 8); };
            std::vector<int> order;
            std::vector<uint32_t> basis;  // reduced slot vectors of the chosen lane bits
            for (int b : free_bits) {
                uint32_t v = slot_vec(b);
                for (uint32_t e : basis)
                    if ((v ^ e) < v) v ^= e;
                if (v && order.size() < 5) {
                    basis.push_back(v);
                    std::sort(basis.rbegin(), basis.rend());
                    order.push_back(b);
                }
            }
            for (int b : free_bits)
                if (std::find(order.begin(), order.end(), b) == order.end()) order.push_back(b);
            for (int j = 0; j < 7; ++j) tb.row[j] = tile_off(1u << order[j]);
            tb.b_offset = (uint32_t)(bimg.size() >> 4);
            bimg.resize(bimg.size() + 2 * kBBytes);
            write_b_image(W, bimg.data() + bimg.size() - 2 * kBBytes, bimg.data() + bimg.size() - kBBytes);
            blocks.push_back(tb);
        }
        step_pass[si] = (int)passes.size();
        passes.push_back(tp);
    }
    const size_t bsz = blocks.size() * sizeof(TcBlock);
    auto al = [](size_t x) { return (x + 1023) / 1024 * 1024; };
    LQ_TRY(ensure_prog(s, al(bsz) + al(bimg.size()) + 1024));
    TcBlock *d_blocks = (TcBlock *)s->d_prog;
    unsigned char *d_bimg = (unsigned char *)s->d_prog + al(bsz);
    LQ_CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (bsz) LQ_CUDA_TRY(cudaMemcpy(d_blocks, blocks.data(), bsz, cudaMemcpyHostToDevice));
    if (!bimg.empty())
        LQ_CUDA_TRY(cudaMemcpy(d_bimg, bimg.data(), bimg.size(), cudaMemcpyHostToDevice));
    static bool attr = false;
    if (!attr) {
        LQ_CUDA_TRY(cudaFuncSetAttribute(k_tc_pass, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kTcSmem));
        attr = true;
    }
    // FP32 accumulation in the tensor cores rounds every block's sums toward
    // zero, which shrinks the state by a near-uniform factor per block; the
    // FP64 norm of the input is restored at the end of the circuit (one
    // reduction before, one reduction and one scaling sweep after).
    const bool restore = tc_restore_norm() && !blocks.empty();
    if (restore) LQ_TRY(norm_snapshot(s));
    int launches = 0;
    for (size_t si = 0; si < steps.size(); ++si) {
        const PlanStep &st = steps[si];
        if (!st.fused) {
            LQ_TRY(launch_gate_op(s, gops[st.gate]));
            if (restore && gops[st.gate].renorm) LQ_TRY(norm_snapshot(s));
            continue;
        }
        const TcPass &tp = passes[step_pass[si]];
        CUtensorMap map;
        LQ_TRY(tc_tile_map(&map, s->d, n, tp.h));
        const int ntiles = 1 << (n - kTcT);
        prof_begin(s->stream, kProfTc);
        k_tc_pass<<<std::min(ntiles, tc_sm_count()), kTcThreads, kTcSmem, s->stream>>>(
            map, tp.h, ntiles, d_blocks + tp.block_begin, tp.nblocks, d_bimg, s->d_flag);
        prof_end(s->stream, kProfTc);
        LQ_CUDA_TRY(cudaGetLastError());
        ++launches;
    }
    if (restore) LQ_TRY(norm_restore(s));
    if (nblocks_out) *nblocks_out = (int)blocks.size();
    if (npasses_out) *npasses_out = launches;
    return LQ_OK;
}

}  // namespace lq

using namespace lq;

extern "C" {

int lq_apply_circuit_tc(lq_state *s, int circuit_qubits, const lq_gate *ops, int nops,
                        const double *theta, int ntheta, int *blocks, int *passes) {
    LQ_TRY(check_state(s));
    if (circuit_qubits != s->n)
        return set_error(LQ_ERR_QUBIT_MISMATCH,
                         "Circuit qubit count mismatch: circuit has %d, state has %d",
                         circuit_qubits, s->n);
    if (nops < 0 || (nops > 0 && !ops)) return set_error(LQ_ERR_INVALID_ARG, "bad op list");
    if (ntheta < 0 || (ntheta > 0 && !theta)) return set_error(LQ_ERR_INVALID_ARG, "bad theta");
    return apply_circuit_tc_impl(s, ops, nops, theta, ntheta, blocks, passes);
}

}  // extern "C"
