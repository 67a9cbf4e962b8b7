// Block-wide FP64 sums in a fixed order, shared by the reductions.
#pragma once

#include "lq_internal.h"

namespace lq {

// Block-wide sum of NC doubles; result valid in thread 0.
template <int NC>
__device__ __forceinline__ void block_sum(double (&x)[NC], double *sh /* 32*NC */) {
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x[c] += __shfl_down_sync(0xffffffffu, x[c], o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < NC; ++c) sh[warp * NC + c] = x[c];
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            x[c] = lane < nw ? sh[lane * NC + c] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x[c] += __shfl_down_sync(0xffffffffu, x[c], o);
        }
    }
}

// v = src (or v, in place) divided by the norm whose squared per-block sums are
// partials, if the norm exceeds 1e-10 (State::normalize, src/states/mod.rs:91-114).
// Every block adds the partials up itself, in the same order, instead of waiting for a
// one-block kernel to do so: one launch of three fewer in a renormalising gate, which
// at 2^14 amplitudes is launch bound (some 2.5 us each).  256 threads.
template <class A>
__global__ void __launch_bounds__(256)
    k_scale_by_partials(A *v, const A *src, uint64_t N,
                        const double *__restrict__ partials, int nparts) {
    __shared__ double sh[32];
    __shared__ double s_norm;
    double acc[1] = {0.0};
    for (int p = threadIdx.x; p < nparts; p += blockDim.x) acc[0] += partials[p];
    block_sum<1>(acc, sh);
    if (threadIdx.x == 0) s_norm = sqrt(acc[0]);
    __syncthreads();
    const double norm = s_norm;
    const bool scale = norm > 1e-10;
    if (!scale && !src) return;
    const A *from = src ? src : v;
    auto put = [&](uint64_t i, A a) {
        if (scale) {
            a.x = a.x / norm;
            a.y = a.y / norm;
        }
        v[i] = a;
    };
    // four loads before the first store (which might be to the same place: 26 qubits
    // 436 us one at a time, 355 so)
    constexpr int kU = 4;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for (; i + (kU - 1) * stride < N; i += kU * stride) {
        A a[kU];
#pragma unroll
        for (int k = 0; k < kU; ++k) a[k] = from[i + k * stride];
#pragma unroll
        for (int k = 0; k < kU; ++k) put(i + k * stride, a[k]);
    }
    for (; i < N; i += stride) put(i, from[i]);
}

// Blocks of a 256-thread grid-stride sweep that leaves one partial sum each.
inline int red_grid(uint64_t N, int threads) {
    uint64_t g = (N + threads - 1) / threads;
    if (g > (uint64_t)kRedBlocks) g = kRedBlocks;
    if (g < 1) g = 1;
    return (int)g;
}

}  // namespace lq
