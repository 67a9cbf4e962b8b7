// Learned warm start and exact ground energies.
//
// 1. A small MLP maps Hamiltonian couplings to ansatz angles: input (Jx, Jy, Jz
//    per bond, padded) + field, `depth` hidden layers of width `hidden` with
//    GELU, linear output of `out` angles.  Training and inference run on
//    hand-written FP32 kernels: a tiled SGEMM with fused bias / GELU epilogue,
//    its transposed forms for the backward pass, a periodic angle loss
//    sum(1 - cos(y - t)) over a validity mask, and Adam.
// 2. FP64 Lanczos on the full 2^n space with a Pauli-sum matrix-vector kernel
//    (textbook Pauli convention: H is real symmetric for X/Y/Z strings with an
//    even number of Y factors), full reorthogonalisation, and a host bisection
//    on the tridiagonal matrix.  This is the "exact" E0 the learned warm start
//    is judged against (the reference has no exact solver).
#include <algorithm>
#include <cmath>
#include <random>

#include "lq_internal.h"

namespace lq {

// ---------------------------------------------------------------------------
// FP32 GEMM: C[M x N] = op(A) op(B), the network's only contraction.
//   op(A) = A (M x K, lda) or A^T (A is K x M);  op(B) likewise
// Epilogues: + bias, then GELU with the pre-activation kept in Z; or times the GELU
// derivative at Z (the next layer's gradient through its activation); row sums of
// op(A) (the bias gradient, whose op(A) is dY^T).
//
// A batch of 256 through 256-wide layers is 17 MFMA a product: the chip would do it
// in under a microsecond, so latency counts and not arithmetic.  32 x 32 output
// tiles (64 blocks for 256 x 256, where 64 x 64 tiles gave 16) of 256 threads, four groups of
// 64 that each take a quarter of every 32-deep K step on 4 x 4 outputs per thread and
// are added at the end; the next K step is loaded into registers meanwhile.  The two
// products of a backward layer, dW and dX, share one launch.  (Measured per product:
// 31-47 us with 64 x 64 tiles of one group.)
// ---------------------------------------------------------------------------
constexpr int GB = 32, GK = 32, GP = GB + 4;

enum GemmEpilogue { EP_NONE = 0, EP_BIAS = 1, EP_BIAS_GELU = 2, EP_GELU_BWD = 3 };

struct GemmJob {
    int M, N, K;
    const float *A;
    int lda, ta;
    const float *B;
    int ldb, tb;
    float *C;
    int ldc;
    int ep;
    const float *bias;
    float *Z;        // written (EP_BIAS_GELU) or read (EP_GELU_BWD), as C
    float *row_sum;  // sums of op(A)'s rows, or null
};

// GELU'(z) = Phi(z) + z phi(z)
__device__ __forceinline__ float gelu_slope(float z) {
    const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

__global__ void __launch_bounds__(256)
    k_gemm(const __grid_constant__ GemmJob j0, const __grid_constant__ GemmJob j1, int blocks0) {
    __shared__ __align__(16) float sm[2][2][GK][GP];  // [buffer][A, B]
    __shared__ float s_row[4][GB];
    const bool second = (int)blockIdx.x >= blocks0;
    const GemmJob &j = second ? j1 : j0;
    const int tid = threadIdx.x, group = tid >> 6, tx = tid & 7, ty = (tid >> 3) & 7;
    const int nt = (j.N + GB - 1) / GB, blk = (int)blockIdx.x - (second ? blocks0 : 0);
    const int m0 = blk / nt * GB, n0 = blk % nt * GB;
    // staging: four elements per thread and operand; consecutive threads run along the
    // contiguous index of the operand
    const int i = tid & 31, o = tid >> 5;
    auto fetch = [&](int k0, float (&ra)[4], float (&rb)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int u = o + 8 * q;
            const int am = m0 + (j.ta ? i : u), ak = k0 + (j.ta ? u : i);
            ra[q] = am < j.M && ak < j.K
                        ? (j.ta ? j.A[(size_t)ak * j.lda + am] : j.A[(size_t)am * j.lda + ak])
                        : 0.f;
            const int bn = n0 + (j.tb ? u : i), bk = k0 + (j.tb ? i : u);
            rb[q] = bn < j.N && bk < j.K
                        ? (j.tb ? j.B[(size_t)bn * j.ldb + bk] : j.B[(size_t)bk * j.ldb + bn])
                        : 0.f;
        }
    };
    auto stash = [&](int buf, const float (&ra)[4], const float (&rb)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int u = o + 8 * q;
            sm[buf][0][j.ta ? u : i][j.ta ? i : u] = ra[q];
            sm[buf][1][j.tb ? i : u][j.tb ? u : i] = rb[q];
        }
    };
    float acc[4][4] = {}, rsum[4] = {};
    float ra[4], rb[4];
    fetch(0, ra, rb);
    stash(0, ra, rb);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < j.K; k0 += GK) {
        const bool more = k0 + GK < j.K;
        if (more) fetch(k0 + GK, ra, rb);
#pragma unroll
        for (int kk = 0; kk < GK / 4; ++kk) {
            const int k = group * (GK / 4) + kk;
            const float4 a4 = *(const float4 *)&sm[buf][0][k][ty * 4];
            const float4 b4 = *(const float4 *)&sm[buf][1][k][tx * 4];
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                rsum[p] += a[p];
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(a[p], b[q], acc[p][q]);
            }
        }
        if (more) stash(buf ^ 1, ra, rb);  // (last read before the previous barrier)
        __syncthreads();
        buf ^= 1;
    }
    // add the four groups
    float(*red)[GB][GB] = (float(*)[GB][GB])sm;
    static_assert(sizeof(float) * 4 * GB * GB <= sizeof(sm), "the groups' sums fit the stages");
#pragma unroll
    for (int p = 0; p < 4; ++p)
        *(float4 *)&red[group][ty * 4 + p][tx * 4] =
            make_float4(acc[p][0], acc[p][1], acc[p][2], acc[p][3]);
    if (tx == 0)
#pragma unroll
        for (int p = 0; p < 4; ++p) s_row[group][ty * 4 + p] = rsum[p];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = o + 8 * q, gm = m0 + r, gn = n0 + i;
        if (gm >= j.M || gn >= j.N) continue;
        float v = (red[0][r][i] + red[1][r][i]) + (red[2][r][i] + red[3][r][i]);
        const size_t at = (size_t)gm * j.ldc + gn;
        if (j.ep == EP_BIAS || j.ep == EP_BIAS_GELU) v += j.bias[gn];
        if (j.ep == EP_BIAS_GELU) {
            j.Z[at] = v;
            v = 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
        } else if (j.ep == EP_GELU_BWD) {
            v *= gelu_slope(j.Z[at]);
        }
        j.C[at] = v;
    }
    if (j.row_sum && n0 == 0 && tid < GB && m0 + tid < j.M)
        j.row_sum[m0 + tid] =
            (s_row[0][tid] + s_row[1][tid]) + (s_row[2][tid] + s_row[3][tid]);
}

static int gemm_blocks(const GemmJob &j) {
    return ((j.M + GB - 1) / GB) * ((j.N + GB - 1) / GB);
}

static void gemm(cudaStream_t st, const GemmJob &j) {
    const int b = gemm_blocks(j);
    k_gemm<<<b, 256, 0, st>>>(j, j, b);
}

static void gemm2(cudaStream_t st, const GemmJob &a, const GemmJob &b) {
    const int n = gemm_blocks(a);
    k_gemm<<<n + gemm_blocks(b), 256, 0, st>>>(a, b, n);
}

// Periodic angle loss: sum mask * (1 - cos(y - t)) / sum(mask); dY = mask sin(y - t) / sum(mask).
// One partial sum per block (the caller adds them in order).
constexpr int kLossBlocks = 148;

__global__ void k_angle_loss(const float *__restrict__ Y, const float *__restrict__ T,
                             const float *__restrict__ Mk, float *__restrict__ dY, int count,
                             float inv_norm, double *__restrict__ loss_part) {
    __shared__ double sh[256];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float d = Y[i] - T[i];
        const float m = Mk[i];
        acc += (double)(m * (1.f - cosf(d)));
        dY[i] = m * sinf(d) * inv_norm;
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss_part[blockIdx.x] = sh[0] * inv_norm;
}

__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, int64_t count, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    }
}

// ---------------------------------------------------------------------------
// Lanczos: y = H x for a Pauli sum (textbook convention, real H).
// For an even number of Y factors, (P x)_i = Re((-i)^ny) (-1)^popcount(i & z) x_{i ^ x}.
// ---------------------------------------------------------------------------
struct RealTerm {
    uint64_t x, z;
    double c;  // coefficient * Re((-i)^ny)
};

__global__ void k_pauli_matvec(const double *__restrict__ in, double *__restrict__ out, int n,
                               const RealTerm *__restrict__ terms, int nt) {
    extern __shared__ RealTerm s_t[];
    for (int t = threadIdx.x; t < nt; t += blockDim.x) s_t[t] = terms[t];
    __syncthreads();
    const uint64_t N = 1ull << n;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        double acc = 0.0;
        for (int t = 0; t < nt; ++t) {
            const double s = (__popcll(i & s_t[t].z) & 1) ? -s_t[t].c : s_t[t].c;
            acc += s * in[i ^ s_t[t].x];
        }
        out[i] = acc;
    }
}

__global__ void k_axpy(double *__restrict__ y, const double *__restrict__ x, double a, uint64_t N) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x)
        y[i] += a * x[i];
}

// partial[j * gridDim.x + b] = block b's share of <V_j, w> for j = blockIdx.y.
__global__ void k_multi_dot(const double *__restrict__ V, const double *__restrict__ w, uint64_t N,
                            double *__restrict__ partial) {
    __shared__ double sh[256];
    const double *vj = V + (size_t)blockIdx.y * N;
    double acc = 0.0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x)
        acc += vj[i] * w[i];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = sh[0];
}

// w -= sum_j c[j] V_j   (classical Gram-Schmidt step against the Lanczos basis)
__global__ void k_multi_sub(const double *__restrict__ V, const double *__restrict__ c, int k,
                            uint64_t N, double *__restrict__ w) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x) {
        double acc = w[i];
        for (int j = 0; j < k; ++j) acc -= c[j] * V[(size_t)j * N + i];
        w[i] = acc;
    }
}

__global__ void k_scale(double *__restrict__ y, const double *__restrict__ x, double a,
                        uint64_t N) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < N;
         i += (uint64_t)gridDim.x * blockDim.x)
        y[i] = a * x[i];
}

// Smallest eigenvalue of the symmetric tridiagonal (alpha, beta) by bisection
// on the Sturm sequence count.
static double tridiag_min_eig(const std::vector<double> &a, const std::vector<double> &b) {
    const int k = (int)a.size();
    double lo = 1e300, hi = -1e300;
    for (int i = 0; i < k; ++i) {
        const double r = (i > 0 ? std::fabs(b[i - 1]) : 0.0) + (i + 1 < k ? std::fabs(b[i]) : 0.0);
        lo = std::min(lo, a[i] - r);
        hi = std::max(hi, a[i] + r);
    }
    auto count_below = [&](double x) {
        int cnt = 0;
        double d = 1.0;
        for (int i = 0; i < k; ++i) {
            d = a[i] - x - (i > 0 ? b[i - 1] * b[i - 1] / d : 0.0);
            if (d == 0.0) d = -1e-300;
            if (d < 0) ++cnt;
        }
        return cnt;
    };
    for (int it = 0; it < 200; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (count_below(mid) >= 1) hi = mid;
        else lo = mid;
        if (hi - lo < 1e-15 * std::max(1.0, std::fabs(mid))) break;
    }
    return 0.5 * (lo + hi);
}

}  // namespace lq

struct lq_mlp {
    int in_dim = 0, hidden = 0, depth = 0, out_dim = 0;
    std::vector<int> dims;           // layer widths: in, hidden x depth, out
    std::vector<size_t> woff, boff;  // offsets in the flat parameter vector
    int64_t nparams = 0;
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // device
    int64_t adam_t = 0;
    // activations for a batch (device), capacity in rows
    int cap = 0;
    std::vector<float *> H, Z;  // H[0] = input, H[l+1] = layer l output; Z pre-activations
    float *target = nullptr, *mask = nullptr, *dA = nullptr, *dB = nullptr;
    double *loss_d = nullptr;
    cudaStream_t stream = nullptr;
};

namespace lq {

static int mlp_reserve(lq_mlp *net, int batch) {
    if (batch <= net->cap) return LQ_OK;
    for (auto p : net->H) cudaFree(p);
    for (auto p : net->Z) cudaFree(p);
    cudaFree(net->target);
    cudaFree(net->mask);
    cudaFree(net->dA);
    cudaFree(net->dB);
    net->target = net->mask = net->dA = net->dB = nullptr;
    net->cap = 0;
    net->H.assign(net->dims.size(), nullptr);
    net->Z.assign(net->dims.size(), nullptr);
    int widest = 0;
    for (size_t l = 0; l < net->dims.size(); ++l) {
        LQ_CUDA_TRY(device_malloc(&net->H[l], sizeof(float) * batch * net->dims[l]));
        LQ_CUDA_TRY(device_malloc(&net->Z[l], sizeof(float) * batch * net->dims[l]));
        widest = std::max(widest, net->dims[l]);
    }
    LQ_CUDA_TRY(device_malloc(&net->target, sizeof(float) * batch * net->out_dim));
    LQ_CUDA_TRY(device_malloc(&net->mask, sizeof(float) * batch * net->out_dim));
    LQ_CUDA_TRY(device_malloc(&net->dA, sizeof(float) * batch * widest));
    LQ_CUDA_TRY(device_malloc(&net->dB, sizeof(float) * batch * widest));
    net->cap = batch;
    return LQ_OK;
}

static int mlp_forward_dev(lq_mlp *net, int batch) {
    const int L = (int)net->dims.size() - 1;
    for (int l = 0; l < L; ++l) {
        const int K = net->dims[l], Nn = net->dims[l + 1];
        const bool last = l == L - 1;
        // H[l+1] = H[l] (batch x K) . W^T (W stored out x in) + b
        gemm(net->stream,
             GemmJob{batch, Nn, K, net->H[l], K, 0, net->p + net->woff[l], K, 1, net->H[l + 1], Nn,
                     last ? EP_BIAS : EP_BIAS_GELU, net->p + net->boff[l], net->Z[l + 1], nullptr});
    }
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

// Backward sweep from dL/dy (in net->dA, batch x out_dim) after a forward pass
// of the same batch; writes dL/dparams to net->g.
static int mlp_backward_dev(lq_mlp *net, int batch) {
    cudaStream_t st = net->stream;
    float *dY = net->dA, *dX = net->dB;
    const int L = (int)net->dims.size() - 1;
    for (int l = L - 1; l >= 0; --l) {
        const int K = net->dims[l], Nn = net->dims[l + 1];
        // dW (Nn x K) = dY^T (Nn x batch) . H[l] (batch x K), and db = dY's column sums
        const GemmJob dw{Nn, K, batch, dY, Nn, 1, net->H[l], K, 0, net->g + net->woff[l], K,
                         EP_NONE, nullptr, nullptr, net->g + net->boff[l]};
        if (l == 0) {
            gemm(st, dw);
            break;
        }
        // dX (batch x K) = dY (batch x Nn) . W (Nn x K), through the GELU of layer l-1
        gemm2(st, dw,
              GemmJob{batch, K, Nn, dY, Nn, 0, net->p + net->woff[l], K, 0, dX, K, EP_GELU_BWD,
                      nullptr, net->Z[l], nullptr});
        std::swap(dY, dX);
    }
    LQ_CUDA_TRY(cudaGetLastError());
    return LQ_OK;
}

}  // namespace lq

using namespace lq;

extern "C" {

int lq_mlp_create(int in_dim, int hidden, int depth, int out_dim, uint64_t seed, lq_mlp **out) {
    if (!out || in_dim < 1 || hidden < 1 || depth < 1 || out_dim < 1)
        return set_error(LQ_ERR_INVALID_ARG, "bad MLP shape");
    lq_mlp *net = new lq_mlp();
    net->in_dim = in_dim;
    net->hidden = hidden;
    net->depth = depth;
    net->out_dim = out_dim;
    net->dims.push_back(in_dim);
    for (int d = 0; d < depth; ++d) net->dims.push_back(hidden);
    net->dims.push_back(out_dim);
    size_t off = 0;
    for (size_t l = 0; l + 1 < net->dims.size(); ++l) {
        net->woff.push_back(off);
        off += (size_t)net->dims[l] * net->dims[l + 1];
        net->boff.push_back(off);
        off += net->dims[l + 1];
    }
    net->nparams = (int64_t)off;
    // He-style uniform init from a seeded generator (host), zero biases; the
    // output layer is scaled down so initial angles start near zero.
    std::vector<float> init(off, 0.f);
    std::mt19937_64 rng(seed);
    for (size_t l = 0; l + 1 < net->dims.size(); ++l) {
        const double bound =
            std::sqrt(6.0 / net->dims[l]) * (l + 2 == net->dims.size() ? 0.1 : 1.0);
        std::uniform_real_distribution<double> u(-bound, bound);
        for (size_t i = 0; i < (size_t)net->dims[l] * net->dims[l + 1]; ++i)
            init[net->woff[l] + i] = (float)u(rng);
    }
    auto fail = [&](cudaError_t e) {
        if (net->stream) cudaStreamDestroy(net->stream);
        cudaFree(net->loss_d);
        cudaFree(net->p);
        cudaFree(net->g);
        cudaFree(net->m);
        cudaFree(net->v);
        delete net;
        return set_error(e == cudaErrorMemoryAllocation ? LQ_ERR_OOM : LQ_ERR_CUDA, "%s",
                         cudaGetErrorString(e));
    };
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking))) return fail(e);
    if ((e = device_malloc(&net->p, off * 4))) return fail(e);
    if ((e = device_malloc(&net->g, off * 4))) return fail(e);
    if ((e = device_malloc(&net->m, off * 4))) return fail(e);
    if ((e = device_malloc(&net->v, off * 4))) return fail(e);
    if ((e = device_malloc(&net->loss_d, sizeof(double) * kLossBlocks))) return fail(e);
    if ((e = cudaMemcpy(net->p, init.data(), off * 4, cudaMemcpyHostToDevice))) return fail(e);
    if ((e = cudaMemset(net->m, 0, off * 4)) || (e = cudaMemset(net->v, 0, off * 4)) ||
        (e = cudaMemset(net->g, 0, off * 4)))
        return fail(e);
    *out = net;
    return LQ_OK;
}

int lq_mlp_destroy(lq_mlp *net) {
    if (!net) return LQ_OK;
    cudaStreamSynchronize(net->stream);
    for (auto p : net->H) cudaFree(p);
    for (auto p : net->Z) cudaFree(p);
    cudaFree(net->target);
    cudaFree(net->mask);
    cudaFree(net->dA);
    cudaFree(net->dB);
    cudaFree(net->loss_d);
    cudaFree(net->p);
    cudaFree(net->g);
    cudaFree(net->m);
    cudaFree(net->v);
    cudaStreamDestroy(net->stream);
    delete net;
    return LQ_OK;
}

int lq_mlp_num_params(const lq_mlp *net, int64_t *out) {
    if (!net || !out) return set_error(LQ_ERR_INVALID_ARG, "null argument");
    *out = net->nparams;
    return LQ_OK;
}

int lq_mlp_get_params(const lq_mlp *net, float *host, int64_t count) {
    if (!net || !host) return set_error(LQ_ERR_INVALID_ARG, "null argument");
    if (count != net->nparams)
        return set_error(LQ_ERR_PARAM_COUNT, "Parameter count mismatch: expected %lld, got %lld",
                         (long long)net->nparams, (long long)count);
    LQ_CUDA_TRY(cudaMemcpy(host, net->p, count * 4, cudaMemcpyDeviceToHost));
    return LQ_OK;
}

int lq_mlp_set_params(lq_mlp *net, const float *host, int64_t count) {
    if (!net || !host) return set_error(LQ_ERR_INVALID_ARG, "null argument");
    if (count != net->nparams)
        return set_error(LQ_ERR_PARAM_COUNT, "Parameter count mismatch: expected %lld, got %lld",
                         (long long)net->nparams, (long long)count);
    LQ_CUDA_TRY(cudaMemcpy(net->p, host, count * 4, cudaMemcpyHostToDevice));
    return LQ_OK;
}

int lq_mlp_get_grads(const lq_mlp *net, float *host, int64_t count) {
    if (!net || !host) return set_error(LQ_ERR_INVALID_ARG, "null argument");
    if (count != net->nparams)
        return set_error(LQ_ERR_PARAM_COUNT, "Parameter count mismatch: expected %lld, got %lld",
                         (long long)net->nparams, (long long)count);
    LQ_CUDA_TRY(cudaMemcpy(host, net->g, count * 4, cudaMemcpyDeviceToHost));
    return LQ_OK;
}

int lq_mlp_forward(lq_mlp *net, const float *x, int batch, float *y) {
    if (!net || !x || !y || batch < 1) return set_error(LQ_ERR_INVALID_ARG, "bad arguments");
    LQ_TRY(mlp_reserve(net, batch));
    LQ_CUDA_TRY(cudaMemcpyAsync(net->H[0], x, sizeof(float) * batch * net->in_dim,
                                cudaMemcpyHostToDevice, net->stream));
    LQ_TRY(mlp_forward_dev(net, batch));
    LQ_CUDA_TRY(cudaMemcpyAsync(y, net->H.back(), sizeof(float) * batch * net->out_dim,
                                cudaMemcpyDeviceToHost, net->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(net->stream));
    return LQ_OK;
}

int lq_mlp_loss_grad(lq_mlp *net, const float *x, const float *target, const float *mask,
                     int batch, double *loss) {
    if (!net || !x || !target || !mask || batch < 1)
        return set_error(LQ_ERR_INVALID_ARG, "bad arguments");
    LQ_TRY(mlp_reserve(net, batch));
    cudaStream_t st = net->stream;
    const int O = net->out_dim;
    // (eight chains: one alone is 40 us of additions for a batch of 256)
    double ms[8] = {0.0}, msum = 0.0;
    const int64_t count = (int64_t)batch * O;
    int64_t mi = 0;
    for (; mi + 8 <= count; mi += 8)
        for (int k = 0; k < 8; ++k) ms[k] += mask[mi + k];
    for (; mi < count; ++mi) msum += mask[mi];
    for (int k = 0; k < 8; ++k) msum += ms[k];
    if (msum <= 0) return set_error(LQ_ERR_INVALID_ARG, "empty mask");
    LQ_CUDA_TRY(cudaMemcpyAsync(net->H[0], x, sizeof(float) * batch * net->in_dim,
                                cudaMemcpyHostToDevice, st));
    LQ_CUDA_TRY(cudaMemcpyAsync(net->target, target, sizeof(float) * batch * O,
                                cudaMemcpyHostToDevice, st));
    LQ_CUDA_TRY(cudaMemcpyAsync(net->mask, mask, sizeof(float) * batch * O,
                                cudaMemcpyHostToDevice, st));
    LQ_TRY(mlp_forward_dev(net, batch));
    const int lb = std::max(1, std::min(kLossBlocks, (batch * O + 255) / 256));
    k_angle_loss<<<lb, 256, 0, st>>>(
        net->H.back(), net->target, net->mask, net->dA, batch * O, (float)(1.0 / msum),
        net->loss_d);
    LQ_TRY(mlp_backward_dev(net, batch));
    double part[kLossBlocks], lv = 0.0;
    LQ_CUDA_TRY(cudaMemcpyAsync(part, net->loss_d, sizeof(double) * lb, cudaMemcpyDeviceToHost,
                                st));
    LQ_CUDA_TRY(cudaStreamSynchronize(st));
    for (int k = 0; k < lb; ++k) lv += part[k];
    if (loss) *loss = lv;
    return LQ_OK;
}

int lq_mlp_backward(lq_mlp *net, const float *x, const float *dy, int batch) {
    if (!net || !x || !dy || batch < 1) return set_error(LQ_ERR_INVALID_ARG, "bad arguments");
    LQ_TRY(mlp_reserve(net, batch));
    cudaStream_t st = net->stream;
    LQ_CUDA_TRY(cudaMemcpyAsync(net->H[0], x, sizeof(float) * batch * net->in_dim,
                                cudaMemcpyHostToDevice, st));
    LQ_TRY(mlp_forward_dev(net, batch));
    LQ_CUDA_TRY(cudaMemcpyAsync(net->dA, dy, sizeof(float) * batch * net->out_dim,
                                cudaMemcpyHostToDevice, st));
    LQ_TRY(mlp_backward_dev(net, batch));
    LQ_CUDA_TRY(cudaStreamSynchronize(st));
    return LQ_OK;
}

int lq_mlp_reset_adam(lq_mlp *net) {
    if (!net) return set_error(LQ_ERR_INVALID_ARG, "null network");
    LQ_CUDA_TRY(cudaMemsetAsync(net->m, 0, net->nparams * 4, net->stream));
    LQ_CUDA_TRY(cudaMemsetAsync(net->v, 0, net->nparams * 4, net->stream));
    LQ_CUDA_TRY(cudaStreamSynchronize(net->stream));
    net->adam_t = 0;
    return LQ_OK;
}

int lq_mlp_adam_step(lq_mlp *net, float lr, float beta1, float beta2, float eps) {
    if (!net) return set_error(LQ_ERR_INVALID_ARG, "null network");
    net->adam_t += 1;
    const float c1 = 1.f / (1.f - std::pow(beta1, (float)net->adam_t));
    const float c2 = 1.f / (1.f - std::pow(beta2, (float)net->adam_t));
    k_adam<<<592, 256, 0, net->stream>>>(net->p, net->g, net->m, net->v, net->nparams, lr, beta1,
                                         beta2, eps, c1, c2);
    LQ_CUDA_TRY(cudaGetLastError());
    LQ_CUDA_TRY(cudaStreamSynchronize(net->stream));
    return LQ_OK;
}

int lq_lanczos_ground_energy(int num_qubits, const lq_pauli_term *terms, int nterms,
                             int max_iter, double tol, uint64_t seed, double *e0, int *iters) {
    if (!terms || nterms < 1 || !e0 || num_qubits < 1 || num_qubits > 26 || max_iter < 2)
        return set_error(LQ_ERR_INVALID_ARG, "bad Lanczos arguments");
    std::vector<RealTerm> rt;
    for (int t = 0; t < nterms; ++t) {
        const int ny = terms[t].ny;
        if (ny & 1)
            return set_error(LQ_ERR_UNSUPPORTED,
                             "Lanczos needs a real Hamiltonian (even number of Y per term)");
        rt.push_back(RealTerm{terms[t].xmask, terms[t].zmask,
                              terms[t].coefficient * ((ny & 3) == 2 ? -1.0 : 1.0)});
    }
    const uint64_t N = 1ull << num_qubits;
    const int kmax = (int)std::min<uint64_t>(max_iter, N);
    if ((double)(kmax + 2) * (double)N * 8.0 > 32e9)
        return set_error(LQ_ERR_OOM, "Lanczos basis of %d vectors of 2^%d doubles exceeds 32 GB",
                         kmax + 1, num_qubits);
    if (rt.size() * sizeof(RealTerm) > 48 * 1024)
        return set_error(LQ_ERR_INVALID_ARG, "too many Pauli terms for the Lanczos matvec");
    constexpr int kDotBlocks = 148;
    cudaStream_t st;
    LQ_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    double *V = nullptr, *w = nullptr, *part = nullptr, *coef = nullptr;
    RealTerm *dterms = nullptr;
    auto cleanup = [&]() {
        cudaFree(V);
        cudaFree(w);
        cudaFree(part);
        cudaFree(coef);
        cudaFree(dterms);
        cudaStreamDestroy(st);
    };
    cudaError_t e;
    if ((e = device_malloc(&V, sizeof(double) * N * (kmax + 1))) ||
        (e = device_malloc(&w, sizeof(double) * N)) ||
        (e = device_malloc(&part, sizeof(double) * kDotBlocks * (kmax + 1))) ||
        (e = device_malloc(&coef, sizeof(double) * (kmax + 1))) ||
        (e = device_malloc(&dterms, sizeof(RealTerm) * rt.size()))) {
        cleanup();
        return set_error(e == cudaErrorMemoryAllocation ? LQ_ERR_OOM : LQ_ERR_CUDA, "%s",
                         cudaGetErrorString(e));
    }
    if ((e = cudaMemcpy(dterms, rt.data(), sizeof(RealTerm) * rt.size(),
                        cudaMemcpyHostToDevice)) != cudaSuccess) {
        cleanup();
        return set_error(LQ_ERR_CUDA, "%s", cudaGetErrorString(e));
    }
    {  // seeded random start vector (host), normalised
        std::vector<double> v0(N);
        std::mt19937_64 rng(seed);
        std::normal_distribution<double> nd(0.0, 1.0);
        double s = 0.0;
        for (auto &x : v0) {
            x = nd(rng);
            s += x * x;
        }
        s = 1.0 / std::sqrt(s);
        for (auto &x : v0) x *= s;
        if ((e = cudaMemcpy(V, v0.data(), sizeof(double) * N, cudaMemcpyHostToDevice)) !=
            cudaSuccess) {
            cleanup();
            return set_error(LQ_ERR_CUDA, "%s", cudaGetErrorString(e));
        }
    }
    // <V_j, x> for j < count, block partials summed on the host in a fixed order.
    std::vector<double> hpart((size_t)kDotBlocks * (kmax + 1)), hc(kmax + 1);
    cudaError_t err = cudaSuccess;  // first failure of any launch or copy below
    auto note = [&](cudaError_t r) {
        if (err == cudaSuccess && r != cudaSuccess) err = r;
    };
    auto dots = [&](const double *Vb, int count, const double *x) {
        k_multi_dot<<<dim3(kDotBlocks, count), 256, 0, st>>>(Vb, x, N, part);
        note(cudaGetLastError());
        note(cudaMemcpyAsync(hpart.data(), part, sizeof(double) * kDotBlocks * count,
                             cudaMemcpyDeviceToHost, st));
        note(cudaStreamSynchronize(st));
        for (int j = 0; j < count; ++j) {
            double s = 0.0;
            for (int b = 0; b < kDotBlocks; ++b) s += hpart[(size_t)j * kDotBlocks + b];
            hc[j] = s;
        }
    };
    const int grid = (int)std::min<uint64_t>(1184, (N + 255) / 256);
    std::vector<double> alpha, beta;
    double prev = 1e300, ev = 0.0;
    int k;
    for (k = 0; k < kmax; ++k) {
        double *vk = V + (size_t)k * N;
        k_pauli_matvec<<<grid, 256, sizeof(RealTerm) * rt.size(), st>>>(vk, w, num_qubits, dterms,
                                                                          (int)rt.size());
        dots(vk, 1, w);
        const double a = hc[0];
        alpha.push_back(a);
        k_axpy<<<grid, 256, 0, st>>>(w, vk, -a, N);
        if (k > 0) k_axpy<<<grid, 256, 0, st>>>(w, V + (size_t)(k - 1) * N, -beta[k - 1], N);
        // full reorthogonalisation against V_0..V_k, classical Gram-Schmidt twice
        for (int pass = 0; pass < 2; ++pass) {
            dots(V, k + 1, w);
            note(cudaMemcpyAsync(coef, hc.data(), sizeof(double) * (k + 1),
                                 cudaMemcpyHostToDevice, st));
            k_multi_sub<<<grid, 256, 0, st>>>(V, coef, k + 1, N, w);
        }
        dots(w, 1, w);
        const double b = std::sqrt(std::max(hc[0], 0.0));
        if (err != cudaSuccess) break;
        ev = tridiag_min_eig(alpha, beta);
        if (std::fabs(ev - prev) < tol || b < 1e-12) {
            ++k;
            break;
        }
        prev = ev;
        beta.push_back(b);
        k_scale<<<grid, 256, 0, st>>>(V + (size_t)(k + 1) * N, w, 1.0 / b, N);
    }
    e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = err;
    cleanup();
    if (e != cudaSuccess) return set_error(LQ_ERR_CUDA, "%s", cudaGetErrorString(e));
    *e0 = ev;
    if (iters) *iters = k;
    return LQ_OK;
}

}  // extern "C"
