// Memory-bound neighbours of the contraction path in a training step, on the layout the contraction
// kernels keep between layers (fp16 NHWC, i.e. a row-major [pixels][channels] matrix):
//   * batch normalisation fused with the activation and the residual add that follow it, forward and
//     backward (replaces the reference's fp32-NCHW Welford / normalize / backward kernels,
//     nectarml/csrc/kernels/tensor/fused/norm.cu, and the separate ReLU / LeakyReLU / add passes
//     around them);
//   * one unscale + finiteness check and one SGD-momentum update over a FLAT parameter buffer
//     (replaces one unscale launch + cudaMalloc + blocking read-back per parameter,
//     nectarml/csrc/ops/amp/amp.cpp:18-37, and one update launch per parameter,
//     nectarml/optim/sgd.py:75-90, nectarml/csrc/kernels/optim/sgd.cu).
// Every reduction is two-stage with a fixed order (no atomics): results are bitwise repeatable.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/nectarml_b200.h"
#include "nml_launch.cuh"

namespace nml_layers {

#define NMLL_CUDA(expr)                              \
    do {                                             \
        cudaError_t e_ = (expr);                     \
        if (e_ != cudaSuccess) return NML_ERR_CUDA;  \
    } while (0)

using nml::launch;
using nml::launch_with;
using nml::load_global;
using nml::load_streaming;
using nml::pdl_enter;

static inline size_t round_up(size_t v, size_t m) { return (v + m - 1) / m * m; }
static std::atomic<long long> g_layer_launches{0};

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 t = __half22float2(h[j]);
        f[2 * j] = t.x;
        f[2 * j + 1] = t.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint4 v;
    __half2* h = reinterpret_cast<__half2*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2half2_rn(f[2 * j], f[2 * j + 1]);
    return v;
}
// Thread layout shared by the kernels below: the matrix is [M][C] fp16 with C a multiple of 8, a
// vector is 8 adjacent channels (16 bytes), cpr = C / 8 vectors per row.  A block has
// (256 / cpr) * cpr threads; thread t owns vector column t % cpr for good (its per-channel
// constants sit in registers) and walks rows t / cpr, + rows-per-pass, ...: consecutive threads read
// consecutive 16-byte vectors, so every access is fully coalesced whatever C is.

// How a backward pass finds the derivative of the activation.
enum {
    D_NONE = 0,  // no activation
    D_Y = 1,     // from the activation's output, which is read again (the C entry point that is given y alone)
    D_X = 2,     // from the normalisation's input, which the pass reads anyway: the sign of gamma * xhat + beta
    D_MASK = 3   // from one bit per element that the forward wrote (a residual was added, so x alone does not tell)
};
// D_X and D_MASK keep y out of the backward: a 256-channel 56 x 56 layer at batch 256 (411 MB per tensor) reads 1.23 -> 0.85
// GB in the reduction and moves 2.05 -> 1.67 GB in the second pass.

// y = half(t) is positive exactly when t is above half of the smallest fp16 subnormal (ties go to zero).
__device__ __forceinline__ bool positive_as_half(float t) { return t > 2.98023223876953125e-8f; }

// The eight values of a vector's channels from a per-channel array, in two loads.  A thread owns its channels for good, so a
// block pays for its constants once, but with one 4-byte load per value (32 bytes apart in a warp) that was eight times
// the L1 wavefronts and cost a block as much as several rows of the tensor.  Callers' arrays may start anywhere.
__device__ __forceinline__ void load8(const float* p, int col, float (&f)[8]) {
    p += col * 8;
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        const float4 a = load_global(reinterpret_cast<const float4*>(p)), b = load_global(reinterpret_cast<const float4*>(p) + 1);
        f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = load_global(p + j);
    }
}
__device__ __forceinline__ void load8_or(const float* p, int col, float otherwise, float (&f)[8]) {
    if (p) {
        load8(p, col, f);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = otherwise;
    }
}

// Per-channel constants of the forward's y = act(sc * x + sh), as the forward computes them.
__device__ __forceinline__ void bn_affine(int col, const float* gamma, const float* beta,
                                          const float* mean, const float* rstd, float (&sc)[8], float (&sh)[8]) {
    float r[8], m[8];
    load8_or(gamma, col, 1.f, sc);
    load8_or(beta, col, 0.f, sh);
    load8(rstd, col, r);
    load8(mean, col, m);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        sc[j] *= r[j];
        sh[j] -= m[j] * sc[j];
    }
}

// dz = dy * act'(.) of one vector.
template <int kDeriv>
__device__ __forceinline__ void act_backward(float (&df)[8], const float (&xf)[8], const uint4& yv, unsigned bits, const float (&sc)[8],
                                             const float (&sh)[8], float below) {
    if (kDeriv == D_Y) {
        float yf[8];
        unpack8(yv, yf);
#pragma unroll
        for (int j = 0; j < 8; ++j) df[j] *= yf[j] > 0.f ? 1.f : below;
    } else if (kDeriv == D_X) {
#pragma unroll
        for (int j = 0; j < 8; ++j) df[j] *= positive_as_half(xf[j] * sc[j] + sh[j]) ? 1.f : below;
    } else if (kDeriv == D_MASK) {
#pragma unroll
        for (int j = 0; j < 8; ++j) df[j] *= ((bits >> j) & 1u) ? 1.f : below;
    }
}

// The gradient of a pass's output: one fp16 tensor, or the sum of two (the output was read by the next layer and, as part of
// the channels of a concatenation, by a later one).  Either may be part of the channels of a wider tensor: rows are `row`
// (`row2`) vectors apart.  Reading both here keeps the slice's copy and the sum out of memory.
struct OutGrad {
    const uint4 *a, *b;
    int row, row2;
};
struct OutGradVector {
    uint4 a, b;
};
template <bool kTwo>
__device__ __forceinline__ OutGradVector load_grad(const OutGrad& g, size_t row, int col) {
    OutGradVector v;
    v.a = load_global(g.a + row * g.row + col);
    if (kTwo) v.b = load_global(g.b + row * g.row2 + col);
    return v;
}
template <bool kTwo>
__device__ __forceinline__ void unpack_grad(const OutGradVector& v, float (&f)[8]) {
    unpack8(v.a, f);
    if (kTwo) {
        float t[8];
        unpack8(v.b, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += t[j];
    }
}

// What a backward pass reads of the forward besides x: see the D_* above.  `below` is the derivative where y <= 0.
struct BnForward {
    const uint4* y;
    const uint8_t* mask;
    const float *gamma, *beta, *mean, *rstd;
    float below;
};

// First stage of a per-channel reduction over rows.  Block p writes its sums to partial[p][0..C) and partial[p][C..2C).
__device__ __forceinline__ void bn_store_partial(float (*sm)[17], const float (&a)[8], const float (&b)[8], int cpr, int rpb, int C,
                                                 float* __restrict__ partial) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        sm[threadIdx.x][j] = a[j];
        sm[threadIdx.x][8 + j] = b[j];
    }
    __syncthreads();
    // fixed order over the block's row lanes, a thread to a sum (in the threads of the first row alone, sixteen sums each: 12544 x 1024 forward
    // 28.8 us instead of 25.4, 262144 x 64 31.1 / 29.0, backward 41.0 / 38.9)
    float* out = partial + static_cast<size_t>(blockIdx.x) * 2 * C;
    for (int o = threadIdx.x; o < 16 * cpr; o += blockDim.x) {
        const int col = o >> 4, j = o & 15;
        float s = 0.f;
#pragma unroll 4
        for (int r = 0; r < rpb; ++r) s += sm[r * cpr + col][j];
        out[(j < 8 ? 0 : C - 8) + col * 8 + j] = s;
    }
}

// Forward statistics: a = sum x, b = sum x^2; four rows in flight per thread.
// (Blocks whose rows follow one another read a tensor of 411 MB in 74 us instead of 83, but sum it in another order: a mean that rounds the
// other way flips single ReLUs behind it, which is not worth half a percent of a block's step.)
__global__ void __launch_bounds__(256) bn_stats_kernel(const uint4* x, float* __restrict__ partial, size_t M, int C) {
    pdl_enter();
    __shared__ float sm[256][17];
    const int cpr = C >> 3;
    const int rpb = blockDim.x / cpr;
    const int col = threadIdx.x % cpr, rsub = threadIdx.x / cpr;
    float a[8], b[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = b[j] = 0.f;
    auto add = [&](const uint4& xv) {
        float xf[8];
        unpack8(xv, xf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            a[j] += xf[j];
            b[j] += xf[j] * xf[j];
        }
    };
    const size_t stride = static_cast<size_t>(gridDim.x) * rpb;
    size_t row = static_cast<size_t>(blockIdx.x) * rpb + rsub;
    for (; row + 3 * stride < M; row += 4 * stride) {
        const uint4 x0 = load_global(x + row * cpr + col), x1 = load_global(x + (row + stride) * cpr + col);
        const uint4 x2 = load_global(x + (row + 2 * stride) * cpr + col), x3 = load_global(x + (row + 3 * stride) * cpr + col);
        add(x0);
        add(x1);
        add(x2);
        add(x3);
    }
    for (; row < M; row += stride) add(load_global(x + row * cpr + col));
    bn_store_partial(sm, a, b, cpr, rpb, C, partial);
}

// Backward sums: with dz = dy * act'(.): a = sum dz, b = sum dz * x (the second stage turns b into
// d gamma = rstd * (b - mean * a), so this pass needs no per-channel constants but those of D_X).  Two rows in flight per
// thread.
template <int kDeriv, bool kTwo>
__global__ void __launch_bounds__(256) bn_grad_sums_kernel(const uint4* x, const OutGrad dy, const BnForward f,
                                                           float* __restrict__ partial, size_t M, int C) {
    pdl_enter();
    __shared__ float sm[256][17];
    const int cpr = C >> 3;
    const int rpb = blockDim.x / cpr;
    const int col = threadIdx.x % cpr, rsub = threadIdx.x / cpr;
    float a[8], b[8], sc[8], sh[8];
    if (kDeriv == D_X) bn_affine(col, f.gamma, f.beta, f.mean, f.rstd, sc, sh);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = b[j] = 0.f;
    auto add = [&](const uint4& xv, const OutGradVector& dv, const uint4& yv, unsigned bits) {
        float xf[8], df[8];
        unpack8(xv, xf);
        unpack_grad<kTwo>(dv, df);
        act_backward<kDeriv>(df, xf, yv, bits, sc, sh, f.below);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            a[j] += df[j];
            b[j] += df[j] * xf[j];
        }
    };
    const size_t stride = static_cast<size_t>(gridDim.x) * rpb;
    size_t row = static_cast<size_t>(blockIdx.x) * rpb + rsub;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (; row + stride < M; row += 2 * stride) {
        const size_t v0 = row * cpr + col, v1 = (row + stride) * cpr + col;
        const uint4 x0 = load_global(x + v0), x1 = load_global(x + v1);
        const OutGradVector d0 = load_grad<kTwo>(dy, row, col), d1 = load_grad<kTwo>(dy, row + stride, col);
        const uint4 y0 = kDeriv == D_Y ? load_global(f.y + v0) : zero, y1 = kDeriv == D_Y ? load_global(f.y + v1) : zero;
        const unsigned m0 = kDeriv == D_MASK ? load_global(f.mask + v0) : 0u, m1 = kDeriv == D_MASK ? load_global(f.mask + v1) : 0u;
        add(x0, d0, y0, m0);
        add(x1, d1, y1, m1);
    }
    if (row < M) {
        const size_t v0 = row * cpr + col;
        add(load_global(x + v0), load_grad<kTwo>(dy, row, col), kDeriv == D_Y ? load_global(f.y + v0) : zero, kDeriv == D_MASK ? load_global(f.mask + v0) : 0u);
    }
    bn_store_partial(sm, a, b, cpr, rpb, C, partial);
}

// Second stage: adds the P rows of partial sums in a fixed order (128 interleaved running sums in double,
// then those 128 in a tree).  mode 0: out0 = mean, out1 = 1 / sqrt(biased variance + eps).
// mode 1: out0 = sum a (d beta), out1 = rstd * (sum b - mean * sum a) (d gamma).  blockDim = (8, 128): the pass is a chain of
// load latencies, so it is spread over many blocks and a thread's few loads are all in flight (32 channels a block and
// 19 rows a thread took 6 us; a U-Net step runs it 26 times).
__global__ void __launch_bounds__(1024) bn_finish_kernel(const float* partial, int P, int C, int mode, double inv_M,
                                                        float eps, const float* mean, const float* rstd,
                                                        float* __restrict__ out0, float* __restrict__ out1) {
    pdl_enter();
    __shared__ double pa[128][9], pb[128][9];
    const int c = blockIdx.x * 8 + threadIdx.x;
    double sa = 0.0, sb = 0.0;
#pragma unroll 5
    for (int p = threadIdx.y; p < P; p += 128) {
        sa += static_cast<double>(load_global(partial + static_cast<size_t>(p) * 2 * C + c));
        sb += static_cast<double>(load_global(partial + static_cast<size_t>(p) * 2 * C + C + c));
    }
    pa[threadIdx.y][threadIdx.x] = sa;
    pb[threadIdx.y][threadIdx.x] = sb;
    for (int half = 64; half > 0; half /= 2) {
        __syncthreads();
        if (threadIdx.y < half) {
            pa[threadIdx.y][threadIdx.x] += pa[threadIdx.y + half][threadIdx.x];
            pb[threadIdx.y][threadIdx.x] += pb[threadIdx.y + half][threadIdx.x];
        }
    }
    if (threadIdx.y == 0) {
        const double ta = pa[0][threadIdx.x], tb = pb[0][threadIdx.x];
        if (mode == 0) {
            const double m = ta * inv_M;
            double var = tb * inv_M - m * m;
            if (var < 0.0) var = 0.0;
            out0[c] = static_cast<float>(m);
            out1[c] = static_cast<float>(1.0 / sqrt(var + static_cast<double>(eps)));
        } else {
            out0[c] = static_cast<float>(ta);
            out1[c] = static_cast<float>(static_cast<double>(load_global(rstd + c)) * (tb - static_cast<double>(load_global(mean + c)) * ta));
        }
    }
}

// y = act(gamma * (x - mean) * rstd + beta [+ residual]), fp16 in and out; two rows in flight per thread.  With `mask`
// one bit per element, set where y > 0, for D_MASK.  The rows are walked from the last to the first: the statistics pass
// has just read x in the other direction, so what of it is still in L2 (126 MB) is read first.
// y (and y2, a second copy) may be part of the channels of a wider tensor: their rows are y_row and y2_row vectors apart.
__global__ void __launch_bounds__(256, 4) bn_apply_kernel(const uint4* x, const uint4* res,
                                                       uint4* __restrict__ y, int y_row, uint4* __restrict__ y2, int y2_row,
                                                       uint8_t* __restrict__ mask, const float* gamma,
                                                       const float* beta, const float* mean,
                                                       const float* rstd, int act, float slope, size_t M, int C) {
    pdl_enter();
    const int cpr = C >> 3;
    const int rpb = blockDim.x / cpr;
    const int col = threadIdx.x % cpr, rsub = threadIdx.x / cpr;
    float sc[8], sh[8];
    bn_affine(col, gamma, beta, mean, rstd, sc, sh);
    auto one = [&](size_t row, const uint4& xv, const uint4& rv) {
        float xf[8], rf[8];
        unpack8(xv, xf);
        if (res) unpack8(rv, rf);
        unsigned bits = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float t = xf[j] * sc[j] + sh[j];
            if (res) t += rf[j];
            bits |= (positive_as_half(t) ? 1u : 0u) << j;
            if (act != 0 && t < 0.f) t = (act == 1) ? 0.f : t * slope;
            xf[j] = t;
        }
        const uint4 out = pack8(xf);
        y[row * y_row + col] = out;
        if (y2) y2[row * y2_row + col] = out;
        if (mask) mask[row * cpr + col] = static_cast<uint8_t>(bits);
    };
    const size_t stride = static_cast<size_t>(gridDim.x) * rpb;
    size_t k = static_cast<size_t>(blockIdx.x) * rpb + rsub;  // rows counted from the end
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (; k + stride < M; k += 2 * stride) {
        const size_t v0 = (M - 1 - k) * cpr + col, v1 = (M - 1 - k - stride) * cpr + col;
        const uint4 x0 = load_global(x + v0), x1 = load_global(x + v1);
        const uint4 r0 = res ? load_global(res + v0) : zero, r1 = res ? load_global(res + v1) : zero;
        one(M - 1 - k, x0, r0);
        one(M - 1 - k - stride, x1, r1);
    }
    if (k < M) {
        const size_t v0 = (M - 1 - k) * cpr + col;
        one(M - 1 - k, load_global(x + v0), res ? load_global(res + v0) : zero);
    }
}

// dx = gamma * rstd * (dz - dbeta / M - xhat * dgamma / M) with dz = dy * act'(.), folded into
// dx = A * dz + B * x + C per channel; optionally dres = dz (the gradient of the residual input that was
// added before the activation).  Two rows in flight per thread, from the last row to the first as in bn_apply_kernel.
template <int kDeriv, bool kTwo>
__global__ void __launch_bounds__(256, 3) bn_dx_kernel(const uint4* x, const OutGrad dy, const BnForward f,
                                                    uint4* __restrict__ dx, uint4* __restrict__ dres, const float* dbeta,
                                                    const float* dgamma, float inv_M, size_t M, int C) {
    pdl_enter();
    const int cpr = C >> 3;
    const int rpb = blockDim.x / cpr;
    const int col = threadIdx.x % cpr, rsub = threadIdx.x / cpr;
    float ka[8], kb[8], kc[8], sc[8], sh[8];
    if (kDeriv == D_X) bn_affine(col, f.gamma, f.beta, f.mean, f.rstd, sc, sh);
    {
        float rs[8], mu[8];
        load8_or(f.gamma, col, 1.f, ka);
        load8(f.rstd, col, rs);
        load8(f.mean, col, mu);
        load8(dbeta, col, kc);
        load8(dgamma, col, kb);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float k1 = kc[j] * inv_M, k2 = kb[j] * inv_M;
            ka[j] *= rs[j];
            kb[j] = -ka[j] * rs[j] * k2;
            kc[j] = ka[j] * (mu[j] * rs[j] * k2 - k1);
        }
    }
    auto one = [&](size_t v, const uint4& xv, const OutGradVector& dv, const uint4& yv, unsigned bits) {
        float xf[8], df[8];
        unpack8(xv, xf);
        unpack_grad<kTwo>(dv, df);
        act_backward<kDeriv>(df, xf, yv, bits, sc, sh, f.below);
#pragma unroll
        for (int j = 0; j < 8; ++j) xf[j] = ka[j] * df[j] + kb[j] * xf[j] + kc[j];
        dx[v] = pack8(xf);
        if (dres) dres[v] = pack8(df);
    };
    const size_t stride = static_cast<size_t>(gridDim.x) * rpb;
    size_t k = static_cast<size_t>(blockIdx.x) * rpb + rsub;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (; k + stride < M; k += 2 * stride) {
        const size_t v0 = (M - 1 - k) * cpr + col, v1 = (M - 1 - k - stride) * cpr + col;
        const uint4 x0 = load_global(x + v0), x1 = load_global(x + v1);
        const OutGradVector d0 = load_grad<kTwo>(dy, M - 1 - k, col), d1 = load_grad<kTwo>(dy, M - 1 - k - stride, col);
        const uint4 y0 = kDeriv == D_Y ? load_global(f.y + v0) : zero, y1 = kDeriv == D_Y ? load_global(f.y + v1) : zero;
        const unsigned m0 = kDeriv == D_MASK ? load_global(f.mask + v0) : 0u, m1 = kDeriv == D_MASK ? load_global(f.mask + v1) : 0u;
        one(v0, x0, d0, y0, m0);
        one(v1, x1, d1, y1, m1);
    }
    if (k < M) {
        const size_t v0 = (M - 1 - k) * cpr + col;
        one(v0, load_global(x + v0), load_grad<kTwo>(dy, M - 1 - k, col), kDeriv == D_Y ? load_global(f.y + v0) : zero, kDeriv == D_MASK ? load_global(f.mask + v0) : 0u);
    }
}

// ---- Small tensors: a whole pass in one launch.
// The three kernels of a pass spend 8 to 10 us on a tensor of a few KB: launches, drains and load latency.
// Here a cluster of eight blocks owns 8 * gv channels: each block reads its eighth of the rows once into shared memory and sums
// as it goes, the blocks exchange their sums through distributed shared memory, and every thread finishes its own vectors.
// No second read, no partial sums in memory, and the order of every sum is fixed.
constexpr int kClusterBlocks = 8, kClusterThreads = 256;
constexpr int kMaxGv = 16;                       // channels: at most 2048, in about 16 clusters
constexpr size_t kClusterShare = 32 * 1024;      // of each tensor per block

// Sums of a thread's (a, b) over its block and the cluster; then finish(channel of the cluster's, sum a, sum b) once per
// channel, before the block goes on.
template <class F>
__device__ __forceinline__ void cluster_sums(const float (&a)[8], const float (&b)[8], int gv, float (*part)[16 * kMaxGv], F&& finish) {
    namespace cg = cooperative_groups;
    auto cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v[16];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = a[j], v[8 + j] = b[j];
    for (int o = 16; o >= gv; o /= 2) {  // lanes of one vector column are gv apart
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
    }
    if (lane < gv) {
#pragma unroll
        for (int j = 0; j < 16; ++j) part[warp][lane * 16 + j] = v[j];
    }
    __syncthreads();
    const int n = 16 * gv;  // at most kClusterThreads
    float* mine = part[kClusterThreads / 32];
    if (threadIdx.x < n) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kClusterThreads / 32; ++w) s += part[w][threadIdx.x];
        mine[threadIdx.x] = s;
    }
    cluster.sync();
    if (threadIdx.x < n / 2) {
        const int i = threadIdx.x / 8 * 16 + threadIdx.x % 8;
        double ta = 0.0, tb = 0.0;
#pragma unroll
        for (int r = 0; r < kClusterBlocks; ++r) {
            const float* theirs = cluster.map_shared_rank(mine, r);
            ta += static_cast<double>(theirs[i]);
            tb += static_cast<double>(theirs[i + 8]);
        }
        finish(static_cast<int>(threadIdx.x), ta, tb);
    }
    __syncthreads();
}

struct ClusterShare {  // a block's share of the tensor and a thread's place in it
    size_t first, last;
    int col, lane, lanes;
};
__device__ __forceinline__ ClusterShare cluster_share(size_t M, int gv) {
    ClusterShare s;
    const int rank = blockIdx.x % kClusterBlocks;
    const size_t per = (M + kClusterBlocks - 1) / kClusterBlocks;
    s.first = min(M, rank * per);
    s.last = min(M, s.first + per);
    s.lanes = kClusterThreads / gv;
    s.lane = threadIdx.x / gv;
    s.col = blockIdx.x / kClusterBlocks * gv + threadIdx.x % gv;
    return s;
}

__global__ void __launch_bounds__(kClusterThreads) bn_cluster_forward_kernel(
    const uint4* x, const uint4* res, uint4* __restrict__ y, int y_row, uint4* __restrict__ y2, int y2_row,
    uint8_t* __restrict__ mask, const float* gamma, const float* beta, float* __restrict__ mean,
    float* __restrict__ rstd, int act, float slope, float eps, double inv_M, size_t M, int C, int gv) {
    pdl_enter();
    extern __shared__ uint4 keep[];
    __shared__ float part[kClusterThreads / 32 + 1][16 * kMaxGv];
    __shared__ float done[2][8 * kMaxGv];  // per channel of the cluster's
    const int cpr = C >> 3;
    const ClusterShare s = cluster_share(M, gv);
    float a[8], b[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = b[j] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    constexpr int kFlight = 8;  // rows a thread has in flight
    int k = threadIdx.x;
    for (size_t row = s.first + s.lane; row < s.last; row += kFlight * s.lanes, k += kFlight * kClusterThreads) {
        uint4 v[kFlight];
#pragma unroll
        for (int i = 0; i < kFlight; ++i) v[i] = row + i * s.lanes < s.last ? load_global(x + (row + i * s.lanes) * cpr + s.col) : zero;
#pragma unroll
        for (int i = 0; i < kFlight; ++i) {
            float f[8];
            unpack8(v[i], f);
            if (row + i * s.lanes < s.last) keep[k + i * kClusterThreads] = v[i];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                a[j] += f[j];
                b[j] += f[j] * f[j];
            }
        }
    }
    const int c0 = blockIdx.x / kClusterBlocks * gv * 8;
    cluster_sums(a, b, gv, part, [&](int c, double ta, double tb) {
        const double m = ta * inv_M;
        double var = tb * inv_M - m * m;
        if (var < 0.0) var = 0.0;
        done[0][c] = static_cast<float>(m);
        done[1][c] = static_cast<float>(1.0 / sqrt(var + static_cast<double>(eps)));
        if (blockIdx.x % kClusterBlocks == 0) {
            mean[c0 + c] = done[0][c];
            rstd[c0 + c] = done[1][c];
        }
    });
    float sc[8], sh[8];
    load8_or(gamma, s.col, 1.f, sc);
    load8_or(beta, s.col, 0.f, sh);
    const int base = threadIdx.x % gv * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        sc[j] *= done[1][base + j];
        sh[j] -= done[0][base + j] * sc[j];
    }
    k = threadIdx.x;
#pragma unroll 2
    for (size_t row = s.first + s.lane; row < s.last; row += s.lanes, k += kClusterThreads) {
        float f[8], rf[8];
        unpack8(keep[k], f);
        if (res) unpack8(load_global(res + row * cpr + s.col), rf);
        unsigned bits = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float t = f[j] * sc[j] + sh[j];
            if (res) t += rf[j];
            bits |= (positive_as_half(t) ? 1u : 0u) << j;
            if (act != 0 && t < 0.f) t = (act == 1) ? 0.f : t * slope;
            f[j] = t;
        }
        const uint4 out = pack8(f);
        y[row * y_row + s.col] = out;
        if (y2) y2[row * y2_row + s.col] = out;
        if (mask) mask[row * cpr + s.col] = static_cast<uint8_t>(bits);
    }
    cooperative_groups::this_cluster().sync();  // no block leaves while another reads its sums
}

template <int kDeriv, bool kTwo>
__global__ void __launch_bounds__(kClusterThreads) bn_cluster_backward_kernel(
    const uint4* x, const OutGrad dy, const BnForward f, uint4* __restrict__ dx, uint4* __restrict__ dres,
    float* __restrict__ dbeta, float* __restrict__ dgamma, double inv_M, size_t M, int C, int gv) {
    pdl_enter();
    extern __shared__ uint4 keep[];  // [x, dy (, second dy)][share]
    __shared__ float part[kClusterThreads / 32 + 1][16 * kMaxGv];
    __shared__ float done[2][8 * kMaxGv];  // per channel of the cluster's
    const int cpr = C >> 3;
    const ClusterShare s = cluster_share(M, gv);
    const size_t share = (M + kClusterBlocks - 1) / kClusterBlocks;
    const int vectors = static_cast<int>((share + s.lanes - 1) / s.lanes) * kClusterThreads;
    float a[8], b[8], sc[8], sh[8];
    if (kDeriv == D_X) bn_affine(s.col, f.gamma, f.beta, f.mean, f.rstd, sc, sh);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = b[j] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    constexpr int kFlight = kTwo ? 2 : 4;
    int k = threadIdx.x;
    for (size_t row = s.first + s.lane; row < s.last; row += kFlight * s.lanes, k += kFlight * kClusterThreads) {
        uint4 xv[kFlight], yv[kFlight];
        OutGradVector dv[kFlight];
        unsigned bits[kFlight];
#pragma unroll
        for (int i = 0; i < kFlight; ++i) {
            const size_t r = row + i * s.lanes, v = r * cpr + s.col;
            const bool in = r < s.last;
            xv[i] = in ? load_global(x + v) : zero;
            dv[i].a = dv[i].b = zero;
            if (in) dv[i] = load_grad<kTwo>(dy, r, s.col);
            yv[i] = kDeriv == D_Y && in ? load_global(f.y + v) : zero;
            bits[i] = kDeriv == D_MASK && in ? load_global(f.mask + v) : 0u;
        }
#pragma unroll
        for (int i = 0; i < kFlight; ++i) {
            if (row + i * s.lanes >= s.last) break;
            float xf[8], df[8];
            unpack8(xv[i], xf);
            unpack_grad<kTwo>(dv[i], df);
            act_backward<kDeriv>(df, xf, yv[i], bits[i], sc, sh, f.below);
            const int at = k + i * kClusterThreads;
            keep[at] = xv[i];
            keep[vectors + at] = dv[i].a;
            if (kTwo) keep[2 * vectors + at] = dv[i].b;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                a[j] += df[j];
                b[j] += df[j] * xf[j];
            }
        }
    }
    const int c0 = blockIdx.x / kClusterBlocks * gv * 8;
    cluster_sums(a, b, gv, part, [&](int c, double ta, double tb) {
        done[0][c] = static_cast<float>(ta);
        done[1][c] = static_cast<float>(static_cast<double>(load_global(f.rstd + c0 + c)) * (tb - static_cast<double>(load_global(f.mean + c0 + c)) * ta));
        if (blockIdx.x % kClusterBlocks == 0) {
            dbeta[c0 + c] = done[0][c];
            dgamma[c0 + c] = done[1][c];
        }
    });
    float ka[8], kb[8], kc[8];
    {
        float rs[8], mu[8];
        load8_or(f.gamma, s.col, 1.f, ka);
        load8(f.rstd, s.col, rs);
        load8(f.mean, s.col, mu);
        const int base = threadIdx.x % gv * 8;
        const float inv = static_cast<float>(inv_M);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float k1 = done[0][base + j] * inv, k2 = done[1][base + j] * inv;
            ka[j] *= rs[j];
            kb[j] = -ka[j] * rs[j] * k2;
            kc[j] = ka[j] * (mu[j] * rs[j] * k2 - k1);
        }
    }
    k = threadIdx.x;
    for (size_t row = s.first + s.lane; row < s.last; row += s.lanes, k += kClusterThreads) {
        const size_t v = row * cpr + s.col;
        OutGradVector dv;
        dv.a = keep[vectors + k];
        if (kTwo) dv.b = keep[2 * vectors + k];
        const uint4 yv = kDeriv == D_Y ? load_global(f.y + v) : zero;
        const unsigned bits = kDeriv == D_MASK ? load_global(f.mask + v) : 0u;
        float xf[8], df[8];
        unpack8(keep[k], xf);
        unpack_grad<kTwo>(dv, df);
        act_backward<kDeriv>(df, xf, yv, bits, sc, sh, f.below);
#pragma unroll
        for (int j = 0; j < 8; ++j) xf[j] = ka[j] * df[j] + kb[j] * xf[j] + kc[j];
        dx[v] = pack8(xf);
        if (dres) dres[v] = pack8(df);
    }
    cooperative_groups::this_cluster().sync();
}

// An activation that no normalisation stands in front of: y = act(x), with a second copy as part of the channels of a wider
// tensor.  rows x C, thread layout and grid as above.
__global__ void __launch_bounds__(256, 4) act_kernel(const uint4* x, uint4* __restrict__ y, uint4* __restrict__ y2,
                                                     int y2_row, float below, size_t M, int C) {
    pdl_enter();
    const int cpr = C >> 3;
    const int rpb = blockDim.x / cpr;
    const int col = threadIdx.x % cpr;
    const size_t stride = static_cast<size_t>(gridDim.x) * rpb;
#pragma unroll 2
    for (size_t row = static_cast<size_t>(blockIdx.x) * rpb + threadIdx.x / cpr; row < M; row += stride) {
        float f[8];
        unpack8(load_global(x + row * cpr + col), f);
#pragma unroll
        for (int j = 0; j < 8; ++j)  // NaN stays NaN, -0 becomes 0; below = 0 is a choice, not a product: of -inf too
            f[j] = f[j] > 0.f ? f[j] : below != 0.f ? f[j] * below + 0.f : f[j] <= 0.f ? 0.f : f[j];
        const uint4 out = pack8(f);
        y[row * cpr + col] = out;
        if (y2) y2[row * y2_row + col] = out;
    }
}
// dx = dy * act'(x).
template <bool kTwo>
__global__ void __launch_bounds__(256, 4) act_backward_kernel(const uint4* x, const OutGrad dy, uint4* __restrict__ dx,
                                                              float below, size_t M, int C) {
    pdl_enter();
    const int cpr = C >> 3;
    const int rpb = blockDim.x / cpr;
    const int col = threadIdx.x % cpr;
    const size_t stride = static_cast<size_t>(gridDim.x) * rpb;
#pragma unroll 2
    for (size_t row = static_cast<size_t>(blockIdx.x) * rpb + threadIdx.x / cpr; row < M; row += stride) {
        float f[8], d[8];
        const OutGradVector g = load_grad<kTwo>(dy, row, col);
        unpack8(load_global(x + row * cpr + col), f);
        unpack_grad<kTwo>(g, d);
#pragma unroll
        for (int j = 0; j < 8; ++j)  // (an overflowed gradient does not pass where the ReLU is shut; NaN inputs let it pass)
            d[j] = f[j] > 0.f ? d[j] : below != 0.f ? d[j] * below : f[j] <= 0.f ? 0.f : d[j];
        dx[row * cpr + col] = pack8(d);
    }
}

// L1 loss sum |a - b| / denom of two fp16 tensors, in fp32 within a thread's share and in double over the blocks, fixed order.
// As separate passes (two conversions, difference, absolute value, sum; sign, product and conversion back) the loss of 16
// images of 256 x 256 took 60 us of small kernels each way and twice as long to issue.
__global__ void __launch_bounds__(256) l1_sum_kernel(const __half2* a, const __half2* b, size_t n, float* __restrict__ partial) {
    pdl_enter();
    float s = 0.f;
    const size_t n2 = n / 2, step = static_cast<size_t>(gridDim.x) * blockDim.x;
#pragma unroll 4
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n2; i += step) {
        const float2 u = __half22float2(load_global(a + i)), v = __half22float2(load_global(b + i));
        s += fabsf(u.x - v.x) + fabsf(u.y - v.y);
    }
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0)
        s += fabsf(__half2float(load_global(reinterpret_cast<const __half*>(a) + n - 1)) - __half2float(load_global(reinterpret_cast<const __half*>(b) + n - 1)));
    __shared__ float sm[8];
#pragma unroll
    for (int o = 16; o > 0; o /= 2) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x / 32] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        s = 0.f;
        for (int w = 0; w < 8; ++w) s += sm[w];
        partial[blockIdx.x] = s;
    }
}
__global__ void __launch_bounds__(32) l1_finish_kernel(const float* partial, int P, float denom, float* __restrict__ loss) {
    pdl_enter();
    double s = 0.0;
    for (int p = threadIdx.x; p < P; p += 32) s += static_cast<double>(load_global(partial + p));
#pragma unroll
    for (int o = 16; o > 0; o /= 2) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *loss = static_cast<float>(s) / denom;
}
// da = sign(a - b) * (*dloss / denom)
__global__ void __launch_bounds__(256) l1_backward_kernel(const __half2* a, const __half2* b, size_t n,
                                                          const float* dloss, float denom, __half2* __restrict__ da) {
    pdl_enter();
    const float g = load_global(dloss) / denom;
    auto one = [&](float d) { return d > 0.f ? g : d < 0.f ? -g : 0.f; };
    const size_t n2 = n / 2, step = static_cast<size_t>(gridDim.x) * blockDim.x;
#pragma unroll 4
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n2; i += step) {
        const float2 u = __half22float2(load_global(a + i)), v = __half22float2(load_global(b + i));
        da[i] = __floats2half2_rn(one(u.x - v.x), one(u.y - v.y));
    }
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0)
        reinterpret_cast<__half*>(da)[n - 1] = __float2half_rn(
            one(__half2float(load_global(reinterpret_cast<const __half*>(a) + n - 1)) - __half2float(load_global(reinterpret_cast<const __half*>(b) + n - 1))));
}

// any(!isfinite(g * inv_scale)) over a flat fp32 buffer -> *found (set, never cleared, here).  Four loads in flight per
// thread; 54 million values 46 -> 45 us.
__global__ void __launch_bounds__(256) grads_check_kernel(const float4* g, size_t n4, float inv_scale, int* found) {
    pdl_enter();
    bool bad = false;
    auto one = [&](const float4& v) {
        bad |= !isfinite(v.x * inv_scale) | !isfinite(v.y * inv_scale) | !isfinite(v.z * inv_scale) | !isfinite(v.w * inv_scale);
    };
    const size_t step = static_cast<size_t>(gridDim.x) * blockDim.x;
    size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
    for (; i + 3 * step < n4; i += 4 * step) {
        const float4 v0 = load_global(g + i), v1 = load_global(g + i + step), v2 = load_global(g + i + 2 * step), v3 = load_global(g + i + 3 * step);
        one(v0);
        one(v1);
        one(v2);
        one(v3);
    }
    for (; i < n4; i += step) one(load_global(g + i));
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *found = 1;  // every writer writes the same value
}

// One SGD-momentum update over the whole flat buffer: g = grad * inv_scale + wd * p; v = momentum * v +
// (1 - dampening) * g; p -= lr * v; and the fp16 copy of p the next forward reads.  Skipped as a whole
// when *found_inf is set (the GradScaler rule: an overflowed step leaves the parameters alone).
// Bound by memory (22 bytes a value).  Walked from the end to the start: the finiteness check has just read the gradients in
// the other direction, so those of the last parameters are in L2, and the fp16 copies of the first layers stay there for the next
// forward; parameters and velocity are streamed past (evict first).  54 million values 190 -> 184 us.
__global__ void __launch_bounds__(256) sgd_momentum_kernel(float4* __restrict__ p, const float4* g, float4* __restrict__ vel,
                                                           uint2* __restrict__ p16, size_t n4, float lr, float momentum, float dampening,
                                                           float wd, float inv_scale, const int* found_inf) {
    pdl_enter();
    if (found_inf && load_global(found_inf)) return;
    auto one = [&](size_t i, float4 pv, float4 vv, const float4& gv) {
        float* pp = reinterpret_cast<float*>(&pv);
        float* vp = reinterpret_cast<float*>(&vv);
        const float* gp = reinterpret_cast<const float*>(&gv);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float gg = gp[j] * inv_scale + wd * pp[j];
            vp[j] = momentum * vp[j] + (1.f - dampening) * gg;
            pp[j] -= lr * vp[j];
        }
        __stcs(p + i, pv);
        __stcs(vel + i, vv);
        if (p16) {
            uint2 h;
            *reinterpret_cast<__half2*>(&h.x) = __floats2half2_rn(pp[0], pp[1]);
            *reinterpret_cast<__half2*>(&h.y) = __floats2half2_rn(pp[2], pp[3]);
            p16[i] = h;
        }
    };
    const size_t step = static_cast<size_t>(gridDim.x) * blockDim.x;
    size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;  // counted from the end
    for (; k + step < n4; k += 2 * step) {
        const size_t i0 = n4 - 1 - k, i1 = i0 - step;
        const float4 p0 = load_streaming(p + i0), p1 = load_streaming(p + i1), v0 = load_streaming(vel + i0), v1 = load_streaming(vel + i1);
        const float4 g0 = load_global(g + i0), g1 = load_global(g + i1);
        one(i0, p0, v0, g0);
        one(i1, p1, v1, g1);
    }
    if (k < n4) {
        const size_t i = n4 - 1 - k;
        one(i, load_streaming(p + i), load_streaming(vel + i), load_global(g + i));
    }
}

// Max pooling over NHWC fp16, 8 channels per thread.  Forward also records, per output value, which tap of
// the window won (kh * k + kw, one byte); backward is a GATHER over the <= ceil(k/s)^2 windows that cover an
// input pixel -- no atomics, so it is bitwise repeatable, and every input gradient is written exactly once
// (no zero-fill pass).  Out-of-image taps are skipped (i.e. padded with -inf).
__global__ void __launch_bounds__(256) maxpool_fwd_kernel(const uint4* x, uint4* __restrict__ y, uint2* __restrict__ idx,
                                                          int N, int H, int W, int C, int k, int s, int p, int Ho, int Wo) {
    pdl_enter();
    const int cpr = C >> 3;
    const size_t total = static_cast<size_t>(N) * Ho * Wo * cpr;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int cv = static_cast<int>(i % cpr);
        size_t r = i / cpr;
        const int ow = static_cast<int>(r % Wo);
        r /= Wo;
        const int oh = static_cast<int>(r % Ho);
        const int n = static_cast<int>(r / Ho);
        float best[8];
        unsigned char who[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            best[j] = -INFINITY;
            who[j] = 0;
        }
        for (int kh = 0; kh < k; ++kh) {
            const int ih = oh * s - p + kh;
            if (ih < 0 || ih >= H) continue;
            for (int kw = 0; kw < k; ++kw) {
                const int iw = ow * s - p + kw;
                if (iw < 0 || iw >= W) continue;
                float f[8];
                unpack8(load_global(x + ((static_cast<size_t>(n) * H + ih) * W + iw) * cpr + cv), f);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (f[j] > best[j]) {
                        best[j] = f[j];
                        who[j] = static_cast<unsigned char>(kh * k + kw);
                    }
            }
        }
        y[i] = pack8(best);
        uint2 w2;
        w2.x = who[0] | (who[1] << 8) | (who[2] << 16) | (who[3] << 24);
        w2.y = who[4] | (who[5] << 8) | (who[6] << 16) | (who[7] << 24);
        idx[i] = w2;
    }
}

__global__ void __launch_bounds__(256) maxpool_bwd_kernel(const uint4* dy, const uint2* idx, uint4* __restrict__ dx,
                                                          int N, int H, int W, int C, int k, int s, int p, int Ho, int Wo) {
    pdl_enter();
    const int cpr = C >> 3;
    const size_t total = static_cast<size_t>(N) * H * W * cpr;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int cv = static_cast<int>(i % cpr);
        size_t r = i / cpr;
        const int iw = static_cast<int>(r % W);
        r /= W;
        const int ih = static_cast<int>(r % H);
        const int n = static_cast<int>(r / H);
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        // windows (oh, ow) with 0 <= ih + p - oh * s < k
        const int oh_hi = min((ih + p) / s, Ho - 1), ow_hi = min((iw + p) / s, Wo - 1);
        for (int oh = oh_hi; oh >= 0 && ih + p - oh * s < k; --oh) {
            const int kh = ih + p - oh * s;
            for (int ow = ow_hi; ow >= 0 && iw + p - ow * s < k; --ow) {
                const int me = kh * k + (iw + p - ow * s);
                const size_t o = ((static_cast<size_t>(n) * Ho + oh) * Wo + ow) * cpr + cv;
                const uint2 w2 = load_global(idx + o);
                float g[8];
                unpack8(load_global(dy + o), g);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned who = ((j < 4 ? w2.x : w2.y) >> (8 * (j & 3))) & 0xffu;
                    if (who == static_cast<unsigned>(me)) acc[j] += g[j];
                }
            }
        }
        dx[i] = pack8(acc);
    }
}

// Blocks of the reductions: four rows a thread (the loads it has in flight), else the second stage reads nearly as much as
// the first; fewer rows where that leaves SMs without a block, and at most four blocks per SM.
static int bn_grid(long long M, int C, int* threads) {
    const int cpr = C / 8;
    *threads = (256 / cpr) * cpr;
    const int rpb = *threads / cpr;
    const long long rows = (M + rpb - 1) / rpb;  // blocks at one row a thread
    const long long want = rows < 4 * 148 ? (rows < 148 ? rows : 148) : (rows + 3) / 4;
    return static_cast<int>(want < 4 * 148 ? want : 4 * 148);
}
// Blocks of the elementwise passes: one wave of as many as fit an SM, so that each pays for its per-channel constants once.
// With sixteen per SM they were a third of the time of tensors of a few MB: 16384 x 256 forward 27.1 -> 14.3 us, backward
// 42.9 -> 17.4; 4096 x 512 20.2 -> 12.7, 28.6 -> 15.8; at 802816 x 256 (411 MB) 245 -> 239, 354 -> 329.
constexpr int kApplyBlocks = 4, kDxBlocks = 3;  // per SM, as the kernels' launch bounds allow
static int bn_grid_elementwise(long long M, int C, int per_sm) {
    const int cpr = C / 8;
    const int rpb = 256 / cpr;
    const long long want = (M + rpb - 1) / rpb;
    return static_cast<int>(want < 148 * per_sm ? want : 148 * per_sm);
}
static bool bn_shape_ok(long long M, int C) { return M > 0 && C > 0 && C % 8 == 0 && C <= 2048; }
// Whether a pass that keeps `tensors` tensors goes through the cluster kernels: gv > 0, and the shared memory of a block.
// gv: so many vectors of a row per cluster that there are about 16 clusters (128 blocks), a power of two.  Above
// kClusterShare a block the three kernels are as fast: their reads run on four blocks per SM.  (Forward / backward, three
// kernels -> one: 64 x 512 7.9 / 9.7 -> 4.2 / 4.3 us, 1024 x 512 11.1 / 14.4 -> 5.8 / 5.9, 4096 x 512, the limit, 11.5 / 14.8 ->
// 9.8 / 9.7, 16384 x 256, twice that, 15.1 / 18.3 -> 15.4 / 21.7; 5000 x 64 9.5 / 12.0 -> 5.1 / 6.2, 32768 x 64 12.3 -> 17.7.)
struct ClusterPlan {
    int gv = 0, grid = 0;
    size_t smem = 0;
};
static ClusterPlan cluster_plan(long long M, int C, int tensors) {
    const int cpr = C / 8;
    int gv = 1;
    while (gv < kMaxGv && cpr / gv > 16 && cpr % (2 * gv) == 0) gv *= 2;
    const long long share = (M + kClusterBlocks - 1) / kClusterBlocks, lanes = kClusterThreads / gv;
    const unsigned long long bytes = 16ull * kClusterThreads * ((share + lanes - 1) / lanes);
    ClusterPlan p;
    if (bytes > kClusterShare) return p;
    p.gv = gv;
    p.grid = cpr / gv * kClusterBlocks;
    p.smem = bytes * tensors;
    return p;
}
// Raises a cluster kernel's shared-memory limit on the current device, once.
static int cluster_ready(const void* kernel, std::atomic<unsigned long long>& devices) {
    int dev = 0;
    NMLL_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (devices.load(std::memory_order_acquire) & bit) return NML_OK;
    NMLL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(3 * kClusterShare)));
    devices.fetch_or(bit, std::memory_order_release);
    return NML_OK;
}

// A row pitch of a tensor of `channels` channels, in elements: 0 for a tensor of its own.
static bool row_ok(int pitch, int channels) { return pitch == 0 || (pitch >= channels && pitch % 8 == 0); }
static int row_vectors(int pitch, int channels) { return (pitch ? pitch : channels) / 8; }
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace nml_layers

using namespace nml_layers;

extern "C" {

int nml_bn_workspace_size(long long rows, int channels, size_t* bytes) {
    if (!bytes || !bn_shape_ok(rows, channels)) return NML_ERR_INVALID;
    int threads;
    const int P = bn_grid(rows, channels, &threads);
    *bytes = round_up(static_cast<size_t>(P) * 2 * channels * sizeof(float), 256);
    return NML_OK;
}

int nml_bn_forward(const void* x, long long rows, int channels, const float* gamma, const float* beta, const void* residual,
                   int act, float slope, float eps, void* y, float* mean, float* rstd, void* workspace,
                   size_t workspace_bytes, void* stream) {
    return nml_bn_forward_masked(x, rows, channels, gamma, beta, residual, act, slope, eps, y, 0, nullptr, 0, nullptr, mean, rstd,
                                 workspace, workspace_bytes, stream);
}

int nml_bn_forward_masked(const void* x, long long rows, int channels, const float* gamma, const float* beta, const void* residual,
                          int act, float slope, float eps, void* y, int y_pitch, void* y2, int y2_pitch, void* mask, float* mean,
                          float* rstd, void* workspace, size_t workspace_bytes, void* stream) {
    if (!x || !y || !mean || !rstd || act < 0 || act > 2) return NML_ERR_INVALID;
    if (!bn_shape_ok(rows, channels)) return NML_ERR_UNSUPPORTED;
    if (!aligned16(x) || !aligned16(y) || (residual && !aligned16(residual)) || (y2 && !aligned16(y2))) return NML_ERR_INVALID;
    if (!row_ok(y_pitch, channels) || !row_ok(y2_pitch, channels)) return NML_ERR_INVALID;
    size_t need = 0;
    nml_bn_workspace_size(rows, channels, &need);
    if (!workspace || workspace_bytes < need) return NML_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t M = static_cast<size_t>(rows);
    const uint4* xv = static_cast<const uint4*>(x);
    const ClusterPlan cp = cluster_plan(rows, channels, 1);
    if (cp.gv) {
        static std::atomic<unsigned long long> ready{0};
        const int rc = cluster_ready(reinterpret_cast<const void*>(bn_cluster_forward_kernel), ready);
        if (rc) return rc;
        launch_with(true, kClusterBlocks, bn_cluster_forward_kernel, cp.grid, kClusterThreads, cp.smem, st, xv,
                    static_cast<const uint4*>(residual), static_cast<uint4*>(y), row_vectors(y_pitch, channels), static_cast<uint4*>(y2),
                    row_vectors(y2_pitch, channels), static_cast<uint8_t*>(mask), gamma, beta, mean, rstd, act, slope, eps,
                    1.0 / static_cast<double>(rows), M, channels, cp.gv);
        NMLL_CUDA(cudaGetLastError());
        ++g_layer_launches;
        return NML_OK;
    }
    int threads;
    const int P = bn_grid(rows, channels, &threads);
    float* partial = static_cast<float*>(workspace);
    launch(bn_stats_kernel, P, threads, 0, st, xv, partial, M, channels);
    launch(bn_finish_kernel, channels / 8, dim3(8, 128), 0, st, partial, P, channels, 0, 1.0 / static_cast<double>(rows), eps,
           nullptr, nullptr, mean, rstd);
    // (overlapping, whatever its grid: the second stage in front of it leaves every SM room for four of its blocks)
    launch_with(true, 1, bn_apply_kernel, bn_grid_elementwise(rows, channels, kApplyBlocks), threads, 0, st, xv, static_cast<const uint4*>(residual),
           static_cast<uint4*>(y), row_vectors(y_pitch, channels), static_cast<uint4*>(y2), row_vectors(y2_pitch, channels),
           static_cast<uint8_t*>(mask), gamma, beta, mean, rstd, act, slope, M, channels);
    NMLL_CUDA(cudaGetLastError());
    g_layer_launches += 3;
    return NML_OK;
}

}  // extern "C"

template <int kDeriv, bool kTwo>
static int bn_backward_launch(const uint4* x, long long rows, int channels, const OutGrad& dy, const BnForward& f, uint4* dx, uint4* dres,
                              float* dgamma, float* dbeta, float* partial, cudaStream_t st) {
    const size_t M = static_cast<size_t>(rows);
    const double inv_M = 1.0 / static_cast<double>(rows);
    const ClusterPlan cp = cluster_plan(rows, channels, kTwo ? 3 : 2);
    if (cp.gv) {
        auto kernel = bn_cluster_backward_kernel<kDeriv, kTwo>;
        static std::atomic<unsigned long long> ready{0};
        const int rc = cluster_ready(reinterpret_cast<const void*>(kernel), ready);
        if (rc) return rc;
        launch_with(true, kClusterBlocks, kernel, cp.grid, kClusterThreads, cp.smem, st, x, dy, f, dx, dres, dbeta, dgamma, inv_M, M,
                    channels, cp.gv);
        ++g_layer_launches;
    } else {
        int threads;
        const int P = bn_grid(rows, channels, &threads);
        launch(bn_grad_sums_kernel<kDeriv, kTwo>, P, threads, 0, st, x, dy, f, partial, M, channels);
        launch(bn_finish_kernel, channels / 8, dim3(8, 128), 0, st, partial, P, channels, 1, 0.0, 0.f, f.mean, f.rstd, dbeta, dgamma);
        launch_with(true, 1, bn_dx_kernel<kDeriv, kTwo>, bn_grid_elementwise(rows, channels, kDxBlocks), threads, 0, st, x, dy, f, dx, dres,
                    dbeta, dgamma, static_cast<float>(inv_M), M, channels);
        g_layer_launches += 3;
    }
    NMLL_CUDA(cudaGetLastError());
    return NML_OK;
}
static int bn_backward(const void* x, long long rows, int channels, int deriv, const OutGrad& dy, const BnForward& f, void* dx, void* dres,
                       float* dgamma, float* dbeta, void* workspace, size_t workspace_bytes, cudaStream_t st) {
    if (!bn_shape_ok(rows, channels)) return NML_ERR_UNSUPPORTED;
    if (!aligned16(dy.a) || (dy.b && !aligned16(dy.b)) || !aligned16(x) || !aligned16(dx) || (f.y && !aligned16(f.y)) ||
        (dres && !aligned16(dres)))
        return NML_ERR_INVALID;
    size_t need = 0;
    nml_bn_workspace_size(rows, channels, &need);
    if (!workspace || workspace_bytes < need) return NML_ERR_WORKSPACE;
    auto run = dy.b ? (deriv == D_NONE ? bn_backward_launch<D_NONE, true> : deriv == D_Y ? bn_backward_launch<D_Y, true>
                       : deriv == D_X ? bn_backward_launch<D_X, true> : bn_backward_launch<D_MASK, true>)
                    : (deriv == D_NONE ? bn_backward_launch<D_NONE, false> : deriv == D_Y ? bn_backward_launch<D_Y, false>
                       : deriv == D_X ? bn_backward_launch<D_X, false> : bn_backward_launch<D_MASK, false>);
    return run(static_cast<const uint4*>(x), rows, channels, dy, f, static_cast<uint4*>(dx), static_cast<uint4*>(dres), dgamma, dbeta,
               static_cast<float*>(workspace), st);
}
static OutGrad out_grad(const void* dy, int pitch, const void* dy2, int pitch2, int channels) {
    return {static_cast<const uint4*>(dy), static_cast<const uint4*>(dy2), row_vectors(pitch, channels), row_vectors(pitch2, channels)};
}

extern "C" {

int nml_bn_backward(const void* dy, const void* y, const void* x, long long rows, int channels, const float* gamma,
                    const float* mean, const float* rstd, int act, float slope, void* dx, void* dres, float* dgamma,
                    float* dbeta, void* workspace, size_t workspace_bytes, void* stream) {
    if (!dy || !x || !mean || !rstd || !dx || !dgamma || !dbeta || act < 0 || act > 2 || (act != 0 && !y)) return NML_ERR_INVALID;
    const BnForward f = {act != 0 ? static_cast<const uint4*>(y) : nullptr, nullptr, gamma, nullptr, mean, rstd, act == 1 ? 0.f : slope};
    return bn_backward(x, rows, channels, act != 0 ? D_Y : D_NONE, out_grad(dy, 0, nullptr, 0, channels), f, dx, dres, dgamma, dbeta,
                       workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

int nml_bn_backward_masked(const void* dy, int dy_pitch, const void* dy2, int dy2_pitch, const void* mask, const void* x, long long rows,
                           int channels, const float* gamma, const float* beta, const float* mean, const float* rstd, int act, float slope,
                           void* dx, void* dres, float* dgamma, float* dbeta, void* workspace, size_t workspace_bytes, void* stream) {
    if (!dy || !x || !mean || !rstd || !dx || !dgamma || !dbeta || act < 0 || act > 2) return NML_ERR_INVALID;
    if (!row_ok(dy_pitch, channels) || !row_ok(dy2_pitch, channels)) return NML_ERR_INVALID;
    const BnForward f = {nullptr, static_cast<const uint8_t*>(mask), gamma, beta, mean, rstd, act == 1 ? 0.f : slope};
    return bn_backward(x, rows, channels, act == 0 ? D_NONE : mask ? D_MASK : D_X, out_grad(dy, dy_pitch, dy2, dy2_pitch, channels), f, dx,
                       dres, dgamma, dbeta, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

int nml_act_forward(const void* x, long long rows, int channels, int act, float slope, void* y, void* y2, int y2_pitch, void* stream) {
    if (!x || !y || act < 1 || act > 2 || !row_ok(y2_pitch, channels)) return NML_ERR_INVALID;
    if (!bn_shape_ok(rows, channels)) return NML_ERR_UNSUPPORTED;
    if (!aligned16(x) || !aligned16(y) || (y2 && !aligned16(y2))) return NML_ERR_INVALID;
    launch(act_kernel, bn_grid_elementwise(rows, channels, kApplyBlocks), 256 / (channels / 8) * (channels / 8), 0,
           static_cast<cudaStream_t>(stream), static_cast<const uint4*>(x), static_cast<uint4*>(y), static_cast<uint4*>(y2),
           row_vectors(y2_pitch, channels), act == 1 ? 0.f : slope, static_cast<size_t>(rows), channels);
    NMLL_CUDA(cudaGetLastError());
    ++g_layer_launches;
    return NML_OK;
}

int nml_act_backward(const void* dy, int dy_pitch, const void* dy2, int dy2_pitch, const void* x, long long rows, int channels, int act,
                     float slope, void* dx, void* stream) {
    if (!dy || !x || !dx || act < 1 || act > 2 || !row_ok(dy_pitch, channels) || !row_ok(dy2_pitch, channels)) return NML_ERR_INVALID;
    if (!bn_shape_ok(rows, channels)) return NML_ERR_UNSUPPORTED;
    if (!aligned16(dy) || (dy2 && !aligned16(dy2)) || !aligned16(x) || !aligned16(dx)) return NML_ERR_INVALID;
    launch(dy2 ? act_backward_kernel<true> : act_backward_kernel<false>, bn_grid_elementwise(rows, channels, kApplyBlocks),
           256 / (channels / 8) * (channels / 8), 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(x),
           out_grad(dy, dy_pitch, dy2, dy2_pitch, channels), static_cast<uint4*>(dx), act == 1 ? 0.f : slope, static_cast<size_t>(rows),
           channels);
    NMLL_CUDA(cudaGetLastError());
    ++g_layer_launches;
    return NML_OK;
}

constexpr int kL1Blocks = 4 * 148;
int nml_l1_workspace_size(size_t* bytes) {
    if (!bytes) return NML_ERR_INVALID;
    *bytes = round_up(kL1Blocks * sizeof(float), 256);
    return NML_OK;
}
static int l1_grid(size_t n) { return static_cast<int>(n / 512 + 1 < kL1Blocks ? n / 512 + 1 : kL1Blocks); }
int nml_l1_forward(const void* a, const void* b, size_t n, float denom, float* loss, void* workspace, size_t workspace_bytes, void* stream) {
    if (!a || !b || !loss || n == 0 || (reinterpret_cast<uintptr_t>(a) & 3) || (reinterpret_cast<uintptr_t>(b) & 3)) return NML_ERR_INVALID;
    size_t need = 0;
    nml_l1_workspace_size(&need);
    if (!workspace || workspace_bytes < need) return NML_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* partial = static_cast<float*>(workspace);
    launch(l1_sum_kernel, l1_grid(n), 256, 0, st, static_cast<const __half2*>(a), static_cast<const __half2*>(b), n, partial);
    launch(l1_finish_kernel, 1, 32, 0, st, partial, l1_grid(n), denom, loss);
    NMLL_CUDA(cudaGetLastError());
    g_layer_launches += 2;
    return NML_OK;
}
int nml_l1_backward(const void* a, const void* b, size_t n, const float* dloss, float denom, void* da, void* stream) {
    if (!a || !b || !dloss || !da || n == 0 || ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(da)) & 3))
        return NML_ERR_INVALID;
    launch(l1_backward_kernel, l1_grid(n), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const __half2*>(a),
           static_cast<const __half2*>(b), n, dloss, denom, static_cast<__half2*>(da));
    NMLL_CUDA(cudaGetLastError());
    ++g_layer_launches;
    return NML_OK;
}

long long nml_layers_launch_count(void) { return g_layer_launches.load(); }

int nml_maxpool_forward(const void* x, int batch, int h, int w, int channels, int k, int stride, int pad, void* y,
                        void* index, void* stream) {
    if (!x || !y || !index || batch <= 0 || h <= 0 || w <= 0 || k <= 0 || k > 15 || stride <= 0 || pad < 0 || pad >= k)
        return NML_ERR_INVALID;
    if (channels <= 0 || channels % 8) return NML_ERR_UNSUPPORTED;
    if (!aligned16(x) || !aligned16(y) || (reinterpret_cast<uintptr_t>(index) & 7)) return NML_ERR_INVALID;
    const int ho = (h + 2 * pad - k) / stride + 1, wo = (w + 2 * pad - k) / stride + 1;
    if (ho <= 0 || wo <= 0) return NML_ERR_INVALID;
    const size_t total = static_cast<size_t>(batch) * ho * wo * (channels / 8);
    const int blocks = static_cast<int>((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    launch(maxpool_fwd_kernel, blocks, 256, 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(x), static_cast<uint4*>(y),
                                                                             static_cast<uint2*>(index), batch, h, w, channels, k,
                                                                             stride, pad, ho, wo);
    NMLL_CUDA(cudaGetLastError());
    ++g_layer_launches;
    return NML_OK;
}

int nml_maxpool_backward(const void* dy, const void* index, int batch, int h, int w, int channels, int k, int stride, int pad,
                         void* dx, void* stream) {
    if (!dy || !dx || !index || batch <= 0 || h <= 0 || w <= 0 || k <= 0 || k > 15 || stride <= 0 || pad < 0 || pad >= k)
        return NML_ERR_INVALID;
    if (channels <= 0 || channels % 8) return NML_ERR_UNSUPPORTED;
    if (!aligned16(dy) || !aligned16(dx) || (reinterpret_cast<uintptr_t>(index) & 7)) return NML_ERR_INVALID;
    const int ho = (h + 2 * pad - k) / stride + 1, wo = (w + 2 * pad - k) / stride + 1;
    if (ho <= 0 || wo <= 0) return NML_ERR_INVALID;
    const size_t total = static_cast<size_t>(batch) * h * w * (channels / 8);
    const int blocks = static_cast<int>((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    launch(maxpool_bwd_kernel, blocks, 256, 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(dy), static_cast<const uint2*>(index),
                                                                             static_cast<uint4*>(dx), batch, h, w, channels, k, stride,
                                                                             pad, ho, wo);
    NMLL_CUDA(cudaGetLastError());
    ++g_layer_launches;
    return NML_OK;
}

int nml_grads_check(const float* grads, size_t n, float inv_scale, int* found_inf, void* stream) {
    if (!grads || !found_inf || n % 4 || !aligned16(grads)) return NML_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    NMLL_CUDA(cudaMemsetAsync(found_inf, 0, sizeof(int), st));
    const size_t n4 = n / 4;
    const int blocks = static_cast<int>(n4 / 256 + 1 < 148 * 8 ? n4 / 256 + 1 : 148 * 8);
    launch(grads_check_kernel, blocks, 256, 0, st, reinterpret_cast<const float4*>(grads), n4, inv_scale, found_inf);
    NMLL_CUDA(cudaGetLastError());
    ++g_layer_launches;
    return NML_OK;
}

int nml_sgd_momentum_step(float* params, const float* grads, float* velocity, void* params_f16, size_t n, float lr,
                          float momentum, float dampening, float weight_decay, float inv_scale, const int* found_inf,
                          void* stream) {
    if (!params || !grads || !velocity || n % 4 || !aligned16(params) || !aligned16(grads) || !aligned16(velocity) ||
        (params_f16 && (reinterpret_cast<uintptr_t>(params_f16) & 7)))
        return NML_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t n4 = n / 4;
    const int blocks = static_cast<int>(n4 / 256 + 1 < 148 * 8 ? n4 / 256 + 1 : 148 * 8);
    launch(sgd_momentum_kernel, blocks, 256, 0, st, reinterpret_cast<float4*>(params), reinterpret_cast<const float4*>(grads),
                                                reinterpret_cast<float4*>(velocity), static_cast<uint2*>(params_f16), n4, lr,
                                                momentum, dampening, weight_decay, inv_scale, found_inf);
    NMLL_CUDA(cudaGetLastError());
    ++g_layer_launches;
    return NML_OK;
}

}  // extern "C"
