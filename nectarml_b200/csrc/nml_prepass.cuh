// Memory-bound helper kernels around the contraction kernel: layout / precision
// conversion of activations (NCHW -> NHWC, fp32 -> fp16 or the tf32 hi/lo pair of the
// 3xTF32 split, with the bias-gradient column sum folded into the same pass over dY),
// weight repacking into the K-major [n][tap][k] operand, and small utilities.
#pragma once
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "nml_launch.cuh"

namespace nml {

__device__ __forceinline__ float to_tf32_rna(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

__device__ __forceinline__ float load_as_float(const float* p, size_t i) { return load_global(p + i); }
__device__ __forceinline__ float load_as_float(const __half* p, size_t i) { return __half2float(load_global(p + i)); }

// Output encodings of the conversion kernels.
enum { ENC_F16 = 0, ENC_TF32_PAIR = 1, ENC_TF32_HI = 2 };

__device__ __forceinline__ void store_enc(int enc, void* out0, void* out1, size_t i, float v) {
    if (enc == ENC_F16) {
        reinterpret_cast<__half*>(out0)[i] = __float2half_rn(v);
    } else {
        float hi = to_tf32_rna(v);
        reinterpret_cast<float*>(out0)[i] = hi;
        if (enc == ENC_TF32_PAIR) reinterpret_cast<float*>(out1)[i] = to_tf32_rna(v - hi);
    }
}

__device__ __forceinline__ float4 load4(const float* p) { return load_global(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load4(const __half* p) {
    const uint2 v = load_global(reinterpret_cast<const uint2*>(p));
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// in  [N][C][HW] (NCHW)  ->  out [N][HW][Cp] (NHWC, channels zero-padded to Cp, whole 16-byte vectors).
// Tiles of 64 channels x 64 pixels through shared memory, several per block: the loads of the next tile are in flight while
// this one is stored.  With one tile per block the last wave was half empty, and eight small blocks fitted an SM, so a grid
// launched beside its predecessor's tail piled up on the SMs that were free first; these registers leave room for four.
// fp32 3x3 64 -> 64 at 56 x 56, batch 8, three passes with four conversions 114.8 -> 108.4 us; 128 channels at 28 x 28, batch
// 64, with three 136.0 -> 131.7.
// Loads run along pixels (four per thread where the rows allow it), stores along channels: 8 threads write the 64 channels
// of one pixel as 16-byte (fp16) or 2 x 16-byte (tf32 planes) pieces, so a warp store covers four whole pixels.  When
// `colsum` is given, the per-channel sums over the tile's pixels (a share of the bias gradient) go to row
// (n * pixel tiles + pixel tile) of that [tiles][C]
// matrix of partial sums; colsum_finish_kernel adds the rows in a fixed order (no atomics, so the
// bias gradient is bitwise repeatable).
template <typename TIn>
__global__ void __launch_bounds__(256) nchw_to_nhwc_kernel(const TIn* in, void* out0,
                                                           void* out1, int enc, int C, int Cp, int HW, int tiles_p, int tiles_c,
                                                           int tiles, float* colsum, int role) {
    pdl_enter(role);
    __shared__ float tile[64][65];
    const bool vec_ok = (HW % 4 == 0) && ((reinterpret_cast<uintptr_t>(in) & (4 * sizeof(TIn) - 1)) == 0);
    const int tx = vec_ok ? (threadIdx.x & 15) * 4 : threadIdx.x & 63;      // 16 x 16 threads: four pixels each; or 64 x 4
    const int ty = vec_ok ? threadIdx.x >> 4 : threadIdx.x >> 6;
    int n, c0, p0;
    auto decode = [&](int t) {
        const int q = t / tiles_p;
        n = q / tiles_c;
        c0 = (q - n * tiles_c) * 64;
        p0 = (t - q * tiles_p) * 64;
    };
    float4 next[4];
    auto load = [&](int t) {
        decode(t);
        const int p = p0 + tx;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int c = c0 + ty + 16 * k;
            next[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c < C && p < HW) next[k] = load4(in + (static_cast<size_t>(n) * C + c) * HW + p);  // HW % 4 == 0: a started quad is complete
        }
    };
    int t = blockIdx.x;
    if (vec_ok && t < tiles) load(t);
    for (; t < tiles; t += gridDim.x) {
        decode(t);
        if (vec_ok) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float* o = &tile[ty + 16 * k][tx];
                o[0] = next[k].x, o[1] = next[k].y, o[2] = next[k].z, o[3] = next[k].w;
            }
        } else {
            const TIn* src = in + static_cast<size_t>(n) * C * HW;
#pragma unroll 8
            for (int c = ty; c < 64; c += 4) {
                float v = 0.f;
                if (c0 + c < C && p0 + tx < HW) v = load_as_float(src, static_cast<size_t>(c0 + c) * HW + p0 + tx);
                tile[c][tx] = v;
            }
        }
        __syncthreads();
        if (vec_ok && t + static_cast<int>(gridDim.x) < tiles) {
            load(t + gridDim.x);
            decode(t);
        }
        if (colsum != nullptr) {  // four threads per channel, 16 pixels each (all lanes of a warp on different banks)
            const int c = threadIdx.x >> 2, q = threadIdx.x & 3;
            float s = 0.f;
#pragma unroll
            for (int p = 0; p < 16; ++p) s += tile[c][4 * p + q];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (q == 0 && c0 + c < C) colsum[(static_cast<size_t>(n) * tiles_p + p0 / 64) * C + c0 + c] = s;
        }
        // store: 8 threads per pixel, 8 channels each
        const int j = threadIdx.x & 7, pp = threadIdx.x >> 3;  // 8 x 32
        const int cb = c0 + 8 * j;
        const bool full8 = (cb + 8 <= Cp) && (Cp % 8 == 0);
        for (int p = pp; p < 64; p += 32) {
            if (p0 + p >= HW || cb >= Cp) continue;
            const size_t o = (static_cast<size_t>(n) * HW + p0 + p) * Cp + cb;
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = tile[8 * j + i][p];
            if (full8 && enc == ENC_F16) {
                uint4 pk;
                __half2 h;
                h = __floats2half2_rn(v[0], v[1]); pk.x = *reinterpret_cast<uint32_t*>(&h);
                h = __floats2half2_rn(v[2], v[3]); pk.y = *reinterpret_cast<uint32_t*>(&h);
                h = __floats2half2_rn(v[4], v[5]); pk.z = *reinterpret_cast<uint32_t*>(&h);
                h = __floats2half2_rn(v[6], v[7]); pk.w = *reinterpret_cast<uint32_t*>(&h);
                *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(out0) + o) = pk;
            } else if (full8) {
                float hi[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) hi[i] = to_tf32_rna(v[i]);
                float4* d0 = reinterpret_cast<float4*>(reinterpret_cast<float*>(out0) + o);
                d0[0] = make_float4(hi[0], hi[1], hi[2], hi[3]);
                d0[1] = make_float4(hi[4], hi[5], hi[6], hi[7]);
                if (enc == ENC_TF32_PAIR) {
                    float4* d1 = reinterpret_cast<float4*>(reinterpret_cast<float*>(out1) + o);
                    d1[0] = make_float4(to_tf32_rna(v[0] - hi[0]), to_tf32_rna(v[1] - hi[1]), to_tf32_rna(v[2] - hi[2]),
                                        to_tf32_rna(v[3] - hi[3]));
                    d1[1] = make_float4(to_tf32_rna(v[4] - hi[4]), to_tf32_rna(v[5] - hi[5]), to_tf32_rna(v[6] - hi[6]),
                                        to_tf32_rna(v[7] - hi[7]));
                }
            } else {
                // fp32 planes of an odd number of four-channel groups (stored value by value: 3x3 67 -> 70 at 36 x 36, batch 8, 40.9 us instead
                // of 28.4; 4x4 s2 input gradient of 64 -> 67 at 168 x 168, batch 65, 2362 instead of 1404)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (cb + 4 * q >= Cp) break;
                    float hi[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) hi[i] = to_tf32_rna(v[4 * q + i]);
                    *reinterpret_cast<float4*>(reinterpret_cast<float*>(out0) + o + 4 * q) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                    if (enc == ENC_TF32_PAIR)
                        *reinterpret_cast<float4*>(reinterpret_cast<float*>(out1) + o + 4 * q) =
                            make_float4(to_tf32_rna(v[4 * q] - hi[0]), to_tf32_rna(v[4 * q + 1] - hi[1]), to_tf32_rna(v[4 * q + 2] - hi[2]),
                                        to_tf32_rna(v[4 * q + 3] - hi[3]));
                }
            }
        }
        __syncthreads();
    }
    pdl_leave(role);
}

// in [N][HW][C] (NHWC, C a multiple of 4) -> out [N][C][HW], no change of values: the way back, in the same manner.
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(__half* p, const float (&v)[4]) {
    uint2 h;
    *reinterpret_cast<__half2*>(&h.x) = __floats2half2_rn(v[0], v[1]);
    *reinterpret_cast<__half2*>(&h.y) = __floats2half2_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = h;
}
template <typename T>
__global__ void __launch_bounds__(256) nhwc_to_nchw_kernel(const T* in, T* __restrict__ out, int C, int HW, int tiles_p,
                                                           int tiles_c, int tiles, int role) {
    pdl_enter(role);
    __shared__ float tile[64][65];  // [pixel][channel]
    const bool vec_ok = (HW % 4 == 0) && ((reinterpret_cast<uintptr_t>(out) & (4 * sizeof(T) - 1)) == 0);
    const int x4 = (threadIdx.x & 15) * 4, y16 = threadIdx.x >> 4;
    int n, c0, p0;
    auto decode = [&](int t) {
        const int q = t / tiles_p;
        n = q / tiles_c;
        c0 = (q - n * tiles_c) * 64;
        p0 = (t - q * tiles_p) * 64;
    };
    float4 next[4];
    auto load = [&](int t) {
        decode(t);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int p = p0 + y16 + 16 * k;
            next[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p < HW && c0 + x4 < C) next[k] = load4(in + (static_cast<size_t>(n) * HW + p) * C + c0 + x4);
        }
    };
    int t = blockIdx.x;
    if (t < tiles) load(t);
    for (; t < tiles; t += gridDim.x) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float* o = &tile[y16 + 16 * k][x4];
            o[0] = next[k].x, o[1] = next[k].y, o[2] = next[k].z, o[3] = next[k].w;
        }
        __syncthreads();
        if (t + static_cast<int>(gridDim.x) < tiles) load(t + gridDim.x);
        decode(t);
        if (vec_ok) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = y16 + 16 * k;
                if (c0 + c < C && p0 + x4 < HW) {  // HW % 4 == 0: a started quad is complete
                    const float v[4] = {tile[x4][c], tile[x4 + 1][c], tile[x4 + 2][c], tile[x4 + 3][c]};
                    store4(out + (static_cast<size_t>(n) * C + c0 + c) * HW + p0 + x4, v);
                }
            }
        } else {
            const int px = threadIdx.x & 63;
            for (int c = threadIdx.x >> 6; c < 64; c += 4)
                if (c0 + c < C && p0 + px < HW) out[(static_cast<size_t>(n) * C + c0 + c) * HW + p0 + px] = static_cast<T>(tile[px][c]);
        }
        __syncthreads();
    }
    pdl_leave(role);
}

// Row-major [R][C] -> [R][Cp] with encoding change (fp32/fp16 -> fp16 / tf32 pair), zero pad; Cp is a multiple of 4.
// Four outputs per thread: a 16-byte load where the rows allow it, one 8-byte (fp16) or one or two 16-byte stores.
// An element per thread with a 64-bit division each ran at 1.8 TB/s on 2 MB; this is bound by the launch there.
template <typename TIn>
__global__ void __launch_bounds__(256) convert_rows_kernel(const TIn* in, void* out0,
                                                           void* out1, int enc, size_t R, int C, int Cp, int role) {
    pdl_enter(role);
    const size_t per_row = Cp / 4, total = R * per_row;
    const bool dense = C == Cp;  // rows follow one another on both sides
    const bool vec = (dense || C % 4 == 0) && (reinterpret_cast<uintptr_t>(in) & (4 * sizeof(TIn) - 1)) == 0;
    const bool small = total < 0xffffffffull;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        size_t src = 4 * i;
        int left = 4;  // source elements under this thread's four outputs
        if (!dense) {
            const size_t r = small ? static_cast<uint32_t>(i) / static_cast<uint32_t>(per_row) : i / per_row;
            const int c = static_cast<int>(i - r * per_row) * 4;
            src = r * C + c;
            left = C - c;
        }
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vec && left >= 4) {
            v = load4(in + src);
        } else {
            if (left > 0) v.x = load_as_float(in, src);
            if (left > 1) v.y = load_as_float(in, src + 1);
            if (left > 2) v.z = load_as_float(in, src + 2);
            if (left > 3) v.w = load_as_float(in, src + 3);
        }
        if (enc == ENC_F16) {
            uint2 h;
            *reinterpret_cast<__half2*>(&h.x) = __floats2half2_rn(v.x, v.y);
            *reinterpret_cast<__half2*>(&h.y) = __floats2half2_rn(v.z, v.w);
            reinterpret_cast<uint2*>(out0)[i] = h;
        } else {
            const float4 hi = make_float4(to_tf32_rna(v.x), to_tf32_rna(v.y), to_tf32_rna(v.z), to_tf32_rna(v.w));
            reinterpret_cast<float4*>(out0)[i] = hi;
            if (enc == ENC_TF32_PAIR)
                reinterpret_cast<float4*>(out1)[i] = make_float4(to_tf32_rna(v.x - hi.x), to_tf32_rna(v.y - hi.y),
                                                                 to_tf32_rna(v.z - hi.z), to_tf32_rna(v.w - hi.w));
        }
    }
    pdl_leave(role);
}

// Column sums of a row-major [R][C] matrix (bias gradient of Linear, or of an NHWC dY), first stage:
// row block blockIdx.y writes its sums to row blockIdx.y of the [row blocks][C] partial-sum matrix.
template <typename TIn>
__global__ void __launch_bounds__(256) colsum_rows_kernel(const TIn* in, float* colsum,
                                                          size_t R, int C, int rows_per_block, int role) {
    pdl_enter(role);
    size_t r0 = static_cast<size_t>(blockIdx.y) * rows_per_block;
    size_t r1 = r0 + rows_per_block < R ? r0 + rows_per_block : R;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        float s = 0.f;
        size_t r = r0;
        for (; r + 8 <= r1; r += 8) {  // (eight loads in flight, added in the rows' order; linear 5000 x 301 -> 333 weight gradient 27.8 -> 26.8 us)
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = load_as_float(in, (r + i) * C + c);
#pragma unroll
            for (int i = 0; i < 8; ++i) s += v[i];
        }
        for (; r < r1; ++r) s += load_as_float(in, r * C + c);
        colsum[static_cast<size_t>(blockIdx.y) * C + c] = s;
    }
    pdl_leave(role);
}

// Vectorised column sums for rows that are whole 16-byte vectors (8 fp16 or 4 fp32 columns each): every thread owns one
// vector column, a warp covers 32 of them, the block's 8 warps take interleaved rows, eight loads in flight each (the pass
// is HBM-bound; four left 16384 x 8192 at 4.9 TB/s), and each block writes its partial sums to its row of the
// partial-sum matrix.
__device__ __forceinline__ void add_vector(float (&acc)[8], const uint4& v, const __half*) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h[j]);
        acc[2 * j] += f.x;
        acc[2 * j + 1] += f.y;
    }
}
__device__ __forceinline__ void add_vector(float (&acc)[4], const uint4& v, const float*) {
    acc[0] += __uint_as_float(v.x); acc[1] += __uint_as_float(v.y); acc[2] += __uint_as_float(v.z); acc[3] += __uint_as_float(v.w);
}
template <typename TIn>
__global__ void __launch_bounds__(256) colsum_vectors_kernel(const TIn* in, float* colsum,
                                                             size_t R, int C, int rows_per_block, int role) {
    pdl_enter(role);
    constexpr int V = 16 / sizeof(TIn);
    __shared__ float part[8][32 * V];
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int c0 = (blockIdx.x * 32 + lane) * V;
    size_t r0 = static_cast<size_t>(blockIdx.y) * rows_per_block;
    size_t r1 = r0 + rows_per_block < R ? r0 + rows_per_block : R;
    float acc[V];
#pragma unroll
    for (int j = 0; j < V; ++j) acc[j] = 0.f;
    if (c0 < C) {
        const TIn* p = in + c0;
        size_t r = r0 + wy;
        for (; r + 56 < r1; r += 64) {
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = load_global(reinterpret_cast<const uint4*>(p + (r + 8 * i) * C));
#pragma unroll
            for (int i = 0; i < 8; ++i) add_vector(acc, v[i], p);
        }
        for (; r < r1; r += 8) add_vector(acc, load_global(reinterpret_cast<const uint4*>(p + r * C)), p);
    }
#pragma unroll
    for (int j = 0; j < V; ++j) part[wy][lane * V + j] = acc[j];
    __syncthreads();
    const int c = blockIdx.x * 32 * V + threadIdx.x;
    if (threadIdx.x < 32 * V && c < C) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += part[w][threadIdx.x];
        colsum[static_cast<size_t>(blockIdx.y) * C + c] = sum;
    }
    pdl_leave(role);
}

// The same in one launch, for matrices of few enough rows: the row blocks of a column block form a cluster, which adds their
// sums through distributed shared memory, in order.  Eight rows are added up by themselves before they join a thread's sum,
// so no chain of additions is longer than in the two stages.
constexpr int kColsumCluster = 8;
template <typename TIn>
__global__ void __launch_bounds__(256) colsum_cluster_kernel(const TIn* in, float* __restrict__ out, int R, int C, int rows_per_block, int role) {
    pdl_enter(role);
    constexpr int V = 16 / sizeof(TIn), kCols = 32 * V, kShare = kCols / kColsumCluster;
    __shared__ float part[8][kCols];
    __shared__ float sum[kCols];
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int rank = blockIdx.x % kColsumCluster, col0 = blockIdx.x / kColsumCluster * kCols, c0 = col0 + lane * V;
    const int r0 = rank * rows_per_block, r1 = min(R, r0 + rows_per_block);
    float acc[V];
#pragma unroll
    for (int j = 0; j < V; ++j) acc[j] = 0.f;
    if (c0 < C) {
        const TIn* p = in + c0;
        for (int r = r0 + wy; r < r1; r += 64) {
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = r + 8 * i < r1 ? load_global(reinterpret_cast<const uint4*>(p + static_cast<size_t>(r + 8 * i) * C)) : make_uint4(0u, 0u, 0u, 0u);
            float eight[V];
#pragma unroll
            for (int j = 0; j < V; ++j) eight[j] = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) add_vector(eight, v[i], p);
#pragma unroll
            for (int j = 0; j < V; ++j) acc[j] += eight[j];
        }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) part[wy][lane * V + j] = acc[j];
    __syncthreads();
    if (threadIdx.x < kCols) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += part[w][threadIdx.x];
        sum[threadIdx.x] = s;
    }
    cooperative_groups::this_cluster().sync();
    const int c = rank * kShare + threadIdx.x;
    if (threadIdx.x < kShare && col0 + c < C) {
        float s = 0.f;
#pragma unroll
        for (int r = 0; r < kColsumCluster; ++r) s += cooperative_groups::this_cluster().map_shared_rank(sum, r)[c];
        out[col0 + c] = s;
    }
    cooperative_groups::this_cluster().sync();  // no block leaves while another reads its sums
    pdl_leave(role);
}

// Weights [D0][D1][T] -> K-major operand dst[n][t][kp]:
//   k_is_dim0 == 0 : n = D0 index, k = D1 index   (Conv2d forward, ConvTranspose2d dgrad)
//   k_is_dim0 == 1 : n = D1 index, k = D0 index   (Conv2d dgrad, ConvTranspose2d forward)
// k is zero-padded to kp per tap so that no K block straddles two taps.  Both cases swap the two inner
// dimensions of a [B][R][Cc] array: out[b][c][r] = in[b][r][c], rows padded to Rp --
//   k_is_dim0 == 0 : B = D0, R = D1 (k), Cc = T          k_is_dim0 == 1 : B = 1, R = D0 (k), Cc = D1 * T
// -- so a tiled transpose through shared memory serves them, with coalesced reads AND writes (a gather
// with one side strided moved a 32-byte sector per 2-byte element).  Two kernels by the width of the
// source rows:
//   repack_weight_tile_kernel  Cc > 64: 64 x 64 tiles, two elements per thread on both sides.
//                              grid (ceil(Cc/64), ceil(Rp/64), B), 256 threads.
//   repack_weight_rows_kernel  Cc <= 64 (the taps of one kernel): 64 source rows are one contiguous run of
//                              64 * Cc elements, read linearly.  grid (ceil(Rp/64), B), 256 threads.
__device__ __forceinline__ void store_enc2(int enc, void* out0, void* out1, size_t i, float a, float b) {
    if (enc == ENC_F16) {
        *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(out0) + i) = __floats2half2_rn(a, b);  // i is even
    } else {
        store_enc(enc, out0, out1, i, a);
        store_enc(enc, out0, out1, i + 1, b);
    }
}

template <typename TIn>
__global__ void __launch_bounds__(256) repack_weight_tile_kernel(const TIn* w, void* out0, void* out1, int enc,
                                                                 int R, int Cc, int Rp, int role) {
    pdl_enter(role);
    __shared__ float tile[64][65];  // [r][c]
    const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
    const size_t b = blockIdx.z;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    float v[8][2];  // (all of a thread's loads in flight: fp32 3x3 s2 128 -> 128 at 28 x 28, batch 64, input gradient 42.1 -> 40.3 us)
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int r = r0 + ty + 8 * k, c = c0 + 2 * tx;
        const size_t src = (b * R + r) * Cc + c;
        v[k][0] = (r < R && c < Cc) ? load_as_float(w, src) : 0.f;
        v[k][1] = (r < R && c + 1 < Cc) ? load_as_float(w, src + 1) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        tile[ty + 8 * k][2 * tx] = v[k][0];
        tile[ty + 8 * k][2 * tx + 1] = v[k][1];
    }
    __syncthreads();
    for (int j = ty; j < 64; j += 8) {
        const int c = c0 + j, r = r0 + 2 * tx;  // Rp is a multiple of the K block, so r + 1 < Rp whenever r < Rp
        if (c < Cc && r < Rp) store_enc2(enc, out0, out1, (b * Cc + c) * Rp + r, tile[2 * tx][j], tile[2 * tx + 1][j]);
    }
    pdl_leave(role);
}

template <typename TIn>
__global__ void __launch_bounds__(256) repack_weight_rows_kernel(const TIn* w, void* out0, void* out1, int enc,
                                                                 int R, int Cc, int Rp, int role) {
    pdl_enter(role);
    __shared__ float tile[64][65];  // [c][r]
    const int r0 = blockIdx.x * 64;
    const size_t b = blockIdx.y;
    const int rows = min(64, R - r0);  // may be <= 0: a block of pure padding
    const int n_valid = rows > 0 ? rows * Cc : 0;
    const size_t base = (b * R + r0) * Cc;
    for (int i = threadIdx.x; i < 64 * Cc; i += 256) {
        const int r = i / Cc, c = i - r * Cc;
        tile[c][r] = (i < n_valid) ? load_as_float(w, base + i) : 0.f;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < Cc * 32; idx += 256) {
        const int c = idx >> 5, r = (idx & 31) * 2;
        if (r0 + r < Rp) store_enc2(enc, out0, out1, (b * Cc + c) * Rp + r0 + r, tile[c][r], tile[c][r + 1]);
    }
    pdl_leave(role);
}

// The same two for fp16 weights that stay fp16 (a training step repacks every layer's weights twice): 16-byte loads, more
// work per block, and no detour through float.  Both want 16-byte aligned source rows and Rp a multiple of 8.
//   [B][R][Cc] -> [B][Cc][Rp], 64 x 64 tiles; Cc a multiple of 8.  2048 x 8192: 29.6 -> 12 us (bytes: 10 us).
__global__ void __launch_bounds__(256) repack_half_tile_kernel(const __half* w, __half* __restrict__ out, int R, int Cc, int Rp, int role) {
    pdl_enter(role);
    __shared__ __half tile[64][66];  // [r][c]; a pitch of 33 words spreads the column reads below over the banks
    const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
    const size_t b = blockIdx.z;
    const int v = threadIdx.x & 7, q = threadIdx.x >> 3;  // 8 vectors of 8 x 32 rows
    uint4 x[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = r0 + q + 32 * h, c = c0 + 8 * v;
        x[h] = (r < R && c < Cc) ? load_global(reinterpret_cast<const uint4*>(w + (b * R + r) * Cc + c)) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t* row = reinterpret_cast<uint32_t*>(&tile[q + 32 * h][8 * v]);
        row[0] = x[h].x; row[1] = x[h].y; row[2] = x[h].z; row[3] = x[h].w;
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int c = q + 32 * h, r = 8 * v;
        if (c0 + c >= Cc || r0 + r >= Rp) continue;
        uint4 y;
        __half* e = reinterpret_cast<__half*>(&y);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = tile[r + i][c];
        *reinterpret_cast<uint4*>(out + (b * Cc + c0 + c) * Rp + r0 + r) = y;
    }
    pdl_leave(role);
}

// Cc <= 64 (the taps of one kernel), R * Cc a multiple of 8: 256 source rows per block, one contiguous run.  Bound by
// instructions, not bytes, so shared memory is written in words where a vector of eight taps stays within a row, and the output
// in 16-byte vectors of eight rows.  A warp takes 8 taps x 4 row groups (4 x 8 where Cc is no multiple of 8): with a pitch of
// Cc + 2 (odd) halves its reads fall on different banks.  512 x 1024 x 16: 9.9 -> 8.7 us.
__host__ __device__ inline int repack_rows_pitch(int Cc) { return Cc % 8 == 0 ? Cc + 2 : (Cc | 1); }
__global__ void __launch_bounds__(256) repack_half_rows_kernel(const __half* w, __half* __restrict__ out, int R, int Cc, int Rp, int role) {
    pdl_enter(role);
    extern __shared__ __half run[];  // [256][pitch]
    const int pitch = repack_rows_pitch(Cc);
    const bool words = Cc % 8 == 0;
    const int r0 = blockIdx.x * 256;
    const size_t b = blockIdx.y;
    const int n_valid = max(0, min(256, R - r0)) * Cc;
    const __half* src = w + (b * R + r0) * Cc;
    const uint32_t inv = (1u << 20) / Cc + 1;  // i / Cc for i < 2^14, Cc <= 64
    for (int i0 = threadIdx.x * 8; i0 < 256 * Cc; i0 += 2 * 256 * 8) {
        uint4 x[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = i0 + h * 256 * 8;
            x[h] = make_uint4(0u, 0u, 0u, 0u);
            __half* e = reinterpret_cast<__half*>(&x[h]);
            if (i + 8 <= n_valid) x[h] = load_global(reinterpret_cast<const uint4*>(src + i));
            else
                for (int k = 0; k < 8; ++k)
                    if (i + k < n_valid) e[k] = load_global(src + i + k);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = i0 + h * 256 * 8;
            if (i >= 256 * Cc) break;
            int r = static_cast<int>((static_cast<uint64_t>(i) * inv) >> 20), c = i - r * Cc;
            if (words) {
                uint32_t* o = reinterpret_cast<uint32_t*>(run + r * pitch + c);
                o[0] = x[h].x; o[1] = x[h].y; o[2] = x[h].z; o[3] = x[h].w;
            } else {
                const __half* e = reinterpret_cast<const __half*>(&x[h]);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    run[r * pitch + c] = e[k];
                    if (++c == Cc) {
                        c = 0;
                        ++r;
                    }
                }
            }
        }
    }
    __syncthreads();
    const int cw = words ? 8 : 4, rw = 32 / cw;  // taps, row groups of a warp
    const int lane = threadIdx.x & 31, col_sets = (Cc + cw - 1) / cw;
    const int dc = lane / rw, dr = lane % rw;
    for (int k = threadIdx.x >> 5; k < col_sets * (32 / rw); k += 8) {
        const int set = k / col_sets;
        const int c = (k - set * col_sets) * cw + dc, r = (set * rw + dr) * 8;
        if (c >= Cc || r0 + r >= Rp) continue;
        uint4 y;
        __half* e = reinterpret_cast<__half*>(&y);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = run[(r + i) * pitch + c];
        *reinterpret_cast<uint4*>(out + (b * Cc + c) * Rp + r0 + r) = y;
    }
    pdl_leave(role);
}

// Few-channel activations (e.g. RGB stems): copy into a zero-padded NHWC image with exactly kCh (4 or 8) fp16 channels per
// pixel, [N][Hp][Wp][kCh], the original at offset (pad_h, pad_w).  A row of 8 consecutive pixels of this image is one K
// slice (64 or 128 bytes) holding (kw, c) for 8 taps, which is what the small-channel contraction path reads.
// A warp takes a padded row at a time, four pixels per lane in flight; an index decoded with 64-bit divisions per
// pixel ran at 2.1 TB/s.
template <typename TIn, int kCh>
__global__ void __launch_bounds__(256) pad_pack_kernel(const TIn* in, int nchw, __half* __restrict__ out,
                                                       int N, int C, int H, int W, int pad_h, int pad_w, int Hp,
                                                       int Wp, float* colsum, int role) {
    pdl_enter(role);
    struct alignas(2 * kCh) Pixel {
        __half2 v[kCh / 2];
    };
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int rows = N * Hp;
    const size_t px = nchw ? 1 : C, ch = nchw ? static_cast<size_t>(H) * W : 1;  // element strides of the source
    float acc[kCh];  // per-channel sums of the values read (bias gradient)
#pragma unroll
    for (int c = 0; c < kCh; ++c) acc[c] = 0.f;
    for (int r = blockIdx.x * 8 + wy; r < rows; r += gridDim.x * 8) {
        const int n = r / Hp, h = r - n * Hp - pad_h;
        const bool row_in = h >= 0 && h < H;
        const TIn* src = in + (nchw ? (static_cast<size_t>(n) * C * H + h) * W : (static_cast<size_t>(n) * H + h) * W * C);
        Pixel* dst = reinterpret_cast<Pixel*>(out) + static_cast<size_t>(r) * Wp;
        for (int p0 = lane; p0 < Wp; p0 += 128) {
            float v[4][kCh];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int w = p0 + 32 * u - pad_w;
                const bool inside = row_in && w >= 0 && w < W;
#pragma unroll
                for (int c = 0; c < kCh; ++c) v[u][c] = (c < C && inside) ? load_as_float(src, w * px + c * ch) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                Pixel q;
#pragma unroll
                for (int c = 0; c < kCh; ++c) acc[c] += v[u][c];  // (the values as given, like every other column-sum path)
#pragma unroll
                for (int c = 0; c < kCh / 2; ++c) q.v[c] = __floats2half2_rn(v[u][2 * c], v[u][2 * c + 1]);
                if (p0 + 32 * u < Wp) dst[p0 + 32 * u] = q;
            }
        }
    }
    if (colsum != nullptr) {  // uniform across the grid
        __shared__ float part[8][8];
#pragma unroll
        for (int c = 0; c < kCh; ++c) {
            float x = acc[c];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == 0) part[wy][c] = x;
        }
        __syncthreads();
        if (threadIdx.x < kCh) {  // row blockIdx.x of the [blocks][8] partial-sum matrix
            float sum = 0.f;
#pragma unroll
            for (int w8 = 0; w8 < 8; ++w8) sum += part[w8][threadIdx.x];
            colsum[static_cast<size_t>(blockIdx.x) * 8 + threadIdx.x] = sum;
        }
    }
    pdl_leave(role);
}

// Weights [C_out][C][KH][KW] -> [C_out][KH][8 * ch] with k = kw * ch + c (zero where c >= C or kw >= KW):
// the K-major operand matching pad_pack's (kw, c) slices.
template <typename TIn>
__global__ void __launch_bounds__(256) repack_weight_window_kernel(const TIn* w, __half* __restrict__ out,
                                                                   int Cout, int C, int KH, int KW, int ch_log2, int role) {
    pdl_enter(role);
    const int total = (Cout * KH) << (3 + ch_log2);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int k = i & ((8 << ch_log2) - 1);
        const int row = i >> (3 + ch_log2);
        const int kh = row % KH, co = row / KH;
        const int kw = k >> ch_log2, c = k & ((1 << ch_log2) - 1);
        float v = 0.f;
        if (c < C && kw < KW) v = load_as_float(w, ((static_cast<size_t>(co) * C + c) * KH + kh) * KW + kw);
        out[i] = __float2half_rn(v);
    }
    pdl_leave(role);
}

// Partial sums of a K-split forward walk, `planes` fp32 planes of [pixels][C] (one per K slice) -> the
// output tensor: the planes are added in slice order (so the result is bitwise repeatable), then bias,
// optional rounding through fp16, cast, and the caller's layout (nchw: out[n][c][pixel of the image]).
// Row-major outputs whose channel count is a multiple of 4 take four values per thread (`vec`).
__device__ __forceinline__ float4 finish4(float4 v, bool has_bias, const float4& b, int round_f16) {
    if (has_bias) {
        v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
    }
    if (round_f16) {
        v.x = __half2float(__float2half_rn(v.x)); v.y = __half2float(__float2half_rn(v.y));
        v.z = __half2float(__float2half_rn(v.z)); v.w = __half2float(__float2half_rn(v.w));
    }
    return v;
}
template <typename TOut>
__global__ void __launch_bounds__(256) finish_rows_kernel(const float* acc, int planes, const float* bias,
                                                          TOut* __restrict__ out, size_t pixels, int C, int hw, int nchw,
                                                          int round_f16, int vec, int role) {
    pdl_enter(role);
    const size_t total = pixels * C;
    if (vec) {
        const uint32_t c4n = static_cast<uint32_t>(C / 4);
        const size_t total4 = total / 4;
        const float4* src = reinterpret_cast<const float4*>(acc);
        for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total4; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
            float4 v = load_global(src + i), bv = make_float4(0.f, 0.f, 0.f, 0.f);
            if (bias != nullptr) {  // (in flight with the planes)
                const float* b = bias + static_cast<uint32_t>(i) % c4n * 4;
                bv = make_float4(load_global(b), load_global(b + 1), load_global(b + 2), load_global(b + 3));
            }
#pragma unroll 8
            for (int z = 1; z < planes; ++z) {
                const float4 b = load_global(src + static_cast<size_t>(z) * total4 + i);
                v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
            }
            v = finish4(v, bias != nullptr, bv, round_f16);
            if (sizeof(TOut) == 2) {
                uint2 h;
                *reinterpret_cast<__half2*>(&h.x) = __floats2half2_rn(v.x, v.y);
                *reinterpret_cast<__half2*>(&h.y) = __floats2half2_rn(v.z, v.w);
                reinterpret_cast<uint2*>(out)[i] = h;
            } else {
                reinterpret_cast<float4*>(out)[i] = v;
            }
        }
        pdl_leave(role);
        return;
    }
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t p = i / C;
        const int c = static_cast<int>(i - p * C);
        float v = load_global(acc + i);
#pragma unroll 4
        for (int z = 1; z < planes; ++z) v += load_global(acc + static_cast<size_t>(z) * total + i);
        if (bias != nullptr) v += load_global(bias + c);
        if (round_f16) v = __half2float(__float2half_rn(v));
        size_t o = i;
        if (nchw) {
            const size_t n = p / hw;
            o = (n * C + c) * hw + (p - n * hw);
        }
        out[o] = static_cast<TOut>(v);
    }
    pdl_leave(role);
}

// The same for many planes of few elements, which a thread would walk one load latency at a time (fp32 4x4 s2 512 -> 64 at 4 x 4, batch 3,
// forward 48.1 -> 16 us; linear 22 x 5248 -> 96 21 -> 13): blockDim = (32, 8), the lanes ty fetch 32 planes at a time into shared memory, where a
// thread per value adds them in the planes' order: results are the same bits.  (Summed by lane instead, a value that rounds the other way in
// an early layer of a net flips activations behind it.)
constexpr int kFinishLanes = 8, kFinishChunk = 32;
template <typename TOut>
__global__ void __launch_bounds__(256) finish_rows_deep_kernel(const float* acc, int planes, const float* bias,
                                                               TOut* __restrict__ out, size_t pixels, int C, int hw, int nchw,
                                                               int round_f16, int vec, int role) {
    pdl_enter(role);
    __shared__ __align__(16) float part[kFinishChunk][128];  // [plane][value of the block: 32 vectors of four, or 32 values]
    const size_t total = pixels * C, items = vec ? total / 4 : total;
    const int t = threadIdx.y * 32 + threadIdx.x, values = vec ? 128 : 32;
    for (size_t i0 = blockIdx.x * 32ull; i0 < items; i0 += gridDim.x * 32ull) {
        const size_t i = i0 + threadIdx.x;
        float v = 0.f;
        for (int z0 = 0; z0 < planes; z0 += kFinishChunk) {
            float4 b[kFinishChunk / kFinishLanes];
#pragma unroll
            for (int k = 0; k < kFinishChunk / kFinishLanes; ++k) {
                const int z = z0 + threadIdx.y + kFinishLanes * k;
                const size_t at = static_cast<size_t>(z) * items + i;
                b[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (z < planes && i < items) {
                    if (vec) b[k] = load_global(reinterpret_cast<const float4*>(acc) + at);
                    else b[k].x = load_global(acc + at);
                }
            }
#pragma unroll
            for (int k = 0; k < kFinishChunk / kFinishLanes; ++k) {
                float* o = part[threadIdx.y + kFinishLanes * k];
                if (vec) *reinterpret_cast<float4*>(o + 4 * threadIdx.x) = b[k];
                else o[threadIdx.x] = b[k].x;
            }
            __syncthreads();
            if (t < values) {
                const int n = min(kFinishChunk, planes - z0);
                if (z0 == 0) v = part[0][t];
                for (int z = z0 == 0 ? 1 : 0; z < n; ++z) v += part[z][t];
            }
            __syncthreads();
        }
        const size_t at = i0 * (vec ? 4 : 1) + t;  // this thread's value
        if (t < values && at < total) {
            const size_t p = at / C;
            const int c = static_cast<int>(at - p * C);
            if (bias != nullptr) v += load_global(bias + c);
            if (round_f16) v = __half2float(__float2half_rn(v));
            size_t o = at;
            if (nchw) {
                const size_t n = p / hw;
                o = (n * C + c) * hw + (p - n * hw);
            }
            out[o] = static_cast<TOut>(v);
        }
    }
    pdl_leave(role);
}

// Phase-packed gather walk: the weights [K][C][KH][KW] of a strided gather (input gradient of a
// convolution, forward of a transposed one; unit dilation) as the weights [N'][K][KH'][KW'] of the
// unit-stride convolution that computes all stride_h x stride_w output phases at once:
// n' = (ph * s_w + pw) * C + c, tap (kh', kw') reads the input at offset (kh' + dh_min, kw' + dw_min),
// which phase ph reaches through kernel row kh = ph + p_h - (kh' + dh_min) * s_h (zero weight if that
// is no kernel row).  Also replicates the bias per phase.
template <typename TIn, typename TBias>
__global__ void __launch_bounds__(256) pack_phase_weights_kernel(const TIn* w, __half* __restrict__ out,
                                                                 const TBias* bias, float* __restrict__ bias_out,
                                                                 int K, int C, int KH, int KW, int s_h, int s_w, int p_h,
                                                                 int p_w, int khp, int kwp, int dh_min, int dw_min, int role) {
    pdl_enter(role);
    const int np = s_h * s_w * C;
    const int total = np * K * khp * kwp;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int kw2 = i % kwp;
        int r = i / kwp;
        const int kh2 = r % khp;
        r /= khp;
        const int k = r % K;
        const int n2 = r / K;
        const int c = n2 % C;
        const int pw = (n2 / C) % s_w;
        const int ph = n2 / (C * s_w);
        const int kh = ph + p_h - (kh2 + dh_min) * s_h;
        const int kw = pw + p_w - (kw2 + dw_min) * s_w;
        float v = 0.f;
        if (kh >= 0 && kh < KH && kw >= 0 && kw < KW)
            v = load_as_float(w, ((static_cast<size_t>(k) * C + c) * KH + kh) * KW + kw);
        out[i] = __float2half_rn(v);
    }
    if (bias_out != nullptr && blockIdx.x == 0 && threadIdx.x < np)
        bias_out[threadIdx.x] = (bias != nullptr) ? load_as_float(bias, threadIdx.x % C) : 0.f;
    pdl_leave(role);
}

// Second stage of the column sums: adds rows [blockIdx.y * rows_per_block, ...) of the [P][stride]
// partial-sum matrix in a fixed order (128 interleaved running sums, then those in a tree) and writes row blockIdx.y of
// `out` ([segments][out_stride]).  Launched again on its own output while more than one segment is left.
// blockDim = (8, 128): few channels and a chain of load latencies, so many threads take few rows each.
__global__ void __launch_bounds__(1024) colsum_finish_kernel(const float* partial, int P, int stride, int C,
                                                             float* __restrict__ out, int out_stride, int rows_per_block, int role) {
    pdl_enter(role);
    __shared__ float part[128][9];
    const int c = blockIdx.x * 8 + threadIdx.x;
    const int p0 = blockIdx.y * rows_per_block;
    const int p1 = min(P, p0 + rows_per_block);
    float s = 0.f;
    if (c < C) {
#pragma unroll 8
        for (int p = p0 + threadIdx.y; p < p1; p += 128) s += load_global(partial + static_cast<size_t>(p) * stride + c);
    }
    part[threadIdx.y][threadIdx.x] = s;
    for (int half = 64; half > 0; half /= 2) {
        __syncthreads();
        if (threadIdx.y < half) part[threadIdx.y][threadIdx.x] += part[threadIdx.y + half][threadIdx.x];
    }
    if (threadIdx.y == 0 && c < C) out[static_cast<size_t>(blockIdx.y) * out_stride + c] = part[0][threadIdx.x];
    pdl_leave(role);
}

// Second stage of a split-K weight gradient: adds the K slices' planes in slice order (bitwise
// repeatable, unlike atomics) and writes dW once.  Row form: dW is `rows` rows of `row_len4` float4,
// plane z holds row r at planes + z * plane_elems + r * src_pitch (floats).
__global__ void __launch_bounds__(256) wgrad_reduce_rows4_kernel(const float* planes, float* __restrict__ dw,
                                                                 int split, size_t plane_elems, size_t rows, int row_len4,
                                                                 size_t src_pitch, int role) {
    pdl_enter(role);
    const size_t total = rows * row_len4;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t r = i / row_len4;
        const int c4 = static_cast<int>(i - r * row_len4);
        const float4* src = reinterpret_cast<const float4*>(planes + r * src_pitch) + c4;
        float4 a = load_global(src);
        const size_t step = plane_elems / 4;
#pragma unroll 4
        for (int z = 1; z < split; ++z) {
            const float4 b = load_global(src + z * step);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
        reinterpret_cast<float4*>(dw)[i] = a;
    }
    pdl_leave(role);
}

// The same for many planes: a thread per element would walk them one load latency at a time (the patch walk cuts K into one slice per
// SM; 1x1 40 -> 16 of 8619 pixels, 135 slices, 27.5 us so and 11.2 with eight lanes).  blockDim = (32, 8): lane ty adds
// planes ty, ty + 8, ... of its float4 in order, then the eight running sums are added in order -- a
// fixed association, so still bitwise repeatable.
__global__ void __launch_bounds__(256) wgrad_reduce_deep4_kernel(const float* planes, float* __restrict__ dw,
                                                                 int split, size_t plane_elems, size_t total4, int row_len4, size_t src_pitch, int role) {
    pdl_enter(role);
    __shared__ float4 part[8][32];
    const size_t i = blockIdx.x * 32ull + threadIdx.x;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < total4) {
        const size_t r = i / row_len4;
        const float4* src = reinterpret_cast<const float4*>(planes + r * src_pitch) + (i - r * row_len4);
        const size_t step = plane_elems / 4;
#pragma unroll 4
        for (int z = threadIdx.y; z < split; z += 8) {
            const float4 b = load_global(src + z * step);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
    }
    part[threadIdx.y][threadIdx.x] = a;
    __syncthreads();
    if (threadIdx.y == 0 && i < total4) {
        float4 t = part[0][threadIdx.x];
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            const float4 b = part[k][threadIdx.x];
            t.x += b.x; t.y += b.y; t.z += b.z; t.w += b.w;
        }
        reinterpret_cast<float4*>(dw)[i] = t;
    }
    pdl_leave(role);
}

// Planes of the tap-by-tile walk ([plain channel][R rows], row (t * c_blocks + pc / kb) * kb + pc % kb = one tap's patch
// channels side by side) -> dW [plain][patch channel][tap].  A block takes one plain channel and 64 patch channels: reads
// run along the patch channels (float4), the tap-fastest order is made in shared memory, and 64 * taps consecutive floats
// are written.  (A thread per element read with a stride of a whole tap row: 4x4 512->128 11 us.)  kPlain plain channels a
// block, their loads in flight together, and 16-byte stores: 4x4 512 x 1024, one plane, 18.8 -> 14 us (bytes: 10 us).
// kGroups groups of threads take every so many planes each, so that no thread of a small gradient walks dozens of them one load latency
// at a time; their sums are added in order.
constexpr int kReducePlain = 2, kReduceGroups = 4;
template <int kGroups>
__global__ void __launch_bounds__(256 * kGroups) wgrad_reduce_taps_kernel(const float* planes, float* __restrict__ dw, int split,
                                                                size_t plane_elems, int c_patch, int c_plain, int n_taps, int c_blocks, int kb,
                                                                int R, int role) {
    pdl_enter(role);
    extern __shared__ float taps[];  // [kGroups][kReducePlain][64][n_taps | 1]
    const int pitch = n_taps | 1, group = kGroups > 1 ? threadIdx.y : 0, group_floats = kReducePlain * 64 * pitch;
    const int plain0 = blockIdx.y * kReducePlain, n_plain = min(kReducePlain, c_plain - plain0);
    const int pc0 = blockIdx.x * 64;
    const int pc = pc0 + 4 * (threadIdx.x & 15);
    if (pc < c_patch) {  // c_patch % 4 == 0
        const float* src = planes + static_cast<size_t>(plain0) * R + (pc / kb) * kb + pc % kb;
        for (int t = threadIdx.x >> 4; t < n_taps; t += 16) {
            const float* p = src + static_cast<size_t>(t) * c_blocks * kb;
            float4 a[kReducePlain];
#pragma unroll
            for (int q = 0; q < kReducePlain; ++q)
                if (q < n_plain) a[q] = load_global(reinterpret_cast<const float4*>(p + group * plane_elems + static_cast<size_t>(q) * R));
#pragma unroll 4
            for (int z = group + kGroups; z < split; z += kGroups) {  // (no more groups than planes)
#pragma unroll
                for (int q = 0; q < kReducePlain; ++q)
                    if (q < n_plain) {
                        const float4 v = load_global(reinterpret_cast<const float4*>(p + z * plane_elems + static_cast<size_t>(q) * R));
                        a[q].x += v.x; a[q].y += v.y; a[q].z += v.z; a[q].w += v.w;
                    }
            }
#pragma unroll
            for (int q = 0; q < kReducePlain; ++q) {
                float* o = taps + group * group_floats + (q * 64 + pc - pc0) * pitch + t;
                if (q < n_plain) o[0] = a[q].x, o[pitch] = a[q].y, o[2 * pitch] = a[q].z, o[3 * pitch] = a[q].w;
            }
        }
    }
    __syncthreads();
    const int n = min(64, c_patch - pc0) * n_taps;  // a multiple of 4
    const bool vec = (reinterpret_cast<uintptr_t>(dw) & 15) == 0;
    for (int q = 0; q < n_plain; ++q) {
        float* out = dw + (static_cast<size_t>(plain0 + q) * c_patch + pc0) * n_taps;
        const float* in = taps + q * 64 * pitch;
        for (int i = (threadIdx.x + 256 * group) * 4; i < n; i += 1024 * kGroups) {
            int c = i / n_taps, t = i - c * n_taps;
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] = in[c * pitch + t];
#pragma unroll
                for (int g = 1; g < kGroups; ++g) v[k] += in[g * group_floats + c * pitch + t];
                if (++t == n_taps) {
                    t = 0;
                    ++c;
                }
            }
            if (vec) {
                *reinterpret_cast<float4*>(out + i) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) out[i + k] = v[k];
            }
        }
    }
    pdl_leave(role);
}

// Where the planes hold element i of dW, in the general form.  layout 0: a plane is laid out like dW.  layout 1: a plane is
// [plain channel][R rows of the tile walk] and dW element (plain, pc, t) sits at row
// (t * c_blocks + pc / kb) * kb + pc % kb.  layout 2 (few-channel window walk): dW element
// (plain, c, kh, kw) sits at row kh * kb + kw * 8 + c.
__device__ __forceinline__ size_t plane_index(size_t i, int layout, int c_patch, int n_taps, int kw_count, int c_blocks, int kb, int R) {
    if (layout == 1) {
        const int t = static_cast<int>(i % n_taps);
        const size_t q = i / n_taps;
        const int pc = static_cast<int>(q % c_patch);
        const size_t plain = q / c_patch;
        return plain * R + static_cast<size_t>(t * c_blocks + pc / kb) * kb + pc % kb;
    }
    if (layout == 2) {
        const int kw = static_cast<int>(i % kw_count);
        size_t q = i / kw_count;
        const int kh = static_cast<int>(q % n_taps);
        q /= n_taps;
        const int c = static_cast<int>(q % c_patch);
        const size_t plain = q / c_patch;
        return plain * R + static_cast<size_t>(kh) * kb + kw * 8 + c;
    }
    return i;
}

// General form, one thread per dW element.  (A kernel of its own: as the one-lane case of the next its guarded loads took 8.2 us instead of 6.8
// for 41 -> 144 5x5 at 16 x 27, batch 5.)
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* planes, float* __restrict__ dw, int split,
                                                           size_t plane_elems, size_t total, int layout, int c_patch,
                                                           int n_taps, int kw_count, int c_blocks, int kb, int R, int role) {
    pdl_enter(role);
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t src = plane_index(i, layout, c_patch, n_taps, kw_count, c_blocks, kb, R);
        float a = load_global(planes + src);
        for (int z = 1; z < split; ++z) a += load_global(planes + z * plane_elems + src);
        dw[i] = a;
    }
    pdl_leave(role);
}

// The same with four threads to an element, for many planes of a small gradient: blockDim = (64, 4), lane ty adds planes ty, ty + 4, ... in
// order (there are no fewer planes than lanes), then the sums are added in order.
constexpr int kReduceLanes = 4;
__global__ void __launch_bounds__(256) wgrad_reduce_lanes_kernel(const float* planes, float* __restrict__ dw, int split,
                                                                 size_t plane_elems, size_t total, int layout, int c_patch,
                                                                 int n_taps, int kw_count, int c_blocks, int kb, int R, int role) {
    pdl_enter(role);
    constexpr unsigned long long kElems = 256 / kReduceLanes;
    __shared__ float part[kReduceLanes][kElems];
    for (size_t i0 = blockIdx.x * kElems; i0 < total; i0 += gridDim.x * kElems) {
        const size_t i = i0 + threadIdx.x;
        const size_t src = plane_index(i, layout, c_patch, n_taps, kw_count, c_blocks, kb, R);
        const int first = threadIdx.y;
        float a = 0.f;
        if (i < total) {
            a = load_global(planes + first * plane_elems + src);
            for (int z = first + kReduceLanes; z < split; z += kReduceLanes) a += load_global(planes + z * plane_elems + src);
        }
        part[threadIdx.y][threadIdx.x] = a;
        __syncthreads();
        if (threadIdx.y == 0) {
#pragma unroll
            for (int k = 1; k < kReduceLanes; ++k) a += part[k][threadIdx.x];
            if (i < total) dw[i] = a;
        }
        __syncthreads();
    }
    pdl_leave(role);
}

// out += add, scaled by `below` where the mask has no bit (null: nowhere), in vectors of eight fp16 values; summed in fp32.
__global__ void __launch_bounds__(256) add_masked_kernel(uint4* out, const uint4* add, const uint8_t* mask, float below, size_t n, int role) {
    pdl_enter(role);
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        uint4 a = load_global(out + i);
        const uint4 b = load_global(add + i);
        const unsigned bits = mask ? load_global(mask + i) : 0xffu;
        __half2* x = reinterpret_cast<__half2*>(&a);
        const __half2* y = reinterpret_cast<const __half2*>(&b);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float2 s = __half22float2(x[j]);
            const float2 t = __half22float2(y[j]);
            s.x += (bits >> (2 * j)) & 1u ? t.x : t.x * below;
            s.y += (bits >> (2 * j + 1)) & 1u ? t.y : t.y * below;
            x[j] = __floats2half2_rn(s.x, s.y);
        }
        out[i] = a;
    }
    pdl_leave(role);
}

template <typename TIn>
__global__ void __launch_bounds__(256) to_float_kernel(const TIn* in, float* out, int n, int role) {
    pdl_enter(role);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = load_as_float(in, i);
    pdl_leave(role);
}

}  // namespace nml
