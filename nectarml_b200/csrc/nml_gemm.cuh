// Products of operands that are read where they lie: out[m + n * out_ns] = sum over k of a(m, k) * b(n, k), one launch, for fp32
// (3xTF32) and fp16 matrices with any strides, of which one per operand is 1.  No conversion pass, no repacked copy, no planes
// in memory: producer warps load the operands with ordinary loads, split or pass them on, and write the K-major, 128-byte
// swizzled tiles that tcgen05.mma reads.
//
// What it is for: small and middling products, where the contraction kernel's preparation was most of the time.  An fp32 Linear
// layer is thirteen launches of 2 to 12 us there for its three passes (conversion of each operand into two planes, the
// product, the sum of its K slices).  What bounds it: launch, set-up and drain, 6.6 us, and 0.5 to 1.3 us a K slice (its loads'
// latency, the split, the fence in front of the MMAs), two slices ahead in registers, two blocks to an SM.
//
// The roles of rows and columns are chosen so that m runs along the result's memory: the lanes of the epilogue are
// consecutive m and store from registers, whatever the alignment.  Where a product has few tiles its K loop is cut over the
// blocks of a cluster: each leaves its partial sums in its own shared memory and adds up a share of the columns of all of them, in
// slice order, so results are bitwise repeatable.  The tensor core truncates as it accumulates, so consecutive slices go to
// accumulators of their own (four of 32 columns, two of 64), which the epilogue adds: no sum has more terms than in the
// contraction kernel's plan for the same product.
//
//   warps 0..7   producers, then the epilogue
//   warp 8       MMA issuer, TMEM
#pragma once
#include "nml_prepass.cuh"
#include "nml_umma.cuh"

namespace nml {

constexpr int kGemmThreads = 288, kGemmProducers = 256;
constexpr int kGemmMaxSplits = 8;

struct GemmParams {
    const void *a, *b, *bias;
    void* out;
    long long a_stride, b_stride, out_ns;       // elements between rows (m, n) where k is contiguous, between k else; between columns of the result
    long long a_batch, b_batch, out_batch;
    int M, N, K;
    int bn, tiles_m, tiles_n;
    int splits, per;                            // blocks that share a tile's K loop (a cluster), slices of each
    int stages;
    int a_vec, b_vec;                           // k-contiguous operand whose rows all start on 16 bytes
    int bias_f16, out_f16, round_f16;
    int role;
    int* err;
    unsigned long long wait_limit_ns;
};

template <typename T>
struct GemmType;
template <>
struct GemmType<float> {
    static constexpr int kPlanes = 2, kChunk = 4, kSlice = 32, kKind = KIND_TF32;  // values in 16 bytes, values of a K slice
};
template <>
struct GemmType<__half> {
    static constexpr int kPlanes = 1, kChunk = 8, kSlice = 64, kKind = KIND_F16;
};

// Sixteen bytes of an operand: values k ... of one row, zeros outside the matrix.
__device__ __forceinline__ uint4 gemm_gather(const float* p, long long step, int n) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (n > 0) v.x = __float_as_uint(load_global(p));
    if (n > 1) v.y = __float_as_uint(load_global(p + step));
    if (n > 2) v.z = __float_as_uint(load_global(p + 2 * step));
    if (n > 3) v.w = __float_as_uint(load_global(p + 3 * step));
    return v;
}
__device__ __forceinline__ uint4 gemm_gather(const __half* p, long long step, int n) {
    uint32_t h[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = i < n ? __half_as_ushort(load_global(p + i * step)) : 0u;
    return make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
}

// One operand as a thread sees it: kRows rows, of which it owns `count` 16-byte chunks of a K slice.  Where k is contiguous
// eight neighbouring threads share a row (one coalesced line), else the lanes are consecutive rows (each of a chunk's loads is
// one); either way a warp's 16-byte stores fall on all banks once.
template <typename T, bool kContiguous>
struct GemmOperand {
    const T* p;         // first value of chunk 0 in the present slice
    long long stride;
    int row0, chunk0, count, groups_log2, rows_left, vec;
    __device__ __forceinline__ GemmOperand(const T* base, long long stride_, int first_row, int rows, int tile_rows, int k0, int vec_)
        : stride(stride_), vec(vec_) {
        const int t = threadIdx.x;
        groups_log2 = tile_rows == 128 ? 2 : tile_rows == 64 ? 1 : 0;
        count = tile_rows / 32;
        if (kContiguous) {
            row0 = t >> 3;
            chunk0 = t & 7;
        } else {
            row0 = (t & 31) + 32 * ((t >> 5) & ((1 << groups_log2) - 1));
            chunk0 = t >> (5 + groups_log2);
        }
        rows_left = rows - first_row;
        const long long r = first_row + row0;
        p = kContiguous ? base + r * stride + k0 + chunk0 * GemmType<T>::kChunk : base + r + (k0 + chunk0 * GemmType<T>::kChunk) * stride;
    }
    __device__ __forceinline__ int row(int i) const { return kContiguous ? row0 + 32 * i : row0; }
    __device__ __forceinline__ int chunk(int i) const { return kContiguous ? chunk0 : chunk0 + (i << (3 - groups_log2)); }
    // the slice whose first k leaves k_left values of the matrix
    __device__ __forceinline__ void load(uint4 (&v)[4], int k_left) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= count) break;
            const int n = row(i) < rows_left ? k_left - chunk(i) * GemmType<T>::kChunk : 0;
            const T* q = kContiguous ? p + 32 * i * stride : p + (static_cast<long long>(i) << (3 - groups_log2)) * GemmType<T>::kChunk * stride;
            if (kContiguous && vec && n >= GemmType<T>::kChunk) v[i] = load_global(reinterpret_cast<const uint4*>(q));
            else v[i] = gemm_gather(q, kContiguous ? 1 : stride, n);
        }
        p += kContiguous ? GemmType<T>::kSlice : GemmType<T>::kSlice * stride;
    }
    // to the tile at `tile` (and the split's second plane plane_bytes behind it)
    __device__ __forceinline__ void store(const uint4 (&v)[4], uint32_t tile, uint32_t plane_bytes) const {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= count) break;
            const int r = row(i), c = chunk(i);
            const uint32_t at = tile + r * 128 + ((c ^ (r & 7)) << 4);
            if constexpr (sizeof(T) == 2) {
                st_shared_v4(at, v[i]);
            } else {
                const float x[4] = {__uint_as_float(v[i].x), __uint_as_float(v[i].y), __uint_as_float(v[i].z), __uint_as_float(v[i].w)};
                float hi[4], lo[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    hi[j] = to_tf32_rna(x[j]);
                    lo[j] = to_tf32_rna(x[j] - hi[j]);
                }
                st_shared_v4(at, make_uint4(__float_as_uint(hi[0]), __float_as_uint(hi[1]), __float_as_uint(hi[2]), __float_as_uint(hi[3])));
                st_shared_v4(at + plane_bytes, make_uint4(__float_as_uint(lo[0]), __float_as_uint(lo[1]), __float_as_uint(lo[2]), __float_as_uint(lo[3])));
            }
        }
    }
};

__device__ __forceinline__ float ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

template <typename T, bool kAContiguous, bool kBContiguous>
__global__ void __launch_bounds__(kGemmThreads, 2) gemm_strided_kernel(const __grid_constant__ GemmParams P) {
    using X = GemmType<T>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const uint32_t a_bytes = X::kPlanes * kStageABytes, b_plane = P.bn * 128, stage_bytes = a_bytes + X::kPlanes * b_plane;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + P.stages * stage_bytes);  // [8]
    uint64_t* empty_bar = full_bar + 8;                                               // [8]
    uint64_t* done_bar = empty_bar + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // main accumulators, then the 3xTF32 split's one for the cross products
    const int mains = P.bn == 32 ? 4 : 2;
    const uint32_t cross = mains * P.bn, tmem_cols = X::kPlanes == 2 ? 256 : 128;
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.stages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), kGemmProducers / 32);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        mbar_init(smem_u32(done_bar), 1);
        abort_state_init(abort_flag, P.wait_limit_ns);
        fence_mbar_init();
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(tmem_slot), tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // (behind the allocation: whoever starts early beside the last blocks of this grid must not have taken their columns)
    pdl_enter(P.role);

    const int rank = blockIdx.x % P.splits;
    int tile = blockIdx.x / P.splits;
    const int batch = tile / (P.tiles_m * P.tiles_n);
    tile -= batch * P.tiles_m * P.tiles_n;
    const int tn = tile / P.tiles_m, m0 = (tile - tn * P.tiles_m) * kTileM, n0 = tn * P.bn;
    const int slices_all = (P.K + X::kSlice - 1) / X::kSlice;
    const int first = rank * P.per, slices = max(min(slices_all, first + P.per) - first, 0);
    bool ok = true;
    if (warp < 8) {
        GemmOperand<T, kAContiguous> A(static_cast<const T*>(P.a) + batch * P.a_batch, P.a_stride, m0, P.M, kTileM, first * X::kSlice, P.a_vec);
        GemmOperand<T, kBContiguous> B(static_cast<const T*>(P.b) + batch * P.b_batch, P.b_stride, n0, P.N, P.bn, first * X::kSlice, P.b_vec);
        uint4 a0[4], b0[4], a1[4], b1[4];
        int k_left = P.K - first * X::kSlice, stage = 0;
        uint32_t parity = 1;
        auto load = [&](uint4 (&a)[4], uint4 (&b)[4]) {
            A.load(a, k_left);
            B.load(b, k_left);
            k_left -= X::kSlice;
        };
        auto store = [&](const uint4 (&a)[4], const uint4 (&b)[4]) -> bool {
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&empty_bar[stage]), parity, abort_flag, P.err, ERR_WAIT_EMPTY))) return false;
            const uint32_t at = smem_u32(smem) + stage * stage_bytes;
            A.store(a, at, kStageABytes);
            B.store(b, at + a_bytes, b_plane);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full_bar[stage]));
            if (++stage == P.stages) {
                stage = 0;
                parity ^= 1;
            }
            return true;
        };
        if (slices > 0) load(a0, b0);
        for (int i = 0; ok && i < slices; i += 2) {
            if (i + 1 < slices) load(a1, b1);
            ok = store(a0, b0);
            if (i + 1 >= slices || !ok) break;
            if (i + 2 < slices) load(a0, b0);
            ok = store(a1, b1);
        }
    } else {
        const uint32_t idesc = make_instr_desc(X::kKind, 0, 0, kTileM, P.bn);
        int stage = 0;
        uint32_t parity = 0;
        for (int i = 0; i < slices; ++i) {
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&full_bar[stage]), parity, abort_flag, P.err, ERR_WAIT_FULL))) {
                ok = false;
                break;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t at = smem_u32(smem) + stage * stage_bytes, d = tmem + (i & (mains - 1)) * P.bn;
                const uint64_t ah = make_smem_desc(at, 16, 1024, 2), bh = make_smem_desc(at + a_bytes, 16, 1024, 2);
                if constexpr (sizeof(T) == 2) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_f16(d, ah + 2 * k, bh + 2 * k, idesc, k || i >= mains ? 1u : 0u);
                } else {  // as in the contraction kernel: the cross products have an accumulator of their own
                    const uint64_t al = ah + (kStageABytes >> 4), bl = bh + (b_plane >> 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_tf32(tmem + cross, ah + 2 * k, bl + 2 * k, idesc, k || i ? 1u : 0u);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_tf32(tmem + cross, al + 2 * k, bh + 2 * k, idesc, 1u);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_tf32(d, ah + 2 * k, bh + 2 * k, idesc, k || i >= mains ? 1u : 0u);
                }
                umma_commit(smem_u32(&empty_bar[stage]));
                if (i + 1 == slices) umma_commit(smem_u32(done_bar));
            }
            if (++stage == P.stages) {
                stage = 0;
                parity ^= 1;
            }
        }
    }

    // ------------------------------------------------------------ epilogue --
    const int quarter = warp & 3, half = warp >> 2;  // (warp 8: none)
    const int m_in = quarter * 32 + lane, m = m0 + m_in;
    float bias = 0.f;
    if (warp < 8 && P.bias != nullptr && m < P.M)
        bias = P.bias_f16 ? __half2float(load_global(static_cast<const __half*>(P.bias) + m)) : load_global(static_cast<const float*>(P.bias) + m);
    auto finish = [&](uint32_t bits) {
        float v = __uint_as_float(bits) + bias;
        if (P.round_f16) v = round_through_f16(v);
        return __float_as_uint(v);
    };
    if (warp < 8 && ok) {
        if (slices > 0) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(done_bar), 0, abort_flag, P.err, ERR_WAIT_TMEM_FULL));
        tc_fence_after();
        for (int c = 32 * half; ok && c < P.bn && n0 + c < P.N; c += 64) {
            uint32_t r[32];
            if (slices > 0) {
                const uint32_t t_row = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + c;
                tmem_ld_32x32(t_row, r);
                tmem_ld_wait();
                const int more = min(mains, slices);  // accumulators in use
#pragma unroll 1
                for (int k = 1; k < more + (X::kPlanes - 1); ++k) {
                    uint32_t x[32];
                    tmem_ld_32x32(t_row + (k < more ? k * P.bn : cross), x);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(x[j]));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) r[j] = 0u;
            }
            if (P.splits == 1) {
#pragma unroll
                for (int j = 0; j < 32; ++j) r[j] = finish(r[j]);
                const int ncols = min(32, P.N - n0 - c);
                const long long at = batch * P.out_batch + m + (n0 + c) * P.out_ns;
                if (m < P.M) {
                    if (P.out_f16) store_columns(static_cast<__half*>(P.out) + at, P.out_ns, r, ncols);
                    else store_columns(static_cast<float*>(P.out) + at, P.out_ns, r, ncols);
                }
                __syncwarp();
            } else {  // [column][row], over the operands' stages: every MMA has read them
                const uint32_t at = smem_u32(smem) + (c * kTileM + m_in) * 4;
#pragma unroll
                for (int j = 0; j < 32; ++j) asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + j * kTileM * 4), "r"(r[j]) : "memory");
            }
        }
    }
    if (P.splits > 1) {
        __syncwarp();
        cluster_sync_all();
        const int share = P.bn / P.splits;  // columns of this block
        // (a block that gave up leaves its partners sums of nothing; the status word tells)
        if (warp < 8) {
            const uint32_t mine = smem_u32(smem) + (rank * share * kTileM + m_in) * 4;
            uint32_t theirs[kGemmMaxSplits];
#pragma unroll
            for (int s = 0; s < kGemmMaxSplits; ++s) theirs[s] = s < P.splits ? map_to_cta(mine, s) : 0u;
            for (int j0 = half; j0 < share; j0 += 8) {
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = 0.f;
#pragma unroll
                for (int s = 0; s < kGemmMaxSplits; ++s) {
                    if (s >= P.splits) break;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (j0 + 2 * u < share) v[u] += ld_cluster(theirs[s] + (j0 + 2 * u) * kTileM * 4);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int n = n0 + rank * share + j0 + 2 * u;
                    if (j0 + 2 * u >= share || n >= P.N || m >= P.M) continue;
                    const float y = __uint_as_float(finish(__float_as_uint(v[u])));
                    const long long at = batch * P.out_batch + m + n * P.out_ns;
                    if (P.out_f16) static_cast<__half*>(P.out)[at] = __float2half_rn(y);
                    else static_cast<float*>(P.out)[at] = y;
                }
            }
        }
        __syncwarp();
        cluster_sync_all();  // no block leaves while another reads its sums
    }
    pdl_leave(P.role);
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, tmem_cols);
    }
}

// ---- Batched fp16 products of short K loops (attention scores) whose rows are no whole vectors.
// A block owns 128 columns of one entry's result and walks down its rows, 64 at a time.  Its columns of B (K x 128, at most two K slices)
// are read once and stay in shared memory; the rows of A come 64 at a time, two groups ahead in registers, three in shared memory, two
// accumulators in TMEM, so that the loads of a group, the MMAs of the one before and the stores of the one before that overlap.  The lanes of
// the epilogue are consecutive columns, as above.  Bound by these stores, 64 bytes of a row that starts anywhere (about eight clocks each), and
// for small products by launch and set-up.  By a conversion that turns B round, and the contraction kernel: 64 x 333 x 64 x 333 14.9 us, here
// 13.1; 25 x 464 x 32 x 170 10.3, 7.3; 49 x 368 x 96 x 230 12.1, 9.3; 128 x 700 x 64 x 41 14.4, 11.3.  Put together in shared memory and stored as
// whole 16-byte vectors, four warps meeting once a group, the same rows left more slowly (18.9 us instead of 13.1).
constexpr int kRowsBn = 64, kRowsStages = 3, kRowsMaxK = 128;

// P: M columns of the result, N rows, per groups of rows a block, splits blocks that share a 128-column strip.
__global__ void __launch_bounds__(kGemmThreads, 2) gemm_rows_kernel(const __grid_constant__ GemmParams P) {
    using X = GemmType<__half>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int slices = (P.K + X::kSlice - 1) / X::kSlice;  // 1 or 2
    constexpr uint32_t kGroupBytes = kRowsBn * 128;        // one K slice of a group of rows
    const uint32_t rows_at = slices * kStageABytes, stage_bytes = slices * kGroupBytes;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + rows_at + kRowsStages * stage_bytes);  // [3]
    uint64_t* empty_bar = full_bar + kRowsStages;                                                  // [3]
    uint64_t* tfull_bar = empty_bar + kRowsStages;                                                 // [2]
    uint64_t* tempty_bar = tfull_bar + 2;                                                          // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr uint32_t tmem_cols = 2 * kRowsBn;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRowsStages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), kGemmProducers / 32);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&tfull_bar[b]), 1);
            mbar_init(smem_u32(&tempty_bar[b]), kGemmProducers / 32);
        }
        abort_state_init(abort_flag, P.wait_limit_ns);
        fence_mbar_init();
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(tmem_slot), tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_enter(P.role);  // (behind the allocation, as above)

    int strip = blockIdx.x / P.splits;
    const int first = (blockIdx.x - strip * P.splits) * P.per;
    const int batch = strip / P.tiles_m, m0 = (strip - batch * P.tiles_m) * kTileM;
    const int groups = max(min(P.tiles_n, first + P.per) - first, 0);
    bool ok = true;
    if (warp < 8) {
        const __half* const rows = static_cast<const __half*>(P.b) + batch * P.b_batch;
        const int row0 = threadIdx.x >> 3, chunk0 = threadIdx.x & 7;
        uint4 v0[4], v1[4];  // [slice][row half] of a group of rows
        auto load = [&](uint4 (&v)[4], int group) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = (first + group) * kRowsBn + row0 + 32 * (i & 1), k = (i >> 1) * X::kSlice + chunk0 * X::kChunk;
                if ((i >> 1) >= slices) break;
                const int n = row < P.N && group < groups ? P.K - k : 0;
                const __half* const q = rows + row * P.b_stride + k;
                if (P.b_vec && n >= X::kChunk) v[i] = load_global(reinterpret_cast<const uint4*>(q));
                else v[i] = gemm_gather(q, 1, n);
            }
        };
        {
            GemmOperand<__half, false> A(static_cast<const __half*>(P.a) + batch * P.a_batch, P.a_stride, m0, P.M, kTileM, 0, 0);
            uint4 a[4];
            A.load(a, P.K);
            load(v0, 0);
            load(v1, 1);
            A.store(a, smem_u32(smem), 0);
            if (slices == 2) {
                A.load(a, P.K - X::kSlice);
                A.store(a, smem_u32(smem) + kStageABytes, 0);
            }
        }
        // ---------------------------------------------------------- epilogue of a group --
        const int quarter = warp & 3, half = warp >> 2, m = m0 + quarter * 32 + lane;
        auto drain = [&](int group) -> bool {
            const int buf = group & 1, n = (first + group) * kRowsBn + 32 * half;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&tfull_bar[buf]), (group >> 1) & 1, abort_flag, P.err, ERR_WAIT_TMEM_FULL))) return false;
            tc_fence_after();
            uint32_t r[32];
            tmem_ld_32x32(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + buf * kRowsBn + 32 * half, r);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[buf]));
            if (m < P.M && n < P.N)
                store_columns(static_cast<__half*>(P.out) + batch * P.out_batch + m + n * P.out_ns, P.out_ns, r, min(32, P.N - n));
            __syncwarp();
            return true;
        };
        int stage = 0;
        uint32_t parity = 1;
        auto step = [&](uint4 (&v)[4], int group) -> bool {
            if (group < groups) {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&empty_bar[stage]), parity, abort_flag, P.err, ERR_WAIT_EMPTY))) return false;
                const uint32_t at = smem_u32(smem) + rows_at + stage * stage_bytes;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if ((i >> 1) >= slices) break;
                    const int r = row0 + 32 * (i & 1);
                    st_shared_v4(at + (i >> 1) * kGroupBytes + r * 128 + ((chunk0 ^ (r & 7)) << 4), v[i]);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&full_bar[stage]));
                if (++stage == kRowsStages) {
                    stage = 0;
                    parity ^= 1;
                }
                load(v, group + 2);
            }
            return group == 0 || drain(group - 1);
        };
        for (int g = 0; ok && g <= groups && groups > 0; g += 2) {
            ok = step(v0, g);
            if (ok && g + 1 <= groups) ok = step(v1, g + 1);
        }
    } else {
        const uint32_t idesc = make_instr_desc(X::kKind, 0, 0, kTileM, kRowsBn);
        int stage = 0;
        uint32_t parity = 0;
        for (int g = 0; g < groups; ++g) {
            const int buf = g & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&tempty_bar[buf]), ((g >> 1) & 1) ^ 1, abort_flag, P.err, ERR_WAIT_TMEM_EMPTY)) ||
                !__all_sync(0xffffffffu, mbar_wait(smem_u32(&full_bar[stage]), parity, abort_flag, P.err, ERR_WAIT_FULL)))
                break;
            tc_fence_after();
            if (elect_one()) {
                for (int s = 0; s < slices; ++s) {
                    const uint64_t a = make_smem_desc(smem_u32(smem) + s * kStageABytes, 16, 1024, 2);
                    const uint64_t b = make_smem_desc(smem_u32(smem) + rows_at + stage * stage_bytes + s * kGroupBytes, 16, 1024, 2);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_f16(tmem + buf * kRowsBn, a + 2 * k, b + 2 * k, idesc, k || s ? 1u : 0u);
                }
                umma_commit(smem_u32(&empty_bar[stage]));
                umma_commit(smem_u32(&tfull_bar[buf]));
            }
            __syncwarp();
            if (++stage == kRowsStages) {
                stage = 0;
                parity ^= 1;
            }
        }
    }
    pdl_leave(P.role);
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, tmem_cols);
    }
}

}  // namespace nml
