// Host side of the C ABI declared in include/nectarml_b200.h: turns a layer description into
// conversion passes, TMA tensor maps, a tile/phase/tap table and one launch of the
// contraction kernel.  No allocation, no synchronisation in the descriptor-based entry
// points; the reference-shaped entry points allocate their result as the reference does.
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "../../include/nectarml_b200.h"
#include "nml_prepass.cuh"
#include "nml_umma.cuh"
#include "nml_gemm.cuh"

namespace nml {

// ------------------------------------------------------------------ utilities --
#define NML_CUDA(expr)                                   \
    do {                                                 \
        cudaError_t e_ = (expr);                         \
        if (e_ != cudaSuccess) {                         \
            set_last_cuda_error(e_, #expr);              \
            return NML_ERR_CUDA;                         \
        }                                                \
    } while (0)

static thread_local char g_last_error[256] = {0};
static thread_local char g_last_scratch_error[256] = {0};
static thread_local char g_last_device_error[96] = {0};
static void set_last_cuda_error(cudaError_t e, const char* what) {
    snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
}

static inline size_t round_up(size_t v, size_t m) { return (v + m - 1) / m * m; }
static inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

struct DeviceState;

// Bump allocator over the caller's workspace; in dry mode it only measures.
struct Bump {
    uint8_t* base;
    size_t off, cap;
    bool dry;
    DeviceState* ds = nullptr;  // when set, used instead of the lazily allocated per-device state
    size_t limit = SIZE_MAX;    // what a plan may ask for in all: regions that only buy speed are left out above it
    void* take(size_t bytes) {
        off = round_up(off, 256);
        void* p = dry ? nullptr : base + off;
        off += bytes;
        return p;
    }
    bool fits() const { return dry || off <= cap; }
    size_t room() const {  // left below the limit, for a region taken next
        const size_t o = round_up(off, 256);
        return o < limit ? limit - o : 0;
    }
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// Tuning overrides for experiments and A/B measurements, read from the environment ONCE, when the
// library is first used (unset in normal use; every default is the measured-best setting):
//   NML_TUNE_STAGES   cap on the ring depth            NML_TUNE_BN        forced tile width (64 / 128 / 256)
//   NML_TUNE_KA       K atoms per stage (1 or 2)       NML_TUNE_L2PROMO   TMA L2 promotion (0..3)
//   NML_TUNE_PAIR     0: no CTA pairs                  NML_TUNE_TMASTORE  0: no TMA-store epilogues
//   NML_TUNE_EPI8     0: never a second epilogue group
//   NML_TUNE_PATCH    0: no forward patch walk, 2: wherever it is legal
//   NML_TUNE_SHUFFLE  0: no phase-packed gather walk
//   NML_TUNE_FSPLIT   0: no K split of the forward walk
//   NML_TUNE_WPATCH   0: no weight-gradient patch walk NML_TUNE_WCOAL     0: its gradient leaves by scattered stores
//   NML_TUNE_WTRANS   0: Linear input-gradients never take a transposed copy of the weights
//   NML_TUNE_PAIR128  0: CTA pairs only for 256-column tiles
//   NML_TUNE_NARROW   0: few-channel layers always take eight channels per pixel
//   NML_TUNE_DEEP     0: finishing passes of K splits always by a thread to a result
struct Tune {
    int stages, bn, ka, l2promo, pair, tmastore, epi8, patch, shuffle, fsplit, wpatch, wcoal, wtrans, pair128, narrow, deep;
};
static const Tune& tune() {
    static Tune t;
    static std::once_flag once;
    std::call_once(once, [] {
        auto env = [](const char* name, int dflt) {
            const char* v = getenv(name);
            return (v && *v) ? atoi(v) : dflt;
        };
        t.stages = env("NML_TUNE_STAGES", 8);
        t.bn = env("NML_TUNE_BN", 0);
        t.ka = env("NML_TUNE_KA", 0);  // 0: chosen per launch
        t.l2promo = env("NML_TUNE_L2PROMO", 3);
        t.pair = env("NML_TUNE_PAIR", 1);
        t.tmastore = env("NML_TUNE_TMASTORE", 1);
        t.epi8 = env("NML_TUNE_EPI8", 1);
        t.patch = env("NML_TUNE_PATCH", 1);
        t.shuffle = env("NML_TUNE_SHUFFLE", 1);
        t.fsplit = env("NML_TUNE_FSPLIT", 1);
        t.wpatch = env("NML_TUNE_WPATCH", 1);
        t.wcoal = env("NML_TUNE_WCOAL", 1);
        t.wtrans = env("NML_TUNE_WTRANS", 1);
        t.pair128 = env("NML_TUNE_PAIR128", 1);
        t.narrow = env("NML_TUNE_NARROW", 1);
        t.deep = env("NML_TUNE_DEEP", 1);
    });
    return t;
}

enum { SWZ_NONE = 0, SWZ_128B = 1, SWZ_128B_ATOM32 = 2, SWZ_64B = 3 };

// Tensor map over a dense tensor given fastest-first dims; strides are the dense ones.
static int encode_map(CUtensorMap* tm, const void* ptr, int elem_bytes, int rank, const uint64_t* dims,
                      const uint32_t* box, const uint32_t* estr, int swizzle,
                      const uint64_t* stride_bytes = nullptr) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) {
        snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled not available");
        return NML_ERR_CUDA;
    }
    cuuint64_t gdim[5], gstr[5];
    cuuint32_t b[5], es[5];
    uint64_t pitch = elem_bytes;
    for (int i = 0; i < rank; ++i) {
        gdim[i] = dims[i];
        b[i] = box[i];
        es[i] = estr[i];
        pitch *= dims[i];
        if (i + 1 < rank) gstr[i] = stride_bytes ? stride_bytes[i] : pitch;  // stride of dim i+1
    }
    CUresult r = fn(tm, elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                    rank, const_cast<void*>(ptr), gdim, gstr, b, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle == SWZ_128B ? CU_TENSOR_MAP_SWIZZLE_128B
                    : swizzle == SWZ_64B ? CU_TENSOR_MAP_SWIZZLE_64B
                    : swizzle == SWZ_128B_ATOM32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B
                                                 : CU_TENSOR_MAP_SWIZZLE_NONE,
                    static_cast<CUtensorMapL2promotion>(tune().l2promo),
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(g_last_error, sizeof(g_last_error),
                 "cuTensorMapEncodeTiled failed (%d): rank %d dims %llu %llu %llu %llu box %u %u %u %u",
                 (int)r, rank, (unsigned long long)dims[0], (unsigned long long)(rank > 1 ? dims[1] : 0),
                 (unsigned long long)(rank > 2 ? dims[2] : 0), (unsigned long long)(rank > 3 ? dims[3] : 0),
                 box[0], rank > 1 ? box[1] : 0, rank > 2 ? box[2] : 0, rank > 3 ? box[3] : 0);
        return NML_ERR_CUDA;
    }
    return NML_OK;
}

// Per-device state: status word the kernels report into, SM count.
struct DeviceState {
    int* err = nullptr;
    int sms = 0;
    bool attr_set = false;
};
static DeviceState g_dev[64];
static std::mutex g_dev_mutex;   // guards g_dev, g_static, g_prof and g_ref_ws
static std::atomic<long long> g_launches{0};
static std::atomic<long long> g_launches_of[9];  // by kind, see nml_debug_launch_count
// Where kernels report an abandoned wait.  The words live in the library image, so set-up needs no
// allocation: their device addresses come from cudaGetSymbolAddress, once per device.
static __device__ int g_status_word;
// Per-launch overrides used by the nml_debug_* entry points only (0 / false in normal use).
static thread_local unsigned long long g_dbg_wait_limit_ns = 0;
static thread_local bool g_dbg_short_a_box = false;

struct Profiler {
    std::atomic<bool> on{false};
    int cap = 0, n = 0;
    std::vector<cudaEvent_t> start, stop;
};
static Profiler g_prof;

// The instances of the contraction kernel, and the one that serves a given launch.
typedef void (*UmmaKernel)(const KParams);
template <int kOut, bool kPair>
static UmmaKernel fprop_instance(bool f16) {
    return f16 ? umma_conv_kernel<MODE_FPROP, kOut, true, kPair> : umma_conv_kernel<MODE_FPROP, kOut, false, kPair>;
}
template <int kOut>
static UmmaKernel stream_instance(bool f16) {
    return f16 ? umma_conv_kernel<MODE_FPROP, kOut, true, false, false, false, true> : umma_conv_kernel<MODE_FPROP, kOut, false, false, false, false, true>;
}
static UmmaKernel kernel_for(const KParams& P) {
    if (P.b_taps) {
        if (P.out_mode == OUT_NHWC_TMA) return stream_instance<OUT_NHWC_TMA>(P.out_f16);
        if (P.out_mode == OUT_NCHW_TMA) return stream_instance<OUT_NCHW_TMA>(P.out_f16);
        return P.out_mode == OUT_NHWC ? stream_instance<OUT_NHWC>(P.out_f16) : stream_instance<OUT_NCHW>(P.out_f16);
    }
    if (P.add) return umma_conv_kernel<MODE_FPROP, OUT_NHWC_TMA, true, false, false, true>;
    if (P.dbl)
        return P.mode == MODE_WGRAD ? umma_conv_kernel<MODE_WGRAD, OUT_NHWC, false, true, true> : umma_conv_kernel<MODE_FPROP, OUT_NHWC_TMA, true, true, true>;
    if (P.mode == MODE_WGRAD)
        return P.pair ? umma_conv_kernel<MODE_WGRAD, OUT_NHWC, false, true> : umma_conv_kernel<MODE_WGRAD, OUT_NHWC, false, false>;
    const bool h = P.out_f16 != 0;
    if (P.pair) {
        if (P.out_mode == OUT_NHWC_TMA) return fprop_instance<OUT_NHWC_TMA, true>(h);
        if (P.out_mode == OUT_NCHW_TMA) return fprop_instance<OUT_NCHW_TMA, true>(h);
        return fprop_instance<OUT_NCHW, true>(h);
    }
    if (P.out_mode == OUT_NHWC_TMA) return fprop_instance<OUT_NHWC_TMA, false>(h);
    if (P.out_mode == OUT_NCHW_TMA) return fprop_instance<OUT_NCHW_TMA, false>(h);
    if (P.out_mode == OUT_NHWC) return fprop_instance<OUT_NHWC, false>(h);
    return fprop_instance<OUT_NCHW, false>(h);
}
typedef void (*GemmKernel)(const GemmParams);
template <typename T>
static GemmKernel gemm_instance(bool a_contiguous, bool b_contiguous) {
    return a_contiguous ? (b_contiguous ? gemm_strided_kernel<T, true, true> : gemm_strided_kernel<T, true, false>)
                        : (b_contiguous ? gemm_strided_kernel<T, false, true> : gemm_strided_kernel<T, false, false>);
}
static int raise_smem_limit() {
    for (int i = 0; i < 4; ++i) {
        NML_CUDA(cudaFuncSetAttribute(gemm_instance<float>(i & 1, i & 2), cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
        NML_CUDA(cudaFuncSetAttribute(gemm_instance<__half>(i & 1, i & 2), cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
    }
    NML_CUDA(cudaFuncSetAttribute(gemm_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
    UmmaKernel all[27] = {stream_instance<OUT_NHWC_TMA>(true), stream_instance<OUT_NHWC_TMA>(false), stream_instance<OUT_NCHW_TMA>(true),
                          stream_instance<OUT_NCHW_TMA>(false), stream_instance<OUT_NHWC>(true), stream_instance<OUT_NHWC>(false),
                          stream_instance<OUT_NCHW>(true), stream_instance<OUT_NCHW>(false),
                          umma_conv_kernel<MODE_FPROP, OUT_NHWC_TMA, true, false, false, true>, umma_conv_kernel<MODE_WGRAD, OUT_NHWC, false, true, true>, umma_conv_kernel<MODE_FPROP, OUT_NHWC_TMA, true, true, true>,
                          umma_conv_kernel<MODE_WGRAD, OUT_NHWC, false, false>, umma_conv_kernel<MODE_WGRAD, OUT_NHWC, false, true>,
                          fprop_instance<OUT_NHWC_TMA, false>(true), fprop_instance<OUT_NHWC_TMA, false>(false),
                          fprop_instance<OUT_NCHW_TMA, false>(true), fprop_instance<OUT_NCHW_TMA, false>(false),
                          fprop_instance<OUT_NHWC, false>(true), fprop_instance<OUT_NHWC, false>(false),
                          fprop_instance<OUT_NCHW, false>(true), fprop_instance<OUT_NCHW, false>(false),
                          fprop_instance<OUT_NHWC_TMA, true>(true), fprop_instance<OUT_NHWC_TMA, true>(false),
                          fprop_instance<OUT_NCHW_TMA, true>(true), fprop_instance<OUT_NCHW_TMA, true>(false),
                          fprop_instance<OUT_NCHW, true>(true), fprop_instance<OUT_NCHW, true>(false)};
    for (UmmaKernel k : all)
        NML_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
    return NML_OK;
}

// Loads every helper kernel of the library (with lazy module loading a kernel is otherwise loaded by
// its first launch, which may allocate and must not happen inside a stream capture).
static int load_helper_kernels() {
    const void* fns[] = {
        (const void*)nchw_to_nhwc_kernel<float>, (const void*)nchw_to_nhwc_kernel<__half>,
        (const void*)nhwc_to_nchw_kernel<float>, (const void*)nhwc_to_nchw_kernel<__half>,
        (const void*)convert_rows_kernel<float>, (const void*)convert_rows_kernel<__half>,
        (const void*)colsum_rows_kernel<float>, (const void*)colsum_rows_kernel<__half>,
        (const void*)colsum_vectors_kernel<float>, (const void*)colsum_vectors_kernel<__half>,
        (const void*)colsum_cluster_kernel<float>, (const void*)colsum_cluster_kernel<__half>,
        (const void*)repack_weight_tile_kernel<float>, (const void*)repack_weight_tile_kernel<__half>,
        (const void*)repack_weight_rows_kernel<float>, (const void*)repack_weight_rows_kernel<__half>,
        (const void*)pad_pack_kernel<float, 4>, (const void*)pad_pack_kernel<__half, 4>,
        (const void*)pad_pack_kernel<float, 8>, (const void*)pad_pack_kernel<__half, 8>,
        (const void*)repack_weight_window_kernel<float>, (const void*)repack_weight_window_kernel<__half>,
        (const void*)finish_rows_kernel<float>, (const void*)finish_rows_kernel<__half>, (const void*)finish_rows_deep_kernel<float>, (const void*)finish_rows_deep_kernel<__half>,
        (const void*)pack_phase_weights_kernel<float, float>, (const void*)pack_phase_weights_kernel<float, __half>,
        (const void*)pack_phase_weights_kernel<__half, float>, (const void*)pack_phase_weights_kernel<__half, __half>,
        (const void*)to_float_kernel<__half>, (const void*)colsum_finish_kernel,
        (const void*)add_masked_kernel, (const void*)repack_half_tile_kernel, (const void*)repack_half_rows_kernel, (const void*)wgrad_reduce_taps_kernel<1>, (const void*)wgrad_reduce_taps_kernel<kReduceGroups>,
        (const void*)wgrad_reduce_rows4_kernel, (const void*)wgrad_reduce_kernel, (const void*)wgrad_reduce_lanes_kernel, (const void*)wgrad_reduce_deep4_kernel,
    };
    for (const void* f : fns) {
        cudaFuncAttributes a;
        NML_CUDA(cudaFuncGetAttributes(&a, f));
    }
    return NML_OK;
}

// One-time set-up of the current device (first use, or nml_init): looks up the status word, loads the
// kernels and raises their shared-memory limit.  Allocates nothing; the cudaMemset is synchronous.
static int device_state(DeviceState** out) {
    int dev = 0;
    NML_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return NML_ERR_INVALID;
    std::lock_guard<std::mutex> lock(g_dev_mutex);
    DeviceState& s = g_dev[dev];
    if (!s.attr_set) {
        void* status = nullptr;
        NML_CUDA(cudaGetSymbolAddress(&status, g_status_word));
        NML_CUDA(cudaMemset(status, 0, sizeof(int)));
        NML_CUDA(cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, dev));
        int rc_attr = raise_smem_limit();
        if (rc_attr) return rc_attr;
        rc_attr = load_helper_kernels();
        if (rc_attr) return rc_attr;
        s.err = static_cast<int*>(status);
        s.attr_set = true;
    }
    *out = &s;
    return NML_OK;
}

// Upper bound on the SMs a launch may occupy (nml_set_sm_limit); 0 = all of them.
static std::atomic<int> g_sm_limit{0};
static inline int limited(int sms) {
    const int lim = g_sm_limit.load(std::memory_order_relaxed);
    return (lim > 0 && lim < sms) ? lim : sms;
}
// SM count the planner assumes: the current device's, or a B200's 148 where no device is present
// (workspace-size queries work on a machine without a GPU).
static int planning_sms() {
    static std::atomic<int> cached{0};
    int v = cached.load();
    if (v > 0) return limited(v);
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        sms <= 0) {
        (void)cudaGetLastError();
        return limited(148);
    }
    cached.store(sms);
    return limited(sms);
}

struct MathInfo {
    int es, kb, enc, planes, kind;
};
static bool math_info(int math, MathInfo* m) {
    switch (math) {
        case NML_MATH_F16: *m = {2, 64, ENC_F16, 1, KIND_F16}; return true;
        case NML_MATH_3XTF32: *m = {4, 32, ENC_TF32_PAIR, 2, KIND_TF32}; return true;
        case NML_MATH_TF32: *m = {4, 32, ENC_TF32_HI, 1, KIND_TF32}; return true;
    }
    return false;
}

// Role (see nml_launch.cuh) of this thread's next helper launch; it falls back to PDL_NORMAL with that launch.
static thread_local int t_role = PDL_NORMAL;
template <typename... P, typename... A>
static void helper_launch(unsigned single_wave_limit, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    const int role = t_role;
    t_role = PDL_NORMAL;
    launch_with(role == PDL_SIBLING || overlaps(grid, single_wave_limit), 1, kernel, grid, block, smem, st, static_cast<A&&>(args)..., role);
}
// The helper launch after this one runs beside it, if both are made.
struct SideBySide {
    SideBySide() { t_role = PDL_LEADER; }
    void second() { t_role = t_role == PDL_NORMAL ? PDL_SIBLING : PDL_NORMAL; }  // (the leader's role is used up once it was launched)
    ~SideBySide() { t_role = PDL_NORMAL; }
};

// Bias gradient = column sums of dY, in two stages so that the result is bitwise repeatable: the pass
// that reads dY writes rows of partial sums ([P][stride], one row per block), colsum_finish_kernel adds
// the rows in a fixed order.  Both scratch matrices come from the workspace.
constexpr int kColsumSegment = 4096;  // rows one block of the second stage adds up
struct ColsumScratch {
    float* partial = nullptr;
    float* second = nullptr;
    int P = 0, stride = 0;
};
static ColsumScratch colsum_scratch(Bump& ws, size_t P, int stride) {
    ColsumScratch c;
    c.P = static_cast<int>(P);
    c.stride = stride;
    c.partial = static_cast<float*>(ws.take(P * stride * sizeof(float)));
    if (P > kColsumSegment) c.second = static_cast<float*>(ws.take(((P + kColsumSegment - 1) / kColsumSegment) * stride * sizeof(float)));
    return c;
}
static int colsum_finish(const ColsumScratch& cs, int C, float* out, cudaStream_t st) {
    const float* src = cs.partial;
    int P = cs.P, stride = cs.stride;
    for (;;) {
        const int S = ceil_div(P, kColsumSegment);
        float* dst = (S == 1) ? out : (src == cs.partial ? cs.second : cs.partial);
        helper_launch(4 * kSms, colsum_finish_kernel, dim3(ceil_div(C, 8), S), dim3(8, 128), 0, st, src, P, stride, C, dst, cs.stride, kColsumSegment);
        ++g_launches;
        if (S == 1) break;
        src = dst;
        P = S;
        stride = cs.stride;
    }
    NML_CUDA(cudaGetLastError());
    return NML_OK;
}

static void convert_rows(const void* src, int dtype, void* p0, void* p1, int enc, size_t rows, int c, int cp, cudaStream_t st) {
    const int blocks = static_cast<int>(std::min<size_t>((rows * (cp / 4) + 255) / 256, 148 * 16));
    if (dtype == NML_F32) helper_launch(4 * kSms, convert_rows_kernel<float>, blocks, 256, 0, st, static_cast<const float*>(src), p0, p1, enc, rows, c, cp);
    else helper_launch(4 * kSms, convert_rows_kernel<__half>, blocks, 256, 0, st, static_cast<const __half*>(src), p0, p1, enc, rows, c, cp);
    ++g_launches;
}

// [B][R][Cc] fp16 -> [B][Cc][Rp] fp16 through the 16-byte kernels; false where the shape does not allow them.
static bool repack_half(const void* src, void* dst, int B, int R, int Cc, int Rp, cudaStream_t st) {
    const __half* w = static_cast<const __half*>(src);
    __half* o = static_cast<__half*>(dst);
    if ((reinterpret_cast<uintptr_t>(src) & 15) || Rp % 8) return false;
    if (Cc > 64) {
        if (Cc % 8) return false;
        helper_launch(4 * kSms, repack_half_tile_kernel, dim3(ceil_div(Cc, 64), ceil_div(Rp, 64), B), 256, 0, st, w, o, R, Cc, Rp);
    } else {
        if ((static_cast<size_t>(R) * Cc) % 8) return false;
        helper_launch(4 * kSms, repack_half_rows_kernel, dim3(ceil_div(Rp, 256), B), 256, 256 * repack_rows_pitch(Cc) * sizeof(__half), st, w, o, R, Cc, Rp);
    }
    ++g_launches;
    return true;
}

// Column sums of a row-major matrix: the first stage's launch, its scratch, and where the sums go.
struct RowsColsum {
    const void* src = nullptr;
    int dtype = 0, c = 0, rows_per_block = 0;
    bool vectors = false;
    size_t pixels = 0;
    dim3 grid;
    ColsumScratch cs;
    float* out = nullptr;  // null: nothing to do
    void plan(const void* s, int dt, size_t px, int ch, float* o) {
        src = s; dtype = dt; pixels = px; c = ch; out = o;
        // enough row blocks to fill the GPU, few enough that the second stage stays negligible
        // (the width of a column block has to follow from the shape alone: workspace queries pass no pointer)
        const int vector = dtype == NML_F16 ? 8 : 4;
        const int col_blocks = ceil_div(c, c % vector == 0 ? 32 * vector : 256);
        vectors = c % vector == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
        rows_per_block = static_cast<int>(std::max<size_t>(64, round_up(ceil_div(static_cast<int>(std::min<size_t>(pixels, 1u << 30)), std::max(1, 1184 / col_blocks)), 8)));
        grid = dim3(col_blocks, static_cast<unsigned>((pixels + rows_per_block - 1) / rows_per_block));
    }
    // Both stages in one launch of eight blocks per column block, up to 1024 rows: a weight gradient with its bias gradient of 64 x
    // 512 -> 512 8.2 -> 6.0 us, 1000 x 304 -> 776 13.7 -> 11.4; more rows are too many for so few blocks (2000 x 512 -> 128 10.5 -> 12.9).
    // On their own between the conversions and the contraction (`serial`: fp32) wide rows are too many from 512 on: 848 x 4 -> 1216 21.4 us in two
    // launches, 23.3 in one; 640 x 512 -> 1216 7 % slower, 1024 x 2048 -> 512 5 %; up to 256 columns 10 to 15 % faster all the way, and beside
    // a product that reads its operands in place, too (824 x 1 -> 348 13.0 and 11.1, 640 x 7 -> 1560 16.5 and 14.3).
    bool serial = false;
    bool one_launch() const { return vectors && pixels <= (serial && dtype == NML_F32 && c > 256 ? 512 : 1024); }
    void first_stage(cudaStream_t st) const {
        if (one_launch()) {
            const int role = t_role, rpb = static_cast<int>(round_up(ceil_div(static_cast<int>(pixels), kColsumCluster), 8));
            t_role = PDL_NORMAL;
            const unsigned blocks = grid.x * kColsumCluster;
            if (dtype == NML_F16)
                launch_with(true, kColsumCluster, colsum_cluster_kernel<__half>, blocks, 256, 0, st, static_cast<const __half*>(src), out, static_cast<int>(pixels), c, rpb, role);
            else
                launch_with(true, kColsumCluster, colsum_cluster_kernel<float>, blocks, 256, 0, st, static_cast<const float*>(src), out, static_cast<int>(pixels), c, rpb, role);
            ++g_launches;
            return;
        }
        if (dtype == NML_F16) {
            auto k = vectors ? colsum_vectors_kernel<__half> : colsum_rows_kernel<__half>;
            helper_launch(kSms, k, grid, 256, 0, st, static_cast<const __half*>(src), cs.partial, pixels, c, rows_per_block);
        } else {
            auto k = vectors ? colsum_vectors_kernel<float> : colsum_rows_kernel<float>;
            helper_launch(kSms, k, grid, 256, 0, st, static_cast<const float*>(src), cs.partial, pixels, c, rows_per_block);
        }
        ++g_launches;
    }
    int second_stage(cudaStream_t st) const {
        if (one_launch()) {
            NML_CUDA(cudaGetLastError());
            return NML_OK;
        }
        return colsum_finish(cs, c, out, st);
    }
};

// Converts an activation tensor into the NHWC operand encoding of `mi` unless it already is one.
// planes[0..1] receive the operand pointers, *cp the padded channel count.  With `colsum` the
// per-channel sums of the tensor (the bias gradient) are produced in the same pass where there is one; for a tensor used
// in place the caller may take them over (`later`) and run them beside the contraction.
static int prepare_activation(const void* src, int dtype, int layout, int batch, int c, int h, int w,
                              const MathInfo& mi, Bump& ws, cudaStream_t st, const void* planes[2], int* cp,
                              float* colsum, RowsColsum* later = nullptr) {
    const int align = 16 / mi.es;
    const bool direct = (mi.enc == ENC_F16) && dtype == NML_F16 && (c % align == 0) &&
                        (layout == NML_NHWC || (h == 1 && w == 1) || c == 1);
    const size_t pixels = static_cast<size_t>(batch) * h * w;
    RowsColsum rows;
    rows.plan(src, dtype, pixels, c, colsum);
    if (direct) {
        planes[0] = src;
        planes[1] = nullptr;
        *cp = c;
        if (colsum) {
            rows.cs = colsum_scratch(ws, rows.grid.y, c);
            if (ws.dry) return NML_OK;
            if (!ws.fits()) return NML_ERR_WORKSPACE;
            if (later) {
                *later = rows;
                return NML_OK;
            }
            rows.first_stage(st);
            return rows.second_stage(st);
        }
        return NML_OK;
    }
    const int Cp = static_cast<int>(round_up(c, align));
    *cp = Cp;
    void* p0 = ws.take(pixels * Cp * mi.es);
    void* p1 = (mi.planes == 2) ? ws.take(pixels * Cp * mi.es) : nullptr;
    planes[0] = p0;
    planes[1] = p1;
    const bool transposing = layout == NML_NCHW && !(h == 1 && w == 1);
    ColsumScratch cs;
    if (colsum) cs = transposing ? colsum_scratch(ws, static_cast<size_t>(batch) * ceil_div(h * w, 64), c) : colsum_scratch(ws, rows.grid.y, c);
    if (ws.dry) return NML_OK;
    if (!ws.fits()) return NML_ERR_WORKSPACE;
    if (transposing) {
        const int tiles_p = ceil_div(h * w, 64), tiles_c = ceil_div(Cp, 64);
        const long long tiles = 1ll * tiles_p * tiles_c * batch;
        if (tiles > INT_MAX / 2) return NML_ERR_UNSUPPORTED;
        const unsigned blocks = static_cast<unsigned>(std::min<long long>(tiles, 6 * kSms));  // (four of them resident)
        auto convert = [&](auto* kernel, auto* in) {
            helper_launch(6 * kSms, kernel, blocks, 256, 0, st, in, p0, p1, mi.enc, c, Cp, h * w, tiles_p, tiles_c, static_cast<int>(tiles),
                          cs.partial);
        };
        if (dtype == NML_F32) convert(nchw_to_nhwc_kernel<float>, static_cast<const float*>(src));
        else convert(nchw_to_nhwc_kernel<__half>, static_cast<const __half*>(src));
        ++g_launches;
        if (colsum) {
            int rc = colsum_finish(cs, c, colsum, st);
            if (rc) return rc;
        }
    } else {
        convert_rows(src, dtype, p0, p1, mi.enc, pixels, c, Cp, st);
        if (colsum) {
            rows.cs = cs;
            rows.serial = true;
            rows.first_stage(st);
            int rc = rows.second_stage(st);
            if (rc) return rc;
        }
    }
    NML_CUDA(cudaGetLastError());
    return NML_OK;
}

// Few-channel path: the activation as a zero-padded [N][Hp][Wp][ch] fp16 image (see pad_pack_kernel).
// Wp leaves room for the 8-pixel window of the last output column.
struct WindowImage {
    const void* ptr;
    int hp, wp;
};
static bool window_eligible(int c, int kw, int d_w, int enc) { return c <= 8 && kw <= 8 && d_w == 1 && enc == ENC_F16; }
// Four channels per pixel halve the MMAs, the patches and the padded image, but consecutive windows start 8 * stride_w
// bytes apart, and TMA wants multiples of 16: odd strides keep eight.
static bool narrow_eligible(int c, int s_w) { return c <= 4 && s_w % 2 == 0 && tune().narrow; }
static int prepare_window(const void* src, int dtype, int layout, int batch, int c, int h, int w, int p_h, int p_w,
                          int s_w, int out_w, int ch, Bump& ws, cudaStream_t st, WindowImage* img, float* colsum = nullptr) {
    img->hp = h + 2 * p_h;
    img->wp = static_cast<int>(round_up(std::max(w + 2 * p_w, (out_w - 1) * s_w + 8), 2));
    const size_t rows = static_cast<size_t>(batch) * img->hp;
    if (rows >= (1u << 31)) return NML_ERR_UNSUPPORTED;
    void* p = ws.take(rows * img->wp * ch * 2);
    img->ptr = p;
    int blocks = static_cast<int>(std::min<size_t>((rows + 7) / 8, 148 * 8));
    ColsumScratch cs;
    if (colsum) cs = colsum_scratch(ws, blocks, 8);  // one row of up to 8 channel sums per block
    if (ws.dry) return NML_OK;
    if (!ws.fits()) return NML_ERR_WORKSPACE;
    const int nchw = (layout == NML_NCHW) ? 1 : 0;
    auto run = [&](auto kernel, auto* in) {
        helper_launch(kSms, kernel, blocks, 256, 0, st, in, nchw, static_cast<__half*>(p), batch, c, h, w, p_h, p_w, img->hp, img->wp, cs.partial);
    };
    if (dtype == NML_F32) run(ch == 4 ? pad_pack_kernel<float, 4> : pad_pack_kernel<float, 8>, static_cast<const float*>(src));
    else run(ch == 4 ? pad_pack_kernel<__half, 4> : pad_pack_kernel<__half, 8>, static_cast<const __half*>(src));
    ++g_launches;
    NML_CUDA(cudaGetLastError());
    if (colsum) return colsum_finish(cs, c, colsum, st);
    return NML_OK;
}

// Picks a power-of-two pixel box (w, h, n) with 2^bits pixels that covers the grid with the
// fewest boxes; ties go to the wider box.  box extents times the element stride stay <= 256.  n_tiles: tiles per box.
static void choose_box(int bits, int gw, int gh, int gn, int s_w, int s_h, int* wl, int* hl, int* nl,
                       int prefer_w_log2 = 0, int n_tiles = 1, int sms = 1, bool split = false, double k_us = 0, double tile_kb = 0, int z_cap = 1) {
    const auto rounds = [&](long long boxes) { return (boxes * n_tiles + sms - 1) / sms; };
    long long best = -1, best_wide = -1, best_narrow = -1;
    int ww = 0, wh = 0, wn = 0, nw = 0, nh = 0, nn = 0;
    for (int a = bits; a >= 0; --a) {
        if ((1 << a) * s_w > 256) continue;
        const bool narrow = prefer_w_log2 > 0 && a < 3 && (1 << a) < gw;  // (see below)
        for (int b = bits - a; b >= 0; --b) {
            if ((1 << b) * s_h > 256) continue;
            int c = bits - a - b;
            if ((1 << c) > 256) continue;
            long long tiles = 1ll * ceil_div(gw, 1 << a) * ceil_div(gh, 1 << b) * ceil_div(gn, 1 << c);
            if (narrow) {
                if (best_narrow < 0 || tiles < best_narrow) {
                    best_narrow = tiles;
                    nw = a;
                    nh = b;
                    nn = c;
                }
                continue;
            }
            if (best < 0 || tiles < best) {
                best = tiles;
                *wl = a;
                *hl = b;
                *nl = c;
            }
            if (a >= prefer_w_log2 && (best_wide < 0 || tiles < best_wide)) {
                best_wide = tiles;
                ww = a;
                wh = b;
                wn = c;
            }
        }
    }
    // A box at least 2^prefer_w_log2 pixels wide (whole 128-byte runs for pixel-major stores) is taken
    // when it costs at most 15 % more tiles and no further round of them, or 3 % more rounds: fp32 1x1 16 -> 832 at 54 x 54, batch 144, boxes
    // of eight pixels in 156 rounds 1337 us, wide ones in 157 452 (of 327 random channel-major layers of many rounds five took 0.56 to 0.95
    // of the time so, none more than 1.04; with 6 % three gain and three lose as much).  3x3 96 -> 96 at 56 x 56, batch 16, fp16 31.1 -> 27.6 us with 392 tiles instead of 448; 128 -> 128 at 28 x 28, batch 16, 112 tiles instead of 98 in one round, 17.1 -> 15.9.
    // 3xTF32 tiles are 128 columns wide: 256 -> 256 at 56 x 56, batch 8, 392 tiles instead of 448 154 -> 124 us.  Their narrow
    // boxes have to save a round of several, though: where all run at once nothing overlaps the drain (`split`; 128 -> 384 at
    // 28 x 28, batch 8, 49.1 us in two rounds of wide boxes, 54.2 in one of narrow ones).
    if (prefer_w_log2 > 0 && best_wide > 0 && best_wide * 100 <= best * 115 &&
        (rounds(best_wide) * 32 <= rounds(best) * 33 || (split && rounds(best) == 1))) {
        *wl = ww;
        *hl = wh;
        *nl = wn;
        best = best_wide;
    }
    // Boxes of fewer than eight pixels of a wider row may save rounds (62 x 62 pixels of 64 images are 1922 boxes of 2 x 1 x 64 and 1984
    // of 64 x 2 x 1), but their pixel-major stores reach 1 TB/s and less (two pixels 0.63) where eight and more reach 3.7: only
    // where the K loop outlasts the stores.  k_us: a tile's K loop, tile_kb: its result.  1x1 64 -> 200 at 62 x 62, batch 64, fp32
    // result of fp16 products 314 -> 54 us without them; 5x5 96 -> 64 at 21 x 21, batch 128, 3xTF32 162 us without, 141 with them; 4x4
    // stride 2 14 -> 3 at 64 x 19, batch 64 23.9 without (two rounds), 15.8 with.  Where fewer boxes leave SMs for a K split (up to z_cap
    // slices) they win by it, and its planes are row-major: input gradient of 4x4 64 -> 200 at 48 x 9, batch 16, 3xTF32 60.8 without, 46.4 with.
    if (best_narrow > 0) {
        const auto launch_us = [&](long long boxes, double store_us) {
            const long long z = z_cap > 1 ? std::min<long long>(z_cap, sms / (boxes * n_tiles)) : 1;
            return z >= 2 ? k_us / z + 3.0 : rounds(boxes) * (std::max(k_us, store_us) + 0.25 * std::min(k_us, store_us));  // (mostly overlapped)
        };
        if (launch_us(best_narrow, tile_kb / (2.4 * (1 << nw))) < 0.97 * launch_us(best, tile_kb / 25.0)) {
            *wl = nw;
            *hl = nh;
            *nl = nn;
        }
    }
}

// Closes the timing bracket of a recorded launch (see nml_profile_begin).
static int profile_stop(int slot, cudaStream_t st) {
    if (slot >= 0) NML_CUDA(cudaEventRecord(g_prof.stop[slot], st));
    return NML_OK;
}

// Launches the contraction kernel.  When `open_slot` is given and the launch is being timed, the
// bracket is left open (slot index returned there) so that the caller can include the kernel's
// second-stage reduction; the caller then closes it with profile_stop.
// Opens a timing bracket before a pass's preparatory kernels (so that they are counted in the pass's
// duration); launch_kernel then continues that bracket instead of opening its own.
static thread_local int g_bracket_slot = -1;
static int profile_open(cudaStream_t st) {
    if (!g_prof.on.load(std::memory_order_relaxed)) return NML_OK;
    std::lock_guard<std::mutex> lock(g_dev_mutex);
    if (g_prof.on.load() && g_prof.n < g_prof.cap) {
        g_bracket_slot = g_prof.n++;
        NML_CUDA(cudaEventRecord(g_prof.start[g_bracket_slot], st));
    }
    return NML_OK;
}

// shared memory besides operands and staging: alignment slack, barriers, bias tiles
constexpr int kFixedSmem = 1024 + 384 + kBiasTileBytes;

static int launch_kernel(KParams& P, DeviceState* ds, cudaStream_t st, int* open_slot = nullptr) {
    // Narrow tiles finish a 64-deep K slice in well under the barrier round trip of a stage, so they
    // take two slices per stage (8 MMAs per round trip); 256-wide tiles already fill 512 clocks.
    // The 3xTF32 split takes one slice: its two planes are 12 MMAs.
    P.ka = P.planes == 2 ? 2 : (P.pair && P.bn == 256) ? 1 : std::max(1, std::min(2, tune().ka ? tune().ka : (P.bn >= 192 ? 1 : 2)));
    if (P.dbl) P.ka = 1;
    const int stage_bytes = P.ka * ((P.dbl ? 2 : 1) * kStageABytes + (P.pair ? P.bn / 2 : P.bn) * 128);
    // Shared memory: the operand ring, then the epilogue's staging buffers (two per warp if that does not
    // cost a ring stage, else one), the per-warp bias tiles, and the barriers.
    const int fixed = kFixedSmem - (P.dbl ? kBiasTileBytes : 0);
    const bool tma_out = (P.mode == MODE_FPROP) && NML_IS_TMA_OUT(P.out_mode);
    // A second group of four epilogue warps (TMA-store and channel-major instances) where a tile's drain outlasts its MMAs.  Clocks,
    // measured: one group needs ~800 per tile plus ~900 per 128-byte piece; four MMAs (one K slice) take 192 at 64 columns
    // and below (shared-memory reads), 512 at 256.  With several tiles per CTA the groups take alternate tiles (one
    // decode per two tiles); with one or two they share each tile, which shortens the last drain.
    const int ctas = P.pair ? limited(ds->sms) / 2 : limited(ds->sms);
    P.epi_warps = 4;
    P.epi_alt = 0;
    if (P.dbl) {
        P.epi_warps = 8;
    } else if ((tma_out || (P.mode == MODE_FPROP && P.out_mode == OUT_NCHW)) && tune().epi8) {
        int k_slices = 0;  // longest phase
        for (int p = 0; p < P.n_phases; ++p) k_slices = std::max(k_slices, P.c_blocks * P.phases[p].tap_count);
        const int pieces = ceil_div(P.bn, P.out_f16 ? 64 : 32);
        const int mma = k_slices * (P.planes == 2 ? 3 : 1) * (P.bn <= 64 ? 192 : P.bn <= 128 ? 288 : 512);
        if (mma * 2 < (800 + 900 * pieces) * 3) {
            // (channel-major stores alternate or have one group; 128 x 300 x 128 x 300 fp16 products 23.7 -> 21.6 us, 8 x 1000 x 64 x
            // 999 fp32 22.9 -> 20.0)
            P.epi_alt = P.num_tiles > (tma_out ? 2 * ctas : ctas) ? 1 : 0;
            P.epi_warps = (P.epi_alt || (tma_out && pieces >= 2)) ? 8 : 4;
        }
    }
    P.tbufs_log2 = 0;
    while (P.tbufs_log2 < (P.epi_alt ? 2 : 1) && ((2 * P.bn * P.planes * (P.dbl ? 2 : 1)) << P.tbufs_log2) <= 512) ++P.tbufs_log2;
    size_t smem;
    if (P.wpatch) {
        // [stages x (patch, box of the other tensor)][staging (unused by this walk)][bias][barriers]
        P.ka = 1;
        P.stg_bufs = 1;
        const int w_stage = P.patch_bytes + P.bn * 128;
        const int avail = 232448 - fixed - P.epi_warps * P.stg_bufs * kStagingBufBytes;
        P.stages = std::max(2, std::min(8, avail / w_stage));
        P.ring_bytes = P.stages * w_stage;
        {
            const long long run = 1ll * P.c_patch * P.n_taps * (P.kw_pack ? P.kw_count : 1);
            P.w_coalesce = (tune().wcoal && 32 * run * 4 <= P.ring_bytes && P.num_tiles <= limited(ds->sms)) ? 1 : 0;
        }
        smem = static_cast<size_t>(P.ring_bytes) + P.epi_warps * P.stg_bufs * kStagingBufBytes + fixed;
    } else if (P.patch && P.b_taps) {
        // [B stages][patch buffers]: two channel blocks' patches, and the taps of as much of a channel block to a stage as two stages
        // have room for.  (What a stage costs besides its MMAs, about 400 clocks, is spread over its taps: 3x3 256 -> 64 at 32 x 32, batch 64,
        // two taps to a stage 44 us, three 38, five 35, nine 33.)
        P.ka = 1;
        const int slice = P.planes * P.bn * 128, patches = P.planes * P.patch_bytes;
        P.stg_bufs = 1;
        int avail = 232448 - fixed - P.epi_warps * kStagingBufBytes - 2 * patches;
        if (avail < 3 * slice && P.epi_warps == 8) {
            P.epi_warps = 4;
            P.epi_alt = 0;
            P.tbufs_log2 = std::min(P.tbufs_log2, 1);
            avail += 4 * kStagingBufBytes;
        }
        if (avail < 2 * slice) return NML_ERR_UNSUPPORTED;  // (two patches of 130 KB at most leave more)
        const int most = std::max(1, std::min(P.planes == 2 ? kStreamTapsSplit : kStreamTaps, avail / slice / 2));
        P.b_taps = ceil_div(P.b_taps, ceil_div(P.b_taps, most));
        P.stages = std::min(8, avail / (P.b_taps * slice));
        avail -= P.stages * P.b_taps * slice;
        P.a_stages = std::min(4, 2 + avail / patches);
        P.a_ring_off = P.stages * P.b_taps * slice;
        P.ring_bytes = P.a_ring_off + P.a_stages * patches;
        P.issuers = 1;
        smem = static_cast<size_t>(P.ring_bytes) + P.epi_warps * P.stg_bufs * kStagingBufBytes + fixed;
    } else if (P.patch) {
        // [resident B slices][patch buffers][staging][bias][barriers]
        P.ka = 1;
        const int res_bytes = P.c_blocks * P.n_taps * P.bn * P.b_row_bytes;  // the taps of every phase
        P.stg_bufs = P.epi_warps == 8 ? 1 : 2;  // (alternate groups return to a buffer after two tiles; patches need the room)
        int avail = 232448 - fixed - P.epi_warps * P.stg_bufs * kStagingBufBytes;
        if (res_bytes + 2 * P.patch_bytes > avail) {  // trade staging for residency
            P.stg_bufs = 1;
            avail = 232448 - fixed - P.epi_warps * P.stg_bufs * kStagingBufBytes;
            if (res_bytes + 2 * P.patch_bytes > avail) {
                P.epi_warps = 4;
                P.epi_alt = 0;
                P.tbufs_log2 = std::min(P.tbufs_log2, 1);
                avail = 232448 - fixed - P.epi_warps * P.stg_bufs * kStagingBufBytes;
            }
        }
        if (res_bytes + 2 * P.patch_bytes > avail) return NML_ERR_UNSUPPORTED;  // (run_fprop_like has checked that they fit)
        P.stages = 1;
        P.a_stages = std::min(4, (avail - res_bytes) / P.patch_bytes);
        if (P.a_stages < (P.c_blocks << P.tbufs_log2)) P.tbufs_log2 = std::min(P.tbufs_log2, 1);
        P.issuers = (P.tbufs_log2 >= 1 && P.a_stages >= (P.c_blocks << P.tbufs_log2)) ? 2 : 1;
        P.a_ring_off = static_cast<int>(round_up(res_bytes, 1024));
        P.ring_bytes = P.a_ring_off + P.a_stages * P.patch_bytes;
        smem = static_cast<size_t>(P.ring_bytes) + P.epi_warps * P.stg_bufs * kStagingBufBytes + fixed;
    } else {
    // (a double tile's warps have one buffer each, or none where they store from registers)
    int stages2 = P.dbl ? 0 : (232448 - fixed - P.epi_warps * 2 * kStagingBufBytes) / stage_bytes;
    const int bufs1 = P.dbl && !tma_out ? 0 : 1;
    int stages1 = (232448 - fixed - P.epi_warps * bufs1 * kStagingBufBytes) / stage_bytes;
    P.stg_bufs = (stages2 >= std::min(stages1, 8) || (P.add && stages2 >= 3)) ? 2 : bufs1;
    int stages = std::min(8, P.stg_bufs == 2 ? stages2 : stages1);
    stages = std::max(2, std::min(stages, tune().stages));
    P.stages = stages;
    P.ring_bytes = stages * stage_bytes;
    smem = static_cast<size_t>(stages) * stage_bytes + P.epi_warps * P.stg_bufs * kStagingBufBytes + fixed;
    }
    smem = std::max<size_t>(smem, 120 * 1024);  // one CTA per SM: each allocates its own TMEM
    P.err = ds->err;
    int grid = P.pair ? 2 * std::min(P.num_tiles, limited(ds->sms) / 2) : std::min(P.num_tiles, limited(ds->sms));
    if (grid <= 0) return NML_OK;
    P.wait_limit_ns = g_dbg_wait_limit_ns;
    int rec_slot = g_bracket_slot;  // a bracket the caller opened, if any
    g_bracket_slot = -1;
    const bool pre_opened = rec_slot >= 0;
    if (!pre_opened && g_prof.on.load(std::memory_order_relaxed)) {
        std::lock_guard<std::mutex> lock(g_dev_mutex);
        if (g_prof.on.load() && g_prof.n < g_prof.cap) rec_slot = g_prof.n++;
    }
    const bool rec = rec_slot >= 0;
    if (rec && !pre_opened) NML_CUDA(cudaEventRecord(g_prof.start[rec_slot], st));
    // No idle second group (352 -> 224 threads: Linear 700 x 300 -> 200 forward 9.0 -> 8.7 us, 32 x 512 -> 2048 input gradient 10.5 -> 9.9),
    // but for the patch walk, which measured 3 % slower without (3x3 64 at 56 x 56, batch 8, channel-major fp16 13.2 -> 13.7).
    const int threads = P.epi_warps == 8 ? kThreadsWide : P.patch ? threads_for(P.out_mode) : kThreads;
    // (under an SM limit not before its predecessor has ended: blocks that wait would sit on the SMs that are to stay free, and
    // a block of this kernel leaves no room beside it)
    if (P.dbl) ++g_launches_of[NML_DEBUG_DOUBLE_TILES];
    if (P.add) ++g_launches_of[NML_DEBUG_SUMS];
    if (P.mode == MODE_FPROP && P.b_taps) ++g_launches_of[NML_DEBUG_STREAMED];
    launch_with(g_sm_limit.load(std::memory_order_relaxed) == 0, P.pair ? 2 : 1, kernel_for(P), grid, threads, smem, st, P);
    NML_CUDA(cudaGetLastError());
    if (open_slot) *open_slot = rec_slot;
    else if (rec) NML_CUDA(cudaEventRecord(g_prof.stop[rec_slot], st));
    ++g_launches;
    return NML_OK;
}

// Microseconds one 128-byte-deep K slice of a 128-row tile keeps an SM busy, by tile width: 512 clocks of MMA at 256
// columns; narrower tiles cost more per column (measured: 1.28x at 128, 2.24x at 64).
static double slice_us(int bn) { return 0.27 * (bn / 256.0) * (bn > 128 ? 1.0 : bn > 64 ? 1.28 : 2.24); }

// Double tiles (see umma_conv_kernel): clocks of a K slice of a pair's tile, one row tile high and two, and what a 256-column
// double tile adds, whose drain nothing overlaps.  Measured on Linear layers: 16384 x 512 -> 2048 (8 slices, 7 rounds of single
// tiles, 4 of double ones) 36.9 us single, 44.3 double; 16384 x 1024 -> 4096 (16; 14 and 7) 110.6 and 116.4; 16384 x 2048 -> 8192
// (32; 28 and 14) 408 and 383; its input gradient (128 slices, 7 rounds of single tiles; three double ones and a single
// one) 421 and 384; 4096 x 2048 -> 8192's (64 tiles in one round of double ones) 123 and 98.
struct PairCost {
    double one, two, drain;
};
static PairCost pair_cost(int bn) { return bn == 256 ? PairCost{575.0, 1060.0, 2000.0} : PairCost{430.0, 690.0, 0.0}; }
// The plan of a launch of `rows` x n_tiles pair tiles of k slices on `units` pairs: 0 double rows, all of them (INT_MAX), or as
// many as fill whole rounds, with single tiles behind them where their last round would be half empty.
static int plan_double_rows(int rows, int n_tiles, int k, int bn, int units, bool may_mix) {
    const PairCost c = pair_cost(bn);
    const double one = k * c.one, two = k * c.two + c.drain;
    const long long single = 1ll * rows * n_tiles, dbl = 1ll * ((rows + 1) / 2) * n_tiles;
    const double all_single = static_cast<double>((single + units - 1) / units) * one;
    const double all_double = static_cast<double>((dbl + units - 1) / units) * two;
    double best = all_single * 0.985;
    int plan = 0;
    if (all_double < best) {
        best = all_double;
        plan = INT_MAX;
    }
    if (may_mix) {
        const int big_rows = static_cast<int>(dbl / units * units / n_tiles);
        const long long big = 1ll * big_rows * n_tiles, total = big + 1ll * (rows - 2 * big_rows) * n_tiles;
        if (big_rows > 0 && rows > 2 * big_rows) {
            double cost = 0;
            for (const long long j : {0ll, big % units}) {  // the first pair, and the first with one double tile less
                const long long b = (big - j + units - 1) / units, t = (total - j + units - 1) / units;
                cost = std::max(cost, b * two + (t - b) * one);
            }
            if (cost < best) plan = big_rows;
        }
    }
    return plan;
}

// ------------------------------------------------------- fprop-like problems --
struct FpropLike {
    const void* a;
    int a_dtype, a_layout, batch, a_c, a_h, a_w;
    const void* w;
    int w_dtype, d0, d1, kh, kw, k_is_dim0;
    int w_direct;  // 0: repacked; 1: read in place where that can be; 2: so if they start on 16 bytes (scratch for a copy is taken anyway)
    int gather;  // 0: output pixel o reads input o*s - p + k*d; 1: output pixel o gathers from (o + p - k*d)/s
    int s_h, s_w, p_h, p_w, d_h, d_w;
    void* out;
    int out_dtype, out_layout, out_c, out_h, out_w;
    const void* bias;
    int bias_dtype;
    int math, round_f16;
    // phase-packed gather walk (set by run_fprop_like itself): the real output behind the packed columns
    int shuf_sh, shuf_sw, shuf_c, shuf_oh, shuf_ow;
    const void* add;  // fp16, laid out like the (fp16 NHWC) result, added to it: see KParams::add
    const void* add_mask;
    float add_below;
    int w_batched;  // every image has its own [d0][d1] weights, one after the other (batched matmul; kh = kw = 1)
};

// choose_box for the tiles of a forward walk: N columns, `slices` K slices (of three products each for the 3xTF32 split) on the
// average of `phases` of as many boxes.  A slice of fewer than 64 columns takes as long as one of 64; where the patch walk could
// take the layer (patch) it counts by its columns all the same: wide boxes leave the layer to that walk, which is worth
// more than a round (7x7 4 -> 2 at 16 x 12, batch 65, input gradient 14.5 us, 26.3 with narrow boxes).
static void choose_tile_box(int gw, int gh, int gn, int s_w, int s_h, int N, int planes, double slices, int phases, int z_cap, bool patch, int out_bytes,
                            int prefer_w_log2, int sms, int* wl, int* hl, int* nl) {
    const int n_tiles = ceil_div(N, planes == 2 ? 128 : 256), bn = ceil_div(N, n_tiles);
    choose_box(7, gw, gh, gn, s_w, s_h, wl, hl, nl, prefer_w_log2, n_tiles * phases, sms, planes == 2,
               slices * slice_us(patch ? bn : std::max(64, bn)) * (planes == 2 ? 3 : 1), bn * out_bytes / 8.0, z_cap);
}

// Whether a few-channel layer with N output channels takes the patch walk with resident weights when its rows are 64
// bytes long (the conditions of run_fprop_like's own choice, which then makes the same one).
static bool narrow_patch_walk(const FpropLike& f, int N) {
    if (tune().patch != 1 || N > 256) return false;
    const int range_h = (f.kh - 1) * f.d_h, pw = 8, ph = 15 * f.s_h + range_h + 1;
    if (f.kh < 2 || ph > 256 || pw * ph * 64 > 48 * 1024) return false;
    int wl = 0, hl = 0, nl = 0;
    const bool nchw = f.out_layout == NML_NCHW && !(f.out_h == 1 && f.out_w == 1);
    choose_tile_box(f.out_w, f.out_h, f.batch, 1, f.s_h, N, 1, f.kh, 1, 1, true, f.out_dtype == NML_F16 ? 2 : 4, nchw ? 5 : 0, planning_sms(), &wl, &hl, &nl);
    const double area = static_cast<double>(f.out_w) * f.out_h;
    const double eff_patch = area / (1.0 * round_up(f.out_w, 8) * round_up(f.out_h, 16));
    const double eff_box = area * f.batch / (1.0 * round_up(f.out_w, 1 << wl) * round_up(f.out_h, 1 << hl) * round_up(f.batch, 1 << nl));
    const int bn = N <= 16 ? 16 : static_cast<int>(round_up(N, 32));
    const long long need = 1ll * f.kh * bn * 64 + 2 * round_up(pw * ph * 64, 1024);
    return eff_patch >= 0.8 * eff_box && need <= 232448 - kFixedSmem - 4 * kStagingBufBytes;
}

// With `open_slot` the timing bracket of a recorded launch is left open, for a caller that launches more of the pass.
static int run_fprop_like(const FpropLike& f, Bump& ws, cudaStream_t st, int* open_slot = nullptr) {
    MathInfo mi;
    if (!math_info(f.math, &mi)) return NML_ERR_INVALID;
    // A column-strided gather into an NCHW result stores single values a stride apart (4 of every 8 bytes, phase after
    // phase).  Where the first (widest) phase's rows are no multiple of eight pixels the tiles' boxes are at most four pixels wide and every
    // store is a part of a sector; those go through an NHWC copy in the workspace (the walk's stores are TMA boxes then), which
    // one pass of full-width stores turns round.  Input gradient of 3x3 s2, fp32 result of fp16 / 3xTF32 products: 128 channels at
    // 28 x 28, batch 64 30.6 -> 28.4 / 48.4 -> 39.9 us; 256 at 28 x 28, batch 64 99.8 -> 54.4 / 131 -> 101; but 64 at 64 x 64 (whole
    // rows of 32) 54.2 -> 49.6 / 68.9 -> 85.5.  Below four million values the extra pass costs more than it saves (64 at 56 x 56,
    // batch 16 13.3 -> 16.9).  Where the caller's workspace has no room for the copy, the walk stores directly; and above 1 GB,
    // because callers keep their workspace and this would double what the result takes.
    const long long out_values = 1ll * f.batch * f.out_h * f.out_w * f.out_c;
    if (f.gather && f.s_w > 1 && f.out_layout == NML_NCHW && f.out_w > 1 && ceil_div(f.out_w, f.s_w) % 8 != 0 &&
        out_values >= (1 << 22) && f.out_c % (f.out_dtype == NML_F16 ? 64 : 32) == 0) {
        FpropLike f2 = f;
        f2.out_layout = NML_NHWC;
        const int hw = f.out_h * f.out_w;
        const size_t bytes = static_cast<size_t>(out_values) * (f.out_dtype == NML_F16 ? 2 : 4);
        Bump probe = ws;
        probe.dry = true;
        probe.take(bytes);
        const int probe_rc = run_fprop_like(f2, probe, st);
        const int tiles_p = ceil_div(hw, 64), tiles_c = ceil_div(f.out_c, 64);
        const long long tiles = 1ll * tiles_p * tiles_c * f.batch;
        if (probe_rc == NML_OK && bytes <= (1ull << 30) && probe.off <= ws.limit && (ws.dry || probe.off <= ws.cap) && tiles < INT_MAX / 2) {
            f2.out = ws.take(bytes);
            int slot = -1;
            const int rc = run_fprop_like(f2, ws, st, &slot);
            if (rc || ws.dry) return rc;
            const unsigned blocks = static_cast<unsigned>(std::min<long long>(tiles, 6 * kSms));
            if (f.out_dtype == NML_F16)
                helper_launch(6 * kSms, nhwc_to_nchw_kernel<__half>, blocks, 256, 0, st, static_cast<const __half*>(f2.out),
                              static_cast<__half*>(f.out), f.out_c, hw, tiles_p, tiles_c, static_cast<int>(tiles));
            else
                helper_launch(6 * kSms, nhwc_to_nchw_kernel<float>, blocks, 256, 0, st, static_cast<const float*>(f2.out),
                              static_cast<float*>(f.out), f.out_c, hw, tiles_p, tiles_c, static_cast<int>(tiles));
            ++g_launches;
            NML_CUDA(cudaGetLastError());
            return profile_stop(slot, st);
        }
    }
    // A strided gather with very few output channels (input gradient of an RGB stem, image-producing
    // transposed layer) would run one mostly empty 16-column pass per output phase.  All phases are
    // packed into the columns instead: one unit-stride pass over the input with stride_h*stride_w*C
    // columns, whose epilogue scatters each row to its stride_h x stride_w block of output pixels.
    if (f.gather && f.k_is_dim0 && !f.shuf_sh && f.d_h == 1 && f.d_w == 1 && f.s_h * f.s_w > 1 &&
        f.s_h * f.s_w * f.d1 <= 16 && f.out_layout == NML_NHWC && mi.enc == ENC_F16 && f.d1 == f.out_c &&
        tune().shuffle) {
        const int C = f.d1, Kc = f.d0;
        int dh_min = 1 << 20, dh_max = -(1 << 20), dw_min = 1 << 20, dw_max = -(1 << 20);
        for (int ph = 0; ph < f.s_h; ++ph)
            for (int kh = 0; kh < f.kh; ++kh) {
                const int nh = ph + f.p_h - kh;
                if (((nh % f.s_h) + f.s_h) % f.s_h != 0) continue;
                const int dh = (nh >= 0) ? nh / f.s_h : -((-nh) / f.s_h);
                dh_min = std::min(dh_min, dh);
                dh_max = std::max(dh_max, dh);
            }
        for (int pw = 0; pw < f.s_w; ++pw)
            for (int kw = 0; kw < f.kw; ++kw) {
                const int nw = pw + f.p_w - kw;
                if (((nw % f.s_w) + f.s_w) % f.s_w != 0) continue;
                const int dw = (nw >= 0) ? nw / f.s_w : -((-nw) / f.s_w);
                dw_min = std::min(dw_min, dw);
                dw_max = std::max(dw_max, dw);
            }
        if (dh_min <= dh_max && dw_min <= dw_max && (dh_max - dh_min + 1) * (dw_max - dw_min + 1) <= kMaxTaps) {
            const int khp = dh_max - dh_min + 1, kwp = dw_max - dw_min + 1;
            const int np = f.s_h * f.s_w * C;
            __half* wp = static_cast<__half*>(ws.take(static_cast<size_t>(np) * Kc * khp * kwp * sizeof(__half)));
            float* bp = f.bias ? static_cast<float*>(ws.take(sizeof(float) * np)) : nullptr;
            if (!ws.dry) {
                if (!ws.fits()) return NML_ERR_WORKSPACE;
                const int total = np * Kc * khp * kwp;
                const int blocks = std::min(ceil_div(total, 256), 148 * 8);
#define NML_PACK(TW, TB)                                                                                            \
    helper_launch(4 * kSms, pack_phase_weights_kernel<TW, TB>, blocks, 256, 0, st, static_cast<const TW*>(f.w), wp,                      \
                                                              static_cast<const TB*>(f.bias), bp, Kc, C, f.kh, f.kw, \
                                                              f.s_h, f.s_w, f.p_h, f.p_w, khp, kwp, dh_min, dw_min)
                if (f.w_dtype == NML_F32) {
                    if (f.bias_dtype == NML_F16) NML_PACK(float, __half); else NML_PACK(float, float);
                } else {
                    if (f.bias_dtype == NML_F16) NML_PACK(__half, __half); else NML_PACK(__half, float);
                }
#undef NML_PACK
                ++g_launches;
                NML_CUDA(cudaGetLastError());
            }
            FpropLike f2 = f;
            f2.w = wp; f2.w_dtype = NML_F16; f2.d0 = np; f2.d1 = Kc; f2.kh = khp; f2.kw = kwp; f2.k_is_dim0 = 0;
            f2.w_direct = 0; f2.gather = 0; f2.s_h = f2.s_w = 1; f2.p_h = -dh_min; f2.p_w = -dw_min;
            f2.out_c = np; f2.out_h = ceil_div(f.out_h, f.s_h); f2.out_w = ceil_div(f.out_w, f.s_w);
            f2.bias = bp; f2.bias_dtype = NML_F32;
            f2.shuf_sh = f.s_h; f2.shuf_sw = f.s_w; f2.shuf_c = C; f2.shuf_oh = f.out_h; f2.shuf_ow = f.out_w;
            return run_fprop_like(f2, ws, st, open_slot);
        }
    }
    const int T = f.kh * f.kw;
    const int K = f.k_is_dim0 ? f.d0 : f.d1;
    const int N = f.k_is_dim0 ? f.d1 : f.d0;
    if (K != f.a_c || N != f.out_c) return NML_ERR_INVALID;
    if (T > kMaxTaps || f.s_h * f.s_w > kMaxPhases) return NML_ERR_UNSUPPORTED;
    if (f.batch <= 0 || f.a_c <= 0 || f.a_h <= 0 || f.a_w <= 0 || f.out_c <= 0 || f.out_h <= 0 || f.out_w <= 0)
        return NML_ERR_INVALID;

    DeviceState* ds = ws.ds;
    if (!ws.dry && !ds) {
        int rc = device_state(&ds);
        if (rc) return rc;
    }
    // Few input channels (RGB stems): one K slice per kernel ROW, holding (kw, c) for 8 taps, read
    // as overlapping 8-pixel windows of a padded image of four or eight channels -- instead of one mostly empty
    // 64-channel slice per tap.
    const bool window = !f.gather && !f.k_is_dim0 && T > 1 && window_eligible(f.a_c, f.kw, f.d_w, mi.enc);
    // (narrow: with four channels per pixel, where the patch walk with resident weights will be taken)
    const bool narrow = window && narrow_eligible(f.a_c, f.s_w) && narrow_patch_walk(f, N);
    const int win_ch = narrow ? 4 : 8, row_bytes = narrow ? 64 : 128;
    WindowImage wimg = {nullptr, 0, 0};
    // activation operand
    const void* a_planes[2] = {nullptr, nullptr};
    int Cp = 0;
    int rc;
    SideBySide operands;  // the two conversions do not depend on one another
    if (window)
        rc = prepare_window(f.a, f.a_dtype, f.a_layout, f.batch, f.a_c, f.a_h, f.a_w, f.p_h, f.p_w, f.s_w, f.out_w, win_ch, ws, st,
                            &wimg);
    else
        rc = prepare_activation(f.a, f.a_dtype, f.a_layout, f.batch, f.a_c, f.a_h, f.a_w, mi, ws, st, a_planes, &Cp,
                                nullptr);
    if (rc) return rc;
    if (window) a_planes[0] = wimg.ptr;
    operands.second();
    // weight operand
    const int c_blocks = window ? 1 : ceil_div(K, mi.kb);
    const int kp = c_blocks * mi.kb;
    const int align = 16 / mi.es;
    bool direct_w = !window && f.w_direct && T == 1 && mi.enc == ENC_F16 && f.w_dtype == NML_F16 &&
                    ((f.k_is_dim0 ? N : K) % align == 0);
    if (direct_w && f.w_direct == 2) {
        if (ws.dry || (reinterpret_cast<uintptr_t>(f.w) & 15) == 0) ws.take(static_cast<size_t>(N) * kp * mi.es);
        else direct_w = false;
    }
    const void* w_planes[2] = {f.w, nullptr};
    int b_mn_major = 0;
    if (window) {
        void* p0 = ws.take(static_cast<size_t>(N) * f.kh * 8 * win_ch * 2);
        w_planes[0] = p0;
        if (!ws.dry) {
            if (!ws.fits()) return NML_ERR_WORKSPACE;
            const int blocks = std::min(ceil_div(N * f.kh * 8 * win_ch, 256), 148 * 8);
            if (f.w_dtype == NML_F32)
                helper_launch(4 * kSms, repack_weight_window_kernel<float>, blocks, 256, 0, st, static_cast<const float*>(f.w), static_cast<__half*>(p0), N, K, f.kh, f.kw, narrow ? 2 : 3);
            else
                helper_launch(4 * kSms, repack_weight_window_kernel<__half>, blocks, 256, 0, st, static_cast<const __half*>(f.w), static_cast<__half*>(p0), N, K, f.kh, f.kw, narrow ? 2 : 3);
            ++g_launches;
            NML_CUDA(cudaGetLastError());
        }
    } else if (direct_w) {
        b_mn_major = f.k_is_dim0 ? 1 : 0;
    } else {
        size_t bytes = static_cast<size_t>(N) * T * kp * mi.es * (f.w_batched ? f.batch : 1);
        void* p0 = ws.take(bytes);
        void* p1 = (mi.planes == 2) ? ws.take(bytes) : nullptr;
        w_planes[0] = p0;
        w_planes[1] = p1;
        if (!ws.dry) {
            if (!ws.fits()) return NML_ERR_WORKSPACE;
            // out[n][t][k] = w[...]: a swap of the two inner dimensions of [B][R][Cc] (see repack_weight_*_kernel)
            // (batched: one such array per image)
            const int rB = f.w_batched ? f.batch : (f.k_is_dim0 || T == 1) ? 1 : f.d0, rR = f.k_is_dim0 ? f.d0 : f.d1, rC = f.k_is_dim0 ? f.d1 * T : T;
            if (rB > 65535) return NML_ERR_UNSUPPORTED;
            // One tap and K innermost already: nothing to transpose, rows are only converted and padded (the repack
            // would have run one 64-element block per row: 24 us for 1000 x 2048).
            const bool rows_only = T == 1 && !f.k_is_dim0;
#define NML_REPACK(T)                                                                                                           \
    do {                                                                                                                        \
        if (rC <= 64)                                                                                                           \
            helper_launch(4 * kSms, repack_weight_rows_kernel<T>, dim3(ceil_div(kp, 64), rB), 256, 0, st, static_cast<const T*>(f.w), p0, p1, mi.enc, \
                                                                                     rR, rC, kp);                               \
        else                                                                                                                    \
            helper_launch(4 * kSms, repack_weight_tile_kernel<T>, dim3(ceil_div(rC, 64), ceil_div(kp, 64), rB), 256, 0, st,                           \
                static_cast<const T*>(f.w), p0, p1, mi.enc, rR, rC, kp);                                                         \
    } while (0)
            if (rows_only) convert_rows(f.w, f.w_dtype, p0, p1, mi.enc, static_cast<size_t>(rB) * f.d0, f.d1, kp, st);
            else if (f.w_dtype == NML_F16 && mi.enc == ENC_F16 && repack_half(f.w, p0, rB, rR, rC, kp, st)) {}
            else {
                if (f.w_dtype == NML_F32) NML_REPACK(float); else NML_REPACK(__half);
                ++g_launches;
            }
#undef NML_REPACK
            NML_CUDA(cudaGetLastError());
        }
    }
    t_role = PDL_NORMAL;
    // Bias as fp32: the TMA-store epilogues read an fp16 bias as it is (they stage the tile's bias values in
    // shared memory once per column tile anyway); the other epilogues and the finishing pass of a K-split walk
    // take a widened copy, made just before the launch once the plan is known.
    const float* bias32 = static_cast<const float*>(f.bias);
    const bool bias_is_f16 = f.bias && f.bias_dtype == NML_F16;
    float* bias_widened = bias_is_f16 ? static_cast<float*>(ws.take(sizeof(float) * N)) : nullptr;
    if (bias_is_f16) bias32 = bias_widened;
    // Few output pixels under a long K loop (the 2x2 ... 8x8 layers of a U-Net, Linear layers on a few hundred rows):
    // room for the fp32 partial sums of a K-split walk.
    const size_t out_pixels = static_cast<size_t>(f.batch) * f.out_h * f.out_w;
    const int k_slices = (mi.planes == 2 ? 3 : 1) * T * c_blocks;
    const double plane_us = static_cast<double>(out_pixels) * N * 4.0 / 6e6;  // one plane through memory
    const auto split_cost_us = [&](int z) { return 3.0 + (2 * z + 1) * plane_us; };  // storing z planes and the finishing pass
    // (the last condition: two slices, the cheapest split, could save at most the K loop itself; no plan below takes one else)
    const bool may_split = !window && !f.shuf_sh && !f.w_batched && out_pixels <= 8192 && k_slices >= 32 && tune().fsplit &&
                           k_slices * slice_us(256) > split_cost_us(2);
    // one fp32 plane per K slice; the bound on the slice count below holds for every plan made further down
    // (tiles >= tiles_lb, at least 4 K iterations per slice)
    int z_cap = 1;
    if (may_split) {
        const long long tiles_lb = 1ll * ((out_pixels + 127) / 128) * ceil_div(N, 256);
        const int sms = ds ? limited(ds->sms) : planning_sms();
        z_cap = static_cast<int>(std::max<long long>(1, std::min<long long>(sms / tiles_lb, k_slices / 4)));
        z_cap = static_cast<int>(std::min<size_t>(z_cap, ws.room() / (out_pixels * N * sizeof(float))));
    }
    const bool can_split = may_split && z_cap >= 2;
    float* split_acc = can_split ? static_cast<float*>(ws.take(static_cast<size_t>(z_cap) * out_pixels * N * sizeof(float))) : nullptr;
    if (ws.dry) return NML_OK;
    if (!ws.fits()) return NML_ERR_WORKSPACE;

    KParams P;
    memset(&P, 0, sizeof(P));
    P.mode = MODE_FPROP;
    P.out_mode = (f.out_layout == NML_NCHW && !(f.out_h == 1 && f.out_w == 1)) ? OUT_NCHW : OUT_NHWC;
    P.kind = mi.kind;
    P.planes = mi.planes;
    P.a_row_bytes = P.b_row_bytes = row_bytes;
    const int products = mi.planes == 2 ? 3 : 1;  // tensor-core products per K slice
    P.kb = mi.kb;
    P.c_blocks = c_blocks;
    P.a_mn_major = 0;
    P.b_mn_major = b_mn_major;
    P.batch = f.batch;
    P.n_tiles = ceil_div(N, 256);  // provisional; the tile width is settled once the row tiles are known
    P.bn = static_cast<int>(round_up(ceil_div(N, P.n_tiles), b_mn_major ? 64 : 32));
    P.out = f.out;
    P.bias = bias32;
    P.out_f16 = (f.out_dtype == NML_F16);
    P.round_f16 = f.round_f16;
    P.c_out = N;
    P.shuf_sh = f.shuf_sh;
    P.shuf_sw = f.shuf_sw;
    P.shuf_c = f.shuf_c;
    P.shuf_oh = f.shuf_oh;
    P.shuf_ow = f.shuf_ow;
    P.out_h = f.out_h;
    P.out_w = f.out_w;
    P.ld_out = N;

    // phases and taps
    int n_taps = 0, n_phases = 0;
    if (window) {
        Phase& ph = P.phases[0];
        ph.ph = ph.pw = 0;
        ph.hq = f.out_h;
        ph.wq = f.out_w;
        ph.tap_begin = 0;
        for (int kh = 0; kh < f.kh; ++kh) {  // the padding is physical: offsets start at 0
            Tap& t = P.taps[n_taps++];
            t.dh = static_cast<short>(kh * f.d_h);
            t.dw = 0;
            t.wk = kh * 8 * win_ch;
        }
        ph.tap_count = static_cast<short>(n_taps);
        n_phases = 1;
        P.a_stride_h = f.s_h;  // rows of the padded image
        P.a_stride_w = 1;      // the window dimension is already indexed by output column
        P.out_stride_h = P.out_stride_w = 1;
    } else if (!f.gather) {
        Phase& ph = P.phases[0];
        ph.ph = ph.pw = 0;
        ph.hq = f.out_h;
        ph.wq = f.out_w;
        ph.tap_begin = 0;
        for (int kh = 0; kh < f.kh; ++kh)
            for (int kw = 0; kw < f.kw; ++kw) {
                Tap& t = P.taps[n_taps++];
                t.dh = static_cast<short>(kh * f.d_h - f.p_h);
                t.dw = static_cast<short>(kw * f.d_w - f.p_w);
                t.wk = direct_w ? 0 : (kh * f.kw + kw) * kp;
            }
        ph.tap_count = static_cast<short>(n_taps);
        n_phases = 1;
        P.a_stride_h = f.s_h;
        P.a_stride_w = f.s_w;
        P.out_stride_h = P.out_stride_w = 1;
    } else {
        for (int ph_ = 0; ph_ < f.s_h; ++ph_)
            for (int pw_ = 0; pw_ < f.s_w; ++pw_) {
                if (ph_ >= f.out_h || pw_ >= f.out_w) continue;
                Phase& ph = P.phases[n_phases++];
                ph.ph = static_cast<short>(ph_);
                ph.pw = static_cast<short>(pw_);
                ph.hq = ceil_div(f.out_h - ph_, f.s_h);
                ph.wq = ceil_div(f.out_w - pw_, f.s_w);
                ph.tap_begin = static_cast<short>(n_taps);
                for (int kh = 0; kh < f.kh; ++kh) {
                    int nh = ph_ + f.p_h - kh * f.d_h;
                    if (((nh % f.s_h) + f.s_h) % f.s_h != 0) continue;
                    for (int kw = 0; kw < f.kw; ++kw) {
                        int nw = pw_ + f.p_w - kw * f.d_w;
                        if (((nw % f.s_w) + f.s_w) % f.s_w != 0) continue;
                        Tap& t = P.taps[n_taps++];
                        t.dh = static_cast<short>(nh / f.s_h);
                        t.dw = static_cast<short>(nw / f.s_w);
                        t.wk = direct_w ? 0 : (kh * f.kw + kw) * kp;
                    }
                }
                ph.tap_count = static_cast<short>(n_taps - ph.tap_begin);
            }
        P.a_stride_h = P.a_stride_w = 1;
        P.out_stride_h = f.s_h;
        P.out_stride_w = f.s_w;
    }
    P.n_phases = n_phases;
    // M-tile box from the largest phase grid
    const int esw = (f.gather || window) ? 1 : f.s_w, esh = f.gather ? 1 : f.s_h;
    // Patch walk: unit-stride walks with several taps load one haloed patch per channel block instead of
    // one box per tap (8 x 16 pixel tiles of a single image).  Taken when the fixed tile shape does not
    // waste much more of the tile than the free-form box does.  Every phase of a gather walk has its own
    // taps and patch origin; the box is sized for the widest phase.
    const int patch_mode = tune().patch;
    int pw_ = 0, ph_ = 0;
    bool patch_fits = false, can_patch = false;
    int taps_max = 0;
    {
        int range_w = 0, range_h = 0;
        bool every_phase_has_taps = true;
        for (int p = 0; p < n_phases; ++p) {
            Phase& ph = P.phases[p];
            if (ph.tap_count == 0) {
                every_phase_has_taps = false;
                continue;
            }
            taps_max = std::max<int>(taps_max, ph.tap_count);
            int dw_min = 0, dw_max = 0, dh_min = 0, dh_max = 0;
            for (int t = 0; t < ph.tap_count; ++t) {
                const Tap& tp = P.taps[ph.tap_begin + t];
                dw_min = t ? std::min<int>(dw_min, tp.dw) : tp.dw;
                dw_max = t ? std::max<int>(dw_max, tp.dw) : tp.dw;
                dh_min = t ? std::min<int>(dh_min, tp.dh) : tp.dh;
                dh_max = t ? std::max<int>(dh_max, tp.dh) : tp.dh;
            }
            ph.org_w = static_cast<short>(dw_min);
            ph.org_h = static_cast<short>(dh_min);
            range_w = std::max(range_w, dw_max - dw_min);
            range_h = std::max(range_h, dh_max - dh_min);
        }
        // (a row stride of the walk only stretches the patch: consecutive output rows are esh patch rows apart)
        pw_ = 8 + range_w;
        ph_ = 15 * esh + range_h + 1;
        can_patch = every_phase_has_taps && n_taps >= 2 && esw == 1 && pw_ <= 256 && ph_ <= 256 &&
                         pw_ * ph_ * row_bytes <= 48 * 1024;
        // Every weight slice stays in shared memory beside two patch buffers and the smallest epilogue staging (else they are streamed, below).
        const int bn_res = N <= 16 ? 16 : static_cast<int>(round_up(N, 32));
        const long long res_need = 1ll * c_blocks * n_taps * bn_res * row_bytes + 2 * round_up(pw_ * ph_ * row_bytes, 1024);
        patch_fits = can_patch && patch_mode && P.planes == 1 && N <= 256 && !b_mn_major && res_need <= 232448 - kFixedSmem - 4 * kStagingBufBytes;
    }
    if (f.w_batched) {  // a tile never straddles two images
        P.b_batched = 1;
        P.wb_log2 = 7;
    } else {
        choose_tile_box(P.phases[0].wq, P.phases[0].hq, f.batch, esw, esh, N, P.planes, static_cast<double>(c_blocks) * n_taps / n_phases, n_phases,
                        can_split ? std::min(z_cap, 8) : 1, patch_fits, P.out_f16 ? 2 : 4, P.out_mode != OUT_NCHW ? 0 : f.gather && f.s_w > 1 ? 1 : 5,
                        limited(ds->sms), &P.wb_log2, &P.hb_log2, &P.nb_log2);
    }
    // Tile width: 256 columns run the tensor pipe best, but when that leaves SMs idle (few row tiles, narrow N) a narrower tile wins.
    // Cost per column relative to a 256-wide tile, measured on B200: 128 -> 1.28, 64 -> 2.24; the makespan is rounds x width x cost.
    struct Width {
        int n_tiles = 0, bn = 0;
        double cost = -1;
    };
    const int k_loop = std::max(1, c_blocks * taps_max);
    const auto tile_width = [&](long long m_tiles, int forced, bool by_tma) {
        const int cand[4] = {256, 128, 64, forced};
        const double cost[3] = {1.0, 1.28, 2.24};
        Width best;
        const auto consider = [&](int nt, int unit, double margin, double extra) {
            const int bn = static_cast<int>(round_up(ceil_div(N, nt), unit));
            // (the split keeps two accumulators per tile; 256 columns would leave one buffer: 16384 x 1024 -> 1024 125 -> 150 us)
            if (bn > 256 || (bn > 128 && P.planes == 2)) return;
            const double rounds = static_cast<double>(ceil_div(static_cast<int>(std::min<long long>(m_tiles * nt, 1 << 30)), limited(ds->sms)));
            const double t = rounds * bn * (bn > 128 ? cost[0] : bn > 64 ? cost[1] : cost[2]) + extra;
            if (best.cost < 0 || t < best.cost * margin) best = {nt, bn, t};
        };
        // (TMA stores take whole pieces of columns, and only a row's last one may be cut off)
        const bool pieces = by_tma && P.out_f16 && !b_mn_major && forced != 16;
        for (int i = forced ? 3 : 0; i < (forced ? 4 : 3); ++i) {
            const int nt = ceil_div(N, cand[i]);
            consider(nt, b_mn_major || (pieces && nt > 1) ? 64 : forced == 16 ? 16 : 32, 0.97, 0.0);  // prefer the wider tile unless the gain is clear
        }
        // Tiles that are no whole pieces have the plain epilogue, about 2 us, which a long K loop outlasts (in the makespan's units, by a slice of 96
        // columns of 0.33 us): 354 x 512 -> 192, eight slices, two tiles of 96 columns 9.3 us, three of 64 6.5; but 5x5 300 -> 152 at 8 x 9,
        // batch 114, 125 slices, two of 96 43.7, one of 160 59.7, and 3x3 175 -> 144, 27 slices, 20.6 and 22.8.  Fewer tiles read the boxes of A less
        // often, which counts where their rows are short: 5x5 88 -> 144 at 90 x 5, batch 9, 24.4 in two tiles of 96, 30.7 in three of 64.
        const bool short_boxes = mi.kb == 64 && K % 64 != 0 && K % 64 <= 40;
        for (int i = 0; pieces && !forced && i < 3; ++i) {
            const int nt = ceil_div(N, cand[i]);
            if (nt > 1) consider(nt, 32, short_boxes ? 1.0 : 0.945, 2.0 / 0.33 * 96 * cost[1] / k_loop);
        }
        return best;
    };
    Width streamed;  // of a patch walk with streamed weights over more than 64 columns
    const int out_es = P.out_f16 ? 2 : 4;
    const bool rows_of_vectors = (static_cast<size_t>(N) * out_es) % 16 == 0 && (reinterpret_cast<uintptr_t>(f.out) & 15) == 0;
    const int forced_width = P.planes == 2 ? std::min(tune().bn, 128) : tune().bn;
    {
        const int wq = P.phases[0].wq, hq = P.phases[0].hq;
        const double eff_patch = static_cast<double>(wq) * hq / (1.0 * round_up(wq, 8) * round_up(hq, 16));
        const double eff_box = static_cast<double>(wq) * hq * f.batch /
                               (1.0 * round_up(wq, 1 << P.wb_log2) * round_up(hq, 1 << P.hb_log2) * round_up(f.batch, 1 << P.nb_log2));
        if (patch_fits && (patch_mode == 2 || eff_patch >= 0.8 * eff_box)) {
            P.patch = 1;
            P.patch_w = pw_;
            P.patch_h = ph_;
            P.patch_bytes = static_cast<int>(round_up(pw_ * ph_ * row_bytes, 1024));
        }
        // The patch walk with streamed weights, where they do not stay: for tiles that do not pair up (pairs of 128 and 256 columns are as
        // fast or faster by boxes), which wait for their operands.  A patch is read once for all taps, but its tiles are 8 x 16 pixels of one
        // image; so by rounds of tiles and the measured ratio of a slice's time, which falls with the taps that share a patch.
        // By boxes / so, us: fp16 3x3 256 -> 64 at 32 x 32, batch 64, 39.2 / 32.7; 256 -> 192 at 64 x 64 222 / 179; 5x5 192 -> 24 at 99 x 99,
        // batch 4, 61.0 / 40.7; fp32 3x3 128 -> 32 at 64 x 64, batch 16, 88.8 / 75.4; 128 -> 128 at 64 x 64, batch 64, 72 / 73.
        // One tap a phase gains nothing (2x2 s2 transposed 960 -> 40 149 / 182); the four of a 4x4 s2 transposed layer a tenth in fp16 (512 ->
        // 64 114 / 102), which is left: their sums then keep the order of boxes, and an image net's activations do not flip by rounding.
        if (!P.patch && can_patch && patch_mode && taps_max >= 2 && !b_mn_major && !window && !f.w_batched && !f.shuf_sh && !f.add && !can_split &&
            (P.planes == 2 ? N <= 64 : P.kind == KIND_F16 && taps_max >= 6 && (N <= 64 || (N > 128 && N <= 224)))) {
            const int bytes = static_cast<int>(round_up(pw_ * ph_ * row_bytes, 1024)), sms = limited(ds->sms);
            const double slice = (P.planes == 2 ? (N <= 32 ? 0.83 : 0.92) : N <= 32 ? 0.75 : 0.86) * (taps_max >= 12 ? 0.85 : 1.0);
            long long patches = 0, boxes = 0;
            for (int p = 0; p < n_phases; ++p) {
                const Phase& ph = P.phases[p];
                patches += 1ll * ceil_div(ph.wq, 8) * ceil_div(ph.hq, 16) * f.batch;
                boxes += 1ll * ceil_div(ph.wq, 1 << P.wb_log2) * ceil_div(ph.hq, 1 << P.hb_log2) * ceil_div(f.batch, 1 << P.nb_log2);
            }
            const auto rounds = [&](long long n) { return static_cast<double>((n + sms - 1) / sms); };
            bool pays;
            if (N <= 64) {
                // (a small gain does not outlast the first patch of a single round: fp32 3x3 40 -> 40 at 52 x 52, batch 3, 17.1 us by boxes, 17.6 so)
                pays = rounds(patches) * slice <= rounds(boxes) * 0.95 && (slice < 0.9 || rounds(boxes) >= 2);
            } else {
                // More than 128 columns are one tile, two, or several of 64, of either walk; by estimated time, of a slice, a column's drain and a round fitted to
                // 420 layers of 129 ... 224 channels (3x3 to 7x7; by boxes with their width / so: 5x5 29 -> 168 at 44 x 9, batch 3, 12.8 / 16.9 in one
                // tile, stays; 40 -> 160 at 24 x 12, batch 8, 21.7 / 13.3 in three).  0.88 of the time by boxes alone in the mean.
                const bool by_tma = rows_of_vectors && P.out_mode == OUT_NHWC;
                const auto us = [&](long long m_tiles, const Width& w, double slice_us) {
                    return rounds(m_tiles * w.n_tiles) * (k_loop * slice_us + 0.012 * w.bn + 0.6);
                };
                const Width box = tile_width(boxes, forced_width, by_tma);
                // (boxes of up to 40 channels, short rows, take longer: 3x3 24 -> 216 at 15 x 85, batch 40, 30.5 / 21.7)
                double best = (f.a_c <= 40 ? 1.1 : 0.92) * us(boxes, box, box.bn <= 64 ? 0.27 : box.bn <= 128 ? 0.34 : 0.5);
                for (int i = 0; i < 3 && !forced_width; ++i) {
                    const int unit = i > 0 && by_tma && P.out_f16 ? 64 : 32, bn = i == 2 ? 64 : static_cast<int>(round_up(ceil_div(N, 1 + i), unit));
                    const Width w = {ceil_div(N, bn), bn, 0.0};
                    const double so = us(patches, w, bn <= 64 ? 0.17 : std::max(0.25, 0.002 * bn));
                    if (so < best) {
                        best = so;
                        streamed = w;
                    }
                }
                pays = streamed.bn > 0;
            }
            if (2ll * P.planes * bytes > 130 * 1024) {
                pays = false;
                streamed = Width();
            }
            if (pays) {
                P.patch = 1;
                P.patch_w = pw_;
                P.patch_h = ph_;
                P.patch_bytes = bytes;
                P.b_taps = taps_max;  // (how many there is room for: launch_kernel)
            }
        }
        if (P.patch) {
            for (int p = 0; p < n_phases; ++p)
                for (int t = 0; t < P.phases[p].tap_count; ++t) {
                    Tap& tp = P.taps[P.phases[p].tap_begin + t];
                    tp.aoff = ((tp.dh - P.phases[p].org_h) * pw_ + (tp.dw - P.phases[p].org_w)) * row_bytes / 16;
                }
            P.n_taps = n_taps;
            P.wb_log2 = 3;
            P.hb_log2 = 4;
            P.nb_log2 = 0;
        }
    }
    // Row-major results by TMA stores (see below), where the geometry allows them.  Up to eight columns have a short epilogue of their own, for
    // fp16 (one vector a row at most) and for the 16-column tiles of the resident patch walk.  Four and eight fp32 columns of other walks leave by
    // TMA where there are many (from a round of tiles of eight columns on: transposed 5x5 s3 5 -> 8 at 128 x 24, batch 58, short 229 us, TMA
    // 162; linear 155624 x 16 -> 8 20.5 and 18.5; below it the short one saves 0.3 us: 1x1 s2 15 -> 4 at 24 x 64, batch 75, 10.4 and
    // 11.9) or have an fp16 bias, of which the short one wants a widened copy, a launch (linear 8 x 640 -> 8 7.4 and 6.2).
    // (Never phase-packed columns: they belong to several output pixels, and the packed image may be larger than the output.)
    const bool short_rows = N <= 8 && (P.out_f16 || (P.patch && !P.b_taps) || (out_pixels * N < 8ull * kTileM * kSms && !bias_is_f16));
    const bool rows_by_tma = P.out_mode == OUT_NHWC && !P.shuf_sh && tune().tmastore && !short_rows && rows_of_vectors;
    int z_plan = 1;  // K slices per tile
    {
        long long m_tiles_all = 0;
        for (int p = 0; p < n_phases; ++p)
            m_tiles_all += 1ll * ceil_div(P.phases[p].wq, 1 << P.wb_log2) * ceil_div(P.phases[p].hq, 1 << P.hb_log2) *
                           ceil_div(f.batch, 1 << P.nb_log2);
        const int forced = P.patch && !P.b_taps ? (N <= 16 ? 16 : static_cast<int>(round_up(N, 32))) : forced_width;
        const Width width = streamed.bn ? streamed : tile_width(m_tiles_all, forced, rows_by_tma);
        P.n_tiles = width.n_tiles;
        P.bn = width.bn;
        // Tiles that leave half the SMs idle under a long K loop: tile width and number of K slices together, against
        // the plan above without a split.
        if (can_split && !P.patch) {
            int k_min = 1 << 30;  // every slice of every phase gets at least 4 K iterations (2 of three products each)
            for (int p = 0; p < n_phases; ++p)
                if (P.phases[p].tap_count > 0) k_min = std::min(k_min, P.c_blocks * P.phases[p].tap_count);
            auto cost_us = [&](int nt, int bn, int z) {
                const long long tiles = m_tiles_all * nt;
                const double rounds = static_cast<double>((tiles * z + limited(ds->sms) - 1) / limited(ds->sms));
                return rounds * (ceil_div(k_min, z) * slice_us(bn) * products + 2.5) + (z > 1 ? split_cost_us(z) : 0.0);
            };
            // (the estimate that the split was fitted against is that of tiles without regard to TMA stores: 7x7 56 -> 152 at 9 x 11, batch 2, whole
            // 17.9 us, in slices 22.7)
            const Width any = tile_width(m_tiles_all, forced, false);
            double best_us = std::min(cost_us(P.n_tiles, P.bn, 1), cost_us(any.n_tiles, any.bn, 1));
            for (int i = 0; i < 4; ++i) {
                if (forced ? i != 3 : i == 3) continue;
                const int nt = ceil_div(N, i == 3 ? forced : 256 >> i);
                const int bn = static_cast<int>(round_up(ceil_div(N, nt), b_mn_major ? 64 : 32));
                if (m_tiles_all * nt * 2 > limited(ds->sms) || (bn > 128 && P.planes == 2)) continue;
                const int z_max = std::min(z_cap, std::min(static_cast<int>(limited(ds->sms) / (m_tiles_all * nt)), k_min / (P.planes == 2 ? 2 : 4)));
                for (int z = 2; z <= z_max; ++z) {
                    const double us = cost_us(nt, bn, z);
                    if (us < best_us) {
                        best_us = us;
                        z_plan = z;
                        P.n_tiles = nt;
                        P.bn = bn;
                    }
                }
            }
        }
    }
    // Row-major output through TMA stores: the box is the 32 consecutive tile rows one epilogue warp owns (a sub-box of the tile's pixel
    // box), 128 bytes of columns wide.  Columns past the row's end are clipped, so the one tile of a narrow result may end anywhere within
    // a piece (its epilogue then stores accumulator columns of nobody's into the clipped part).  354 x 512 -> 80 forward, whose
    // 96-column tile went through the plain epilogue and took a widened copy of the bias, 9.2 -> 6.3 us.
    if (rows_by_tma) {
        const int esz = out_es;
        const int cpi = 128 / esz;
        if (P.bn % cpi == 0 || P.n_tiles == 1) {
            const int wbx = 1 << P.wb_log2, hbx = 1 << P.hb_log2;
            const int bw = std::min(wbx, 32), bh = std::min(hbx, 32 / bw), bnn = 32 / (bw * bh);
            uint64_t cd[4] = {static_cast<uint64_t>(N), static_cast<uint64_t>(f.out_w), static_cast<uint64_t>(f.out_h),
                              static_cast<uint64_t>(f.batch)};
            uint32_t cb[4] = {static_cast<uint32_t>(cpi), static_cast<uint32_t>(bw * P.out_stride_w),
                              static_cast<uint32_t>(bh * P.out_stride_h), static_cast<uint32_t>(bnn)};
            uint32_t ce[4] = {1, static_cast<uint32_t>(P.out_stride_w), static_cast<uint32_t>(P.out_stride_h), 1};
            if (cb[1] <= 256 && cb[2] <= 256 && encode_map(&P.tmC, f.out, esz, 4, cd, cb, ce, SWZ_128B) == NML_OK &&
                (!f.add || encode_map(&P.tmD, f.add, esz, 4, cd, cb, ce, SWZ_128B) == NML_OK))
                P.out_mode = OUT_NHWC_TMA;
        }
    }
    // Channel-major (NCHW) output through TMA stores: box = the (w, h) sub-box of the warp's 32 pixels x 64 fp16 / 32 fp32 channels, staged channel-major.  Needs
    // unit output stride (TMA cannot stride the innermost dimension) and 16-byte aligned rows.
    if (P.out_mode == OUT_NCHW && tune().tmastore && P.out_stride_w == 1 && P.out_stride_h == 1) {
        const int esz = P.out_f16 ? 2 : 4;
        const int cpi = 128 / esz;
        const int wbx = 1 << P.wb_log2, hbx = 1 << P.hb_log2;
        const int bw = std::min(wbx, 32), bh = std::min(hbx, 32 / bw), bnn = 32 / (bw * bh);
        if (P.bn % cpi == 0 && (bw * esz) % 16 == 0 && (static_cast<size_t>(f.out_w) * esz) % 16 == 0 &&
            (reinterpret_cast<uintptr_t>(f.out) & 15) == 0) {
            uint64_t cd[4] = {static_cast<uint64_t>(f.out_w), static_cast<uint64_t>(f.out_h), static_cast<uint64_t>(N),
                              static_cast<uint64_t>(f.batch)};
            uint32_t cb[4] = {static_cast<uint32_t>(bw), static_cast<uint32_t>(bh), static_cast<uint32_t>(cpi),
                              static_cast<uint32_t>(bnn)};
            uint32_t ce[4] = {1, 1, 1, 1};
            if (encode_map(&P.tmC, f.out, esz, 4, cd, cb, ce, SWZ_NONE) == NML_OK) {
                P.out_mode = OUT_NCHW_TMA;
                int l = 0;
                while ((1 << l) < bw) ++l;
                P.cm_bw_log2 = l;
                l = 0;
                while ((1 << l) < bh) ++l;
                P.cm_bh_log2 = l;
            }
        }
    }
    // Pairs of CTAs (cta_group::2) for 256-wide tiles of problems large enough to fill the pairs: a
    // tile id then names two consecutive row tiles of one phase.
    // (short K loops are epilogue-bound, where pairing only halves the number of independent tiles)
    const int k_iters_min = products * P.c_blocks * std::max<int>(1, P.phases[0].tap_count);
    long long tiles_single = 0;
    for (int p = 0; p < n_phases; ++p)
        tiles_single += 1ll * ceil_div(P.phases[p].wq, 1 << P.wb_log2) * ceil_div(P.phases[p].hq, 1 << P.hb_log2) *
                        ceil_div(f.batch, 1 << P.nb_log2) * P.n_tiles;
    // 128-column tiles pair up too (two K slices per stage, see launch_kernel) where every phase has a K loop
    // of at least four slices and the tiles fill most of the GPU: measured 5-15 % on such layers, a loss on
    // the short phases of strided gathers and on few-tile problems.
    int k_iters_all = k_iters_min;
    for (int p = 0; p < n_phases; ++p)
        if (P.phases[p].tap_count > 0) k_iters_all = std::min(k_iters_all, products * P.c_blocks * P.phases[p].tap_count);
    const bool pair_width = P.bn == 256 || (tune().pair128 && P.bn == 128 && k_iters_all >= 4 && tiles_single * 4 >= 3ll * limited(ds->sms));
    // Pairs save operand feed, which shows over a long K loop or many tiles: with 4 slices, or with 8 and one or two tiles per
    // SM, single CTAs measured 3-14 % faster (they drain twice as many independent tiles).
    const bool pair_k = k_iters_min >= 12 || (k_iters_min >= 5 && tiles_single > 2ll * limited(ds->sms));
    P.pair = (tune().pair && !P.patch && !P.b_batched && z_plan == 1 && pair_width && (!b_mn_major || N % mi.kb == 0) && pair_k &&
              (P.out_mode == OUT_NHWC_TMA || P.out_mode == OUT_NCHW_TMA || P.out_mode == OUT_NCHW) && limited(ds->sms) >= 2) ? 1 : 0;
    // A sum is taken by single CTAs, whose staging buffers have room for the addend.  Under a long K loop pairs (and double tiles) save
    // more than the pass costs that adds behind them: per million values 5.3e-4 us a K term at 256 columns (7.5e-4 at 128, where
    // single CTAs are slower) against 0.92 us, and 2 us for its launch.  Single CTAs / pairs and the pass, us: 3x3 512 at 28 x 28, batch 16
    // 69 / 64; at 7 x 7, batch 256 79 / 69; at 14 x 14, batch 64 79 / 66; 5x5 256 at 28 x 28, batch 64 138 / 122; 1x1 2048 -> 512 at 28 x 28,
    // batch 64 117 / 109; even 3x3 256 at 14 x 14, batch 256 73 / 73; 3x3 128 at 56 x 56, batch 64 90 / 91; but 3x3 256 at 28 x 28, batch 16
    // 30 / 34; 3x3 128 at 28 x 28, batch 64 27 / 29; 1x1 1024 -> 512 at 28 x 28, batch 64 70 / 72; 3x3 stride 2 512 at 28 x 28 69 / 76.
    if (f.add && P.pair) {
        long long slices = 0;
        for (int p = 0; p < n_phases; ++p) slices += P.c_blocks * P.phases[p].tap_count;
        const double mvalues = static_cast<double>(out_pixels) * N * 1e-6, terms = static_cast<double>(slices) * P.kb / n_phases;
        P.pair = mvalues * terms * (P.bn == 256 ? 5.3e-4 : 7.5e-4) > 2.0 + 0.92 * mvalues ? 1 : 0;
    }
    // Double tiles: pairs that write fp16 rows by TMA stores.  The phases of a gather are planned by their sum.
    if (P.pair && P.out_mode == OUT_NHWC_TMA && P.out_f16 && P.planes == 1 && (P.bn == 256 || P.bn == 128)) {
        int rows = 0, slices = 0;
        for (int p = 0; p < n_phases; ++p) {
            rows += ceil_div(ceil_div(P.phases[p].wq, 1 << P.wb_log2) * ceil_div(P.phases[p].hq, 1 << P.hb_log2) * ceil_div(f.batch, 1 << P.nb_log2), 2);
            slices += P.c_blocks * P.phases[p].tap_count;
        }
        P.big_rows = plan_double_rows(rows, P.n_tiles, slices / n_phases, P.bn, limited(ds->sms) / 2, n_phases == 1);
        P.dbl = P.big_rows > 0 ? 1 : 0;
        P.big_tiles = P.big_rows == INT_MAX ? INT_MAX : P.big_rows * P.n_tiles;
    }
    int tiles = 0;
    for (int p = 0; p < n_phases; ++p) {
        Phase& ph = P.phases[p];
        ph.tiles_w = ceil_div(ph.wq, 1 << P.wb_log2);
        ph.tiles_h = ceil_div(ph.hq, 1 << P.hb_log2);
        ph.tile_begin = tiles;
        int m_tiles = ph.tiles_w * ph.tiles_h * ceil_div(f.batch, 1 << P.nb_log2);
        if (P.pair) m_tiles = ceil_div(m_tiles, 2);
        if (P.dbl) m_tiles = P.big_rows == INT_MAX ? ceil_div(m_tiles, 2) : m_tiles - P.big_rows;
        tiles += m_tiles * P.n_tiles;
    }
    P.num_tiles = tiles;
    P.base_tiles = tiles;
    {   // division by multiplication in the kernels' tile decode: exact while tile index x divisor < 2^32
        auto reciprocal = [](int d) { return d > 1 ? static_cast<uint32_t>((1ull << 32) / static_cast<unsigned>(d) + 1) : 0u; };
        long long dmax = P.n_tiles;
        P.mul_nt = reciprocal(P.n_tiles);
        for (int p = 0; p < n_phases; ++p) {
            Phase& ph = P.phases[p];
            ph.mul_w = reciprocal(ph.tiles_w);
            ph.mul_h = reciprocal(ph.tiles_h);
            dmax = std::max<long long>(dmax, std::max(ph.tiles_w, ph.tiles_h));
        }
        // (a pair doubles the row-tile index before it is divided, a double tile once more)
        P.fastdiv = ((P.dbl ? 4ll : 2ll) * (tiles + 1) * dmax < (1ll << 32)) ? 1 : 0;
    }
    P.fsplit = 1;
    if (z_plan >= 2) {
        P.fsplit = z_plan;
        P.num_tiles = tiles * z_plan;
        // slice z stores into plane z of the scratch; the finishing pass adds the planes in order and
        // applies bias, rounding, cast and layout
        P.plane_elems = out_pixels * N;
        P.out = split_acc;
        P.out_mode = OUT_NHWC;
        P.out_f16 = 0;
        P.round_f16 = 0;
        P.bias = nullptr;
        P.ld_out = N;
    }

    // tensor maps
    for (int pl = 0; pl < mi.planes; ++pl) {
        uint64_t adims[4] = {static_cast<uint64_t>(Cp), static_cast<uint64_t>(f.a_w), static_cast<uint64_t>(f.a_h),
                             static_cast<uint64_t>(f.batch)};
        uint32_t abox[4] = {static_cast<uint32_t>(mi.kb), static_cast<uint32_t>((1 << P.wb_log2) * esw),
                            static_cast<uint32_t>((1 << P.hb_log2) * esh), static_cast<uint32_t>(1 << P.nb_log2)};
        uint32_t aes[4] = {1, static_cast<uint32_t>(esw), static_cast<uint32_t>(esh), 1};
        if (P.patch) {  // contiguous rows: the row stride is applied by the MMA descriptors
            abox[1] = static_cast<uint32_t>(P.patch_w);
            abox[2] = static_cast<uint32_t>(P.patch_h);
            abox[3] = 1;
            aes[1] = aes[2] = 1;
        }
        if (window) {
            // dims: (8 pixels x 8 or 4 channels, output column, padded row, image); consecutive
            // output columns start s_w pixels apart, so the windows overlap
            const uint64_t pix = 2ull * win_ch;
            uint64_t wd[4] = {8ull * win_ch, static_cast<uint64_t>(f.out_w), static_cast<uint64_t>(wimg.hp), static_cast<uint64_t>(f.batch)};
            uint64_t wstr[3] = {f.s_w * pix, wimg.wp * pix, static_cast<uint64_t>(wimg.hp) * wimg.wp * pix};
            abox[0] = static_cast<uint32_t>(8 * win_ch);
            rc = encode_map(&P.tmA[pl], a_planes[pl], 2, 4, wd, abox, aes, narrow ? SWZ_64B : SWZ_128B, wstr);
        } else {
            rc = encode_map(&P.tmA[pl], a_planes[pl], mi.es, 4, adims, abox, aes, SWZ_128B);
        }
        if (rc) return rc;
        uint32_t one[2] = {1, 1};
        if (f.w_batched) {  // as below, with the image as the outermost dimension
            const uint64_t images = static_cast<uint64_t>(f.batch), es = static_cast<uint64_t>(mi.es);
            const uint32_t kb = static_cast<uint32_t>(mi.kb), bn = static_cast<uint32_t>(P.bn);
            uint32_t one4[4] = {1, 1, 1, 1};
            if (!b_mn_major) {
                uint64_t d[3] = {static_cast<uint64_t>(direct_w ? K : kp), static_cast<uint64_t>(N), images};
                uint32_t box[3] = {kb, bn, 1};
                rc = encode_map(&P.tmB[pl], w_planes[pl], mi.es, 3, d, box, one4, SWZ_128B);
            } else if (N % mi.kb == 0) {
                P.b_grouped = 1;
                uint64_t d[4] = {kb, static_cast<uint64_t>(K), static_cast<uint64_t>(N / mi.kb), images};
                uint64_t str[3] = {N * es, kb * es, static_cast<uint64_t>(K) * N * es};
                uint32_t box[4] = {kb, kb, bn / kb, 1};
                rc = encode_map(&P.tmB[pl], w_planes[pl], mi.es, 4, d, box, one4, SWZ_128B, str);
            } else {
                uint64_t d[3] = {static_cast<uint64_t>(N), static_cast<uint64_t>(K), images};
                uint32_t box[3] = {kb, kb, 1};
                rc = encode_map(&P.tmB[pl], w_planes[pl], mi.es, 3, d, box, one4, SWZ_128B);
            }
        } else if (!b_mn_major) {
            uint64_t bdims[2] = {static_cast<uint64_t>(direct_w ? K : (window ? f.kh * 8 * win_ch : T * kp)), static_cast<uint64_t>(N)};
            uint32_t bbox[2] = {static_cast<uint32_t>(row_bytes / mi.es), static_cast<uint32_t>(P.pair ? P.bn / 2 : P.bn)};
            rc = encode_map(&P.tmB[pl], w_planes[pl], mi.es, 2, bdims, bbox, one, narrow ? SWZ_64B : SWZ_128B);
        } else if (N % mi.kb == 0) {
            // one box per stage: the outermost dimension walks the 128-byte column groups
            P.b_grouped = 1;
            uint64_t bdims[3] = {static_cast<uint64_t>(mi.kb), static_cast<uint64_t>(K), static_cast<uint64_t>(N / mi.kb)};
            uint64_t bstr[2] = {static_cast<uint64_t>(N) * mi.es, static_cast<uint64_t>(mi.kb) * mi.es};
            uint32_t bbox[3] = {static_cast<uint32_t>(mi.kb), static_cast<uint32_t>(mi.kb),
                                static_cast<uint32_t>((P.pair ? P.bn / 2 : P.bn) / mi.kb)};
            uint32_t one3[3] = {1, 1, 1};
            rc = encode_map(&P.tmB[pl], w_planes[pl], mi.es, 3, bdims, bbox, one3, SWZ_128B, bstr);
        } else {
            uint64_t bdims[2] = {static_cast<uint64_t>(N), static_cast<uint64_t>(K)};
            uint32_t bbox[2] = {static_cast<uint32_t>(mi.kb), static_cast<uint32_t>(mi.kb)};
            rc = encode_map(&P.tmB[pl], w_planes[pl], mi.es, 2, bdims, bbox, one, SWZ_128B);
        }
        if (rc) return rc;
    }
    if (g_dbg_short_a_box) {
        // nml_debug_stalled_linear_forward only: A boxes half as tall as the kernel expects, so no stage
        // ever receives all its bytes and the bounded waits run out
        uint64_t adims[4] = {static_cast<uint64_t>(Cp), static_cast<uint64_t>(f.a_w), static_cast<uint64_t>(f.a_h),
                             static_cast<uint64_t>(f.batch)};
        uint32_t abox[4] = {static_cast<uint32_t>(mi.kb), static_cast<uint32_t>((1 << P.wb_log2) / 2), 1, 1};
        uint32_t aes[4] = {1, 1, 1, 1};
        rc = encode_map(&P.tmA[0], a_planes[0], mi.es, 4, adims, abox, aes, SWZ_128B);
        if (rc) return rc;
    }
    if (bias_is_f16) {
        if (NML_IS_TMA_OUT(P.out_mode) && P.fsplit <= 1 && P.bias != nullptr) {
            P.bias = static_cast<const float*>(f.bias);  // read as __half by the kernel
            P.bias_f16 = 1;
        } else {
            helper_launch(4 * kSms, to_float_kernel<__half>, ceil_div(N, 256), 256, 0, st, static_cast<const __half*>(f.bias), bias_widened, N);
            ++g_launches;
        }
    }
    if (f.add && P.out_mode == OUT_NHWC_TMA && !P.pair) {
        P.add = 1;
        P.add_mask = static_cast<const uint8_t*>(f.add_mask);
        P.add_below = f.add_below;
    }
    int slot = -1;
    rc = launch_kernel(P, ds, st, &slot);
    if (rc) return rc;
    if (P.fsplit > 1) {
        const size_t total = out_pixels * N;
        const int nchw = (f.out_layout == NML_NCHW && !(f.out_h == 1 && f.out_w == 1)) ? 1 : 0;
        const int vec = (!nchw && N % 4 == 0 && (reinterpret_cast<uintptr_t>(f.out) & 15) == 0) ? 1 : 0;
        const size_t items = vec ? total / 4 : total;
        // (from 64 x 2 x 2 pixels of 512 channels, 32768 items of 9 planes, a thread an item is as fast: 18.6 us, eight 19.5)
        const bool deep = P.fsplit >= kFinishLanes && items <= 16384 && tune().deep;
        // (values one by one: a thread each while the grid still overlaps its predecessor; 3x3 s2 72 -> 77 at 58 x 58, batch 9, 34.1 us, a grid above
        // that limit 38.3)
        const size_t quarter = (total + 1023) / 1024;
        const size_t wanted = deep ? (items + 31) / 32 : vec ? quarter : std::min<size_t>((total + 255) / 256, std::max<size_t>(4 * kSms, quarter));
        const int blocks = static_cast<int>(std::min<size_t>(wanted, 148 * 8));
        const auto finish = [&](auto* kernel, auto* out, int round_f16) {
            helper_launch(4 * kSms, kernel, blocks, deep ? dim3(32, kFinishLanes) : dim3(256), 0, st, split_acc, P.fsplit, bias32, out, out_pixels, N,
                          f.out_h * f.out_w, nchw, round_f16, vec);
        };
        if (f.out_dtype == NML_F16) finish(deep ? finish_rows_deep_kernel<__half> : finish_rows_kernel<__half>, static_cast<__half*>(f.out), 0);
        else finish(deep ? finish_rows_deep_kernel<float> : finish_rows_kernel<float>, static_cast<float*>(f.out), f.round_f16);
        if (deep) ++g_launches_of[NML_DEBUG_DEEP_FINISH];
        ++g_launches;
        NML_CUDA(cudaGetLastError());
    }
    if (f.add && !P.add) {  // a K-split walk, pairs, a result that TMA does not store
        const size_t vectors = out_pixels * N / 8;
        const int blocks = static_cast<int>(std::min<size_t>((vectors + 255) / 256, 148 * 16));
        helper_launch(4 * kSms, add_masked_kernel, blocks, 256, 0, st, static_cast<uint4*>(f.out), static_cast<const uint4*>(f.add),
                      static_cast<const uint8_t*>(f.add_mask), f.add_below, vectors);
        ++g_launches;
        NML_CUDA(cudaGetLastError());
    }
    if (open_slot) {
        *open_slot = slot;
        return NML_OK;
    }
    return profile_stop(slot, st);
}

// ------------------------------------------------------- wgrad-like problems --
struct WgradLike {
    const void* patch;  // tensor the (tap-shifted, strided) patches are cut from
    int patch_c, patch_h, patch_w;
    const void* plain;  // tensor indexed by the pixel itself
    int plain_c, plain_h, plain_w;
    int dtype, layout, batch;
    int kh, kw, s_h, s_w, p_h, p_w, d_h, d_w;
    float* dw;  // [plain_c][patch_c][kh*kw]
    float* colsum;
    int colsum_of_patch;
    int math;
    // A 1x1 layer's images that are walked as one row: their own batch, height and width (0: as walked).  The tensor core truncates as it
    // accumulates, so the error of a sum grows with its K blocks; fewer blocks, none of which hangs over an image, would be cut into fewer slices of
    // the same length, or none.  So the slices are planned for the images' blocks, and each gets fewer: relative error against
    // float64 of 126 -> 248 at 104 x 3, batch 2, 8.0e-7 in one slice of ten blocks, 1.2e-7 in the images' thirteen slices.
    int plan_batch, plan_h, plan_w;
};

// Microseconds of a K block (64 pixels) of a double 256-column pair tile, and of its prologue and drain (256 KB of fp32 per SM,
// all SMs at once).  Measured: 16384 x 2048 -> 8192, 256 blocks, four rounds of single tiles 468 us, two of double ones 422;
// transposed 4x4 512 -> 128 at 32 x 32, batch 64 110 -> 99; but 16384 x 512 -> 2048 cut into nine slices of 29 blocks 48 -> 52.
constexpr double kDoubleBlockUs = 0.57, kDoubleTileUs = 8.0;

static int run_wgrad_like(const WgradLike& g, Bump& ws, cudaStream_t st) {
    MathInfo mi;
    if (!math_info(g.math, &mi)) return NML_ERR_INVALID;
    const int T = g.kh * g.kw;
    if (T > kMaxTaps) return NML_ERR_UNSUPPORTED;
    if (g.batch <= 0 || g.patch_c <= 0 || g.plain_c <= 0 || g.patch_h <= 0 || g.patch_w <= 0 || g.plain_h <= 0 ||
        g.plain_w <= 0)
        return NML_ERR_INVALID;
    DeviceState* ds = nullptr;
    if (!ws.dry) {
        int rc = device_state(&ds);
        if (rc) return rc;
    }
    const int sms = ds ? limited(ds->sms) : planning_sms();
    const void* pa[2] = {nullptr, nullptr};
    const void* pb[2];
    int cpa = 0, cpb = 0;
    // Few-channel layer input (RGB stems): patches come as 8-pixel windows of the padded image,
    // one kernel row per tap, (kw, c) packed in the 64 patch columns.
    const bool window = T > 1 && window_eligible(g.patch_c, g.kw, g.d_w, mi.enc);
    // (narrow: with four channels per pixel, where the patch walk below will be taken: the same conditions)
    bool narrow = window && narrow_eligible(g.patch_c, g.s_w) && tune().wpatch && round_up(g.plain_c, 8) % 64 == 0 && g.kh >= 2 && g.kh <= 32;
    if (narrow) {
        const int ph = 7 * g.s_h + (g.kh - 1) * g.d_h + 1;
        const double eff = static_cast<double>(g.plain_w) * g.plain_h / (1.0 * round_up(g.plain_w, 8) * round_up(g.plain_h, 8));
        // (a row tile always reads four kernel rows: the ones past the last have to stay within the stage's other box)
        const int past = static_cast<int>(round_up(g.kh, 4) - g.kh) * g.d_h * 8 * 64;
        narrow = ph <= 256 && 8 * ph * 64 <= 40 * 1024 && eff >= 0.7 && past <= 64 * 128;
    }
    const int win_ch = narrow ? 4 : 8, row_bytes = narrow ? 64 : 128;
    WindowImage wimg = {nullptr, 0, 0};
    int rc;
    // (the two conversions do not depend on one another; column sums taken with the first would stand between them)
    SideBySide operands;
    if (g.colsum && g.colsum_of_patch) t_role = PDL_NORMAL;
    RowsColsum later;
    // Column sums of a tensor used in place run beside the contraction and its reduction (on the SMs these leave, or as
    // their CTAs finish) -- not while launches are being timed, which would count them in.
    RowsColsum* const defer = g_prof.on.load(std::memory_order_relaxed) ? nullptr : &later;
    if (window) {
        rc = prepare_window(g.patch, g.dtype, g.layout, g.batch, g.patch_c, g.patch_h, g.patch_w, g.p_h, g.p_w, g.s_w,
                            g.plain_w, win_ch, ws, st, &wimg, g.colsum_of_patch ? g.colsum : nullptr);
        pa[0] = wimg.ptr;
        cpa = 8;
    } else {
        rc = prepare_activation(g.patch, g.dtype, g.layout, g.batch, g.patch_c, g.patch_h, g.patch_w, mi, ws, st, pa,
                                &cpa, g.colsum_of_patch ? g.colsum : nullptr, defer);
    }
    if (rc) return rc;
    if (!(g.colsum && g.colsum_of_patch)) operands.second();
    rc = prepare_activation(g.plain, g.dtype, g.layout, g.batch, g.plain_c, g.plain_h, g.plain_w, mi, ws, st, pb, &cpb,
                            g.colsum_of_patch ? nullptr : g.colsum, defer);
    if (rc) return rc;
    t_role = PDL_NORMAL;

    KParams P;
    memset(&P, 0, sizeof(P));
    P.mode = MODE_WGRAD;
    P.kind = mi.kind;
    P.planes = mi.planes;
    P.a_row_bytes = row_bytes;
    P.b_row_bytes = 128;
    P.a_cols_log2 = narrow ? 5 : 6;
    P.ch_log2 = narrow ? 2 : 3;
    P.kb = mi.kb;
    P.a_mn_major = 1;
    P.b_mn_major = 1;
    P.batch = g.batch;
    P.c_blocks = window ? 1 : ceil_div(g.patch_c, mi.kb);
    P.groups_total = (window ? g.kh : T) * P.c_blocks;
    P.c_patch = g.patch_c;
    P.c_plain = g.plain_c;
    P.n_taps = window ? g.kh : T;
    P.kw_pack = window ? 1 : 0;
    P.kw_count = g.kw;
    P.n_tiles = ceil_div(g.plain_c, 256);
    P.bn = static_cast<int>(round_up(ceil_div(g.plain_c, P.n_tiles), 64));
    P.c_out = g.plain_c;
    P.a_stride_h = g.s_h;
    P.a_stride_w = window ? 1 : g.s_w;
    P.out_stride_h = P.out_stride_w = 1;
    if (window) {
        for (int kh = 0; kh < g.kh; ++kh) {
            Tap& t = P.taps[kh];
            t.dh = static_cast<short>(kh * g.d_h);
            t.dw = 0;
            t.wk = kh;
        }
    } else
    for (int kh = 0; kh < g.kh; ++kh)
        for (int kw = 0; kw < g.kw; ++kw) {
            Tap& t = P.taps[kh * g.kw + kw];
            t.dh = static_cast<short>(kh * g.d_h - g.p_h);
            t.dw = static_cast<short>(kw * g.d_w - g.p_w);
            t.wk = kh * g.kw + kw;
        }
    const int bits = (mi.kb == 64) ? 6 : 5;
    choose_box(bits, g.plain_w, g.plain_h, g.batch, window ? 1 : g.s_w, g.s_h, &P.wb_log2, &P.hb_log2, &P.nb_log2);
    // Patch walk: one 64-channel group per tap, unit column stride, few enough row tiles for TMEM, 8 x 8 pixel
    // K blocks that do not waste much of the image, the other tensor fetched as grouped boxes.
    {
        const int groups = P.groups_total;
        const int mt = ceil_div(groups, narrow ? 4 : 2);
        int dw_min = 0, dw_max = 0, dh_min = 0, dh_max = 0;
        for (int t = 0; t < P.n_taps; ++t) {
            dw_min = t ? std::min<int>(dw_min, P.taps[t].dw) : P.taps[t].dw;
            dw_max = t ? std::max<int>(dw_max, P.taps[t].dw) : P.taps[t].dw;
            dh_min = t ? std::min<int>(dh_min, P.taps[t].dh) : P.taps[t].dh;
            dh_max = t ? std::max<int>(dh_max, P.taps[t].dh) : P.taps[t].dh;
        }
        const int pw_ = 8 + dw_max - dw_min, ph_ = 7 * g.s_h + dh_max - dh_min + 1;
        const int bn_w = std::min(256, (512 / std::max(mt, 1)) / 64 * 64);
        const double eff = static_cast<double>(g.plain_w) * g.plain_h / (1.0 * round_up(g.plain_w, 8) * round_up(g.plain_h, 8));
        if (tune().wpatch && mi.enc == ENC_F16 && P.c_blocks == 1 && groups >= 2 && mt <= 8 &&
            (window || g.s_w == 1) && bn_w >= 64 && cpb % 64 == 0 && pw_ <= 256 && ph_ <= 256 &&
            pw_ * ph_ * row_bytes <= 40 * 1024 && eff >= 0.7) {
            P.wpatch = 1;
            P.w_mtiles = mt;
            P.bn = std::min(bn_w, static_cast<int>(round_up(g.plain_c, 64)));
            P.n_tiles = ceil_div(g.plain_c, P.bn);
            P.patch_w = pw_;
            P.patch_h = ph_;
            P.patch_bytes = static_cast<int>(round_up(pw_ * ph_ * row_bytes, 1024));
            P.phases[0].org_w = static_cast<short>(dw_min);
            P.phases[0].org_h = static_cast<short>(dh_min);
            for (int t = 0; t < P.n_taps; ++t)
                P.taps[t].aoff = ((P.taps[t].dh - dh_min) * pw_ + (P.taps[t].dw - dw_min)) * row_bytes / 16;
            P.wb_log2 = 3;
            P.hb_log2 = 3;
            P.nb_log2 = 0;
        }
    }
    P.ktiles_w = ceil_div(g.plain_w, 1 << P.wb_log2);
    P.ktiles_h = ceil_div(g.plain_h, 1 << P.hb_log2);
    P.kblocks_total = P.ktiles_w * P.ktiles_h * ceil_div(g.batch, 1 << P.nb_log2);
    int plan_blocks = P.kblocks_total;
    if (g.plan_w) {
        int wl, hl, nl;
        choose_box(bits, g.plan_w, g.plan_h, g.plan_batch, 1, 1, &wl, &hl, &nl);
        plan_blocks = std::max(plan_blocks, ceil_div(g.plan_w, 1 << wl) * ceil_div(g.plan_h, 1 << hl) * ceil_div(g.plan_batch, 1 << nl));
    }
    // Tile width and K split so that the CTAs finish together.  Microseconds, measured over widths 64 / 128 / 256 and 1 ... 32
    // slices on 18 layers: a K block costs the same at 64 and 128 columns (0.32; operand feed, not MMAs), little more as a
    // 256-column CTA pair (0.36, 0.41 with the whole GPU busy); twice that for the 3xTF32 split's blocks of half the
    // pixels.  A tile adds its prologue and drain, more than one slice (and any multi-tap gradient) the second-stage
    // reduction, which writes and re-reads one plane of dW per slice and then writes dW, from L2 while the planes fit.
    const int G_ = kTileM / mi.kb;
    const bool a_grp = !window && (cpa % mi.kb == 0) && (P.c_blocks % G_ == 0);
    const bool b_grp = (cpb % mi.kb == 0);
    const int row_tiles = ceil_div(P.groups_total * mi.kb, kTileM);
    int split = 1, m_tiles = 1;
    long long launch_tiles = 0;
    if (!P.wpatch) {
        const double dw_us = 4.0 * g.plain_c * g.patch_c * T / 8e6;  // one pass over dW at 8 TB/s
        // at most 192 slices, as many as leave each at least one block (a count that the loop below does not pass over, so
        // that there is a plan whatever else is refused)
        const int max_split = ceil_div(plan_blocks, ceil_div(plan_blocks, std::min(plan_blocks, 192)));
        const bool may_pair = tune().pair;  // (read once: the loop runs up to 500 times per plan)
        double best = -1;
        for (int width = 256; width >= 64; width /= 2) {
            const int nt = ceil_div(g.plain_c, width);
            const int bn = static_cast<int>(round_up(ceil_div(g.plain_c, nt), 64));
            const bool pair = may_pair && bn == 256 && a_grp && b_grp && sms >= 2;
            if ((width < 256 && bn > width) || (bn > 128 && P.planes == 2 && !pair)) continue;
            const int mt = pair ? ceil_div(row_tiles, 2) : row_tiles;
            const int units = pair ? sms / 2 : sms;
            for (int sp = 1; sp <= max_split; ++sp) {
                const long long tiles = 1ll * mt * nt * sp;
                if (best >= 0 && sp > 1 && tiles > 3ll * units) break;
                const int per_sp = ceil_div(plan_blocks, sp);
                // every slice gets at least one K block: the next split that leaves each one block less
                if (ceil_div(plan_blocks, per_sp) != sp) continue;
                // the tensor core truncates as it accumulates: at most 4096 terms per sum of the 3xTF32 split, or as few
                // as the most slices leave
                if (P.planes == 2 && per_sp * mi.kb > 4096 && sp < max_split) continue;
                const double block_us = (pair ? (tiles * 8 >= units * 7ll ? 0.41 : 0.36) : 0.32) * (P.planes == 2 ? 2.3 : 1.0);
                const double tile_us = per_sp * block_us + 1.0 + bn / 128.0;
                const double reduce_us = sp > 1 || T > 1 ? 2.5 + (2.0 * sp + 1.0) * dw_us * (sp * dw_us > 8.0 ? 1.6 : 1.0) : 0.0;
                const auto rounds = [&](long long n) { return static_cast<double>((n + units - 1) / units); };
                const auto consider = [&](double us, int big_rows, long long n, int rows) {
                    if (best >= 0 && us >= best * (width == 256 ? 1.0 : 0.98)) return;
                    best = us;
                    split = sp;
                    m_tiles = rows;
                    launch_tiles = n;
                    P.n_tiles = nt;
                    P.bn = bn;
                    P.pair = pair ? 1 : 0;
                    P.big_rows = big_rows;
                };
                consider(rounds(tiles) * tile_us + reduce_us, 0, tiles, mt);
                // double tiles, with single ones behind them where K is whole (for 3 % and more)
                if (pair && P.planes == 1) {
                    const double double_us = per_sp * kDoubleBlockUs + kDoubleTileUs;
                    const int rows2 = ceil_div(mt, 2);
                    const long long doubles = 1ll * rows2 * nt * sp;
                    consider((rounds(doubles) * double_us + reduce_us) * 1.03, INT_MAX, doubles, 2 * rows2);
                    const int big_rows = static_cast<int>(doubles / units * units / nt);
                    if (sp == 1 && big_rows > 0 && mt > 2 * big_rows) {
                        const long long big = 1ll * big_rows * nt, total = big + 1ll * (mt - 2 * big_rows) * nt;
                        double us = 0;
                        for (const long long j : {0ll, big % units}) {  // the first pair, and the first with one double tile less
                            const double b = rounds(big - j), t = rounds(total - j);
                            us = std::max(us, b * double_us + (t - b) * tile_us);
                        }
                        consider((us + reduce_us) * 1.03, big_rows, total, mt);
                    }
                }
            }
        }
    }
    P.dbl = P.big_rows > 0 ? 1 : 0;
    P.big_tiles = P.big_rows == INT_MAX ? INT_MAX : P.big_rows * P.n_tiles;
    if (P.wpatch) {  // one tile per CTA, no empty slice
        split = std::max(1, std::min(P.kblocks_total, sms / std::max(1, P.n_tiles)));
        split = ceil_div(P.kblocks_total, ceil_div(P.kblocks_total, split));
    }
    if (plan_blocks > P.kblocks_total) {  // as many slices of the blocks that there are, at least one block to each
        const int slices = ceil_div(P.kblocks_total, ceil_div(P.kblocks_total, split));
        launch_tiles = launch_tiles / split * slices;
        split = slices;
    }
    P.split_k = split;
    P.num_tiles = P.wpatch ? P.n_tiles * split : static_cast<int>(launch_tiles);
    // One K slice of a one-tap layer writes dW itself.  With several taps the rows of a tile are 4 * taps bytes apart in dW
    // (a store instruction would touch 32 sectors: 4x4 512->512 on 4x4 images took 29 us for its 17 MB of gradient), so
    // they go through a plane even when there is one slice.  Several slices store their partial sums into one fp32 plane each
    // (like dW for the patch walk, else [plain channel][rows of the tile walk]); wgrad_reduce_* then adds
    // the planes in slice order and writes dW once -- no zero-fill, no atomics, bitwise repeatable.
    const size_t dw_elems = static_cast<size_t>(g.plain_c) * g.patch_c * T;
    const int plane_rows = P.wpatch ? 0 : m_tiles * (P.pair ? 2 : 1) * kTileM;
    const bool staged = split > 1 || (!P.wpatch && !P.kw_pack && T > 1);
    const size_t plane_elems = !staged ? 0 : P.wpatch ? round_up(dw_elems, 4) : static_cast<size_t>(g.plain_c) * plane_rows;
    float* planes = staged ? static_cast<float*>(ws.take(static_cast<size_t>(split) * plane_elems * sizeof(float))) : nullptr;
    if (ws.dry) return NML_OK;
    if (!ws.fits()) return NML_ERR_WORKSPACE;
    P.out = staged ? planes : g.dw;
    P.plane_elems = plane_elems;
    P.ld_plane = staged ? plane_rows : 0;
    // A wave of CTAs re-reads one operand in full; make that the smaller tensor.
    {
        const double patch_bytes = static_cast<double>(g.batch) * g.patch_h * g.patch_w * cpa * mi.es;
        const double plain_bytes = static_cast<double>(g.batch) * g.plain_h * g.plain_w * cpb * mi.es;
        P.m_fastest = (patch_bytes < plain_bytes) ? 1 : 0;
    }

    // MN-major tf32 operands need the 32-byte-chunk swizzle, fp16 ones the plain 128-byte swizzle
    const int mn_swz = (mi.es == 4) ? SWZ_128B_ATOM32 : SWZ_128B;
    for (int pl = 0; pl < mi.planes; ++pl) {
        uint64_t adims[4] = {static_cast<uint64_t>(cpa), static_cast<uint64_t>(g.patch_w),
                             static_cast<uint64_t>(g.patch_h), static_cast<uint64_t>(g.batch)};
        uint32_t abox[4] = {static_cast<uint32_t>(mi.kb), static_cast<uint32_t>((1 << P.wb_log2) * g.s_w),
                            static_cast<uint32_t>((1 << P.hb_log2) * g.s_h), static_cast<uint32_t>(1 << P.nb_log2)};
        uint32_t aes[4] = {1, static_cast<uint32_t>(g.s_w), static_cast<uint32_t>(g.s_h), 1};
        const int G = kTileM / mi.kb;
        if (P.wpatch) {  // contiguous patch rows; the row stride of the walk lives in the MMA descriptors
            abox[1] = static_cast<uint32_t>(P.patch_w);
            abox[2] = static_cast<uint32_t>(P.patch_h);
            abox[3] = 1;
            aes[1] = aes[2] = 1;
        }
        if (window) {
            const uint64_t pix = 2ull * win_ch;
            uint64_t wd[4] = {8ull * win_ch, static_cast<uint64_t>(g.plain_w), static_cast<uint64_t>(wimg.hp), static_cast<uint64_t>(g.batch)};
            uint64_t wstr[3] = {g.s_w * pix, wimg.wp * pix, static_cast<uint64_t>(wimg.hp) * wimg.wp * pix};
            uint32_t wbox[4] = {static_cast<uint32_t>(8 * win_ch), static_cast<uint32_t>(1 << P.wb_log2), static_cast<uint32_t>((1 << P.hb_log2) * g.s_h),
                                static_cast<uint32_t>(1 << P.nb_log2)};
            uint32_t wes[4] = {1, 1, static_cast<uint32_t>(g.s_h), 1};
            if (P.wpatch) {
                wbox[1] = abox[1];
                wbox[2] = abox[2];
                wbox[3] = 1;
                wes[2] = 1;
            }
            rc = encode_map(&P.tmA[pl], pa[pl], 2, 4, wd, wbox, wes, narrow ? SWZ_64B : mn_swz, wstr);
        } else if (P.wpatch) {
            rc = encode_map(&P.tmA[pl], pa[pl], mi.es, 4, adims, abox, aes, mn_swz);
        } else if (cpa % mi.kb == 0 && P.c_blocks % G == 0) {
            P.a_grouped = 1;
            uint64_t d5[5] = {static_cast<uint64_t>(mi.kb), adims[1], adims[2], adims[3], static_cast<uint64_t>(cpa / mi.kb)};
            uint64_t s5[4] = {static_cast<uint64_t>(cpa) * mi.es, adims[1] * cpa * mi.es, adims[1] * adims[2] * cpa * mi.es,
                              static_cast<uint64_t>(mi.kb) * mi.es};
            uint32_t b5[5] = {abox[0], abox[1], abox[2], abox[3], static_cast<uint32_t>(G)};
            uint32_t e5[5] = {1, aes[1], aes[2], 1, 1};
            rc = encode_map(&P.tmA[pl], pa[pl], mi.es, 5, d5, b5, e5, mn_swz, s5);
        } else {
            rc = encode_map(&P.tmA[pl], pa[pl], mi.es, 4, adims, abox, aes, mn_swz);
        }
        if (rc) return rc;
        uint64_t bdims[4] = {static_cast<uint64_t>(cpb), static_cast<uint64_t>(g.plain_w),
                             static_cast<uint64_t>(g.plain_h), static_cast<uint64_t>(g.batch)};
        uint32_t bbox[4] = {static_cast<uint32_t>(mi.kb), static_cast<uint32_t>(1 << P.wb_log2),
                            static_cast<uint32_t>(1 << P.hb_log2), static_cast<uint32_t>(1 << P.nb_log2)};
        uint32_t bes[4] = {1, 1, 1, 1};
        if (cpb % mi.kb == 0) {
            P.b_grouped = 1;
            uint64_t d5[5] = {static_cast<uint64_t>(mi.kb), bdims[1], bdims[2], bdims[3], static_cast<uint64_t>(cpb / mi.kb)};
            uint64_t s5[4] = {static_cast<uint64_t>(cpb) * mi.es, bdims[1] * cpb * mi.es, bdims[1] * bdims[2] * cpb * mi.es,
                              static_cast<uint64_t>(mi.kb) * mi.es};
            uint32_t b5[5] = {bbox[0], bbox[1], bbox[2], bbox[3], static_cast<uint32_t>((P.pair ? P.bn / 2 : P.bn) / mi.kb)};
            uint32_t e5[5] = {1, 1, 1, 1, 1};
            rc = encode_map(&P.tmB[pl], pb[pl], mi.es, 5, d5, b5, e5, mn_swz, s5);
        } else {
            rc = encode_map(&P.tmB[pl], pb[pl], mi.es, 4, bdims, bbox, bes, mn_swz);
        }
        if (rc) return rc;
    }
    int slot = -1;
    P.pdl_role = later.out ? PDL_LEADER : PDL_NORMAL;
    rc = launch_kernel(P, ds, st, &slot);
    if (rc) return rc;
    if (later.out) {
        t_role = PDL_SIBLING;
        later.first_stage(st);
        if (staged && !later.one_launch()) t_role = PDL_LEADER;  // the planes' reduction, with the sums' second stage beside it
    }
    if (staged) {
        const bool vec_ok = (reinterpret_cast<uintptr_t>(g.dw) & 15) == 0;
        // planes whose rows are float4s of dW's, in order: of the patch walk (laid out like dW) and of one tap
        const bool rows4 = vec_ok && (P.wpatch ? dw_elems % 4 == 0 : !P.kw_pack && T == 1 && g.patch_c % 4 == 0);
        const size_t total4 = dw_elems / 4;
        const int row_len4 = P.wpatch ? static_cast<int>(total4) : g.patch_c / 4;
        const size_t group_bytes = kReducePlain * 64 * (P.n_taps | 1) * sizeof(float);
        // Many planes of a small gradient: several threads an element, or a few blocks walk the planes one load latency at a time.
        bool several = false;
        if (rows4 && split > 8 && (P.wpatch || total4 <= 16384)) {
            several = true;
            helper_launch(4 * kSms, wgrad_reduce_deep4_kernel, static_cast<unsigned>((total4 + 31) / 32), dim3(32, 8), 0, st, planes, g.dw, split, plane_elems, total4,
                          row_len4, static_cast<size_t>(plane_rows));
        } else if (rows4) {
            const int blocks = static_cast<int>(std::min<size_t>((total4 + 255) / 256, 148 * 16));
            helper_launch(4 * kSms, wgrad_reduce_rows4_kernel, blocks, 256, 0, st, planes, g.dw, split, plane_elems, total4 / row_len4, row_len4, plane_rows);
        } else if (!P.wpatch && !P.kw_pack && g.patch_c % 4 == 0 && g.plain_c <= 65535 && group_bytes <= 48 * 1024) {
            const dim3 blocks(ceil_div(g.patch_c, 64), ceil_div(g.plain_c, kReducePlain));
            const bool deep = split >= 4 * kReduceGroups && blocks.x * blocks.y <= kSms && kReduceGroups * group_bytes <= 48 * 1024;
            several = deep;
            helper_launch(4 * kSms, deep ? wgrad_reduce_taps_kernel<kReduceGroups> : wgrad_reduce_taps_kernel<1>, blocks, dim3(256, deep ? kReduceGroups : 1),
                         (deep ? kReduceGroups : 1) * group_bytes, st, planes, g.dw, split, plane_elems, g.patch_c, g.plain_c, P.n_taps, P.c_blocks, mi.kb, plane_rows);
        } else {
            const int layout = P.wpatch ? 0 : P.kw_pack ? 2 : 1;
            // (one tap: the planes are read in dW's order, so that a thread an element is as fast from the size on where a grid of four no longer starts
            // beside its predecessor: 307 x 177 20.5 us so, 18.1 with a thread each, 238 x 200 28.1 and 24.9; 83 x 30 x 25 21.8 and 28.1)
            const bool deep = split >= 16 && dw_elems <= (T > 1 ? 65536 : 256 / kReduceLanes * 4 * kSms);
            several = deep;
            const int elems = deep ? 256 / kReduceLanes : 256;
            const int blocks = static_cast<int>(std::min<size_t>((dw_elems + elems - 1) / elems, 148 * 16));
            helper_launch(4 * kSms, deep ? wgrad_reduce_lanes_kernel : wgrad_reduce_kernel, blocks, dim3(elems, deep ? kReduceLanes : 1), 0, st, planes, g.dw, split, plane_elems,
                          dw_elems, layout, g.patch_c, P.n_taps, P.kw_count, P.c_blocks, mi.kb, plane_rows);
        }
        ++g_launches;
        if (several) ++g_launches_of[NML_DEBUG_DEEP_SUMS];
        NML_CUDA(cudaGetLastError());
    }
    if (later.out) {
        t_role = staged && !later.one_launch() ? PDL_SIBLING : PDL_NORMAL;
        rc = later.second_stage(st);
        t_role = PDL_NORMAL;
        if (rc) return rc;
    }
    return profile_stop(slot, st);
}

// ------------------------------------------------------------ strided products --
// out[m + n * out_ns] (+ entry * out_batch) = sum over k of a(m, k) * b(n, k) [+ bias[m]]: see nml_gemm.cuh.
struct StridedProduct {
    int M, N, K, batch;
    int dtype;  // of both operands; fp32 runs as 3xTF32
    const void *a, *b;
    bool a_contiguous, b_contiguous;  // k is the inner dimension (else m or n is)
    long long a_stride, b_stride, out_ns, a_batch, b_batch, out_batch;
    void* out;
    int out_dtype;
    const void* bias;
    int bias_dtype, round_f16;
};

struct StridedPlan {
    int bn = 0, splits = 1;
    double us = 0, waves = 0, loop_us = 0;  // in all, waves of blocks, the K loops of all of them
};
// Tile width and blocks per tile by estimated time: 6.6 us for launch, set-up and drain, then a K slice by how full the SMs are
// (alone 0.5 us at 32 columns, 0.6 at 64; with two blocks to every SM 1.1 and 1.3; 30 % more for an operand whose rows are the
// inner dimension, which is four loads a chunk), and for every further wave of blocks its own set-up and drain.
static StridedPlan plan_strided(const StridedProduct& g, int sms) {
    const int slices = ceil_div(g.K, g.dtype == NML_F32 ? 32 : 64);
    StridedPlan best;
    for (int bn = 64; bn >= 32; bn /= 2) {
        const long long tiles = 1ll * ceil_div(g.M, kTileM) * ceil_div(g.N, bn) * g.batch;
        for (int z = 1; z <= kGemmMaxSplits && (z == 1 || slices >= 2 * z); z *= 2) {
            const double blocks = static_cast<double>(tiles) * z, waves = std::ceil(blocks / (2.0 * sms));
            const double slice_us = (bn == 32 ? 0.5 : 0.6) * (1.0 + 0.6 * std::min(2.0, blocks / sms)) * (g.a_contiguous ? 1.0 : 1.3) *
                                    (g.b_contiguous ? 1.0 : 1.3);
            const double loop_us = waves * ceil_div(slices, z) * slice_us, us = 6.6 + loop_us + (waves - 1.0) * 4.0;
            if (best.bn == 0 || us < best.us) best = {bn, z, us, waves, loop_us};
        }
    }
    return best;
}

static void fill_strided(GemmParams* P, const StridedProduct& g, const DeviceState* ds, int role) {
    memset(P, 0, sizeof(*P));
    P->a = g.a; P->b = g.b; P->bias = g.bias; P->out = g.out;
    P->a_stride = g.a_stride; P->b_stride = g.b_stride; P->out_ns = g.out_ns;
    P->a_batch = g.a_batch; P->b_batch = g.b_batch; P->out_batch = g.out_batch;
    P->M = g.M; P->N = g.N; P->K = g.K;
    P->tiles_m = ceil_div(g.M, kTileM);
    const int es = g.dtype == NML_F32 ? 4 : 2;
    const auto vec = [&](const void* p, long long stride, long long batch) {
        return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && stride * es % 16 == 0 && batch * es % 16 == 0 ? 1 : 0;
    };
    P->a_vec = vec(g.a, g.a_stride, g.a_batch);
    P->b_vec = vec(g.b, g.b_stride, g.b_batch);
    P->bias_f16 = g.bias_dtype == NML_F16;
    P->out_f16 = g.out_dtype == NML_F16;
    P->round_f16 = g.round_f16;
    P->role = role;
    P->err = ds->err;
    P->wait_limit_ns = g_dbg_wait_limit_ns;
}

// ds: the state of the entry point (Bump::ds), nullptr for the device's own.
static int run_strided(const StridedProduct& g, const StridedPlan& plan, DeviceState* ds, int role, cudaStream_t st) {
    const bool f32 = g.dtype == NML_F32;
    const int slice = f32 ? 32 : 64;
    int rc = ds ? NML_OK : device_state(&ds);
    if (rc) return rc;
    GemmParams P;
    fill_strided(&P, g, ds, role);
    P.bn = plan.bn;
    P.tiles_n = ceil_div(g.N, plan.bn);
    P.splits = plan.splits;
    P.per = ceil_div(ceil_div(g.K, slice), plan.splits);
    const int stage_bytes = (f32 ? 2 : 1) * (kStageABytes + plan.bn * 128);
    P.stages = f32 ? 2 : 4;  // (80 to 96 KB: two blocks to an SM)
    const long long blocks = 1ll * P.tiles_m * P.tiles_n * g.batch * plan.splits;
    if (blocks > INT_MAX) return NML_ERR_UNSUPPORTED;
    rc = profile_open(st);
    if (rc) return rc;
    const int slot = g_bracket_slot;
    g_bracket_slot = -1;
    // Two blocks to an SM, and none beside a block of the contraction kernel (120 KB and more): blocks of clusters that wait for
    // TMEM columns behind one another on two SMs would wait for good.
    const size_t smem = std::max<size_t>(static_cast<size_t>(P.stages) * stage_bytes + 1024 + 256, 110 * 1024);
    launch_with(true, plan.splits, f32 ? gemm_instance<float>(g.a_contiguous, g.b_contiguous) : gemm_instance<__half>(g.a_contiguous, g.b_contiguous),
                static_cast<unsigned>(blocks), kGemmThreads, smem, st, P);
    NML_CUDA(cudaGetLastError());
    ++g_launches;
    ++g_launches_of[NML_DEBUG_IN_PLACE];
    return profile_stop(slot, st);
}

// A batched fp16 product with K <= kRowsMaxK by gemm_rows_kernel: b's rows are contiguous along k, a's columns along m.
struct RowsPlan {
    int splits = 1, per = 0;
    double us = 0;
};
// Blocks that share a strip of 128 columns, by estimated time: two blocks to an SM, what starts and ends one, and its groups of 64 rows.
// (By the groups of the busiest SM, which asks for fewer and longer blocks: 25 x 464 x 32 x 170 7.3 -> 9.5 us, 108 x 443 x 32 x 51 9.4 -> 13.0.)
static RowsPlan plan_rows(const StridedProduct& g, int sms) {
    const int groups = ceil_div(g.N, kRowsBn), slices = ceil_div(g.K, 64);
    const double strips = static_cast<double>(g.batch) * ceil_div(g.M, kTileM);
    RowsPlan best;
    for (int z = 1; z <= groups; ++z) {
        const int per = ceil_div(groups, z);
        if (ceil_div(groups, per) != z) continue;
        const double blocks = strips * z, waves = std::ceil(blocks / (2.0 * sms));
        const double us = 2.5 + waves * (2.0 + 0.7 * slices) + waves * per * (blocks > sms ? 0.6 : 0.4);
        if (best.per == 0 || us < best.us) best = {z, per, us};
    }
    return best;
}
static int run_rows(const StridedProduct& g, cudaStream_t st) {
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    const RowsPlan plan = plan_rows(g, limited(ds->sms));
    GemmParams P;
    fill_strided(&P, g, ds, PDL_NORMAL);
    P.bn = kRowsBn;
    P.tiles_n = ceil_div(g.N, kRowsBn);
    P.splits = plan.splits;
    P.per = plan.per;
    const long long blocks = 1ll * P.tiles_m * g.batch * plan.splits;
    if (blocks > INT_MAX) return NML_ERR_UNSUPPORTED;
    rc = profile_open(st);
    if (rc) return rc;
    const int slot = g_bracket_slot;
    g_bracket_slot = -1;
    // (two blocks to an SM and none beside a block of the contraction kernel, as in run_strided)
    launch_with(true, 1, gemm_rows_kernel, static_cast<unsigned>(blocks), kGemmThreads, 110 * 1024, st, P);
    NML_CUDA(cudaGetLastError());
    ++g_launches;
    return profile_stop(slot, st);
}

// Estimated microseconds of n products [M][K] x [K][N], as images of one launch of the contraction kernel, by rows of the result or
// turned round (see nml_ref_matmul): what starts and ends it, the conversions of both operands (per million values written), the
// K loops and, per 32 columns, the drains of the rounds of tiles, and the result; no less than the host takes for the launches.
// Fitted to 1372 random fp32 products and 944 of fp16 with N not of whole vectors, of 7 to 500 us: a standard error of 9 to 22 %.
// The fastest of the two and of the in-place kernel by these estimates took 13.2 us in the (geometric) mean where the best takes 13.1,
// always by rows 20.5, always turned 20.8, always in place 14.3; fp16 11.7, 11.6, 17.5, 15.4 and 14.6.
static double batched_us(bool turned, double n, int M, int K, int N, int es, int sms) {
    struct Cost { double fixed, a, b, loop, drain, ragged_round, ragged, result; };
    static constexpr Cost kCost[2][2] = {{{8.3, 2.4, 2.6, 0.86, 0.27, 0.69, 0.91, 0.27}, {9.8, 2.35, 3.6, 0.77, 0.07, 0.0, 0.0, 0.69}},
                                         {{7.7, 1.2, 1.05, 1.33, 0.55, 2.0, 0.0, 0.27}, {9.1, 0.87, 1.55, 1.37, 0.165, 0.0, 0.0, 0.24}}};
    const bool f32 = es == 4;
    const Cost& c = kCost[f32 ? 0 : 1][turned ? 1 : 0];
    const int kb = f32 ? 32 : 64, vector = 16 / es, slices = ceil_div(K, kb) * (f32 ? 3 : 1);
    const double row_tiles = n * ceil_div(turned ? N : M, kTileM);
    const int columns = turned ? M : N;
    double best = 0, rounds = 0, bn = 0;
    for (int width = f32 ? 128 : 256; width >= 64; width /= 2) {  // (as run_fprop_like chooses)
        const int nt = ceil_div(columns, width);
        const double b = static_cast<double>(round_up(ceil_div(columns, nt), 32)), r = std::ceil(row_tiles * nt / sms);
        const double t = r * b * (b > 128 ? 1.0 : b > 64 ? 1.28 : 2.24);
        if (bn == 0 || t < best * 0.97) best = t, rounds = r, bn = b;
    }
    const double a_values = f32 || K % 8 ? n * M * round_up(K, turned ? kb : vector) * 1e-6 : 0.0;
    const double b_values = n * N * round_up(K, turned ? vector : kb) * 1e-6;
    const double drains = rounds * std::ceil(bn / 32);
    const double ragged = !turned && N > 8 && N % vector ? 1.0 : 0.0;
    const double us = c.fixed + c.a * a_values + c.b * b_values + c.loop * rounds * slices * slice_us(std::max(64, static_cast<int>(bn))) + c.drain * drains +
                      ragged * (c.ragged_round * rounds + c.ragged * drains) + c.result * n * M * N * 1e-6;
    return std::max(f32 || K % 8 ? 13.0 : 10.0, us);
}

// --------------------------------------------------------- layer -> problems --
static bool conv_out_size(const nml_conv_desc* d, int* ho, int* wo) {
    if (!d || d->stride_h <= 0 || d->stride_w <= 0 || d->dil_h <= 0 || d->dil_w <= 0 || d->kh <= 0 || d->kw <= 0 ||
        d->pad_h < 0 || d->pad_w < 0)
        return false;
    if (!d->transposed) {
        int nh = d->h + 2 * d->pad_h - d->dil_h * (d->kh - 1) - 1;
        int nw = d->w + 2 * d->pad_w - d->dil_w * (d->kw - 1) - 1;
        if (nh < 0 || nw < 0) return false;
        *ho = nh / d->stride_h + 1;
        *wo = nw / d->stride_w + 1;
    } else {
        *ho = (d->h - 1) * d->stride_h - 2 * d->pad_h + d->dil_h * (d->kh - 1) + 1 + d->outpad_h;
        *wo = (d->w - 1) * d->stride_w - 2 * d->pad_w + d->dil_w * (d->kw - 1) + 1 + d->outpad_w;
    }
    return *ho > 0 && *wo > 0;
}

struct Pointwise {  // a 1x1 convolution as a Linear layer: its weights may start anywhere, and its input gradient may have an addend (KParams::add)
    const void *add, *add_mask;
    float add_below;
    int batch, h, w;
};
static int linear_pass(const nml_linear_desc* d, int pass, const void* in0, const void* in1, const void* bias, void* out, float* db, Bump& ws,
                       cudaStream_t st, const Pointwise* conv = nullptr);

static int conv_pass(const nml_conv_desc* d, int pass, const void* in0, const void* in1, const void* bias, void* out,
                     float* db, Bump& ws, cudaStream_t st, const void* add = nullptr, const void* add_mask = nullptr, float add_below = 0.f) {
    int ho, wo;
    nml_conv_desc flattened;
    const nml_conv_desc* image = nullptr;  // of a layer that is walked as images of one row
    g_last_scratch_error[0] = 0;  // a workspace error reported from here on is not the static entry point's
    if (!conv_out_size(d, &ho, &wo)) return NML_ERR_INVALID;
    const bool tr = d->transposed != 0;
    // 1x1 layers of unit stride without padding have no geometry.  fp16 rows of pixels are a Linear layer's: its rules, weights read in place,
    // no tile hanging over an image.  Forward / input gradient, us: 448 -> 192 at 5 x 5,
    // batch 14, 9.3 -> 6.3 (forward); 1024 -> 256 at 9 x 9, batch 24, 10.0 / 9.5 -> 8.4 / 6.6; 512 -> 2048 at 7 x 7, batch 64, 16.8 / 16.6 -> 12.4 / 13.9;
    // 256 -> 64 at 56 x 56, batch 256, 80.7 / 96.4 -> 79.0 / 95.0.
    const bool pointwise = d->kh == 1 && d->kw == 1 && d->stride_h == 1 && d->stride_w == 1 && d->pad_h == 0 && d->pad_w == 0 && !tr;
    const bool weights = pass == NML_PASS_BACKWARD_WEIGHT;
    const long long pixels = 1ll * d->batch * d->h * d->w;
    if (pointwise && d->batch > 0 && d->h > 0 && d->w > 0 && pixels <= INT_MAX / 2 && d->in_layout == NML_NHWC && (weights || d->out_layout == NML_NHWC) &&
        d->math == NML_MATH_F16 && d->in_dtype == NML_F16 && (weights || d->w_dtype == NML_F16)) {
        nml_linear_desc l;
        memset(&l, 0, sizeof(l));
        l.rows = static_cast<int>(pixels); l.in_features = d->c_in; l.out_features = d->c_out;
        l.in_dtype = d->in_dtype; l.out_dtype = d->out_dtype; l.w_dtype = d->w_dtype; l.math = d->math; l.round_out_f16 = d->round_out_f16;
        const Pointwise conv = {add, add_mask, add_below, d->batch, d->h, d->w};
        if (!ws.dry) ++g_launches_of[NML_DEBUG_POINTWISE];
        return linear_pass(&l, pass, in0, in1, bias, out, db, ws, st, &conv);
    }
    // Other tensors become images of one row, so that channel-major stores run on over the ends of the rows (small images find better
    // boxes in two dimensions: fp32 96 -> 384 at 14 x 14, batch 60, 20.0 us, flat 22.3).  Where the one row would be whole 16-byte vectors
    // and the image's are not, the result would go to the TMA epilogue, which takes longer than the direct one for small results (24 -> 90
    // at 22 x 174, batch 4, 10.5 us, flat 11.8; 272 -> 5 input gradient at 104 x 6, batch 3, 8.3 and 9.5; of 68 such layers below two million
    // values 25 lost more than 5 %, three gained as much).
    const auto flat_pays = [&] {
        const long long es = d->out_dtype == NML_F16 ? 2 : 4, image_pixels = 1ll * d->h * d->w;
        const bool turns_tma = d->out_layout == NML_NCHW && d->w * es % 16 != 0 && image_pixels * es % 16 == 0;
        return image_pixels >= 512 && !(turns_tma && pixels * (pass == NML_PASS_FORWARD ? d->c_out : d->c_in) < 2000000);
    };
    if (pointwise && d->batch > 0 && d->h > 0 && d->w > 0 && 1ll * d->h * d->w <= INT_MAX / 2 && (weights || flat_pays())) {
        flattened = *d;
        image = d;
        flattened.w *= d->h;
        flattened.h = 1;
        d = &flattened;
        wo *= ho;
        ho = 1;
    }
    if (weights) {
        // in0 = x, in1 = dy
        WgradLike g;
        memset(&g, 0, sizeof(g));
        if (!tr) {
            g.patch = in0; g.patch_c = d->c_in; g.patch_h = d->h; g.patch_w = d->w;
            g.plain = in1; g.plain_c = d->c_out; g.plain_h = ho; g.plain_w = wo;
            g.colsum_of_patch = 0;
        } else {
            g.patch = in1; g.patch_c = d->c_out; g.patch_h = ho; g.patch_w = wo;
            g.plain = in0; g.plain_c = d->c_in; g.plain_h = d->h; g.plain_w = d->w;
            g.colsum_of_patch = 1;
        }
        g.dtype = d->in_dtype; g.layout = d->in_layout; g.batch = d->batch;
        g.kh = d->kh; g.kw = d->kw; g.s_h = d->stride_h; g.s_w = d->stride_w;
        g.p_h = d->pad_h; g.p_w = d->pad_w; g.d_h = d->dil_h; g.d_w = d->dil_w;
        g.dw = static_cast<float*>(out);
        g.colsum = db;
        g.math = d->math;
        if (image) g.plan_batch = image->batch, g.plan_h = image->h, g.plan_w = image->w;
        return run_wgrad_like(g, ws, st);
    }
    FpropLike f;
    memset(&f, 0, sizeof(f));
    // conv forward and convT backward-data are strided reads; conv backward-data and convT forward gather.
    const bool forward = (pass == NML_PASS_FORWARD);
    const bool reads_layer_input = forward;  // A is the layer input for forward, the output gradient otherwise
    f.a = in0;
    f.a_dtype = d->in_dtype; f.a_layout = d->in_layout; f.batch = d->batch;
    if (reads_layer_input) { f.a_c = d->c_in; f.a_h = d->h; f.a_w = d->w; f.out_c = d->c_out; f.out_h = ho; f.out_w = wo; }
    else                   { f.a_c = d->c_out; f.a_h = ho; f.a_w = wo; f.out_c = d->c_in; f.out_h = d->h; f.out_w = d->w; }
    f.w = in1; f.w_dtype = d->w_dtype;
    // weight source dims: conv [c_out][c_in][T], convT [c_in][c_out][T]
    f.d0 = tr ? d->c_in : d->c_out;
    f.d1 = tr ? d->c_out : d->c_in;
    f.kh = d->kh; f.kw = d->kw;
    // contraction channel is a_c: it is dim0 exactly when a_c names d0
    f.k_is_dim0 = (forward == tr) ? 1 : 0;  // conv fwd: k=c_in=d1; conv bwd: k=c_out=d0; convT fwd: k=c_in=d0; convT bwd: k=c_out=d1
    f.w_direct = 0;
    f.gather = (forward == tr) ? 1 : 0;     // conv fwd 0, conv bwd 1, convT fwd 1, convT bwd 0
    f.s_h = d->stride_h; f.s_w = d->stride_w; f.p_h = d->pad_h; f.p_w = d->pad_w; f.d_h = d->dil_h; f.d_w = d->dil_w;
    f.out = out; f.out_dtype = d->out_dtype; f.out_layout = d->out_layout;
    f.bias = forward ? bias : nullptr; f.bias_dtype = d->w_dtype;
    f.math = d->math;
    f.round_f16 = forward ? d->round_out_f16 : 0;
    f.add = add; f.add_mask = add_mask; f.add_below = add_below;
    return run_fprop_like(f, ws, st);
}

// Whether TMA takes an fp16 matrix of `rows` rows of `inner` values, as the contraction kernel's own maps of it would find.
static int rows_for_tma(const void* p, int inner, int rows) {
    CUtensorMap tm;
    const uint64_t dims[2] = {static_cast<uint64_t>(inner), static_cast<uint64_t>(rows)};
    const uint32_t box[2] = {8, 1}, steps[2] = {1, 1};
    return encode_map(&tm, p, 2, 2, dims, box, steps, SWZ_NONE);
}

static int linear_pass(const nml_linear_desc* d, int pass, const void* in0, const void* in1, const void* bias,
                       void* out, float* db, Bump& ws, cudaStream_t st, const Pointwise* conv) {
    if (!d || d->rows <= 0 || d->in_features <= 0 || d->out_features <= 0) return NML_ERR_INVALID;
    g_last_scratch_error[0] = 0;
    const int operands = d->math == NML_MATH_3XTF32 ? NML_F32 : d->math == NML_MATH_F16 ? NML_F16 : -1;
    if (d->in_dtype == operands && (pass == NML_PASS_BACKWARD_WEIGHT || d->w_dtype == operands) &&
        g_sm_limit.load(std::memory_order_relaxed) == 0) {
        const int R = d->rows, I = d->in_features, O = d->out_features;
        StridedProduct g;
        memset(&g, 0, sizeof(g));
        g.dtype = operands;
        g.batch = 1;
        g.out = out;
        g.out_dtype = pass == NML_PASS_BACKWARD_WEIGHT ? NML_F32 : d->out_dtype;
        if (pass == NML_PASS_FORWARD) {          // y[r][o] = x[r][i] * w[o][i]
            g.M = O; g.N = R; g.K = I;
            g.a = in1; g.a_contiguous = true; g.a_stride = I;
            g.b = in0; g.b_contiguous = true; g.b_stride = I;
            g.out_ns = O;
            g.bias = bias; g.bias_dtype = d->w_dtype; g.round_f16 = d->round_out_f16;
        } else if (pass == NML_PASS_BACKWARD_DATA) {  // dx[r][i] = dy[r][o] * w[o][i]
            g.M = I; g.N = R; g.K = O;
            g.a = in1; g.a_contiguous = false; g.a_stride = I;
            g.b = in0; g.b_contiguous = true; g.b_stride = O;
            g.out_ns = I;
        } else {                                 // dw[o][i] = dy[r][o] * x[r][i]
            g.M = I; g.N = O; g.K = R;
            g.a = in0; g.a_contiguous = false; g.a_stride = I;
            g.b = in1; g.b_contiguous = false; g.b_stride = O;
            g.out_ns = I;
        }
        // The conversions and the contraction kernel take (forward / input gradient / weight gradient, us, with this path in
        // brackets) 64 x 512 -> 512 12.0 / 13.6 / 12.3 (7.6 / 8.1 / 8.5), 128 x 768 -> 256 12.5 / 13.6 / 12.3 (8.6 / 7.8 / 10.4), 300 x 1500 ->
        // 300 20.7 / 16.1 / 18.7 (15.7 / 12.6 / 17.0), 256 x 2048 -> 1000 22.4 / 24.3 / 18.9 (20.1 / 20.9 / 24.7), 2000 x 90 -> 400
        // 10.2 / 25.0 / 18.4 (9.6 / 12.9 / 21.9), 20 x 4000 -> 200 17.4 / 13.6 / 12.5 (18.3 / 9.3 / 7.8): the estimates up to which
        // this path was the faster.
        // (a weight gradient of fewer than eight tiles is the contraction kernel's: it cuts K into up to 192 shares)
        // fp16 operands that are read in place by TMA need no conversions in the first place, and an operand whose rows are the inner
        // dimension is eight 2-byte loads a chunk here: forward only, with one or two K slices (500 x 128 -> 512 5.8 -> 4.7 us, 2000 x
        // 90 -> 400 9.1 -> 7.8; four slices, 4000 x 256 -> 100, 8.4 and 8.5; 32 x 512 -> 2048, whose loop blocks would share, 6.8 and
        // 6.5 from L2 but 6.4 and 6.6 from HBM).  Rows that TMA is to read and cannot, because the matrix does not start on 16 bytes,
        // stay refused, by the map's own error (the plan's scratch, none, is no room for the contraction kernel to find out).
        StridedPlan plan;
        bool in_place;
        if (operands == NML_F32) {
            plan = plan_strided(g, planning_sms());
            const bool few = pass == NML_PASS_BACKWARD_WEIGHT && ceil_div(I, kTileM) * ceil_div(O, 32) < 8;
            // (of one to four tiles, which the contraction kernel cuts over all SMs and eight blocks each take long for: 1 x 3456 -> 6 forward
            // 12.4 us there and 15.6 here, input gradient of 2 x 3 -> 3877 12.5 and 19.8, of 85 x 1 -> 3328 12.8 and 17.9)
            const double tiles = static_cast<double>(ceil_div(g.M, kTileM)) * ceil_div(g.N, plan.bn);
            const double limit_us = pass == NML_PASS_BACKWARD_WEIGHT ? 13.0 : tiles <= 4 ? 12.5 : pass == NML_PASS_FORWARD ? 14.0 : 20.0;
            in_place = !few && plan.us <= limit_us;
        } else {
            // (a launch that is to stall is the contraction kernel's)
            in_place = pass == NML_PASS_FORWARD && I <= 128 && 1ll * ceil_div(O, kTileM) * ceil_div(R, 64) <= 2 * planning_sms() && !g_dbg_short_a_box;
            if (in_place && !ws.dry && I % 8 == 0 && ((reinterpret_cast<uintptr_t>(in0) | reinterpret_cast<uintptr_t>(in1)) & 15) != 0) {
                int rc = rows_for_tma(in0, I, R);
                if (!rc && !conv) rc = rows_for_tma(in1, I, O);
                if (rc) return rc;
            }
        }
        if (in_place) {
            RowsColsum sums;
            if (pass == NML_PASS_BACKWARD_WEIGHT && db) {
                sums.plan(in1, operands, R, O, db);
                sums.cs = colsum_scratch(ws, sums.grid.y, O);
            }
            if (ws.dry) return NML_OK;
            if (!ws.fits()) return NML_ERR_WORKSPACE;
            if (operands == NML_F16) plan = plan_strided(g, planning_sms());
            const bool beside = sums.out && !g_prof.on.load(std::memory_order_relaxed);
            if (sums.out && !beside) {
                sums.first_stage(st);
                const int rc = sums.second_stage(st);
                if (rc) return rc;
            }
            const int rc = run_strided(g, plan, ws.ds, beside ? PDL_LEADER : PDL_NORMAL, st);
            if (rc || !beside) return rc;
            t_role = PDL_SIBLING;
            sums.first_stage(st);
            return sums.second_stage(st);
        }
    }
    if (pass == NML_PASS_BACKWARD_WEIGHT) {
        WgradLike g;
        memset(&g, 0, sizeof(g));
        g.patch = in0; g.patch_c = d->in_features; g.patch_h = 1; g.patch_w = d->rows;
        g.plain = in1; g.plain_c = d->out_features; g.plain_h = 1; g.plain_w = d->rows;
        g.dtype = d->in_dtype; g.layout = NML_NHWC; g.batch = 1;
        g.kh = g.kw = 1; g.s_h = g.s_w = 1; g.d_h = g.d_w = 1;
        g.dw = static_cast<float*>(out);
        g.colsum = db; g.colsum_of_patch = 0;
        g.math = d->math;
        if (conv) g.plan_batch = conv->batch, g.plan_h = conv->h, g.plan_w = conv->w;
        return run_wgrad_like(g, ws, st);
    }
    FpropLike f;
    memset(&f, 0, sizeof(f));
    const bool forward = (pass == NML_PASS_FORWARD);
    f.a = in0; f.a_dtype = d->in_dtype; f.a_layout = NML_NHWC; f.batch = 1; f.a_h = 1; f.a_w = d->rows;
    f.a_c = forward ? d->in_features : d->out_features;
    f.w = in1; f.w_dtype = d->w_dtype; f.d0 = d->out_features; f.d1 = d->in_features; f.kh = f.kw = 1;
    f.k_is_dim0 = forward ? 0 : 1;
    // Short rows of weights take TMA long to read in place, which a 1x1 convolution's copy (rows of whole slices) pays for where many tiles read
    // them: 8 -> 96, 82650 rows, 18.0 us in place, copied 11.1; 104 -> 176, 105560 rows, 22.6 and 17.4; 8 -> 77, 27522 rows, 15.3 and 13.7; but
    // 24 -> 150, 57876 rows, 27.3 and 26.6, 64 -> 313, 86848 rows, 59.8 and 61.7.
    const long long row_tiles = 1ll * ceil_div(d->rows, kTileM) * ceil_div(d->out_features, 256);
    const bool short_k = d->in_features <= 128 && d->in_features % 64 != 0 && row_tiles >= (d->in_features == 8 && d->out_features >= 48 ? 1 : 4) * static_cast<long long>(kSms);
    f.w_direct = !conv ? 1 : forward && short_k ? 0 : 2;
    // Input gradient: W [out][in] read in place is an MN-major B operand.  Where its rows are no whole groups of 64 it takes a load per
    // group and excludes CTA pairs, and a transposed fp16 copy W^T [in][out] (one coalesced pass over the weights, counted in the
    // pass's duration) pays from 2.2e9 products on, with 128 outputs (two K slices) and more: 12000 x 520 -> 2048 55.6 -> 36.4 us, 8192 x 328
    // -> 1024 18.7 -> 16.0, 4096 x 520 -> 1024 18.6 -> 15.0, 16384 x 520 -> 320 18.6 -> 16.9; 4096 x 1000 -> 512 12.6 -> 13.5; 65536 x 1000 -> 64
    // 36.5 -> 42.2.  Less than one group is mostly fill: from 8192 rows on for up to 32 inputs, 16384 x 8 -> 512 15.9 -> 8.3, 81664 x 40 -> 320
    // 20.3 -> 16.0, 16384 x 40 -> 1024 13.0 -> 12.0, -> 512 10.1 -> 10.2.  Whole groups are read almost as fast as a K-major
    // operand: only very wide layers of many rows gain a little (16384 x 3072 -> 1024 93.5 -> 88.5, 8192 x 4096 -> 4096 213 -> 205;
    // but 16384 x 3072 -> 512 52.1 -> 54.3, 16384 x 512 -> 2048 33.3 -> 37.2, 16384 x 2048 -> 8192 360 -> 371).
    const long long out_rows = 1ll * d->rows * d->out_features;
    const bool pays = d->in_features % 64 == 0 ? d->in_features >= 3072 && d->rows >= 8192 && d->out_features >= 1024
                      : d->out_features < 128 ? false
                      : d->in_features <= 32 ? d->rows >= 8192
                      : d->in_features < 64 ? out_rows >= 16000000ll
                                            : out_rows * d->in_features >= 2200000000ll;
    // Weights that do not start on 16 bytes are no operand for TMA, but the copy's kernel takes them: from 8192 rows on, with whole groups
    // of outputs, such a layer has its copy (and a workspace query, which sees no pointer, counts it); elsewhere it is refused.
    const bool any_start = d->rows >= 8192 && d->out_features % 64 == 0;
    const bool starts = (reinterpret_cast<uintptr_t>(in1) & 15) == 0;
    // 1x1 convolutions have scratch for the copy anyway, and take it also where a last group of inputs that is far from whole meets many rows of tiles,
    // by K slices (104 <- 24 at 62 x 29, batch 66, in place 19.4 us, copied 13.1; 72 <- 688, 42408 rows, 24.5 and 17.6; 8 <- 72, 44556 rows, 13.0
    // and 8.5; but 56 <- 576, 12980 rows, 9.3 and 10.9, 456 <- 16, 16968 rows, 10.1 and 10.6), or a long K loop (208 <- 1920, 4 rows, 14.2 and 12.2),
    // or where the output gradient is converted anyway, beside the copy (392 <- 4, 46560 rows, 22.7 and 17.1; 512 <- 2, 113344 rows, 37.0 and 29.1).
    const int last = d->in_features % 64;
    const bool short_last = last != 0 && last <= (d->in_features < 64 ? 40 : d->in_features < 256 ? 56 : 48);
    const bool copied = conv && !forward && d->math == NML_MATH_F16 &&
                        ((last != 0 && d->rows >= 120000) || (short_last && d->in_features < 256 && 1ll * d->rows * ceil_div(d->out_features, 64) >= 60000) ||
                         (short_last && last <= 40 && d->in_features < 1000 && d->out_features >= 1300) ||
                         (d->out_features < 64 && d->out_features % 8 != 0 && 1ll * ceil_div(d->rows, kTileM) * ceil_div(d->in_features, 256) >= 2 * kSms));
    if (conv && !forward && (pays || copied || conv->add)) {
        f.w_direct = 0;  // (repacked: that is the same copy)
        f.add = conv->add; f.add_mask = conv->add_mask; f.add_below = conv->add_below;
    } else
    if (!forward && !conv && d->math == NML_MATH_F16 && d->w_dtype == NML_F16 && d->in_features % 8 == 0 && d->out_features % 8 == 0 &&
        (ws.dry ? pays || any_start : starts ? pays : any_start) && tune().wtrans) {
        __half* wt = static_cast<__half*>(ws.take(static_cast<size_t>(d->in_features) * d->out_features * sizeof(__half)));
        if (!ws.dry) {
            if (!ws.fits()) return NML_ERR_WORKSPACE;
            int rc = profile_open(st);
            if (rc) return rc;
            if (!repack_half(in1, wt, 1, d->out_features, d->in_features, d->out_features, st)) {
                const dim3 grid(ceil_div(d->in_features, 64), ceil_div(d->out_features, 64), 1);
                helper_launch(4 * kSms, repack_weight_tile_kernel<__half>, grid, 256, 0, st, static_cast<const __half*>(in1), wt, nullptr, ENC_F16,
                             d->out_features, d->in_features, d->out_features);
                ++g_launches;
            }
            NML_CUDA(cudaGetLastError());
        }
        f.w = wt; f.d0 = d->in_features; f.d1 = d->out_features; f.k_is_dim0 = 0;
    }
    f.gather = 0;
    f.s_h = f.s_w = 1; f.d_h = f.d_w = 1;
    f.out = out; f.out_dtype = d->out_dtype; f.out_layout = NML_NHWC;
    f.out_c = forward ? d->out_features : d->in_features; f.out_h = 1; f.out_w = d->rows;
    f.bias = forward ? bias : nullptr; f.bias_dtype = d->w_dtype;
    f.math = d->math;
    f.round_f16 = forward ? d->round_out_f16 : 0;
    return run_fprop_like(f, ws, st);
}

// Grow-only per-device workspace for the reference-shaped entry points.
constexpr size_t kRefScratchLimit = 1ull << 30;  // what a batched product takes of it at most
struct RefWorkspace {
    void* ptr = nullptr;
    size_t bytes = 0;
};
static RefWorkspace g_ref_ws[64];

static int ref_workspace(size_t need, void** out) {
    int dev = 0;
    NML_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_dev_mutex);
    RefWorkspace& w = g_ref_ws[dev];
    if (need > w.bytes) {
        if (w.ptr) {
            NML_CUDA(cudaDeviceSynchronize());
            NML_CUDA(cudaFree(w.ptr));
            w.ptr = nullptr;
            w.bytes = 0;
        }
        size_t grow = round_up(need + need / 4, 1 << 20);
        NML_CUDA(cudaMalloc(&w.ptr, grow));
        w.bytes = grow;
    }
    *out = w.ptr;
    return NML_OK;
}

// Results of the reference-shaped entry points come from the device's stream-ordered pool
// (cudaMallocAsync on the legacy default stream the entry points run on): no device-wide
// synchronisation per call, freed memory is kept for the next result (release threshold = never).
// cudaFree accepts such pointers, so the reference's own `free_cuda` path keeps working; where a
// device has no memory pools the plain cudaMalloc / cudaFree pair is used.
static bool g_pool_ready[64] = {false};
static bool g_pool_usable[64] = {false};
static int ref_alloc(void** out, size_t bytes) {
    int dev = 0;
    NML_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return NML_ERR_INVALID;
    {
        std::lock_guard<std::mutex> lock(g_dev_mutex);
        if (!g_pool_ready[dev]) {
            int supported = 0;
            cudaMemPool_t pool;
            if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && supported &&
                cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
                unsigned long long keep = ~0ull;
                g_pool_usable[dev] = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess;
            }
            (void)cudaGetLastError();
            g_pool_ready[dev] = true;
        }
    }
    if (g_pool_usable[dev]) NML_CUDA(cudaMallocAsync(out, bytes ? bytes : 1, cudaStreamLegacy));
    else NML_CUDA(cudaMalloc(out, bytes ? bytes : 1));
    return NML_OK;
}
static void ref_release(void* p) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && g_pool_usable[dev]) cudaFreeAsync(p, cudaStreamLegacy);
    else cudaFree(p);
}

__global__ void tma_box_probe_kernel(const __grid_constant__ CUtensorMap tm, int c0, int c1, int c2, int c3,
                                     uint32_t bytes, uint8_t* out, int* err) {
    extern __shared__ __align__(1024) uint8_t box_smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ __align__(8) int abort_flag[4];
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_state_init(abort_flag, 0);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_arrive_expect_tx(smem_u32(&bar), bytes);
        tma_load_4d(smem_u32(box_smem), &tm, smem_u32(&bar), c0, c1, c2, c3);
    }
    bool ok = mbar_wait(smem_u32(&bar), 0, abort_flag, err, ERR_WAIT_FULL);
    if (ok)
        for (uint32_t i = threadIdx.x; i < bytes; i += blockDim.x) out[i] = box_smem[i];
}

// One warp waits, with the library's bounded wait, on an mbarrier that nothing ever arrives on.  The
// wait runs out after limit_ns, records ERR_WAIT_FULL in *err and the kernel returns: the give-up path
// of every kernel here, exercised without a fault, a trap or an unbounded spin.
__global__ void wait_limit_probe_kernel(unsigned long long limit_ns, int* err, int* gave_up) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ __align__(8) int abort_flag[4];
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_state_init(abort_flag, limit_ns);
        fence_mbar_init();
    }
    __syncthreads();
    const bool ok = mbar_wait(smem_u32(&bar), 0, abort_flag, err, ERR_WAIT_FULL);
    if (threadIdx.x == 0 && gave_up) *gave_up = ok ? 0 : 1;
}

}  // namespace nml

using namespace nml;

// ---------------------------------------------------------------- C ABI -------
extern "C" {

const char* nml_status_string(int status) {
    switch (status) {
        case NML_OK: return "ok";
        case NML_ERR_INVALID: return "invalid argument";
        case NML_ERR_WORKSPACE: return g_last_scratch_error[0] ? g_last_scratch_error : "workspace too small";
        case NML_ERR_CUDA: return g_last_error[0] ? g_last_error : "CUDA error";
        case NML_ERR_UNSUPPORTED: return "unsupported configuration";
        case NML_ERR_DEVICE: return g_last_device_error[0] ? g_last_device_error : "a kernel abandoned a bounded wait";
    }
    return "unknown status";
}

int nml_conv_output_size(const nml_conv_desc* d, int* h_out, int* w_out) {
    if (!d || !h_out || !w_out) return NML_ERR_INVALID;
    return conv_out_size(d, h_out, w_out) ? NML_OK : NML_ERR_INVALID;
}

int nml_conv_workspace_size(const nml_conv_desc* d, int pass, size_t* bytes) {
    if (!d || !bytes) return NML_ERR_INVALID;
    Bump ws{nullptr, 0, 0, true};
    // (bias and db stand in as non-null so that the scratch behind them is counted)
    float db_stand_in;
    int rc = conv_pass(d, pass, nullptr, nullptr, d, nullptr, &db_stand_in, ws, nullptr);
    *bytes = round_up(ws.off, 256);
    return rc;
}

int nml_linear_workspace_size(const nml_linear_desc* d, int pass, size_t* bytes) {
    if (!d || !bytes) return NML_ERR_INVALID;
    Bump ws{nullptr, 0, 0, true};
    float db_stand_in;
    int rc = linear_pass(d, pass, nullptr, nullptr, d, nullptr, &db_stand_in, ws, nullptr);
    *bytes = round_up(ws.off, 256);
    return rc;
}

int nml_conv_forward(const nml_conv_desc* d, const void* x, const void* w, const void* bias, void* y,
                     void* workspace, size_t workspace_bytes, void* stream) {
    if (!d || !x || !w || !y) return NML_ERR_INVALID;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    return conv_pass(d, NML_PASS_FORWARD, x, w, bias, y, nullptr, ws, static_cast<cudaStream_t>(stream));
}

int nml_conv_backward_data(const nml_conv_desc* d, const void* dy, const void* w, void* dx, void* workspace,
                           size_t workspace_bytes, void* stream) {
    if (!d || !dy || !w || !dx) return NML_ERR_INVALID;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    return conv_pass(d, NML_PASS_BACKWARD_DATA, dy, w, nullptr, dx, nullptr, ws, static_cast<cudaStream_t>(stream));
}

int nml_conv_backward_data_add(const nml_conv_desc* d, const void* dy, const void* w, const void* add, const void* add_mask, float add_below,
                               void* dx, void* workspace, size_t workspace_bytes, void* stream) {
    if (!d || !dy || !w || !dx || !add || ((reinterpret_cast<uintptr_t>(add) | reinterpret_cast<uintptr_t>(dx)) & 15)) return NML_ERR_INVALID;
    // dx is written before add is read where the sum is a pass of its own
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(add), d0 = reinterpret_cast<uintptr_t>(dx);
    const uintptr_t bytes = 2ull * std::max(d->batch, 0) * std::max(d->h, 0) * std::max(d->w, 0) * std::max(d->c_in, 0);
    if (a0 < d0 + bytes && d0 < a0 + bytes) return NML_ERR_INVALID;
    // (phase-packed columns have their own stores, which do not add)
    if (d->out_dtype != NML_F16 || d->out_layout != NML_NHWC || d->math != NML_MATH_F16 || d->c_in % 8 || d->stride_h * d->stride_w * d->c_in <= 16)
        return NML_ERR_UNSUPPORTED;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    return conv_pass(d, NML_PASS_BACKWARD_DATA, dy, w, nullptr, dx, nullptr, ws, static_cast<cudaStream_t>(stream), add, add_mask, add_below);
}

int nml_conv_backward_weight(const nml_conv_desc* d, const void* x, const void* dy, float* dw, float* db,
                             void* workspace, size_t workspace_bytes, void* stream) {
    if (!d || !x || !dy || !dw) return NML_ERR_INVALID;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    return conv_pass(d, NML_PASS_BACKWARD_WEIGHT, x, dy, nullptr, dw, db, ws, static_cast<cudaStream_t>(stream));
}

int nml_linear_forward(const nml_linear_desc* d, const void* x, const void* w, const void* bias, void* y,
                       void* workspace, size_t workspace_bytes, void* stream) {
    if (!d || !x || !w || !y) return NML_ERR_INVALID;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    return linear_pass(d, NML_PASS_FORWARD, x, w, bias, y, nullptr, ws, static_cast<cudaStream_t>(stream));
}

int nml_linear_backward_data(const nml_linear_desc* d, const void* dy, const void* w, void* dx, void* workspace,
                             size_t workspace_bytes, void* stream) {
    if (!d || !dy || !w || !dx) return NML_ERR_INVALID;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    return linear_pass(d, NML_PASS_BACKWARD_DATA, dy, w, nullptr, dx, nullptr, ws,
                       static_cast<cudaStream_t>(stream));
}

int nml_linear_backward_weight(const nml_linear_desc* d, const void* x, const void* dy, float* dw, float* db,
                               void* workspace, size_t workspace_bytes, void* stream) {
    if (!d || !x || !dy || !dw) return NML_ERR_INVALID;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    return linear_pass(d, NML_PASS_BACKWARD_WEIGHT, x, dy, nullptr, dw, db, ws, static_cast<cudaStream_t>(stream));
}

int nml_set_sm_limit(int sms) {
    if (sms < 0) return NML_ERR_INVALID;
    g_sm_limit.store(sms);
    return NML_OK;
}

int nml_init(void) {
    DeviceState* ds = nullptr;
    return device_state(&ds);
}

// Reads and clears one status word; the code of an abandoned wait goes into *code and into the
// message nml_status_string returns for NML_ERR_DEVICE.
static int read_status_word(int* word, int* code) {
    NML_CUDA(cudaDeviceSynchronize());
    int v = 0;
    NML_CUDA(cudaMemcpy(&v, word, sizeof(int), cudaMemcpyDeviceToHost));
    if (code) *code = v;
    if (v == 0) return NML_OK;
    NML_CUDA(cudaMemset(word, 0, sizeof(int)));
    snprintf(g_last_device_error, sizeof(g_last_device_error), "a kernel abandoned bounded wait %d (%s)", v,
             v == ERR_WAIT_EMPTY ? "producer: free stage" : v == ERR_WAIT_FULL ? "operands to land"
             : v == ERR_WAIT_TMEM_EMPTY ? "accumulator to drain" : v == ERR_WAIT_TMEM_FULL ? "accumulator to fill"
             : v == ERR_WAIT_DRAIN ? "copies in flight at unwinding" : "unknown");
    return NML_ERR_DEVICE;
}

int nml_device_status(int* code) {
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    return read_status_word(ds->err, code);
}

long long nml_launch_count(void) { return g_launches.load() + nml_layers_launch_count(); }

long long nml_debug_launch_count(int kind) { return kind >= 0 && kind < 9 ? g_launches_of[kind].load() : -1; }

int nml_profile_begin(int max_records) {
    if (max_records <= 0 || max_records > 1 << 16) return NML_ERR_INVALID;
    while (static_cast<int>(g_prof.start.size()) < max_records) {
        cudaEvent_t a, b;
        NML_CUDA(cudaEventCreate(&a));
        NML_CUDA(cudaEventCreate(&b));
        g_prof.start.push_back(a);
        g_prof.stop.push_back(b);
    }
    std::lock_guard<std::mutex> lock(g_dev_mutex);
    g_prof.cap = max_records;
    g_prof.n = 0;
    g_prof.on = true;
    return NML_OK;
}

int nml_profile_end(float* ms_out, int capacity, int* count) {
    if (!ms_out || !count) return NML_ERR_INVALID;
    g_prof.on = false;
    NML_CUDA(cudaDeviceSynchronize());
    int n = std::min(g_prof.n, capacity);
    for (int i = 0; i < n; ++i) NML_CUDA(cudaEventElapsedTime(&ms_out[i], g_prof.start[i], g_prof.stop[i]));
    *count = n;
    return NML_OK;
}

// ---- forward entry point that allocates nothing ----
// Scratch for the converted operands lives in the library image instead of caller memory.
// kStaticScratchBytes of every GPU that loads this library are held until the process exits.
constexpr size_t kStaticScratchBytes = 64ull << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
static __device__ int g_static_status;  // where kernels launched by this entry point report a give-up (see g_status_word)

struct StaticState {
    bool ready = false;
    void* scratch = nullptr;  // DEVICE address of g_static_scratch on this device
    DeviceState ds;           // status word = device address of g_static_status
};
static StaticState g_static[64];

// Once per device, with that device current.  In host code `g_static_scratch` is only a handle for
// the symbol, not an address a kernel may use: the device address comes from cudaGetSymbolAddress.
static int static_state(StaticState** out) {
    int dev = 0;
    NML_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return NML_ERR_INVALID;
    std::lock_guard<std::mutex> lock(g_dev_mutex);
    StaticState& s = g_static[dev];
    if (!s.ready) {
        void* scratch = nullptr;
        void* status = nullptr;
        NML_CUDA(cudaGetSymbolAddress(&scratch, g_static_scratch));
        NML_CUDA(cudaGetSymbolAddress(&status, g_static_status));
        NML_CUDA(cudaMemset(status, 0, sizeof(int)));
        NML_CUDA(cudaDeviceGetAttribute(&s.ds.sms, cudaDevAttrMultiProcessorCount, dev));
        int rc_attr = raise_smem_limit();
        if (rc_attr) return rc_attr;
        rc_attr = load_helper_kernels();  // so that no later call is the first use (= the loading) of a kernel
        if (rc_attr) return rc_attr;
        s.scratch = scratch;
        s.ds.err = static_cast<int*>(status);
        s.ds.attr_set = true;
        s.ready = true;
    }
    *out = &s;
    return NML_OK;
}

int nml_conv_forward_static(const nml_conv_desc* d, const void* x, const void* w, const void* bias, void* y,
                            void* stream) {
    StaticState* ss = nullptr;
    if (!d) {  // query form: wait for the device, report and clear a recorded give-up
        int rc = static_state(&ss);
        if (rc) return rc;
        return read_status_word(ss->ds.err, nullptr);  // the code is in nml_status_string(NML_ERR_DEVICE)
    }
    if (!x || !w || !y) return NML_ERR_INVALID;
    // (both runs plan within the array: a K split or an output copy that does not fit is left out)
    Bump dry{nullptr, 0, 0, true, nullptr, kStaticScratchBytes};
    int rc = conv_pass(d, NML_PASS_FORWARD, nullptr, nullptr, bias ? d : nullptr, nullptr, nullptr, dry, nullptr);
    if (rc) return rc;
    const size_t need = round_up(dry.off, 256);
    if (need > kStaticScratchBytes) {
        snprintf(g_last_scratch_error, sizeof(g_last_scratch_error),
                 "this layer needs %zu bytes of scratch; the built-in scratch array holds %zu "
                 "(use nml_conv_forward with a caller workspace)", need, kStaticScratchBytes);
        return NML_ERR_WORKSPACE;
    }
    rc = static_state(&ss);
    if (rc) return rc;
    // Every region of the scratch that the contraction reads is rewritten in full by the conversion
    // passes of this call (channel and K padding included), so nothing from the last call survives.
    Bump ws{static_cast<uint8_t*>(ss->scratch), 0, kStaticScratchBytes, false, &ss->ds, kStaticScratchBytes};
    return conv_pass(d, NML_PASS_FORWARD, x, w, bias, y, nullptr, ws, static_cast<cudaStream_t>(stream));
}

// ---- reference-shaped entry points ----
static void fill_conv_desc(nml_conv_desc* d, int transposed, int B, int C_in, int H, int W, int C_out, int KH,
                           int KW, int sh, int sw, int ph, int pw, int dh, int dw, int oph, int opw) {
    memset(d, 0, sizeof(*d));
    d->batch = B; d->c_in = C_in; d->h = H; d->w = W; d->c_out = C_out; d->kh = KH; d->kw = KW;
    d->stride_h = sh; d->stride_w = sw; d->pad_h = ph; d->pad_w = pw; d->dil_h = dh; d->dil_w = dw;
    d->outpad_h = oph; d->outpad_w = opw; d->transposed = transposed;
    d->in_layout = d->out_layout = NML_NCHW;
}

static int ref_run_conv(nml_conv_desc* d, int pass, const void* in0, const void* in1, const void* bias,
                        size_t out_bytes, uintptr_t* result) {
    if (!result) return NML_ERR_INVALID;
    size_t need = 0;
    int rc = nml_conv_workspace_size(d, pass, &need);
    if (rc) return rc;
    void* ws = nullptr;
    rc = ref_workspace(need, &ws);
    if (rc) return rc;
    void* out = nullptr;
    rc = ref_alloc(&out, out_bytes);
    if (rc) return rc;
    Bump b{static_cast<uint8_t*>(ws), 0, need, false};
    rc = conv_pass(d, pass, in0, in1, bias, out, nullptr, b, nullptr);
    if (rc) {
        ref_release(out);
        return rc;
    }
    *result = reinterpret_cast<uintptr_t>(out);
    return NML_OK;
}

static int ref_forward(int transposed, uintptr_t input_ptr, uintptr_t weight_ptr, uintptr_t bias_ptr,
                       size_t output_size, int B, int C_in, int H, int W, int C_out, int KH, int KW, int sh, int sw,
                       int ph, int pw, int dh, int dw, int oph, int opw, int groups, int dtype, int half_precision,
                       uintptr_t* result) {
    if (groups != 1) return NML_ERR_UNSUPPORTED;
    if (dtype != NML_F32 && dtype != NML_F16) return NML_ERR_INVALID;
    nml_conv_desc d;
    fill_conv_desc(&d, transposed, B, C_in, H, W, C_out, KH, KW, sh, sw, ph, pw, dh, dw, oph, opw);
    d.in_dtype = d.out_dtype = d.w_dtype = dtype;
    d.math = (half_precision || dtype == NML_F16) ? NML_MATH_F16 : NML_MATH_3XTF32;
    d.round_out_f16 = half_precision ? 1 : 0;
    int ho, wo;
    if (!conv_out_size(&d, &ho, &wo)) return NML_ERR_INVALID;
    size_t elems = static_cast<size_t>(B) * C_out * ho * wo;
    if (output_size != 0 && output_size != elems) return NML_ERR_INVALID;
    return ref_run_conv(&d, NML_PASS_FORWARD, reinterpret_cast<const void*>(input_ptr),
                        reinterpret_cast<const void*>(weight_ptr), reinterpret_cast<const void*>(bias_ptr),
                        elems * (dtype == NML_F16 ? 2 : 4), result);
}

int nml_ref_conv2d(uintptr_t input_ptr, size_t input_size, uintptr_t weight_ptr, size_t weight_size,
                   uintptr_t bias_ptr, size_t bias_size, size_t output_size, int B, int C_in, int H, int W, int C_out,
                   int KH, int KW, int stride_h, int stride_w, int padding_h, int padding_w, int dilation_h,
                   int dilation_w, int groups, int dtype, int half_precision, uintptr_t* result) {
    (void)input_size; (void)weight_size; (void)bias_size;
    return ref_forward(0, input_ptr, weight_ptr, bias_ptr, output_size, B, C_in, H, W, C_out, KH, KW, stride_h,
                       stride_w, padding_h, padding_w, dilation_h, dilation_w, 0, 0, groups, dtype, half_precision,
                       result);
}

int nml_ref_conv_transpose2d(uintptr_t input_ptr, size_t input_size, uintptr_t weight_ptr, size_t weight_size,
                             uintptr_t bias_ptr, size_t bias_size, size_t output_size, int B, int C_in, int H, int W,
                             int C_out, int KH, int KW, int stride_h, int stride_w, int padding_h, int padding_w,
                             int dilation_h, int dilation_w, int output_padding_h, int output_padding_w, int groups,
                             int dtype, int half_precision, uintptr_t* result) {
    (void)input_size; (void)weight_size; (void)bias_size;
    return ref_forward(1, input_ptr, weight_ptr, bias_ptr, output_size, B, C_in, H, W, C_out, KH, KW, stride_h,
                       stride_w, padding_h, padding_w, dilation_h, dilation_w, output_padding_h, output_padding_w,
                       groups, dtype, half_precision, result);
}

// The backward entry points receive H_out/W_out explicitly; for ConvTranspose2d they determine
// the output padding, which the reference's signature does not pass.
static int ref_backward(int transposed, int pass, uintptr_t p0, uintptr_t p1, int B, int C_in, int H, int W,
                        int C_out, int KH, int KW, int H_out, int W_out, int sh, int sw, int ph, int pw, int dh,
                        int dw, int dtype, uintptr_t* result) {
    if (dtype != NML_F32 && dtype != NML_F16) return NML_ERR_INVALID;
    nml_conv_desc d;
    fill_conv_desc(&d, transposed, B, C_in, H, W, C_out, KH, KW, sh, sw, ph, pw, dh, dw, 0, 0);
    int ho, wo;
    if (!conv_out_size(&d, &ho, &wo)) return NML_ERR_INVALID;
    if (transposed) {
        d.outpad_h = H_out - ho;
        d.outpad_w = W_out - wo;
        if (d.outpad_h < 0 || d.outpad_w < 0 || d.outpad_h >= sh + dh || d.outpad_w >= sw + dw) return NML_ERR_INVALID;
    } else if (ho != H_out || wo != W_out) {
        return NML_ERR_INVALID;
    }
    d.in_dtype = d.w_dtype = dtype;
    d.out_dtype = NML_F32;
    d.math = (dtype == NML_F16) ? NML_MATH_F16 : NML_MATH_3XTF32;
    size_t elems;
    const void *in0, *in1;
    if (pass == NML_PASS_BACKWARD_DATA) {
        elems = static_cast<size_t>(B) * C_in * H * W;
        in0 = reinterpret_cast<const void*>(p0);  // out_grad
        in1 = reinterpret_cast<const void*>(p1);  // weight
    } else {
        elems = static_cast<size_t>(C_out) * C_in * KH * KW;
        in0 = reinterpret_cast<const void*>(p1);  // input
        in1 = reinterpret_cast<const void*>(p0);  // out_grad
    }
    return ref_run_conv(&d, pass, in0, in1, nullptr, elems * 4, result);
}

int nml_ref_conv2d_backward_input(uintptr_t out_grad_ptr, uintptr_t weight_ptr, int B, int C_in, int H, int W,
                                  int C_out, int KH, int KW, int H_out, int W_out, int stride_h, int stride_w,
                                  int padding_h, int padding_w, int dilation_h, int dilation_w, int groups, int dtype,
                                  uintptr_t* result) {
    if (groups != 1) return NML_ERR_UNSUPPORTED;
    return ref_backward(0, NML_PASS_BACKWARD_DATA, out_grad_ptr, weight_ptr, B, C_in, H, W, C_out, KH, KW, H_out,
                        W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w, dtype, result);
}

int nml_ref_conv_transpose2d_backward_input(uintptr_t out_grad_ptr, uintptr_t weight_ptr, int B, int C_in, int H,
                                            int W, int C_out, int KH, int KW, int H_out, int W_out, int stride_h,
                                            int stride_w, int padding_h, int padding_w, int dilation_h,
                                            int dilation_w, int groups, int dtype, uintptr_t* result) {
    if (groups != 1) return NML_ERR_UNSUPPORTED;
    return ref_backward(1, NML_PASS_BACKWARD_DATA, out_grad_ptr, weight_ptr, B, C_in, H, W, C_out, KH, KW, H_out,
                        W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w, dtype, result);
}

int nml_ref_conv2d_backward_weight(uintptr_t out_grad_ptr, uintptr_t input_ptr, int B, int C_in, int H, int W,
                                   int C_out, int KH, int KW, int H_out, int W_out, int stride_h, int stride_w,
                                   int padding_h, int padding_w, int dilation_h, int dilation_w, int dtype,
                                   uintptr_t* result) {
    return ref_backward(0, NML_PASS_BACKWARD_WEIGHT, out_grad_ptr, input_ptr, B, C_in, H, W, C_out, KH, KW, H_out,
                        W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w, dtype, result);
}

int nml_ref_conv_transpose2d_backward_weight(uintptr_t out_grad_ptr, uintptr_t input_ptr, int B, int C_in, int H,
                                             int W, int C_out, int KH, int KW, int H_out, int W_out, int stride_h,
                                             int stride_w, int padding_h, int padding_w, int dilation_h,
                                             int dilation_w, int dtype, uintptr_t* result) {
    return ref_backward(1, NML_PASS_BACKWARD_WEIGHT, out_grad_ptr, input_ptr, B, C_in, H, W, C_out, KH, KW, H_out,
                        W_out, stride_h, stride_w, padding_h, padding_w, dilation_h, dilation_w, dtype, result);
}

// 1-D convolutions are the same walks over an image of height 1 ([B, C, L] is [B, C, 1, L]).
int nml_ref_conv1d(uintptr_t input_ptr, uintptr_t weight_ptr, uintptr_t bias_ptr, int B, int C_in, int L, int C_out,
                   int K, int stride, int padding, int dilation, int groups, int dtype, uintptr_t* result) {
    return ref_forward(0, input_ptr, weight_ptr, bias_ptr, 0, B, C_in, 1, L, C_out, 1, K, 1, stride, 0, padding, 1,
                       dilation, 0, 0, groups, dtype, 0, result);
}

int nml_ref_conv_transpose1d(uintptr_t input_ptr, uintptr_t weight_ptr, uintptr_t bias_ptr, int B, int C_in, int L,
                             int C_out, int K, int stride, int padding, int dilation, int output_padding, int groups,
                             int dtype, uintptr_t* result) {
    return ref_forward(1, input_ptr, weight_ptr, bias_ptr, 0, B, C_in, 1, L, C_out, 1, K, 1, stride, 0, padding, 1,
                       dilation, 0, output_padding, groups, dtype, 0, result);
}

int nml_ref_conv1d_backward_input(uintptr_t out_grad_ptr, uintptr_t weight_ptr, int B, int C_in, int L, int C_out,
                                  int K, int L_out, int stride, int padding, int dilation, int groups, int dtype,
                                  uintptr_t* result) {
    if (groups != 1) return NML_ERR_UNSUPPORTED;
    return ref_backward(0, NML_PASS_BACKWARD_DATA, out_grad_ptr, weight_ptr, B, C_in, 1, L, C_out, 1, K, 1, L_out, 1,
                        stride, 0, padding, 1, dilation, dtype, result);
}

int nml_ref_conv_transpose1d_backward_input(uintptr_t out_grad_ptr, uintptr_t weight_ptr, int B, int C_in, int L,
                                            int C_out, int K, int L_out, int stride, int padding, int dilation,
                                            int groups, int dtype, uintptr_t* result) {
    if (groups != 1) return NML_ERR_UNSUPPORTED;
    return ref_backward(1, NML_PASS_BACKWARD_DATA, out_grad_ptr, weight_ptr, B, C_in, 1, L, C_out, 1, K, 1, L_out, 1,
                        stride, 0, padding, 1, dilation, dtype, result);
}

int nml_ref_conv1d_backward_weight(uintptr_t out_grad_ptr, uintptr_t input_ptr, int B, int C_in, int L, int C_out,
                                   int K, int L_out, int stride, int padding, int dilation, int dtype,
                                   uintptr_t* result) {
    return ref_backward(0, NML_PASS_BACKWARD_WEIGHT, out_grad_ptr, input_ptr, B, C_in, 1, L, C_out, 1, K, 1, L_out, 1,
                        stride, 0, padding, 1, dilation, dtype, result);
}

int nml_ref_conv_transpose1d_backward_weight(uintptr_t out_grad_ptr, uintptr_t input_ptr, int B, int C_in, int L,
                                             int C_out, int K, int L_out, int stride, int padding, int dilation,
                                             int dtype, uintptr_t* result) {
    return ref_backward(1, NML_PASS_BACKWARD_WEIGHT, out_grad_ptr, input_ptr, B, C_in, 1, L, C_out, 1, K, 1, L_out, 1,
                        stride, 0, padding, 1, dilation, dtype, result);
}

int nml_ref_matmul(uintptr_t a_ptr, uintptr_t b_ptr, const int* a_shape, int a_rank, const int* b_shape, int b_rank,
                   int dtype, uintptr_t* result) {
    if (!a_shape || !b_shape || a_rank < 2 || b_rank < 2 || !result) return NML_ERR_INVALID;
    if (dtype != NML_F32 && dtype != NML_F16) return NML_ERR_INVALID;
    const int M = a_shape[a_rank - 2], K = a_shape[a_rank - 1], N = b_shape[b_rank - 1];
    if (b_shape[b_rank - 2] != K) return NML_ERR_INVALID;
    size_t batch = 1;
    for (int i = 0; i < a_rank - 2; ++i) batch *= a_shape[i];
    size_t b_batch = 1;
    for (int i = 0; i < b_rank - 2; ++i) b_batch *= b_shape[i];
    // A 2-D right operand is shared by every batch entry; a batched one must match.
    if (b_batch != 1 && b_batch != batch) return NML_ERR_INVALID;
    const int es = (dtype == NML_F16) ? 2 : 4;
    if (batch == 0 || M <= 0 || K <= 0 || N <= 0) return NML_ERR_INVALID;
    // C = A * B with B [K][N]: the input-gradient form of a Linear layer whose weight is B.  A shared B makes all
    // rows of A one problem.  Otherwise the entries run as the images of ONE launch, each with its own B (tiles of one
    // entry each), because an entry of an attention-sized product fills a handful of SMs for a few microseconds:
    // 64 x [333 x 64] x [64 x 333] in fp16 took 1740 us as 64 launches.  Entries that fill the GPU by themselves
    // keep their own launches, where the planner may pair CTAs and split K.
    const int math = (dtype == NML_F16) ? NML_MATH_F16 : NML_MATH_3XTF32;
    const bool shared_b = b_batch == 1 && batch * static_cast<size_t>(M) < (1u << 30);
    const long long tiles = 1ll * ceil_div(M, 128) * ceil_div(N, 256);
    const size_t c_entry = static_cast<size_t>(M) * N * es, a_entry = static_cast<size_t>(M) * K * es, b_entry = static_cast<size_t>(K) * N * es;
    size_t per_call = 1;  // entries per launch
    if (!shared_b && b_batch != 1 && tiles < 2ll * planning_sms()) per_call = std::min<size_t>(batch, 32768);  // (the grid of the weight repack)
    auto in_place = [&](const uint8_t* A, const uint8_t* B, uint8_t* C, size_t n) {
        StridedProduct g;
        memset(&g, 0, sizeof(g));
        g.M = N; g.N = M; g.K = K; g.batch = static_cast<int>(n);
        g.dtype = g.out_dtype = dtype;
        g.a = B; g.a_contiguous = false; g.a_stride = N; g.a_batch = 1ll * K * N;
        g.b = A; g.b_contiguous = true; g.b_stride = K; g.b_batch = 1ll * M * K;
        g.out = C; g.out_ns = N; g.out_batch = 1ll * M * N;
        return g;
    };
    // The way `n` entries of one launch go, by estimated time.  By rows, as the layer above; turned round, the columns of the
    // result being the pixels of an image whose channels are its rows (B [K][N] is that image's input, channel-major, and A its
    // weights), so that the lanes of the epilogue are consecutive columns and store from their registers, on any alignment;
    // in place (see nml_gemm.cuh).  fp16 rows of whole vectors leave by TMA stores and go by rows (64 x 512 x 64 x 512 11.1 us, turned 19.8).
    // Turned round, results of eight columns and fewer store a few bytes a line (64 x 18571 x 8 x 1 fp16 55 us by rows, 244 turned).
    // Us by rows / turned / in place: fp16 24 x 192 x 471 x 33 18.7 / 13.3 / 21.0; 64 x 333 x 64 x 333 25.7 / 16.0 / -; 128 x 33 x 64 x 33
    // 15.6 / 9.8 / 6.4; fp32 64 x 333 x 64 x 333 43.9 / 25.4 / 28.7; 3 x 800 x 96 x 801 - / 16.3 / 10.4; 85 x 12 x 284 x 1200 127 / 337 / 52;
    // 20 x 19698 x 6 x 1 29 / 166 / 91; 103 x 14010 x 2 x 39 323 / 191 / 341.
    enum Way { BY_ROWS, TURNED, IN_PLACE, STRIPS };
    auto way_of = [&](size_t n) -> Way {
        if (es == 2 && N % 8 == 0) return BY_ROWS;
        const int sms = planning_sms();
        const double rows_us = batched_us(false, n, M, K, N, es, sms);
        const double turned_us = N <= 8 ? 1e30 : batched_us(true, n, M, K, N, es, sms);
        double place_us = 1e30;
        if (g_sm_limit.load(std::memory_order_relaxed) == 0) {
            // Strips of 128 columns, read in place (gemm_rows_kernel), for K loops of one or two slices.  Stores of 64 bytes that start anywhere bound
            // large results whichever way they go, and two slices of both operands then cost more here than a conversion (28 x 726 x 96 x 844
            // 24.6 us, turned 19.6; 128 x 511 x 128 x 513 57 and 51).  From eight groups of rows an SM on, by estimate against the conversions
            // (110 x 855 x 20 x 324, whose strips make 1.1 waves, 39.7 and 32.6; 88 x 682 x 55 x 451 42.1 and 35.1; of 567 random products 5 are
            // slower so by more than 5 %, without the estimate 12).
            const StridedProduct g = in_place(nullptr, nullptr, nullptr, n);
            const double result = n * static_cast<double>(M) * N * 1e-6;
            const double groups = static_cast<double>(n) * ceil_div(N, kTileM) * ceil_div(M, kRowsBn) / sms;
            if (es == 2 && K <= kRowsMaxK && N >= 32 && M >= 32 && groups <= (K <= 64 ? 32.0 : 8.0) &&
                (groups < 8.0 || 1.33 * plan_rows(g, sms).us + 0.32 * result - 0.7 <= 0.95 * std::min(rows_us, turned_us)))
                return STRIPS;
            const StridedPlan plan = plan_strided(g, sms);
            place_us = es == 4 ? 5.9 + 0.92 * plan.loop_us + 2.0 * (plan.waves - 1.0) + 0.32 * result
                               : 5.65 + 1.4 * plan.loop_us + 1.8 * (plan.waves - 1.0) + 0.28 * result;
        }
        return place_us < std::min(rows_us, turned_us) ? IN_PLACE : turned_us < rows_us ? TURNED : BY_ROWS;
    };
    Way way = BY_ROWS;
    auto entries = [&](const uint8_t* A, const uint8_t* B, uint8_t* C, size_t n, Bump& bump) -> int {
        if (per_call == 1 || shared_b) {
            nml_linear_desc d;
            memset(&d, 0, sizeof(d));
            d.rows = static_cast<int>(n * M); d.out_features = K; d.in_features = N;
            d.in_dtype = d.out_dtype = d.w_dtype = dtype;
            d.math = math;
            return linear_pass(&d, NML_PASS_BACKWARD_DATA, A, B, nullptr, C, nullptr, bump, nullptr);
        }
        if (way == IN_PLACE || way == STRIPS) {
            if (bump.dry) return NML_OK;
            // (fp16 rows that TMA was to read and cannot stay refused)
            const int rc = es == 2 && K % 8 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) != 0 ? rows_for_tma(A, K, M) : NML_OK;
            const StridedProduct g = in_place(A, B, C, n);
            if (way == STRIPS && !rc) ++g_launches_of[NML_DEBUG_STRIPS];
            return rc ? rc : way == STRIPS ? run_rows(g, nullptr) : run_strided(g, plan_strided(g, planning_sms()), bump.ds, PDL_NORMAL, nullptr);
        }
        FpropLike f;
        memset(&f, 0, sizeof(f));
        if (way == TURNED) {
            if (!bump.dry) ++g_launches_of[NML_DEBUG_TURNED];
            f.a = B; f.a_dtype = dtype; f.a_layout = NML_NCHW; f.batch = static_cast<int>(n); f.a_h = 1; f.a_w = N; f.a_c = K;
            f.w = A; f.w_dtype = dtype; f.d0 = M; f.d1 = K; f.kh = f.kw = 1; f.k_is_dim0 = 0; f.w_direct = 1; f.w_batched = 1;
            f.s_h = f.s_w = f.d_h = f.d_w = 1;
            f.out = C; f.out_dtype = dtype; f.out_layout = NML_NCHW; f.out_c = M; f.out_h = 1; f.out_w = N;
            f.math = math;
            return run_fprop_like(f, bump, nullptr);
        }
        f.a = A; f.a_dtype = dtype; f.a_layout = NML_NHWC; f.batch = static_cast<int>(n); f.a_h = 1; f.a_w = M; f.a_c = K;
        f.w = B; f.w_dtype = dtype; f.d0 = K; f.d1 = N; f.kh = f.kw = 1; f.k_is_dim0 = 1; f.w_direct = 1; f.w_batched = 1;
        f.s_h = f.s_w = f.d_h = f.d_w = 1;
        f.out = C; f.out_dtype = dtype; f.out_layout = NML_NHWC; f.out_c = N; f.out_h = 1; f.out_w = M;
        f.math = math;
        return run_fprop_like(f, bump, nullptr);
    };
    if (shared_b) per_call = batch;
    // The converted operands of many small entries can be far larger than the operands (K is padded to a slice of 32 or 64, fp32
    // becomes two planes), and the workspace stays for good: at most 1 GB of it, or one entry's.
    size_t need = 0;
    int rc;
    for (;;) {
        Bump dry{nullptr, 0, 0, true};
        way = way_of(per_call);  // (for all launches: a last one of fewer entries has this one's scratch)
        rc = entries(nullptr, nullptr, nullptr, per_call, dry);
        if (rc) return rc;
        need = round_up(dry.off, 256);
        if (shared_b || per_call == 1 || need <= kRefScratchLimit) break;
        per_call = std::max<size_t>(1, std::min(per_call - 1, static_cast<size_t>(static_cast<double>(per_call) * kRefScratchLimit / need)));
    }
    void* ws = nullptr;
    rc = ref_workspace(need, &ws);
    if (rc) return rc;
    void* out = nullptr;
    rc = ref_alloc(&out, batch * c_entry);
    if (rc) return rc;
    for (size_t b = 0; b < batch; b += per_call) {
        Bump bump{static_cast<uint8_t*>(ws), 0, need, false};
        rc = entries(reinterpret_cast<const uint8_t*>(a_ptr) + b * a_entry,
                     reinterpret_cast<const uint8_t*>(b_ptr) + (b_batch == 1 ? 0 : b) * b_entry, static_cast<uint8_t*>(out) + b * c_entry,
                     std::min(per_call, batch - b), bump);
        if (rc) {
            ref_release(out);
            return rc;
        }
    }
    *result = reinterpret_cast<uintptr_t>(out);
    return NML_OK;
}

int nml_ref_free(uintptr_t ptr) {
    if (ptr) ref_release(reinterpret_cast<void*>(ptr));
    NML_CUDA(cudaGetLastError());
    return NML_OK;
}

int nml_debug_tma_box(const void* tensor, int elem_bytes, const int dims[4], const int box[4],
                      const int elem_strides[4], const int coords[4], void* out, size_t out_bytes, void* stream) {
    if (!tensor || !out || (elem_bytes != 2 && elem_bytes != 4)) return NML_ERR_INVALID;
    DeviceState* ds = nullptr;
    int rc = device_state(&ds);
    if (rc) return rc;
    uint64_t gd[4];
    uint32_t bx[4], es[4];
    size_t bytes = elem_bytes;
    for (int i = 0; i < 4; ++i) {
        gd[i] = dims[i];
        bx[i] = box[i];
        es[i] = elem_strides[i];
        bytes *= (box[i] + elem_strides[i] - 1) / elem_strides[i];
    }
    if (bytes > 96 * 1024 || bytes > out_bytes || bytes % 16) return NML_ERR_INVALID;
    CUtensorMap tm;
    rc = encode_map(&tm, tensor, elem_bytes, 4, gd, bx, es, SWZ_NONE);
    if (rc) return rc;
    static bool attr = false;
    if (!attr) {
        NML_CUDA(cudaFuncSetAttribute(tma_box_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
        attr = true;
    }
    tma_box_probe_kernel<<<1, 128, bytes + 1024, static_cast<cudaStream_t>(stream)>>>(
        tm, coords[0], coords[1], coords[2], coords[3], static_cast<uint32_t>(bytes), static_cast<uint8_t*>(out),
        ds->err);
    NML_CUDA(cudaGetLastError());
    return NML_OK;
}

int nml_debug_wait_timeout(unsigned long long limit_ns, int use_static_word, void* stream) {
    if (limit_ns == 0 || limit_ns > 100000000ull) return NML_ERR_INVALID;  // at most 0.1 s
    int* word = nullptr;
    if (use_static_word) {
        StaticState* ss = nullptr;
        int rc = static_state(&ss);
        if (rc) return rc;
        word = ss->ds.err;
    } else {
        DeviceState* ds = nullptr;
        int rc = device_state(&ds);
        if (rc) return rc;
        word = ds->err;
    }
    wait_limit_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(limit_ns, word, nullptr);
    NML_CUDA(cudaGetLastError());
    return NML_OK;
}

int nml_debug_stalled_linear_forward(const nml_linear_desc* d, const void* x, const void* w, void* y, void* workspace,
                                     size_t workspace_bytes, unsigned long long limit_ns, void* stream) {
    if (!d || !x || !w || !y || limit_ns == 0 || limit_ns > 100000000ull) return NML_ERR_INVALID;
    // only the plain stage-ring walk of a small fp16 layer (one CTA per tile, no pairs): every wait in it is
    // bounded and no MMA is ever issued
    if (d->math != NML_MATH_F16 || d->in_dtype != NML_F16 || d->w_dtype != NML_F16 || d->rows > 4096 ||
        d->in_features > 1024 || d->out_features > 128 || d->in_features % 8 || d->out_features % 8)
        return NML_ERR_UNSUPPORTED;
    Bump ws{static_cast<uint8_t*>(workspace), 0, workspace ? workspace_bytes : 0, false};
    g_dbg_wait_limit_ns = limit_ns;
    g_dbg_short_a_box = true;
    int rc = linear_pass(d, NML_PASS_FORWARD, x, w, nullptr, y, nullptr, ws, static_cast<cudaStream_t>(stream));
    g_dbg_wait_limit_ns = 0;
    g_dbg_short_a_box = false;
    return rc;
}

int nml_debug_copy_to_host(void* host_dst, uintptr_t device_src, size_t bytes) {
    if (!host_dst || !device_src) return NML_ERR_INVALID;
    NML_CUDA(cudaMemcpy(host_dst, reinterpret_cast<const void*>(device_src), bytes, cudaMemcpyDeviceToHost));
    return NML_OK;
}

}  // extern "C"
