// Launches with programmatic stream serialization.  A pass is a chain of short kernels (conversion, repack, contraction,
// reduction), so a good part of a small layer's time was the gap between one kernel's last block and the next one's
// first instruction.  Every kernel of the library is launched so that it may start while its predecessor in the stream
// still runs; it calls pdl_enter() before it touches global memory, which waits until the predecessor has finished
// and its writes are visible, and lets its own successor start.  Block scheduling, barrier and TMEM set-up then overlap the
// predecessor's tail.  A kernel that waits for its predecessor has waited for everything before it (the predecessor did
// too, or was serialised in full), so the order of a stream is kept, for writes and for ordinary loads (see load_global).
//
// Which grids overlap: those of at most one block per SM, and those of many waves.  In between, blocks that arrive while
// the predecessor still fills some SMs pile up on the others, and a bandwidth-bound kernel of one or two waves then runs
// on part of the GPU (the batch-norm passes of a 56 x 56 x 256 block at batch 256 +4 %); there only kernels whose blocks do a
// few KB of work each overlap (launch_short, up to 4 blocks per SM), and those of whose blocks no more fit an SM than the grid has
// for it.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace nml {

__device__ __forceinline__ void pdl_enter() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

// Two neighbours in a stream that do not depend on one another (the conversions of a pass's two operands, a
// contraction and the column sums of one of its operands) run side by side as a leader and a sibling.  The leader lets
// the sibling start only after its own wait, so everything in front of the leader is over when the sibling starts
// working without a wait; the sibling waits at its end, so that it ends after the leader and whoever waits for the
// sibling has waited for both.  The sibling is always launched as an overlapping grid.
enum { PDL_NORMAL = 0, PDL_LEADER = 1, PDL_SIBLING = 2 };
__device__ __forceinline__ void pdl_enter(int role) {
    if (role == PDL_LEADER) cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    if (role == PDL_NORMAL) cudaGridDependencySynchronize();
}
__device__ __forceinline__ void pdl_leave(int role) {
    if (role == PDL_SIBLING) cudaGridDependencySynchronize();
}

// Loads of global memory in the helper kernels and epilogues, all of them.  What they read, an earlier grid may have written after
// this one became resident: grids trigger before they wait, so a pass's reduction may sit on an SM while the last pass's still
// reads the same planes and the contraction between the two has yet to write them.  The wait makes those writes visible to
// ordinary loads; a read-only load (ld.global.nc: __ldg, and what the compiler makes of a const __restrict__ pointer) is for
// data that does not change while its grid lives, and may be answered from a line cached before.  Hence ordinary loads,
// volatile so that none moves above the wait.
__device__ __forceinline__ uint4 load_global(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ uint2 load_global(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ float4 load_global(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ float load_global(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ int load_global(const int* p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ unsigned load_global(const uint8_t* p) {
    unsigned v;
    asm volatile("ld.global.u8 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ __half load_global(const __half* p) {
    __half_raw v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v.x) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ __half2 load_global(const __half2* p) {
    unsigned v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
    return *reinterpret_cast<__half2*>(&v);
}
// The same for what is read once and written back (evict first).
__device__ __forceinline__ float4 load_streaming(const float4* p) {
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
}

constexpr unsigned kSms = 148;
inline bool overlaps(dim3 grid, unsigned single_wave_limit) {
    const unsigned long long blocks = 1ull * grid.x * grid.y * grid.z;
    return blocks <= single_wave_limit || blocks >= 32ull * kSms;
}

// cluster: blocks per cluster along x (1: none).  Errors surface in cudaGetLastError like those of <<< >>>.
template <typename... P, typename... A>
inline void launch_with(bool overlap, int cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    if (overlap) {
        cudaLaunchAttribute& a = attr[cfg.numAttrs++];
        a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        a.val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        cudaLaunchAttribute& a = attr[cfg.numAttrs++];
        a.id = cudaLaunchAttributeClusterDimension;
        a.val.clusterDim.x = cluster;
        a.val.clusterDim.y = 1;
        a.val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    launch_with(overlaps(grid, kSms), 1, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}
template <typename... P, typename... A>
inline void launch_short(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    launch_with(overlaps(grid, 4 * kSms), 1, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}

}  // namespace nml
