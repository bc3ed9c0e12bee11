// Launches with programmatic stream serialization.  A pass is a chain of short kernels (conversion, repack, contraction,
// reduction), so a good part of a small layer's time was the gap between one kernel's last block and the next one's
// first instruction.  Every kernel of the library is launched so that it may start while its predecessor in the stream
// still runs; it calls pdl_enter() before it touches global memory, which waits until the predecessor has finished
// and its writes are visible, and lets its own successor start.  Block scheduling, barrier and TMEM set-up then overlap the
// predecessor's tail.  A kernel that waits for its predecessor has waited for everything before it (the predecessor did
// too, or was serialised in full), so the order of a stream is kept.
//
// Which grids overlap: those of at most one block per SM, and those of many waves.  In between, blocks that arrive while
// the predecessor still fills some SMs pile up on the others, and a bandwidth-bound kernel of one or two waves then runs
// on part of the GPU (the batch-norm passes of a 56 x 56 x 256 block at batch 256 +4 %); there only kernels whose blocks do a
// few KB of work each overlap (launch_short, up to 4 blocks per SM), and those of whose blocks no more fit an SM than the grid has
// for it.
#pragma once
#include <cuda_runtime.h>

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
