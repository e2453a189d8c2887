// Launches that may begin while the kernel in front of them still runs (programmatic dependent launch), for the short
// kernels of a decoding step, where launch latency and the ramp of the first loads are a good part of each.
//
// A kernel launched this way calls `wait_for_predecessor()` in EVERY thread block before it reads or writes anything an
// earlier kernel may touch; it may then be sure that everything before it in the stream is done, because each kernel in
// such a chain waits for its own predecessor before it can finish.  `let_successor_start()` allows the next one in.  Before
// the wait only addresses may be prefetched into L2: that is coherent, so even data the predecessor writes stays right.
#pragma once
#include <cuda_runtime.h>

#include "neox_b200.h"

namespace launch {

__device__ __forceinline__ void let_successor_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// 16 bytes that the kernel in front may have written, read after the wait: a coherent load.  (Read-only loads, which the
// compiler also makes of `const __restrict__` pointers, assume data that is constant for the kernel's whole life; a kernel that
// starts early lives through its predecessor's writes.)
__device__ __forceinline__ uint4 load_16(const void* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// cluster: thread blocks per cluster along x (1: none)
template <typename... Params, typename... Args>
int overlapped(void (*kernel)(Params...), dim3 grid, dim3 block, int cluster, cudaStream_t stream, Args... args) {
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = cluster;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = stream;
    cfg.attrs = attrs;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...) == cudaSuccess ? 0 : NEOX_ERR_LAUNCH;
}

}  // namespace launch
