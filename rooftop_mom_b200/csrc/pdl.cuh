// Programmatic dependent launch (sm_90 and later), used by the kernels of products, preconditioner applies and COCG
// iterations: a kernel launched with the programmatic stream-serialisation attribute is set up while its predecessor on
// the stream is still running; its CTAs then block in griddep_wait() until the predecessor has completed and its memory
// is visible. Each kernel launched this way calls griddep_wait() before anything else, so it reads no data of its
// predecessor early (nor of that one's predecessors, which completed before it). After a predecessor that is a copy, or
// outside such a launch, the wait is the ordinary one or none.
//
// griddep_launch_dependents() lets a kernel's dependents start once all its CTAs have called it. Only the passes of
// grid_reg.cu do: their long straight code then starts to load behind the predecessor (a 64 x 64 circulant apply: 8.4 us
// against 10.1 without). Elsewhere the dependents' CTAs would fill the SMs whose CTAs end first, several on one SM, and
// run the slower for it (with triggers a block-Jacobi apply and a product on 256 x 256 faces take 22.4 us instead of
// 17.4, the product alone 17.6 instead of 14.2, an FP32 512 x 512 product 30.1 instead of 25.1).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace rtm {

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// The same for a kernel whose clusters are rows of `cluster` CTAs.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent_clusters(void (*kernel)(KArgs...), int cluster, dim3 grid, dim3 block, cudaStream_t s,
                                             Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                    Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace rtm
