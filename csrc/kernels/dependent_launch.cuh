// Launches whose start overlaps the end of the kernel in front of them in the stream (programmatic dependent launch).
//
// A plain launch starts when the kernel before it has ended and its end has been seen, and back to back that happens in
// steps: launches of spinning kernels of 0.5 .. 8.4 us follow one another every 2.1, 4.2, 6.2, 8.2 or 10.3 us on a B200,
// never in between, which is half a step, about a microsecond, lost per launch beside the start itself.  A kernel launched
// with the attribute below is set up while its predecessor ends, and holds at DependencyWait() until the predecessor has
// completed and its writes are visible: kernel time + 0.8 us each, + 0.55 us where the predecessor calls AllowDependents().
//
// Rules.  Every thread of a kernel launched this way calls DependencyWait() before it touches global memory (kernel
// parameters, shared and tensor memory are free), and so before it ends: a kernel is complete only after all kernels in front
// of it are, and what follows may rely on the whole stream as with plain launches.  AllowDependents() lets the next kernel's
// blocks take what this kernel leaves free of an SM; kernels that wait for another rank do not call it, so that blocks which
// wait hold nothing that a kernel on another stream may need for that rank to get on.  A kernel calls it only when it has all that
// it will ever ask of its SM, its tensor memory above all: a follower, this library's or another's, may take the columns and then
// hold at its own wait, for a kernel that cannot go on without them.
#pragma once
#include <cuda_runtime.h>
#include <cstring>

namespace hccl {

__device__ __forceinline__ void DependencyWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void AllowDependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `cluster`: CTAs per cluster; 0 for a kernel without clusters or with a compiled-in cluster size.
template <class... Params, class... Args>
cudaError_t LaunchDependent(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, unsigned cluster, Args&&... args)
{
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = cluster;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = cluster > 0 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
    if (e != cudaSuccess) cudaGetLastError();             // the caller has it: the check behind the next <<<>>> shall not find it
    return e;
}

}  // namespace hccl
