// HcclMoeExpertOffsetsNoAlloc: the expert offsets for callers that cannot allocate (see hccl/hccl_moe_noalloc.h for who they
// are).  The kernel keeps its counters in shared memory; nothing in this file allocates: no cudaMalloc / cudaFree, no
// containers that grow on the call path, no library routine that allocates device memory.
#include <cuda_runtime.h>
#include "../core/log.h"
#include "hccl/hccl_moe_noalloc.h"
#include "moe_route.cuh"

extern "C" HcclResult HcclMoeExpertOffsetsNoAlloc(const int32_t* topkIdx, uint64_t nPairs, uint32_t nExperts, uint32_t* offsets,
                                                  hcclStream_t stream)
{
    using namespace hccl;
    CHK_PTR_NULL(topkIdx);
    CHK_PTR_NULL(offsets);
    if (nExperts == 0 || nExperts > HCCL_MOE_NOALLOC_MAX_EXPERTS) {
        HCCL_ERROR("HcclMoeExpertOffsetsNoAlloc: nExperts = %u is outside 1..%u; use HcclMoeExpertOffsets for more experts", nExperts,
                   HCCL_MOE_NOALLOC_MAX_EXPERTS);
        return HCCL_E_PARA;
    }
    const cudaError_t e = LaunchDependent(MoeExpertOffsetsKernel, kRouteCtas, kRouteThreads, 0, (cudaStream_t)stream, 0, topkIdx, nPairs, nExperts, offsets);
    if (e != cudaSuccess) { HCCL_ERROR("HcclMoeExpertOffsetsNoAlloc: launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}
