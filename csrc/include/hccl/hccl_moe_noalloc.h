// Allocation-free variant of HcclMoeExpertOffsets.
//
// This entry point has no counterpart in the HCCL reference; it exists for callers of this library that are not
// allowed to allocate device memory at the moment they need the routing offsets: code running under a memory
// budget that has already handed every byte to a framework's caching allocator, plugins loaded into a serving
// process whose operator forbids cudaMalloc after start-up, and code on a latency path where the implicit device
// synchronisation of cudaMalloc / cudaFree is not acceptable.
//
// Neither this entry point nor HcclMoeExpertOffsets allocates: the kernel they launch keeps its counters in shared memory.
// What the variant promises beyond that is its limit: the number of experts is capped at HCCL_MOE_NOALLOC_MAX_EXPERTS (a
// larger value is rejected with HCCL_E_PARA and a log line that names the limit).
//
// Behaviour to know about:
//   * A call launches one kernel and nothing else.  Calls may overlap on the GPU, on any streams and in graphs.
//   * Inputs and outputs are the caller's, exactly as for HcclMoeExpertOffsets: topkIdx [nPairs] int32 and
//     offsets [nExperts + 1] uint32 in device memory; ids outside [0, nExperts) are ignored.
#ifndef HCCL_B200_MOE_NOALLOC_H_
#define HCCL_B200_MOE_NOALLOC_H_

#include "hccl_types.h"

#ifdef __cplusplus
extern "C" {
#endif

#define HCCL_MOE_NOALLOC_MAX_EXPERTS 4096u

HcclResult HcclMoeExpertOffsetsNoAlloc(const int32_t* topkIdx, uint64_t nPairs, uint32_t nExperts, uint32_t* offsets, hcclStream_t stream);

#ifdef __cplusplus
}
#endif
#endif  // HCCL_B200_MOE_NOALLOC_H_
