// Host interface of the MoE dispatch / combine kernels.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cuda_bf16.h>
#include "dev_types.h"
#include "launch.h"

namespace hccl {

constexpr int kMoeMaxExperts = 512;
constexpr int kMoeMaxTopk = 8;
constexpr int kMoeMaxHidden = 8192;
// Pairs up to which the dispatch kernel counts them itself.  Against one counting launch in front, which is what a rank with a GPU of
// its own saves (one rank, rows of 7168, top-8, us, in the kernel and with the launch): launched one by one 8 pairs 14.6 and 18.0, 512
// 16.8 and 20.4, 2048 28.0 and 30.6, 4096 40.0 and 40.8, where the two meet; in a CUDA graph, where a launch costs less, 8 pairs 14.6 and
// 15.3, 512 19.8 and 20.2, 1024 23.7 and 23.4, 2048 31.6 and 30.7, 4096 43.4 and 41.1.  Two emulated ranks, whose launches run one after the other,
// gain at every size and either way (4096 pairs 42.5 and 48.0, in a graph 45.7 and 46.7).
constexpr int kMoeCountInDispatch = 4096;
constexpr size_t kMoeTableBytes = (size_t)kMaxBlocks * kMaxDevRanks * kMoeMaxExperts * sizeof(uint32_t);

struct MoeDispatchArgs {
    const __nv_bfloat16* x;            // [nTokens, hidden]
    const int32_t* topkIdx;            // [nTokens, topk] global expert ids (negative = dropped)
    const uint32_t* counts;            // [nExperts] pairs per expert on this rank; null: the kernel counts
    const uint32_t* pos;               // [nTokens * topk] position of the pair among this rank's pairs of that expert; null likewise
    uint64_t* slotMap;                 // [nTokens * topk] out: (destination rank << 32) | slot
    uint32_t* recvOffsets;             // [nExperts / nRanks + 1] out: where each local expert starts in the receive buffer
    uint32_t* table[kMaxDevRanks];     // count exchange table of every rank (symmetric)
    uint8_t* recvX[kMaxDevRanks];      // [capacity, hidden] fp8 e4m3 (symmetric)
    float* recvScale[kMaxDevRanks];    // [capacity, hidden / 128] (symmetric)
    uint64_t* recvSrc[kMaxDevRanks];   // [capacity] (source rank << 32) | (token * topk + k) (symmetric)
    int nTokens, hidden, topk, nExperts;
    uint32_t capacity;
};

struct MoeCombineArgs {
    const __nv_bfloat16* y[kMaxDevRanks];   // expert outputs [capacity, hidden] of every rank (symmetric)
    const float* topkWeight;                // [nTokens, topk]
    const uint64_t* slotMap;                // from dispatch
    __nv_bfloat16* out;                     // [nTokens, hidden]
    int nTokens, hidden, topk;
    uint32_t capacity;
};

HcclResult LaunchMoeCount(const int32_t* topkIdx, int nPairs, int nExperts, uint32_t* counts, uint32_t* pos, cudaStream_t stream);
HcclResult LaunchMoeDispatch(const LaunchTarget& t, const MoeDispatchArgs& a, int nBlocks);
HcclResult LaunchMoeCombine(const LaunchTarget& t, const MoeCombineArgs& a, int nBlocks);

}  // namespace hccl
