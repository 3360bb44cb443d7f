// Host interface of the MC2 (matmul + collective) kernels.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "../core/symmem.h"
#include "hccl/hccl_types.h"

namespace hccl {

class CommImpl;

// Per-communicator resources of the fused kernels: the device control block, tile flags (symmetric) and the
// exchange buffer for partial tiles (symmetric, two parities), grown on demand.
struct Mc2State {
    uint32_t* ctl = nullptr;            // device, zero-initialised
    SymSegment flags;                   // [nRanks][kMaxTiles] uint64
    SymSegment xchg;                    // 2 * parityBytes
    uint64_t xchgParityBytes = 0;
    void* resCtxDev = nullptr;          // device copy of HcclMc2ResCtx (HcclCreateOpResCtx)
    ~Mc2State();
};
constexpr int kMc2MaxTiles = 16384;
constexpr int kMc2AgBlocks = 8 * 512;   // arrival counters of the push-form AllGather: ranks x 128-row blocks per rank
constexpr int kMc2CtlWords = 16 + 8 * 512;

// How a plain matmul runs, from its sizes, the number of SMs and the switches of the environment.
enum class MatmulRoute { SPLIT, ONE_SM, TWO_SM, WIDE, TWO_SM_SPLIT };
struct MatmulSwitches {
    bool twoSm = true;                  // HCCL_MC2_2SM
    int wide = -1;                      // HCCL_MC2_WIDE: 0 never, 1 wherever one full round runs, -1 by the rule
    bool l2Hints = false;               // HCCL_MC2_L2_HINTS
};
struct MatmulPlan {
    MatmulRoute route = MatmulRoute::ONE_SM;
    int bn = 0, tilesM = 0, tilesN = 0, grid = 0;
    int bt = 0, split = 0;              // SPLIT: tokens per tile (bn: weight rows), CTAs per tile; TWO_SM_SPLIT: CTA pairs per tile
    int ring = 0;                       // SPLIT: bytes of shared memory for stages
    int wide = 0, singles = 0;          // WIDE: wide items, single ones
    int rasterGroup = 0, l2HintA = 0, l2HintB = 0;
};
MatmulSwitches MatmulSwitchesOfEnv();
// `outAlign`: bytes the output is aligned to, 16 for more.
MatmulPlan PlanMatmul(uint64_t m, uint64_t n, uint64_t k, bool aMn, bool bMn, int sms, const MatmulSwitches& sw, uint32_t outAlign = 16);
uint32_t MatmulOutAlign(const MatmulPlan& plan);      // what the route asks for

// Tests of a wait that runs out, on a matmul with few output tiles: CTA `cta` loads nothing, all waits end after waitLimitNs.
struct Mc2StalledCta { int cta; uint64_t waitLimitNs; };
HcclResult Mc2Matmul(const void* a, const void* b, void* out, uint64_t m, uint64_t n, uint64_t k, int transA, int transB,
                     cudaStream_t stream, const Mc2StalledCta* stalled = nullptr);
HcclResult Mc2AllGatherMatmul(CommImpl* comm, const void* aShard, const void* b, void* out, void* gathered, uint64_t mPerRank,
                              uint64_t n, uint64_t k, int transB, cudaStream_t stream);
HcclResult Mc2MatmulReduceScatter(CommImpl* comm, const void* a, const void* b, void* out, uint64_t m, uint64_t n, uint64_t k,
                                  int transB, cudaStream_t stream);
HcclResult Mc2MatmulAllReduce(CommImpl* comm, const void* a, const void* b, void* out, uint64_t m, uint64_t n, uint64_t k,
                              int transB, cudaStream_t stream);
// Collective: makes sure the exchange buffer can hold `parityBytes` per parity (reallocates symmetric memory).
HcclResult Mc2EnsureState(CommImpl* comm, uint64_t parityBytes);

}  // namespace hccl
