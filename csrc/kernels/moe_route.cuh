// Expert histogram + exclusive scan for MoE routing: from the [tokens, topk]
// expert ids of this rank, the row range every expert's tokens occupy when the
// (token, expert) pairs are grouped by expert (what a grouped GEMM consumes).
// The kernel needs `nExperts + 1` 32-bit words of scratch that are zero when it
// starts: per-expert counters and an exit ticket.  Blocks add their pairs to
// the counters; the last block to finish turns the counters into offsets and
// leaves the scratch zeroed again for the next call.
//
// Latency bound: a table of 64 Ki pairs is 256 KiB.  A block counts its pairs in
// shared memory and adds only the sums to the counters (up to kRouteSharedExperts
// experts; beyond that an expert meets few pairs and the counters take them
// directly), and the last block scans all counters together, kRouteThreads at a
// time; one thread that walks them pays a round trip to L2 per expert.  Measured
// against that: 8192 x 8 pairs and 256 experts 40.8 -> 6.3 us, 16 x 8 24.7 -> 4.3
// us, 32768 x 8 and 512 experts 82.0 -> 7.2 us, 100000 x 2 and 4096 experts 637 ->
// 14.5 us, 20000 x 2 and 60000 experts 9156 -> 132 us.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hccl {

constexpr int kRouteThreads = 256;
constexpr uint32_t kRouteSharedExperts = 4096;      // 16 KiB of counters per block
constexpr int kRoutePairs = 8;                      // ids a thread requests before it counts the first

static __global__ void __launch_bounds__(kRouteThreads) MoeExpertOffsetsKernel(const int32_t* __restrict__ topkIdx, uint64_t nPairs, uint32_t nExperts,
                                                                               uint32_t* __restrict__ scratch, uint32_t* __restrict__ offsets)
{
    uint32_t* counters = scratch;
    uint32_t* ticket = scratch + nExperts;
    __shared__ uint32_t s_count[kRouteSharedExperts];
    __shared__ uint32_t s_warp[kRouteThreads / 32];
    __shared__ bool s_last;
    const bool shared = nExperts <= kRouteSharedExperts;
    if (shared) {
        for (uint32_t e = threadIdx.x; e < nExperts; e += kRouteThreads) s_count[e] = 0;
        __syncthreads();
    }
    const uint64_t step = (uint64_t)gridDim.x * kRouteThreads;
    for (uint64_t i = (uint64_t)blockIdx.x * kRouteThreads + threadIdx.x; i < nPairs; i += step * kRoutePairs) {
        int32_t e[kRoutePairs];
#pragma unroll
        for (int k = 0; k < kRoutePairs; ++k) e[k] = i + k * step < nPairs ? topkIdx[i + k * step] : -1;
#pragma unroll
        for (int k = 0; k < kRoutePairs; ++k)
            if (e[k] >= 0 && (uint32_t)e[k] < nExperts) atomicAdd(shared ? &s_count[e[k]] : &counters[e[k]], 1u);
    }
    if (shared) {
        __syncthreads();
        for (uint32_t e = threadIdx.x; e < nExperts; e += kRouteThreads)
            if (s_count[e] != 0) atomicAdd(&counters[e], s_count[e]);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t run = 0;                               // pairs of all experts before this pass of the loop
    for (uint32_t base = 0; base < nExperts; base += kRouteThreads) {
        const uint32_t e = base + threadIdx.x;
        uint32_t c = 0;
        if (e < nExperts) {
            c = *reinterpret_cast<volatile uint32_t*>(&counters[e]);
            counters[e] = 0;                        // the scratch is zero again when the kernel ends
        }
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (int q = 0; q < kRouteThreads / 32; ++q) {
            if (q < warp) before += s_warp[q];
            all += s_warp[q];
        }
        if (e < nExperts) offsets[e] = run + before + incl - c;
        run += all;
        __syncthreads();                            // s_warp is read before the next pass writes it
    }
    if (threadIdx.x == 0) {
        offsets[nExperts] = run;
        *ticket = 0;
    }
}

// One block per 2048 pairs (every thread's ids in one request), 64 at most.
inline int MoeExpertOffsetsBlocks(uint64_t nPairs)
{
    uint64_t b = (nPairs + kRouteThreads * kRoutePairs - 1) / (kRouteThreads * kRoutePairs);
    return (int)(b < 1 ? 1 : (b > 64 ? 64 : b));
}

}  // namespace hccl
