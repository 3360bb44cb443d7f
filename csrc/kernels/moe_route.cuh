// Expert histogram + exclusive scan for MoE routing: from the [tokens, topk]
// expert ids of this rank, the row range every expert's tokens occupy when the
// (token, expert) pairs are grouped by expert (what a grouped GEMM consumes).
//
// One cluster of kRouteCtas CTAs does the whole job, with its counters in
// shared memory: a launch owns everything it writes, so calls on any number of
// streams, in graphs and from several threads do not meet.
//
// Latency bound: a table of 64 Ki pairs is 256 KiB.  Up to kRouteCounters
// experts every CTA counts its share of the pairs on its own, and CTA r adds
// up the CTAs' counters of its eighth of the experts through distributed
// shared memory; with more experts an expert meets few pairs and its counter
// lives only in the CTA that owns it, where all CTAs add to it.  Each CTA
// scans its experts, the CTAs' totals give it its first row; up to 1024
// experts the first CTA adds up and scans them all, which saves that exchange
// (in a graph 8192 x 8 and 256 experts 4.20 -> 3.64 us, 132 x 2 and 64 3.70 -> 3.00,
// 32768 x 8 and 512 6.14 -> 5.59).  Measured (back to back on
// one B200, 6.3 us is what an empty table takes), against blocks that share counters in
// memory and a last block that scans them: 8192 x 8 pairs and 256 experts 6.3 us both,
// 32768 x 8 and 512 8.3 both, 100000 x 2 and 4096 14.5 -> 8.3, 20000 x 2 and 60000 131 ->
// 18.6 us.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "dependent_launch.cuh"

namespace hccl {

constexpr int kRouteCtas = 8;                       // the largest cluster every GPU grants
constexpr int kRouteThreads = 1024;
constexpr uint32_t kRouteCounters = 8192;           // 32 KiB per CTA
constexpr uint32_t kRouteMaxExperts = kRouteCtas * kRouteCounters;
static_assert(kRouteThreads == 32 * 32, "one warp total per lane");
constexpr int kRouteVecs = 4;                       // 16-byte loads a thread requests before it counts the first id

namespace route {
__device__ __forceinline__ uint32_t ClusterRank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void ClusterBarrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void ClusterArrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void ClusterWait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t PeerAddr(const uint32_t* p, uint32_t rank)      // `p` of CTA `rank`
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t LoadPeer(const uint32_t* p, uint32_t rank)
{
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(PeerAddr(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ void StorePeer(const uint32_t* p, uint32_t rank, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(PeerAddr(p, rank)), "r"(v) : "memory");
}
__device__ __forceinline__ void AddPeer(const uint32_t* p, uint32_t rank)
{
    asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], 1;" ::"r"(PeerAddr(p, rank)) : "memory");
}
}  // namespace route

static __global__ void __cluster_dims__(kRouteCtas, 1, 1) __launch_bounds__(kRouteThreads, 1)
    MoeExpertOffsetsKernel(const int32_t* __restrict__ topkIdx, uint64_t nPairs, uint32_t nExperts, uint32_t* __restrict__ offsets)
{
    __shared__ uint32_t s_count[kRouteCounters];
    __shared__ uint32_t s_warp[kRouteThreads / 32];
    __shared__ uint32_t s_before[kRouteCtas];                    // pairs of the experts of each CTA before this one
    const uint32_t rank = route::ClusterRank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool everyCta = nExperts <= kRouteCounters;            // every CTA counts all experts
    const bool oneScans = nExperts <= kRouteThreads;             // the first CTA adds up and scans them all
    const uint32_t perCta = oneScans ? nExperts : (nExperts + kRouteCtas - 1) / kRouteCtas;
    const uint32_t nCounters = everyCta ? nExperts : perCta;
    for (uint32_t e = tid; e < nCounters; e += kRouteThreads) s_count[e] = 0;
    AllowDependents();
    DependencyWait();                                            // the counters are cleared under the end of the kernel in front
    __syncthreads();
    if (!everyCta) route::ClusterBarrier();
    auto count = [&](int32_t id) {
        const uint32_t e = (uint32_t)id;
        if (id < 0 || e >= nExperts) return;
        if (everyCta) atomicAdd(&s_count[e], 1u);
        else route::AddPeer(&s_count[e % perCta], e / perCta);
    };
    const uint64_t me = (uint64_t)rank * kRouteThreads + tid, step = (uint64_t)kRouteCtas * kRouteThreads;
    const uint64_t nVecs = (reinterpret_cast<uintptr_t>(topkIdx) & 15u) == 0 ? nPairs / 4 : 0;
    const int4* vecs = reinterpret_cast<const int4*>(topkIdx);
    for (uint64_t i = me; i < nVecs; i += step * kRouteVecs) {
        int4 v[kRouteVecs];
#pragma unroll
        for (int k = 0; k < kRouteVecs; ++k) v[k] = i + k * step < nVecs ? vecs[i + k * step] : make_int4(-1, -1, -1, -1);
#pragma unroll
        for (int k = 0; k < kRouteVecs; ++k) { count(v[k].x); count(v[k].y); count(v[k].z); count(v[k].w); }
    }
    // the ids after the last whole vector, or all of them where the table does not start on 16 bytes
    for (uint64_t i = nVecs * 4 + me; i < nPairs; i += step * kRouteVecs) {
        int32_t v[kRouteVecs];
#pragma unroll
        for (int k = 0; k < kRouteVecs; ++k) v[k] = i + k * step < nPairs ? topkIdx[i + k * step] : -1;
#pragma unroll
        for (int k = 0; k < kRouteVecs; ++k) count(v[k]);
    }
    route::ClusterBarrier();                                     // every pair is counted
    // this CTA's experts [first, last), `mine` consecutive ones per thread
    const uint32_t first = rank * perCta < nExperts ? rank * perCta : nExperts;
    const uint32_t last = first + perCta < nExperts ? first + perCta : nExperts;
    const uint32_t mine = (perCta + kRouteThreads - 1) / kRouteThreads;
    constexpr uint32_t kMost = kRouteCounters / kRouteThreads;
    uint32_t c[kMost], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < kMost; ++j) {
        const uint32_t e = first + tid * mine + j;
        c[j] = 0;
        if (j < mine && e < last) {
            if (everyCta) {
#pragma unroll
                for (uint32_t r = 0; r < kRouteCtas; ++r) c[j] += route::LoadPeer(&s_count[e], r);
            } else {
                c[j] = s_count[e - first];
            }
        }
        sum += c[j];
    }
    if (oneScans) {
        route::ClusterArrive();                                  // this thread reads no peer after this
        if (rank != 0) {
            route::ClusterWait();                                // the first CTA has this one's counters
            return;
        }
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += up;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    const uint32_t ofWarp = s_warp[lane];                        // as many warps as lanes
    uint32_t run = incl - sum + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? ofWarp : 0u);      // before this thread's, in this CTA
    const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, ofWarp);
    if (!oneScans) {
        if (tid > rank && tid < kRouteCtas) route::StorePeer(&s_before[rank], tid, all);
        route::ClusterBarrier();                                 // the totals are there; nobody reads a peer after this
        for (uint32_t r = 0; r < rank; ++r) run += s_before[r];
    }
#pragma unroll
    for (uint32_t j = 0; j < kMost; ++j) {
        const uint32_t e = first + tid * mine + j;
        if (j < mine && e < last) offsets[e] = run;
        run += c[j];
    }
    if (rank == (oneScans ? 0 : kRouteCtas - 1) && tid == kRouteThreads - 1) offsets[nExperts] = run;
    if (oneScans) route::ClusterWait();
}

}  // namespace hccl
