// Plain matmul for outputs too small to fill the chip with 256-wide tiles (decode steps, short prompts): the inner
// dimension is split over the CTAs of a cluster and the partial tiles are added through distributed shared memory.
//
// What bounds these shapes is the weight stream from HBM: at 16 tokens x 8192 x 8192 a pass reads 134 MB of weights for
// 2 GFLOP.  A one-tile-per-SM kernel leaves most SMs idle (64 tiles of 128 columns) and pads the tokens to a 128-row
// operand.  So here
//   * the WEIGHT is the 128-row operand of tcgen05.mma (cta_group::1, M = 128) and the tokens are the narrow one
//     (N = bt, a multiple of 16): a stage is 16 KiB of weights plus bt * 128 bytes of activations;
//   * a cluster of `split` CTAs (at most 4) works on one 128 x bt tile, CTA r on the r-th share of the k-blocks, until
//     about two CTAs per SM are busy: the stage ring takes at most half of an SM's shared memory, so that one CTA's
//     start and end run under its neighbour's main loop;
//   * each CTA leaves its fp32 partial in its own shared memory ([token][column], the idle stage ring) and, after one
//     cluster barrier, CTA r adds its share of the tokens over all CTAs in rank order (one fixed order, no atomics, no
//     workspace) and stores them as bf16, 256 contiguous bytes per token row.  The order depends on the number of CTAs
//     per tile and so on the shape: a row's fp32 sum may differ in its last place from that of a call with more rows.
// Measured against the one-SM kernel on 128 x 128 tiles (us, bf16, weight [N, K]): 16 x 8192 x 8192 47.5 -> 26.8 (5.0
// TB/s), 64 x 8192 x 8192 48.4 -> 28.8, 16 x 8192 x 1024 12.4 -> 8.4, 128 x 4096 x 4096 26.7 -> 16.5, 32 x 4096 x 14336
// 73.9 -> 26.6, 300 x 2048 x 4096 24.7 -> 16.5; against its 256-wide form 16 x 57344 x 8192 160.6 -> 142.4 (6.6 TB/s), 64
// x 57344 x 8192 162.3 -> 151.0.
// Warp roles and waits are those of the other kernels (mc2_gemm.cuh): warp 0 TMA producer, warp 1 MMA issuer, warps 2-5
// drain the accumulator; every wait is bounded, and a CTA that gave one up tells its cluster, which then stores nothing of
// the tile: what its shared memory holds is no partial sum.
#pragma once
#include "mc2_gemm.cuh"

namespace hccl {
namespace mc2 {

constexpr int kSplitMaxBt = 128;
constexpr int kSplitMaxCluster = 4;               // more CTAs per tile read more activations and wait for one another longer
constexpr int kSplitMaxStages = 6;
constexpr int kSplitWBytes = 128 * kBK * 2;                  // 16 KiB of weights per stage
constexpr int kSplitRingBytes = 108 * 1024;                  // two CTAs per SM
constexpr int kSplitBarBytes = 256;

struct SplitArgs {
    int M, N, K;               // out[M, N] = X[M, K] x W[N, K]^T   (operand storage is described by the tensor maps)
    __nv_bfloat16* out;
    int bt;                    // tokens per tile
    int tilesM;                // token tiles; the tile index runs over them first, so that they share a weight tile in L2
    int stages;
    uint32_t* ctl;             // control block: the abort word of bounded waits
    uint64_t waitLimitNs;      // of every wait
    int stalledCta;            // tests: this CTA's producer loads nothing (-1: none)
};

__host__ __device__ constexpr int SplitStageBytes(int bt) { return kSplitWBytes + bt * kBK * 2; }
inline int SplitStages(int bt)
{
    const int n = kSplitRingBytes / SplitStageBytes(bt);
    return n < kSplitMaxStages ? n : kSplitMaxStages;
}
// the ring also has to hold the fp32 partial tile
inline int SplitSmemBytes(int bt)
{
    const int ring = SplitStages(bt) * SplitStageBytes(bt), partial = bt * 128 * 4;
    return (ring > partial ? ring : partial) + kSplitBarBytes + 1024;      // + slack for the 1024-byte alignment
}
constexpr int kSplitMaxSmemBytes = kSplitRingBytes + kSplitBarBytes + 1024;
static_assert(kSplitMaxBt * 128 * 4 <= kSplitRingBytes, "the largest partial tile is no larger than the ring");

__device__ __forceinline__ uint32_t SplitClusterRank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t SplitClusterSize()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void SplitClusterSync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t LdCluster1(uint32_t localAddr, uint32_t rank)
{
    uint32_t a, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(localAddr), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 LdCluster4(uint32_t localAddr, uint32_t rank)
{
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(localAddr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
// 32 lanes x 16 consecutive 32-bit columns (see TmemLd32x32)
__device__ __forceinline__ void TmemLd32x16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

template <bool W_MN, bool X_MN>
__global__ void __launch_bounds__(kThreads) GemmSplitKernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SplitArgs g)
{
    extern __shared__ uint8_t smemRaw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
    const int stageBytes = SplitStageBytes(g.bt);
    const int ringBytes = g.stages * stageBytes, partialBytes = g.bt * 128 * 4;
    uint64_t* fullBar = reinterpret_cast<uint64_t*>(smem + (ringBytes > partialBytes ? ringBytes : partialBytes));
    uint64_t* emptyBar = fullBar + kSplitMaxStages;
    uint64_t* tmemFull = fullBar + 2 * kSplitMaxStages;
    uint32_t* tmemBaseSlot = reinterpret_cast<uint32_t*>(fullBar + 2 * kSplitMaxStages + 1);
    volatile uint32_t* gaveUp = tmemBaseSlot + 1;      // a role of this CTA left before its work was done
    volatile uint32_t* abortWord = g.ctl + kCtlAbort;

    const int warp = threadIdx.x / 32;
    const int split = (int)SplitClusterSize(), crank = (int)SplitClusterRank();
    const int tile = (int)blockIdx.x / split;
    const int row0 = (tile % g.tilesM) * g.bt, col0 = (tile / g.tilesM) * 128;
    const int kBlocks = (g.K + kBK - 1) / kBK;
    const int kFirst = (int)((long long)kBlocks * crank / split), kLast = (int)((long long)kBlocks * (crank + 1) / split);
    const uint32_t tmemCols = g.bt <= 32 ? 32u : (g.bt <= 64 ? 64u : 128u);

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; ++s) { MbarInit(&fullBar[s], 1); MbarInit(&emptyBar[s], 1); }
        MbarInit(tmemFull, 1);
        *gaveUp = 0;
        MbarInitFence();
        PrefetchTensorMap(&tmW);
        PrefetchTensorMap(&tmX);
    }
    if (warp == 1) {
        TmemAlloc(tmemBaseSlot, tmemCols);
        TmemRelinquish();
    }
    TcFenceBefore();
    __syncthreads();
    TcFenceAfter();
    const uint32_t tmemBase = *tmemBaseSlot;
    AllowDependents();
    DependencyWait();

    if (warp == 0) {
        if (ElectOne()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kFirst; kb < kLast && (int)blockIdx.x != g.stalledCta; ++kb) {
                ok = MbarWait(&emptyBar[stage], phase ^ 1u, abortWord, g.waitLimitNs);
                if (!ok) break;
                uint8_t* sw = smem + stage * stageBytes;
                uint8_t* sx = sw + kSplitWBytes;
                MbarExpectTx(&fullBar[stage], (uint32_t)stageBytes);
                if (!W_MN) {
                    TmaLoad2D(sw, &tmW, &fullBar[stage], kb * kBK, col0);
                } else {
#pragma unroll
                    for (int j = 0; j < 2; ++j) TmaLoad2D(sw + j * (64 * kBK * 2), &tmW, &fullBar[stage], col0 + j * 64, kb * kBK);
                }
                if (!X_MN) {
                    TmaLoad2D(sx, &tmX, &fullBar[stage], kb * kBK, row0);
                } else {
                    for (int j = 0; j < g.bt / 64; ++j) TmaLoad2D(sx + j * (64 * kBK * 2), &tmX, &fullBar[stage], row0 + j * 64, kb * kBK);
                }
                if (++stage == g.stages) { stage = 0; phase ^= 1u; }
            }
            if (!ok) { *gaveUp = 1; GiveUp(g.ctl); }
        }
    } else if (warp == 1) {
        if (ElectOne()) {
            const uint32_t idesc = InstrDescF16(128, g.bt, true, W_MN, X_MN);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kFirst; kb < kLast; ++kb) {
                ok = MbarWait(&fullBar[stage], phase, abortWord, g.waitLimitNs);
                if (!ok) break;
                TcFenceAfter();
                const uint32_t sw = SmemAddr(smem + stage * stageBytes);
                const uint32_t sx = sw + kSplitWBytes;
                const uint64_t dw = W_MN ? SmemDescMnMajor(sw, 64 * kBK * 2) : SmemDescKMajor(sw);
                const uint64_t dx = X_MN ? SmemDescMnMajor(sx, 64 * kBK * 2) : SmemDescKMajor(sx);
#pragma unroll
                for (int k = 0; k < kBK / kUmmaK; ++k) {
                    const uint64_t wStep = (uint64_t)((W_MN ? kUmmaK * 128 : kUmmaK * 2) >> 4) * k;
                    const uint64_t xStep = (uint64_t)((X_MN ? kUmmaK * 128 : kUmmaK * 2) >> 4) * k;
                    UmmaF16(tmemBase, dw + wStep, dx + xStep, idesc, (kb != kFirst || k != 0) ? 1u : 0u);
                }
                UmmaCommit(&emptyBar[stage]);
                if (++stage == g.stages) { stage = 0; phase ^= 1u; }
            }
            if (ok) UmmaCommit(tmemFull);
            else { *gaveUp = 1; GiveUp(g.ctl); }
        }
    } else {
        // accumulator lanes = weight rows (output columns), accumulator columns = tokens; the MMAs that read the ring
        // have completed, so the partial tile may take its place
        const int quarter = warp & 3, lane = threadIdx.x & 31;
        if (__all_sync(0xFFFFFFFFu, MbarWait(tmemFull, 0, abortWord, g.waitLimitNs))) {
            TcFenceAfter();
            const uint32_t taddr = tmemBase + ((uint32_t)(quarter * 32) << 16);
            float* part = reinterpret_cast<float*>(smem) + quarter * 32 + lane;
            for (int c = 0; c < g.bt; c += 16) {
                uint32_t v[16];
                TmemLd32x16(taddr + (uint32_t)c, v);
                TmemLdWait();
#pragma unroll
                for (int j = 0; j < 16; ++j) part[(c + j) * 128] = __uint_as_float(v[j]);
            }
            TcFenceBefore();
        } else if (lane == 0) {
            *gaveUp = 1;
            GiveUp(g.ctl);
        }
    }
    __syncthreads();
    if (split > 1) SplitClusterSync();               // every CTA's partial is in its shared memory
    {
        // this CTA's share of the tokens: every CTA's piece of 4 columns is requested before the first is added
        const int tokens = (g.M - row0) < g.bt ? (g.M - row0) : g.bt;
        const int t0 = tokens * crank / split, t1 = tokens * (crank + 1) / split;
        const uint32_t base = SmemAddr(smem);
        uint32_t lost = 0;
#pragma unroll
        for (int r = 0; r < kSplitMaxCluster; ++r)
            if (r < split) lost |= LdCluster1(SmemAddr(const_cast<uint32_t*>(gaveUp)), (uint32_t)r);
        for (int i = t0 * 32 + (int)threadIdx.x; i < t1 * 32; i += kThreads) {
            const int t = i >> 5, c = (i & 31) * 4;
            float4 p[kSplitMaxCluster];
#pragma unroll
            for (int r = 0; r < kSplitMaxCluster; ++r)
                if (r < split) p[r] = LdCluster4(base + (uint32_t)(t * 128 + c) * 4, (uint32_t)r);
            float4 s = p[0];
#pragma unroll
            for (int r = 1; r < kSplitMaxCluster; ++r)
                if (r < split) { s.x += p[r].x; s.y += p[r].y; s.z += p[r].z; s.w += p[r].w; }
            if (col0 + c < g.N && lost == 0) {         // N is a multiple of 8
                __nv_bfloat162 lo = __floats2bfloat162_rn(s.x, s.y), hi = __floats2bfloat162_rn(s.z, s.w);
                *reinterpret_cast<uint2*>(g.out + (size_t)(row0 + t) * g.N + col0 + c) =
                    make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            }
        }
    }
    __syncthreads();
    if (split > 1) SplitClusterSync();               // nobody leaves while a peer still reads its partial
    if (warp == 1) {
        TcFenceAfter();
        TmemDealloc(tmemBase, tmemCols);
    }
}

}  // namespace mc2
}  // namespace hccl
