// Plain matmul for outputs too small to fill the chip with 256-wide tiles (decode steps, short prompts): the inner
// dimension is split over the CTAs of a cluster and the partial tiles are added through distributed shared memory.
//
// What bounds these shapes is the weight stream from HBM: at 16 tokens x 8192 x 8192 a pass reads 134 MB of weights for
// 2 GFLOP.  A one-tile-per-SM kernel leaves most SMs idle (64 tiles of 128 columns) and pads the tokens to a 128-row
// operand.  So here
//   * the WEIGHT is the 128- or 64-row operand of tcgen05.mma (cta_group::1) and the tokens are the narrow one (N = bt, a multiple
//     of 16): a stage is 16 or 8 KiB of weights plus bt * 128 bytes of activations;
//   * a cluster of `split` CTAs (at most 8) works on one 128 x bt tile, CTA r on the r-th share of the k-blocks.  Long streams of
//     weights want about two CTAs per SM: the stage ring takes at most half of an SM's shared memory, so that one CTA's start and
//     end run under its neighbour's main loop.  Outputs of few tiles are bound by what one CTA gets through (a k-block of 64 takes
//     0.14 us however small its tile is): there the cut has more CTAs, smaller tiles and a ring as large as an SM (PlanMatmul);
//   * alone on its tile, a CTA stores it straight from tensor memory.  Otherwise each CTA leaves its fp32 partial in its own shared
//     memory ([token][column], the idle stage ring) and, after one cluster barrier, CTA r adds its share of the tokens over all
//     CTAs in rank order (one fixed order, no atomics, no workspace) and stores them as bf16.  The order depends on the number of
//     CTAs per tile and so on the shape: a row's fp32 sum may differ in its last place from that of a call with more rows.
// The drain is a serial chain of a few warps: with more than 32 tokens eight warps share it, and a tile that nobody shares does not
// pass through shared memory (101 x 288 x 72 5.2 -> 2.8 us, 128 x 2048 x 512 7.0 -> 3.4).  Sending the partials to their owner
// instead of fetching them was slower (128 x 10240 x 8192 35.6 against 34.4 us).
// Measured against the one-SM kernel on 128 x 128 tiles (us, bf16, weight [N, K]): 16 x 8192 x 8192 47.5 -> 26.8 (5.0
// TB/s), 64 x 8192 x 8192 48.4 -> 28.8; against its 256-wide form 16 x 57344 x 8192 160.6 -> 142.4 (6.6 TB/s), 64 x 57344 x 8192
// 162.3 -> 151.0.  Clusters of at most four, 128 x 128 tiles and 108 KiB rings -> chosen per shape (back to back in a graph): 128 x 2048 x
// 8192 18.2 -> 11.4 (3.4 TB/s), 128 x 1024 x 8192 13.8 -> 9.2, 16 x 1024 x 8192 7.5 -> 5.7, 64 x 4096 x 8192 17.7 -> 14.9, 128 x 8192 x 1024
// 9.4 -> 5.6, 64 x 2048 x 512 5.1 -> 3.6, 128 x 4096 x 4096 14.6 -> 11.4, 33 x 128 x 13048 15.9 -> 10.0.
// Warp roles and waits are those of the other kernels (mc2_gemm.cuh): warp 0 TMA producer, warp 1 MMA issuer, warps 2-5
// or 2-9 drain the accumulator; every wait is bounded, and a CTA that gave one up tells its cluster, or the warps of its
// own that would store, and nothing of the tile is stored: what its shared memory holds is no partial sum.
#pragma once
#include "mc2_gemm.cuh"

namespace hccl {
namespace mc2 {

constexpr int kSplitMaxBt = 128;
constexpr int kSplitMaxCluster = 8;               // the portable cluster size
constexpr int kSplitMaxThreads = 320;
constexpr int kSplitMaxStages = 12;
constexpr int kSplitRingBytes = 108 * 1024;                  // two CTAs per SM
constexpr int kSplitLoneRingBytes = 200 * 1024;              // one CTA per SM
// One warp per quarter of the accumulator lanes to drain it, 16 tokens at a time; two where there is more to drain and no neighbour on the
// SM whose main loop runs meanwhile.  128 x 8192 x 1024 6.33 us with one, 5.64 with two; 32 x 8192 x 256 3.10 and 2.78; in clusters, whose CTAs drain
// into shared memory, only from 32 tokens on (20 x 1728 x 3064 5.50 and 5.62); with a neighbour 64 x 10240 x 8192 30.04 and 30.30.
inline int SplitThreads(int tokens, int split, int ringBytes)
{
    return tokens <= (split == 1 ? 16 : 32) || ringBytes == kSplitRingBytes ? 192 : kSplitMaxThreads;
}
constexpr int kSplitBarBytes = 256;

struct SplitArgs {
    int M, N, K;               // out[M, N] = X[M, K] x W[N, K]^T   (operand storage is described by the tensor maps)
    __nv_bfloat16* out;
    int bt;                    // tokens per tile
    int tilesM;                // token tiles; the tile index runs over them first, so that they share a weight tile in L2
    int stages;
    int barOffset;             // barriers behind the ring and the partial tile
    uint32_t* ctl;             // control block: the abort word of bounded waits
    uint64_t waitLimitNs;      // of every wait
    int stalledCta;            // tests: this CTA's producer loads nothing (-1: none)
};

__host__ __device__ constexpr int SplitStageBytes(int bt, int wr) { return (wr + bt) * kBK * 2; }
inline int SplitStages(int bt, int wr, int ringBytes)
{
    const int n = ringBytes / SplitStageBytes(bt, wr);
    return n < kSplitMaxStages ? n : kSplitMaxStages;
}
// The ring also has to hold the CTA's fp32 partial tile.
__host__ __device__ constexpr int SplitPartialBytes(int bt, int wr) { return bt * wr * 4; }
inline int SplitBarOffset(int bt, int wr, int stages, int split)
{
    const int ring = stages * SplitStageBytes(bt, wr), partial = split > 1 ? SplitPartialBytes(bt, wr) : 0;
    return ring > partial ? ring : partial;
}
inline int SplitSmemBytes(int barOffset) { return barOffset + kSplitBarBytes + 1024; }      // + slack for the 1024-byte alignment
constexpr int kSplitMaxSmemBytes = kSplitLoneRingBytes + kSplitBarBytes + 1024;
static_assert(SplitPartialBytes(kSplitMaxBt, 128) <= kSplitRingBytes, "the largest partial tile is no larger than the ring");
static_assert((2 * kSplitMaxStages + 1) * 8 + 8 <= kSplitBarBytes, "barriers, tensor memory address and flag");

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

// This CTA's share of the tokens: the partial tiles of the cluster's R CTAs added in rank order, every CTA's piece of 4 columns
// requested before the first is added.
template <int R, int WR>
__device__ __forceinline__ void SplitAddPartials(const SplitArgs& g, uint8_t* smem, uint32_t* gaveUp, int crank, int tokens, int row0, int col0)
{
    uint32_t lost = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) lost |= LdCluster1(SmemAddr(gaveUp), (uint32_t)r);
    constexpr int quadBits = WR == 128 ? 5 : 4;
    const int t0 = tokens * crank / R, t1 = tokens * (crank + 1) / R;
    const uint32_t base = SmemAddr(smem);
#pragma unroll 1
    for (int i = (t0 << quadBits) + (int)threadIdx.x; i < t1 << quadBits; i += (int)blockDim.x) {
        const int t = i >> quadBits, c = (i - (t << quadBits)) * 4;
        float4 p[R];
#pragma unroll
        for (int r = 0; r < R; ++r) p[r] = LdCluster4(base + (uint32_t)i * 16, (uint32_t)r);
        float4 a = p[0];
#pragma unroll
        for (int r = 1; r < R; ++r) { a.x += p[r].x; a.y += p[r].y; a.z += p[r].z; a.w += p[r].w; }
        if (col0 + c < g.N && lost == 0) {               // N is a multiple of 8
            const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
            *reinterpret_cast<uint2*>(g.out + (size_t)(row0 + t) * g.N + col0 + c) =
                make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        }
    }
}

// One kernel for every height of a weight tile (WR) and cluster size (R), with loops that are not unrolled over tokens: what a launch of a
// few microseconds fetches of its code shows.  As values of the launch they cost 0.1 .. 0.3 us (us, values -> kernels: 16 x 7168 x 2048 8.27 -> 8.14, 256 x 128 x 8192
// 6.38 -> 6.18, 128 x 2048 x 8192 11.74 -> 11.37, 64 x 10240 x 8192 30.67 -> 30.26, 128 x 8192 x 1024 5.83 -> 5.61).
template <bool W_MN, bool X_MN, int WR, int R>
__global__ void __launch_bounds__(kSplitMaxThreads, 2) GemmSplitKernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SplitArgs g)
{
    extern __shared__ uint8_t smemRaw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
    const int stageBytes = SplitStageBytes(g.bt, WR);
    constexpr int wBytes = WR * kBK * 2;
    uint64_t* fullBar = reinterpret_cast<uint64_t*>(smem + g.barOffset);
    uint64_t* emptyBar = fullBar + kSplitMaxStages;
    uint64_t* tmemFull = fullBar + 2 * kSplitMaxStages;
    uint32_t* tmemBaseSlot = reinterpret_cast<uint32_t*>(fullBar + 2 * kSplitMaxStages + 1);
    volatile uint32_t* gaveUp = tmemBaseSlot + 1;      // a role of this CTA left before its work was done
    volatile uint32_t* abortWord = g.ctl + kCtlAbort;

    const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const int crank = R == 1 ? 0 : (int)SplitClusterRank();
    const int tile = (int)blockIdx.x / R;
    const int row0 = (tile % g.tilesM) * g.bt, col0 = (tile / g.tilesM) * WR;
    const int kBlocks = (g.K + kBK - 1) / kBK;
    const int kFirst = (int)((long long)kBlocks * crank / R), kLast = (int)((long long)kBlocks * (crank + 1) / R);
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
    bool drained = false;                              // epilogue warps: the accumulator is complete

    if (warp == 0) {
        if (ElectOne()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kFirst; kb < kLast && (int)blockIdx.x != g.stalledCta; ++kb) {
                ok = MbarWait(&emptyBar[stage], phase ^ 1u, abortWord, g.waitLimitNs);
                if (!ok) break;
                uint8_t* sw = smem + stage * stageBytes;
                uint8_t* sx = sw + wBytes;
                MbarExpectTx(&fullBar[stage], (uint32_t)stageBytes);
                if (!W_MN) {
                    TmaLoad2D(sw, &tmW, &fullBar[stage], kb * kBK, col0);
                } else {
                    TmaLoad2D(sw, &tmW, &fullBar[stage], col0, kb * kBK);
                    if (WR > 64) TmaLoad2D(sw + 64 * kBK * 2, &tmW, &fullBar[stage], col0 + 64, kb * kBK);
                }
                if (!X_MN) {
                    TmaLoad2D(sx, &tmX, &fullBar[stage], kb * kBK, row0);
                } else {
                    TmaLoad2D(sx, &tmX, &fullBar[stage], row0, kb * kBK);
                    if (g.bt > 64) TmaLoad2D(sx + 64 * kBK * 2, &tmX, &fullBar[stage], row0 + 64, kb * kBK);
                }
                if (++stage == g.stages) { stage = 0; phase ^= 1u; }
            }
            if (!ok) { *gaveUp = 1; GiveUp(g.ctl); }
        }
    } else if (warp == 1) {
        if (ElectOne()) {
            const uint32_t idesc = InstrDescF16(WR, g.bt, true, W_MN, X_MN);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kFirst; kb < kLast; ++kb) {
                ok = MbarWait(&fullBar[stage], phase, abortWord, g.waitLimitNs);
                if (!ok) break;
                TcFenceAfter();
                const uint32_t sw = SmemAddr(smem + stage * stageBytes);
                const uint32_t sx = sw + wBytes;
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
        drained = __all_sync(0xFFFFFFFFu, MbarWait(tmemFull, 0, abortWord, g.waitLimitNs));
        TcFenceAfter();
        if (!drained && lane == 0) { *gaveUp = 1; GiveUp(g.ctl); }
    }
    // accumulator lanes = weight rows (output columns), accumulator columns = tokens; two warps per quarter of the lanes take
    // every second stretch of 16 tokens
    const int tokens = (g.M - row0) < g.bt ? (g.M - row0) : g.bt;
    const int quarter = warp & 3, part = (warp - 2) >> 2, threads = (int)blockDim.x, chunkStep = (threads - 64) / 8;
    const uint32_t taddr = tmemBase + ((uint32_t)(quarter * 32) << 16);
    const bool odd = (lane & 1) != 0;
    // 64 rows lie in the first 16 lanes of every quarter
    constexpr int perQuarter = WR / 4;
    const int myRow = quarter * perQuarter + lane;
    const bool hasRow = lane < perQuarter;
    if (R == 1) {
        // straight to memory: a pair of lanes swaps halves, so that each stores two columns of every second token.  All of the tile or nothing:
        // of two warps that wait for the same accumulator, one may have given up just before it was complete.
        __syncthreads();
        drained = drained && *gaveUp == 0;
        const int col = hasRow ? col0 + (myRow & ~1) : g.N;
#pragma unroll 1
        for (int c = part * 16; drained && c < tokens; c += chunkStep) {
            uint32_t v[16];
            TmemLd32x16(taddr + (uint32_t)c, v);
            TmemLdWait();
            __nv_bfloat16* o = g.out + (size_t)(row0 + c + (odd ? 1 : 0)) * g.N + col;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float even0 = __uint_as_float(v[2 * j]), odd0 = __uint_as_float(v[2 * j + 1]);
                const float other = __shfl_xor_sync(0xFFFFFFFFu, odd ? even0 : odd0, 1);
                const __nv_bfloat162 two = odd ? __floats2bfloat162_rn(other, odd0) : __floats2bfloat162_rn(even0, other);
                if (c + 2 * j + (odd ? 1 : 0) < tokens && col < g.N) *reinterpret_cast<__nv_bfloat162*>(o + (size_t)(2 * j) * g.N) = two;
            }
        }
        TcFenceBefore();
        __syncthreads();                                 // the accumulator is read
    } else {
        // every CTA leaves its partial tile in its own idle ring, [token][column], before the cluster meets
        float* mine = reinterpret_cast<float*>(smem) + myRow;
#pragma unroll 1
        for (int c = part * 16; drained && c < tokens; c += chunkStep) {
            uint32_t v[16];
            TmemLd32x16(taddr + (uint32_t)c, v);
            TmemLdWait();
            if (hasRow) {
#pragma unroll
                for (int j = 0; j < 16; ++j) mine[(c + j) * WR] = __uint_as_float(v[j]);
            }
        }
        TcFenceBefore();
        __syncthreads();
        SplitClusterSync();
        SplitAddPartials<R, WR>(g, smem, const_cast<uint32_t*>(gaveUp), crank, tokens, row0, col0);
        __syncthreads();
        SplitClusterSync();                              // nobody leaves while a peer still reads its partial
    }
    if (warp == 1) {
        TcFenceAfter();
        TmemDealloc(tmemBase, tmemCols);
    }
}

}  // namespace mc2
}  // namespace hccl
