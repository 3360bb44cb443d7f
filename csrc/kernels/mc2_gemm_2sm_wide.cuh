// Wide-tile variant of the two-SM matmul (plain matmul only): a CTA pair works on 256 rows x TWO adjacent column
// tiles, one in each of its two TMEM accumulators, so that a k-block of A is loaded once for 512 output columns
// instead of once for 256.
//
// Why: a GPU at its power limit finishes a matmul when the matmul's energy has been spent, and with 256 x 256 tiles the
// shared-memory fill traffic from L2 (64 KiB per pair and k-block) is a large part of what is spent beyond the tensor
// cores.  The wide tile needs 48 KiB per CTA and k-block for twice the math (A 16 KiB + two B halves of 16 KiB): a
// quarter less L2 -> SM traffic per FLOP.
//
// Both accumulators belong to the tile in flight, so the epilogue can only overlap if the two halves end at different
// times.  They are skewed by `skew` k-blocks: the left half runs k-blocks [0, skew) alone, both run [skew, K) together,
// the right half catches up with [0, skew) alone.  The left accumulator is drained under the right half's catch-up, the
// right one under the next tile's left-only stretch; the price is `skew` k-blocks of A loaded twice per tile.
//
// Work items: full rounds of wide tiles over all pairs, then the rest as single 256-row x one-column-tile items in
// alternating accumulators, so the launch takes as many column-tile times as the narrow kernel.  Left-over positions give
// a pair at most two singles, an odd last column tile adds one per row tile, spread over the pairs.
//
// A column's sum runs over k in the order 0 .. K where it is a left half or a single item, and skew .. K, 0 .. skew where
// it is a right half: results depend on the shape of the product (not on timing) in the last place of their fp32 sums.
//
// Pipeline: four stages of 48 KiB; otherwise the roles, barriers and hand-over of mc2_gemm_2sm.cuh (full[stage] in
// the leader, empty[stage] and tmemFull[acc] per CTA through the multicast commit, tmemEmpty[acc] in the leader with
// eight arrivals).
#pragma once
#include "mc2_gemm_2sm.cuh"

namespace hccl {
namespace mc2 {

constexpr int kStagesWide = 4;
struct SmemLayoutWide {
    static constexpr int kABytes = kBM * kBK * 2;            // 16 KiB: this CTA's 128 rows of A
    static constexpr int kBBytes = (kBN2 / 2) * kBK * 2;     // 16 KiB: this CTA's half of ONE column tile of B
    static constexpr int kStageBytes = kABytes + 2 * kBBytes;
    static constexpr int kTileBytes = kStagesWide * kStageBytes;   // 192 KiB
    static constexpr int kStagingOff = kTileBytes + 256;
    static constexpr int kTotal = kStagingOff + kEpilogueStagingBytes + 1024;
};

constexpr int kWideSkew = 12;                         // k-blocks: about the time 256 accumulator columns take to drain

// Item t of the launch -> what a pair does.  Full rounds of wide tiles come first: `wide` of them, a multiple of the
// pairs; a wide position that is left over becomes two singles, an odd last column tile one.
struct WideItem { int mt2, nt; bool both; int acc; };
struct WideOrder {
    int tilesM2, cols, tilesN, positions, wide, items, nPairs, group;
    __host__ __device__ WideOrder(int tilesM2_, int tilesN_, int nPairs_, int group_)
        : tilesM2(tilesM2_), cols(tilesN_ / 2), tilesN(tilesN_), positions(tilesM2_ * (tilesN_ / 2)), nPairs(nPairs_), group(group_)
    {
        wide = positions / nPairs * nPairs;
        items = wide + 2 * (positions - wide) + (tilesN & 1) * tilesM2;
    }
    // grouped raster over (256-row tile, pair of column tiles): bands of `group` row tiles, rows fastest
    __host__ __device__ void Position(int q, int* mt2, int* col) const
    {
        GroupedTile(q, tilesM2, cols, group, mt2, col);
    }
    __host__ __device__ WideItem Get(int t) const
    {
        WideItem w;
        int col;
        if (t < wide) {
            Position(t, &w.mt2, &col);
            w.nt = 2 * col; w.both = true; w.acc = 0;
            return w;
        }
        const int s = t - wide, split = 2 * (positions - wide);
        w.both = false;
        w.acc = (s / nPairs) & 1;                      // this pair's singles take the accumulators in turn
        if (s < split) {
            Position(wide + s / 2, &w.mt2, &col);
            w.nt = 2 * col + (s & 1);
        } else {
            w.mt2 = s - split;
            w.nt = tilesN - 1;
        }
        return w;
    }
};

template <bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    GemmKernel2SmWide(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g)
{
    using L = SmemLayoutWide;
    extern __shared__ uint8_t smemRaw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kTileBytes);
    uint64_t* fullBar = bars;                          // [kStagesWide]  (used in the leader)
    uint64_t* emptyBar = bars + kStagesWide;           // [kStagesWide]
    uint64_t* tmemFull = bars + 2 * kStagesWide;       // [2]
    uint64_t* tmemEmpty = bars + 2 * kStagesWide + 2;  // [2]            (used in the leader)
    uint32_t* tmemBaseSlot = reinterpret_cast<uint32_t*>(bars + 2 * kStagesWide + 4);
    volatile uint32_t* abortWord = g.ctl + kCtlAbort;

    const int warp = threadIdx.x / 32;
    const int cta = (int)blockIdx.x;
    const uint32_t crank = ClusterCtaRank();

    constexpr uint32_t kTmemCols = 2 * kBN2;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStagesWide; ++s) { MbarInit(&fullBar[s], 1); MbarInit(&emptyBar[s], 1); }
        for (int a = 0; a < 2; ++a) { MbarInit(&tmemFull[a], 1); MbarInit(&tmemEmpty[a], 2 * (kEpilogueThreads / 32)); }
        MbarInitFence();
        PrefetchTensorMap(&tmA);
        PrefetchTensorMap(&tmB);
    }
    if (warp == 1) {
        TmemAlloc2(tmemBaseSlot, kTmemCols);
        TmemRelinquish2();
    }
    TcFenceBefore();
    __syncthreads();
    ClusterSync();
    TcFenceAfter();
    const uint32_t tmemBase = *tmemBaseSlot;
    AllowDependents();
    DependencyWait();
    const int BN = g.bn;
    const int pair = cta >> 1, nPairs = g.nGemmCtas >> 1;
    const int kBlocks = (g.K + kBK - 1) / kBK;
    const WideOrder order((g.M + 255) / 256, g.tilesN, nPairs, g.rasterGroup > 0 ? g.rasterGroup : kRasterGroup);
    const int skew = kBlocks / 2 < kWideSkew ? kBlocks / 2 : kWideSkew;

    if (warp == 0) {
        // ===== TMA producer (both CTAs)
        if (ElectOne()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            // whole boxes of 64 columns for an MN-major half tile of B (see mc2_gemm_2sm.cuh)
            const uint32_t bHalfBytes = (uint32_t)((B_MN ? (BN / 2 + 63) / 64 * 64 : BN / 2) * kBK * 2);
            for (int t = pair; t < order.items && ok; t += nPairs) {
                const WideItem w = order.Get(t);
                const int mt = w.mt2 * 2 + (int)crank;
                // steps of a wide item: left only, both, right only; of a single one: its column tile only
                const int steps = w.both ? kBlocks + skew : kBlocks;
                for (int i = 0; i < steps; ++i) {
                    const bool left = !w.both || i < kBlocks, right = w.both && i >= skew;
                    const int kb = i < kBlocks ? i : i - kBlocks;
                    ok = MbarWait(&emptyBar[stage], phase ^ 1u, abortWord, kWaitLimitNs);
                    if (!ok) break;
                    uint8_t* sa = smem + stage * L::kStageBytes;
                    const uint32_t leaderFull = SmemAddr(&fullBar[stage]) & kPeerBitMask;
                    if (crank == 0) MbarExpectTx(&fullBar[stage], 2u * ((uint32_t)L::kABytes + (left && right ? 2u : 1u) * bHalfBytes));
                    if (!A_MN) {
                        TmaLoad2D2Sm(sa, &tmA, leaderFull, kb * kBK, mt * kBM);
                    } else {
#pragma unroll
                        for (int j = 0; j < kBM / 64; ++j) TmaLoad2D2Sm(sa + j * (64 * kBK * 2), &tmA, leaderFull, mt * kBM + j * 64, kb * kBK);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (!(h == 0 ? left : right)) continue;
                        uint8_t* sb = sa + L::kABytes + h * L::kBBytes;
                        const int nRow = (w.nt + h) * BN + (int)crank * (BN / 2);
                        if (!B_MN) {
                            TmaLoad2D2Sm(sb, &tmB, leaderFull, kb * kBK, nRow);
                        } else {
#pragma unroll
                            for (int j = 0; j < (kBN2 / 2) / 64; ++j)
                                if (j * 64 < BN / 2) TmaLoad2D2Sm(sb + j * (64 * kBK * 2), &tmB, leaderFull, nRow + j * 64, kb * kBK);
                        }
                    }
                    if (++stage == kStagesWide) { stage = 0; phase ^= 1u; }
                }
            }
            if (!ok) GiveUp(g.ctl);
        }
    } else if (warp == 1) {
        // ===== MMA issuer: leader CTA only
        if (crank == 0 && ElectOne()) {
            const uint32_t idesc = InstrDescF16(256, BN, true, A_MN, B_MN);
            int stage = 0;
            uint32_t phase = 0;
            uint32_t accPhase[2] = {0, 0};
            bool ok = true;
            for (int t = pair; t < order.items && ok; t += nPairs) {
                const WideItem w = order.Get(t);
                const int steps = w.both ? kBlocks + skew : kBlocks;
                const int first = w.both ? 0 : w.acc;      // accumulator of the left (or only) half
                for (int i = 0; i < steps; ++i) {
                    const bool left = !w.both || i < kBlocks, right = w.both && i >= skew;
                    if (i == 0) ok = MbarWait(&tmemEmpty[first], accPhase[first] ^ 1u, abortWord, kWaitLimitNs);
                    if (ok && w.both && i == skew) ok = MbarWait(&tmemEmpty[1], accPhase[1] ^ 1u, abortWord, kWaitLimitNs);
                    if (ok) ok = MbarWait(&fullBar[stage], phase, abortWord, kWaitLimitNs);
                    if (!ok) break;
                    TcFenceAfter();
                    const uint32_t sa = SmemAddr(smem + stage * L::kStageBytes);
                    const uint64_t da = A_MN ? SmemDescMnMajor(sa, 64 * kBK * 2) : SmemDescKMajor(sa);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (!(h == 0 ? left : right)) continue;
                        const uint32_t sb = sa + L::kABytes + h * L::kBBytes;
                        const uint64_t db = B_MN ? SmemDescMnMajor(sb, 64 * kBK * 2) : SmemDescKMajor(sb);
                        const uint32_t tmemD = tmemBase + (uint32_t)((h == 0 ? first : 1) * kBN2);
                        const int start = h == 0 ? 0 : skew;
#pragma unroll
                        for (int k = 0; k < kBK / kUmmaK; ++k) {
                            const uint64_t aStep = (uint64_t)((A_MN ? kUmmaK * 128 : kUmmaK * 2) >> 4) * k;
                            const uint64_t bStep = (uint64_t)((B_MN ? kUmmaK * 128 : kUmmaK * 2) >> 4) * k;
                            UmmaF16_2Sm(tmemD, da + aStep, db + bStep, idesc, (i != start || k != 0) ? 1u : 0u);
                        }
                    }
                    UmmaCommit2Sm(&emptyBar[stage]);
                    if (i == kBlocks - 1) { UmmaCommit2Sm(&tmemFull[first]); accPhase[first] ^= 1u; }
                    if (w.both && i == steps - 1) { UmmaCommit2Sm(&tmemFull[1]); accPhase[1] ^= 1u; }
                    if (++stage == kStagesWide) { stage = 0; phase ^= 1u; }
                }
            }
            if (!ok) GiveUp(g.ctl);
        }
    } else {
        // ===== epilogue warps 2..5 of both CTAs: each CTA drains its own 128 accumulator rows
        const int quarter = warp & 3;
        const int lane = threadIdx.x & 31;
        uint32_t accPhase[2] = {0, 0};
        bool ok = true;
        for (int t = pair; t < order.items && ok; t += nPairs) {
            const WideItem w = order.Get(t);
            const int row0 = (w.mt2 * 2 + (int)crank) * kBM + quarter * 32;
            uint8_t* stg = smem + L::kStagingOff + quarter * kStgWarpBytes;
            for (int h = 0; h < (w.both ? 2 : 1); ++h) {
                const int acc = w.both ? h : w.acc, nt = w.nt + h;
                ok = __all_sync(0xFFFFFFFFu, MbarWait(&tmemFull[acc], accPhase[acc], abortWord, kWaitLimitNs));
                if (!ok) break;
                TcFenceAfter();
                const uint32_t taddr = tmemBase + (uint32_t)(acc * kBN2) + ((uint32_t)(quarter * 32) << 16);
                DrainTileRows(taddr, BN, stg, lane, g.N - nt * BN, g.M - row0, g.out + (size_t)row0 * g.ldc + (size_t)nt * BN, (size_t)g.ldc);
                TcFenceBefore();
                __syncwarp();
                if (lane == 0) MbarArriveCluster(SmemAddr(&tmemEmpty[acc]) & kPeerBitMask);
                accPhase[acc] ^= 1u;
            }
        }
        if (!ok && lane == 0) GiveUp(g.ctl);
    }
    TcFenceBefore();
    __syncthreads();
    ClusterSync();
    if (warp == 1) {
        TcFenceAfter();
        TmemDealloc2(tmemBase, kTmemCols);
    }
}

}  // namespace mc2
}  // namespace hccl
