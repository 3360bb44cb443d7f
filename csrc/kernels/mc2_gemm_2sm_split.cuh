// Two-SM matmul with the inner dimension split over a cluster (plain matmul only): `split` CTA pairs work on one
// 256 x bn output tile, pair q on the q-th share of the k-blocks, and add their partial tiles through distributed shared
// memory.  One tile per cluster; stages as small as the tile allows, so that a 128-wide one has eight in flight.
//
// For outputs of 129 rows and more that give the CTA pairs no tile each (or just one): there a pair is bound by the latency and
// the rate of its own loads (24 KiB per SM and k-block of a 128-wide tile: 0.20 us, while the math takes 0.14), and by what
// comes before and after them, about 5 us a launch.  So the inner dimension is cut until most SMs have a share, and the drain,
// with no other tile's math to hide under, has eight warps.
// Partial sums go to the pair that owns their columns with stores into its idle stage ring (remote loads there wait for a
// round trip each: 2 .. 4 us more), and are added in pair order.
// Measured before -> after (us, back to back, weight [N, K]): 256 x 8192 x 8192 38.0 -> 34.0, 200 x 8192 x 8192 37.8 -> 33.3,
// 512 x 4096 x 4096 20.4 -> 18.4, 1000 x 2048 x 8192 34.0 -> 29.0 (one pair per tile); 256 x 4096 x 4096 16.7 -> 14.6, 300 x
// 2048 x 4096 14.7 -> 13.5, 1024 x 1024 x 16384 36.7 -> 31.3 (two); 256 x 2048 x 8192 20.9 -> 17.1 (three); 1000 x 2048 x 2048
// 12.6 -> 12.4, 256 x 1024 x 2048 8.9 -> 8.7; shorter inner dimensions lose: 256 x 1024 x 1024 6.1 -> 7.6.
#pragma once
#include "mc2_gemm_2sm.cuh"
#include "mc2_gemm_splitk.cuh"

namespace hccl {
namespace mc2 {

constexpr int kSplit2MaxPairs = 4;                 // clusters of at most eight CTAs, the portable size
constexpr int kSplit2MaxStages = 8;
constexpr int kSplit2RingBytes = 192 * 1024;
constexpr int kSplit2EpilogueWarps = 8;            // two per quarter of the accumulator rows
constexpr int kSplit2Threads = 64 + 32 * kSplit2EpilogueWarps;
constexpr int kSplit2StgRowBytes = 64 + 16, kSplit2StgWarpBytes = 32 * kSplit2StgRowBytes;      // 32 rows x 32 columns of bf16, padded

struct Split2Args {
    int M, N, K;               // out[M, N] = A[M, K] x B[K, N]   (operand storage is described by the tensor maps)
    __nv_bfloat16* out;
    int bn;                    // column tile width, a multiple of 32, at most 256 (launched with 128 and 256)
    int tilesM2, tilesN;
    int stages;
    uint32_t* ctl;             // control block: the abort word of bounded waits
    uint64_t waitLimitNs;      // of every wait
    int stalledCta;            // tests: this CTA's producer loads nothing (-1: none)
};

// A stage of one CTA: its 128 rows of A and its half of the tile's B rows (MN-major: whole boxes of 64 columns).
__host__ __device__ constexpr int Split2BBytes(int bn, bool bMn) { return (bMn ? (bn / 2 + 63) / 64 * 64 : bn / 2) * kBK * 2; }
inline int Split2Stages(int bn, bool bMn)
{
    const int n = kSplit2RingBytes / (SmemLayout2::kABytes + Split2BBytes(bn, bMn));
    return n < kSplit2MaxStages ? n : kSplit2MaxStages;
}
struct SmemLayout2Split {
    static constexpr int kStagingOff = kSplit2RingBytes + 256;
    static constexpr int kTotal = kStagingOff + kSplit2EpilogueWarps * kSplit2StgWarpBytes + 1024;
};

__device__ __forceinline__ void StCluster4(uint32_t localAddr, uint32_t rank, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(localAddr), "r"(rank));
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// First 32-column chunk of a tile that pair q of `split` adds up and stores.
__device__ __forceinline__ int Split2FirstChunk(int bn, int q, int split) { return (bn / 32) * q / split; }

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kSplit2Threads, 1)
    GemmKernel2SmSplit(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Split2Args g)
{
    using L = SmemLayout2Split;
    extern __shared__ uint8_t smemRaw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
    uint64_t* fullBar = reinterpret_cast<uint64_t*>(smem + kSplit2RingBytes);   // [stages]  (used in the pair's leader)
    uint64_t* emptyBar = fullBar + kSplit2MaxStages;                            // [stages]
    uint64_t* tmemFull = fullBar + 2 * kSplit2MaxStages;
    uint32_t* tmemBaseSlot = reinterpret_cast<uint32_t*>(tmemFull + 1);
    volatile uint32_t* gaveUp = tmemBaseSlot + 1;      // a role of this CTA left before its work was done
    volatile uint32_t* abortWord = g.ctl + kCtlAbort;

    const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const int split = (int)SplitClusterSize() / 2, crank = (int)ClusterCtaRank();
    const int pair = crank >> 1, half = crank & 1;     // this CTA: rows half * 128 .. + 127 of the tile, the pair's share of K
    int mt2, nt;
    GroupedTile((int)blockIdx.x / (2 * split), g.tilesM2, g.tilesN, kRasterGroup, &mt2, &nt);
    const int BN = g.bn, mt = mt2 * 2 + half;
    const int kBlocks = (g.K + kBK - 1) / kBK;
    const int kFirst = (int)((long long)kBlocks * pair / split), kLast = (int)((long long)kBlocks * (pair + 1) / split);
    const int bBytes = Split2BBytes(BN, B_MN), stageBytes = SmemLayout2::kABytes + bBytes;
    const uint32_t tmemCols = BN <= 128 ? 128u : 256u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; ++s) { MbarInit(&fullBar[s], 1); MbarInit(&emptyBar[s], 1); }
        MbarInit(tmemFull, 1);
        *gaveUp = 0;
        MbarInitFence();
        PrefetchTensorMap(&tmA);
        PrefetchTensorMap(&tmB);
    }
    if (warp == 1) {
        TmemAlloc2(tmemBaseSlot, tmemCols);
        TmemRelinquish2();
    }
    TcFenceBefore();
    __syncthreads();
    ClusterSync();                                     // the peer's barriers exist before anything arrives on them
    TcFenceAfter();
    const uint32_t tmemBase = *tmemBaseSlot;
    DependencyWait();
    AllowDependents();
    const int quarter = warp & 3, part = (warp - 2) >> 2;      // warps 2..9: rows, and every second chunk of columns
    const uint32_t taddr = tmemBase + ((uint32_t)(quarter * 32) << 16);
    bool drained = false;                              // warps 2..9: the accumulator is complete

    if (warp == 0) {
        // ===== TMA producer: own 128 rows of A, own half of the tile's B rows, completion on the pair leader's barrier
        if (ElectOne()) {
            const int nRow = nt * BN + half * (BN / 2);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kFirst; kb < kLast && (int)blockIdx.x != g.stalledCta; ++kb) {
                ok = MbarWait(&emptyBar[stage], phase ^ 1u, abortWord, g.waitLimitNs);
                if (!ok) break;
                uint8_t* sa = smem + stage * stageBytes;
                uint8_t* sb = sa + SmemLayout2::kABytes;
                const uint32_t leaderFull = SmemAddr(&fullBar[stage]) & kPeerBitMask;
                if (half == 0) MbarExpectTx(&fullBar[stage], (uint32_t)(2 * stageBytes));
                if (!A_MN) {
                    TmaLoad2D2Sm(sa, &tmA, leaderFull, kb * kBK, mt * kBM);
                } else {
#pragma unroll
                    for (int j = 0; j < kBM / 64; ++j) TmaLoad2D2Sm(sa + j * (64 * kBK * 2), &tmA, leaderFull, mt * kBM + j * 64, kb * kBK);
                }
                if (!B_MN) {
                    TmaLoad2D2Sm(sb, &tmB, leaderFull, kb * kBK, nRow);
                } else {
#pragma unroll
                    for (int j = 0; j < (kBN2 / 2) / 64; ++j)
                        if (j * 64 < BN / 2) TmaLoad2D2Sm(sb + j * (64 * kBK * 2), &tmB, leaderFull, nRow + j * 64, kb * kBK);
                }
                if (++stage == g.stages) { stage = 0; phase ^= 1u; }
            }
            if (!ok) { *gaveUp = 1; GiveUp(g.ctl); }
        }
    } else if (warp == 1) {
        // ===== MMA issuer: the leader of every pair
        if (half == 0 && ElectOne()) {
            const uint32_t idesc = InstrDescF16(256, BN, true, A_MN, B_MN);
            const uint16_t both = (uint16_t)(3u << (crank & ~1));
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kb = kFirst; kb < kLast; ++kb) {
                ok = MbarWait(&fullBar[stage], phase, abortWord, g.waitLimitNs);
                if (!ok) break;
                TcFenceAfter();
                const uint32_t sa = SmemAddr(smem + stage * stageBytes), sb = sa + SmemLayout2::kABytes;
                const uint64_t da = A_MN ? SmemDescMnMajor(sa, 64 * kBK * 2) : SmemDescKMajor(sa);
                const uint64_t db = B_MN ? SmemDescMnMajor(sb, 64 * kBK * 2) : SmemDescKMajor(sb);
#pragma unroll
                for (int k = 0; k < kBK / kUmmaK; ++k) {
                    const uint64_t aStep = (uint64_t)((A_MN ? kUmmaK * 128 : kUmmaK * 2) >> 4) * k;
                    const uint64_t bStep = (uint64_t)((B_MN ? kUmmaK * 128 : kUmmaK * 2) >> 4) * k;
                    UmmaF16_2Sm(tmemBase, da + aStep, db + bStep, idesc, (kb != kFirst || k != 0) ? 1u : 0u);
                }
                UmmaCommitPair(&emptyBar[stage], both);
                if (++stage == g.stages) { stage = 0; phase ^= 1u; }
            }
            if (ok) UmmaCommitPair(tmemFull, both);
            else { *gaveUp = 1; GiveUp(g.ctl); }
        }
    } else {
        drained = __all_sync(0xFFFFFFFFu, MbarWait(tmemFull, 0, abortWord, g.waitLimitNs));
        TcFenceAfter();
        if (!drained && lane == 0) { *gaveUp = 1; GiveUp(g.ctl); }
    }
    const int cLo = Split2FirstChunk(BN, pair, split), cHi = Split2FirstChunk(BN, pair + 1, split);
    const int row = quarter * 32 + lane;
    uint32_t lost = 0;
    __syncthreads();
    ClusterSync();                                     // all rings of the cluster are idle: partial sums may take their place
    if (split > 1) {
        // chunks of other pairs go to their owner, slot [sender][float4 of columns][row]: rows are lanes here and where they are
        // read, so both sides are free of bank conflicts
        if (drained) {
            for (int q = 0; q < split; ++q) {
                if (q == pair) continue;
                const int lo = Split2FirstChunk(BN, q, split), hi = Split2FirstChunk(BN, q + 1, split);
                const int slot = pair < q ? pair : pair - 1;
                for (int c = lo + part; c < hi; c += kSplit2EpilogueWarps / 4) {
                    uint32_t v[32];
                    TmemLd32x32(taddr + (uint32_t)(c * 32), v);
                    TmemLdWait();
                    const uint32_t at = SmemAddr(smem) + (uint32_t)((slot * (hi - lo) + (c - lo)) * 8 * kBM + row) * 16;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        StCluster4(at + (uint32_t)(i * kBM * 16), (uint32_t)(2 * q + half), v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
            }
        }
        __syncthreads();
        ClusterSync();                                 // every partial sum is with its owner
    }
    for (int r = 0; r < 2 * split; ++r) lost |= LdCluster1(SmemAddr(const_cast<uint32_t*>(gaveUp)), (uint32_t)r);
    if (warp >= 2 && lost == 0) {
        // own chunks: accumulator + the other pairs' partials, added in pair order, then rows of 64 bytes through the staging area
        uint8_t* stg = smem + L::kStagingOff + (warp - 2) * kSplit2StgWarpBytes;
        const int validCols = g.N - nt * BN, validRows = g.M - mt * kBM - quarter * 32;
        __nv_bfloat16* base = g.out + (size_t)(mt * kBM + quarter * 32) * g.N + (size_t)nt * BN;
        for (int c = cLo + part; c < cHi; c += kSplit2EpilogueWarps / 4) {
            uint32_t v[32];
            TmemLd32x32(taddr + (uint32_t)(c * 32), v);
            TmemLdWait();
            const uint8_t* got = smem + (size_t)((c - cLo) * 8 * kBM + row) * 16;
            const size_t perSlot = (size_t)(cHi - cLo) * 8 * kBM * 16;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 own = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
                float4 s = pair == 0 ? own : *reinterpret_cast<const float4*>(got + i * kBM * 16);
#pragma unroll
                for (int q = 1; q < kSplit2MaxPairs; ++q) {
                    if (q >= split) continue;
                    const float4 p = q == pair ? own : *reinterpret_cast<const float4*>(got + (q < pair ? q : q - 1) * perSlot + i * kBM * 16);
                    s.x += p.x; s.y += p.y; s.z += p.z; s.w += p.w;
                }
                __nv_bfloat162 lo = __floats2bfloat162_rn(s.x, s.y), hi = __floats2bfloat162_rn(s.z, s.w);
                *reinterpret_cast<uint2*>(stg + lane * kSplit2StgRowBytes + i * 8) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            }
            __syncwarp();
            // four 16-byte pieces per row, eight rows at a time
            const int pc = lane & 3, col = c * 32 + pc * 8;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = (lane >> 2) + 8 * k;
                const uint4 o = *reinterpret_cast<const uint4*>(stg + r * kSplit2StgRowBytes + pc * 16);
                if (col < validCols && r < validRows) *reinterpret_cast<uint4*>(base + (size_t)r * g.N + col) = o;
            }
            __syncwarp();
        }
    }
    TcFenceBefore();
    __syncthreads();
    ClusterSync();                                     // nobody leaves while a peer may still read its words or use its TMEM
    if (warp == 1) {
        TcFenceAfter();
        TmemDealloc2(tmemBase, tmemCols);
    }
}

}  // namespace mc2
}  // namespace hccl
