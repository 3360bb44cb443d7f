// Expert-parallel MoE dispatch and combine (sm_100a).
//
// HCCL serves MoE expert parallelism with AlltoAllV / AlltoAllVC
// (src/ops/all_to_all_v, staging protocol aiv_all_to_all_v_mesh_1D.h:105-266);
// token permutation, quantisation and the weighted sum run as separate operators
// around it.  Here the two directions are ONE kernel each:
//   dispatch  count exchange -> per (token, expert) slot assignment -> the token row is read once, quantised to
//             fp8 e4m3 with one fp32 scale per 1x128 block, and written straight into the destination rank's
//             receive buffer, grouped by local expert and, inside an expert, by source rank (ready for a grouped
//             GEMM); the variable per-peer counts never go through the host
//   combine   every rank pulls the expert outputs of its own tokens from the peers' (symmetric) output buffers and
//             accumulates sum_k gate[t, k] * y[slot(t, k)] in fp32 -> bf16, in token order: permutation back,
//             transfer and gate-weighted sum in one pass, no intermediate buffer
// Synchronisation, epochs, bounded waits: the same block-row protocol as the collectives (dev_comm.cuh).
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include "coll_bodies.cuh"
#include "launch.h"
#include "moe_launch.h"
#include "../core/log.h"
#include "../core/per_device.h"

namespace hccl {

namespace {

constexpr int kMoeThreads = 512;
constexpr int kMoeWarps = kMoeThreads / 32;

// ------------------------------------------------------------------ count + local positions
// counts[e] = number of (token, k) pairs routed to global expert e; pos[t * K + k] = rank of the pair among this
// rank's pairs for the same expert.  Up to kMoeCountInDispatch pairs (a decode step) the dispatch kernel does this itself
// (CountPairs); then up to kMoeCountOneBlock pairs (a short prompt) one block counts in shared memory and writes every count;
// more pairs are spread over blocks that share cleared global counters.
constexpr int kMoeCountOneBlock = 16384;
__global__ void __launch_bounds__(1024) MoeCountOneBlockKernel(const int32_t* __restrict__ topkIdx, int nPairs, int nExperts, uint32_t* __restrict__ counts,
                                                               uint32_t* __restrict__ pos)
{
    __shared__ uint32_t s_count[kMoeMaxExperts];
    for (int e = threadIdx.x; e < nExperts; e += blockDim.x) s_count[e] = 0;
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < nPairs; i += blockDim.x) {
        const int e = topkIdx[i];
        pos[i] = (e >= 0 && e < nExperts) ? atomicAdd(&s_count[e], 1u) : 0xFFFFFFFFu;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nExperts; e += blockDim.x) counts[e] = s_count[e];
}
__global__ void MoeCountKernel(const int32_t* __restrict__ topkIdx, int nPairs, int nExperts, uint32_t* __restrict__ counts,
                               uint32_t* __restrict__ pos)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nPairs; i += gridDim.x * blockDim.x) {
        const int e = topkIdx[i];
        pos[i] = (e >= 0 && e < nExperts) ? atomicAdd(&counts[e], 1u) : 0xFFFFFFFFu;
    }
}

// The same inside one block for up to kMoeCountInDispatch pairs, in an order that depends on the pairs alone, so that every
// block of a launch counts for itself and all agree: a warp takes a run of consecutive pairs, 32 at a time (lanes with the
// same expert find each other by match.any), and a scan over the warps' counters gives each run its start.  It saves the
// counting launch in front (2.1 .. 2.9 us and the boundary between the two) for 1 .. 5 us of the dispatch kernel; up to where that
// pays stands beside kMoeCountInDispatch.  Eight emulated ranks, whose counting launches run one after the other, take 1149 -> 1120
// us for a whole layer of 256 tokens.
struct CountScratch {
    uint16_t before[kMoeWarps][kMoeMaxExperts];       // pairs of an expert in a warp's run, then in the runs before it
    uint16_t pos[kMoeCountInDispatch];                // position of a pair among the pairs of its expert in its warp's run
    uint32_t count[kMoeMaxExperts];
};
__device__ __forceinline__ int CountRun(int nPairs) { return ((nPairs + kMoeWarps - 1) / kMoeWarps + 31) / 32 * 32; }
__device__ __forceinline__ void CountPairs(const int32_t* __restrict__ topkIdx, int nPairs, int nExperts, CountScratch& s)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, run = CountRun(nPairs);
    for (int e = lane; e < nExperts; e += 32) s.before[warp][e] = 0;
    __syncwarp();
    for (int i0 = warp * run; i0 < min((warp + 1) * run, nPairs); i0 += 32) {
        const int i = i0 + lane, e = i < nPairs ? topkIdx[i] : -1;
        const bool ok = e >= 0 && e < nExperts;
        const uint32_t same = __match_any_sync(0xffffffffu, ok ? e : -1), below = same & ((1u << lane) - 1u);
        const uint16_t start = ok ? s.before[warp][e] : 0;
        __syncwarp();
        if (ok && below == 0) s.before[warp][e] = (uint16_t)(start + __popc(same));
        if (ok) s.pos[i] = (uint16_t)(start + __popc(below));
        __syncwarp();
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nExperts; e += kMoeThreads) {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < kMoeWarps; ++w) {
            const uint16_t n = s.before[w][e];
            s.before[w][e] = (uint16_t)sum;
            sum += n;
        }
        s.count[e] = sum;
    }
    __syncthreads();
}

// ------------------------------------------------------------------ dispatch
// Bound by the bytes written (topk fp8 copies of every row, over NVLink to the peers).  A WARP owns a token, or a part of
// one while there are warps for it: a lane takes 16 elements of the row (two 16-byte loads), eight lanes share a
// 128-element block's maximum, and the lane quantises its 16 elements in registers and stores them to all topk
// destinations, 512 contiguous bytes per warp and destination.  No block-wide step inside a token, so all warps' loads and
// stores overlap.  Measured against a block per token with three barriers, 8 emulated ranks, rows of 7168, top-8: 256 tokens
// (150 MB) 133 -> 52 us, 64 82 -> 33, 8 72 -> 28, 1 28 -> 17 (with whole tokens only 49, 41, 36 and 34 us).  A stretch of a row is
// requested while the one before it is quantised and stored, a warp's first one before the block counts and waits for its
// peers: 256 tokens 47.7 -> 41.4 us, 64 19.4 -> 19.3, rows of 5120 with top-2 21.7 -> 21.7.
struct DispatchBody {
    using Args = MoeDispatchArgs;
    static constexpr int kThreads = kMoeThreads;
    __device__ static void Run(const DevComm& c, const Args& a, int b, int nb)
    {
        __shared__ uint32_t s_cnt[kMaxDevRanks * kMoeMaxExperts];   // [src][expert]
        __shared__ uint32_t s_base[kMoeMaxExperts];                 // slot base in the destination rank for (expert, src = me)
        __shared__ CountScratch s_pairs;
        OpHead(c, b);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        // Token rows.  16 elements per lane: nPiece is a multiple of 8 (hidden is one of 128).  A warp requests the first stretch of its
        // first item before it counts and waits for the peers.
        const int H = a.hidden, nScale = H / 128, nPiece = H / 16;
        constexpr int U = 2;                                        // pieces a lane requests at a time
        const int nStretch = (nPiece + 32 * U - 1) / (32 * U);
        const int parts = min(max(nb * kMoeWarps / max(a.nTokens, 1), 1), nStretch), perPart = (nStretch + parts - 1) / parts;
        const uint32_t items = (uint32_t)a.nTokens * parts;         // at most eight parts of rows that fit the GPU: far below 2^32
        uint4 ahead[U][2];
        auto request = [&](int t, int w0) {
            const uint4* row = reinterpret_cast<const uint4*>(a.x + (size_t)t * H);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int w = w0 + u * 32 + lane;
                ahead[u][0] = ahead[u][1] = make_uint4(0, 0, 0, 0);
                if (w < nPiece) { ahead[u][0] = row[2 * w]; ahead[u][1] = row[2 * w + 1]; }
            }
        };
        auto requestItem = [&](uint32_t it) {
            const int t = (int)(it / (uint32_t)parts);
            request(t, ((int)it - t * parts) * perPart * 32 * U);
        };
        if ((uint32_t)(b + warp * nb) < items) requestItem((uint32_t)(b + warp * nb));
        const bool counted = a.counts != nullptr;
        if (!counted) CountPairs(a.topkIdx, a.nTokens * a.topk, a.nExperts, s_pairs);
        const int run = CountRun(a.nTokens * a.topk);
        const int p = c.nRanks, me = c.rank;
        const int E = a.nExperts, perRank = E / p;
        const uint64_t e0 = LoadEpoch(c, b);
        // phase 0: publish my counts in every rank's table, row `me` (each block row owns a private copy of the table)
        for (int i = threadIdx.x; i < p * E; i += kThreads) {
            const int q = i / E, e = i - q * E;
            a.table[q][((size_t)b * kMaxDevRanks + me) * kMoeMaxExperts + e] = counted ? a.counts[e] : s_pairs.count[e];
        }
        bool ok = RankBarrier(c, b, 0, e0 + 1, K_MOE_DISPATCH);
        // phase 1: slot bases.  Destination rank d = e / perRank holds its experts one after the other; inside an expert the
        // sources are ordered by rank.
        const uint32_t* mine = a.table[me] + (size_t)b * kMaxDevRanks * kMoeMaxExperts;
        for (int i = threadIdx.x; i < p * E; i += kThreads) {
            const int s = i / E, e = i - s * E;
            s_cnt[s * kMoeMaxExperts + e] = mine[(size_t)s * kMoeMaxExperts + e];
        }
        __syncthreads();
        // one warp per destination rank scans its experts, 32 at a time
        for (int d = warp; d < p; d += kMoeWarps) {
            uint32_t run = 0;
            for (int le0 = 0; le0 < perRank; le0 += 32) {
                const int le = le0 + lane, e = d * perRank + le;
                uint32_t total = 0, before = 0;
                if (le < perRank) {
                    for (int s = 0; s < p; ++s) {
                        const uint32_t n = s_cnt[s * kMoeMaxExperts + e];
                        total += n;
                        if (s < me) before += n;
                    }
                }
                uint32_t incl = total;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += up;
                }
                const uint32_t off = run + incl - total;            // where the expert starts in rank d's receive buffer
                if (le < perRank) {
                    s_base[e] = off + before;
                    if (b == 0 && d == me) a.recvOffsets[le] = off;  // for the grouped GEMM that follows
                }
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (b == 0 && d == me && lane == 0) {
                a.recvOffsets[perRank] = run;
                if (run > a.capacity) ReportWaitFailure(c, K_MOE_DISPATCH, b, 0, me, a.capacity, run, DEV_ERR_BOUNDS);
            }
        }
        __syncthreads();
        // phase 2: token rows
        for (uint32_t it = b + warp * nb; it < items && ok; it += nb * kMoeWarps) {
            const int t = (int)(it / (uint32_t)parts), part = (int)it - t * parts;
            // lane k < topk: where the row's k-th copy goes
            uint64_t sm = ~0ull;
            if (lane < a.topk) {
                const int pair = t * a.topk + lane;
                const int e = a.topkIdx[pair];
                if (e >= 0 && e < E) sm = ((uint64_t)(e / perRank) << 32) | (uint64_t)(s_base[e] + (counted ? a.pos[pair] : (uint32_t)s_pairs.before[pair / run][e] + s_pairs.pos[pair]));
                if (part == 0) a.slotMap[pair] = sm;
                if (sm != ~0ull && (uint32_t)sm >= a.capacity) sm = ~0ull;      // overflow: reported by the receiver's bounds check above
                if (sm != ~0ull && part == 0) a.recvSrc[sm >> 32][(uint32_t)sm] = ((uint64_t)me << 32) | (uint32_t)pair;
            }
            const int begin = part * perPart * 32 * U, end = min(begin + perPart * 32 * U, nPiece);
            const uint32_t next = it + nb * kMoeWarps;
            if (begin >= end && next < items) requestItem(next);    // the parts before this one cover the row
            for (int w0 = begin; w0 < end; w0 += 32 * U) {
                uint4 raw[U][2];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    raw[u][0] = ahead[u][0];
                    raw[u][1] = ahead[u][1];
                }
                // the next stretch, of this item or the warp's next one, is on its way while this one is quantised and stored
                if (w0 + 32 * U < end) request(t, w0 + 32 * U);
                else if (next < items) requestItem(next);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int w = w0 + u * 32 + lane;
                    float f[16];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u][j]);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float2 v = __bfloat1622float2(h[k]);
                            f[j * 8 + 2 * k] = v.x;
                            f[j * 8 + 2 * k + 1] = v.y;
                        }
                    }
                    float amax = 0.f;
#pragma unroll
                    for (int k = 0; k < 16; ++k) amax = fmaxf(amax, fabsf(f[k]));
                    // 8 consecutive lanes cover one block of 128
#pragma unroll
                    for (int o = 4; o >= 1; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                    const float scale = fmaxf(amax, 1e-10f) / 448.f;
                    const float inv = 1.f / scale;
                    uint32_t outw[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j] * inv, f[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
                        const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j + 2] * inv, f[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
                        outw[j] = (uint32_t)lo | ((uint32_t)hi << 16);
                    }
                    const uint4 q = make_uint4(outw[0], outw[1], outw[2], outw[3]);
                    for (int k = 0; k < a.topk; ++k) {
                        const uint64_t to = __shfl_sync(0xffffffffu, sm, k);
                        if (to == ~0ull || w >= nPiece) continue;
                        reinterpret_cast<uint4*>(a.recvX[to >> 32] + (size_t)(uint32_t)to * H)[w] = q;
                        if ((lane & 7) == 0) a.recvScale[to >> 32][(size_t)(uint32_t)to * nScale + w / 8] = scale;
                    }
                }
            }
        }
        RankBarrier(c, b, 0, e0 + 2, K_MOE_DISPATCH);
        StoreEpoch(c, b, e0 + 2);
        OpTail(c, b);
    }
};

// ------------------------------------------------------------------ combine
// A pull over NVLink, bound by the bytes in flight.  Work item of a WARP: pieces (32 vectors of 16 bytes) of one token's row,
// whole rows where there are tokens enough, else as many parts as finish first.  Every thread owns a ring
// of kCombineRing vectors in shared memory that asynchronous copies fill, 3 pieces of 8 copies (or 6 of 4, 12 of 2) ahead of
// the arithmetic; it reads what it copied itself, so there is no hand-over.  The ring keeps up to 192 KiB per SM requested all
// the time, where loads into registers (8 a thread: sixteen spilled) had 64 KiB, and nothing between a piece's sum and the
// next piece's loads.  Lane k keeps the k-th copy's address and weight and hands them round by shuffle.
// Measured against loads into registers, 8 emulated ranks, rows of 7168, top-8: 256 tokens (264 MB, the expert rows still being
// written back) 83.6 -> 73.5 us, 64 50.4 -> 34.1, 8 41.9 -> 29.2, 1 16.4 -> 15.9; rows of 4096, top-2: 256 29.6 -> 28.4, 1 14.9 -> 14.0.
constexpr int kCombineRing = 24;                                    // vectors per thread
constexpr size_t kCombineSmem = (size_t)kCombineRing * kMoeThreads * 16;
struct CombineBody {
    using Args = MoeCombineArgs;
    static constexpr int kThreads = kMoeThreads;
    template <int COPIES>
    __device__ static void Tokens(const Args& a, int b, int nb)
    {
        extern __shared__ __align__(16) uint8_t s_ring[];
        constexpr int D = kCombineRing / COPIES;
        const int H = a.hidden, vecPerRow = H / 8, nPieces = (vecPerRow + 31) / 32;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const uint32_t stride = (uint32_t)nb * kMoeWarps;
        // parts per row: lane l weighs l + 1 of them by rounds of all warps x (pieces of a part + about two for its addresses)
        static_assert(kMoeMaxHidden / 8 <= 32 * 32, "no row has more pieces, and so parts to weigh, than a warp has lanes");
        const uint32_t p = (uint32_t)lane + 1, rounds = ((uint32_t)a.nTokens * p + stride - 1) / stride;
        const uint32_t cost = p <= (uint32_t)nPieces ? rounds * (((uint32_t)nPieces + p - 1) / p + 2) : 0x3FFFFFFu;      // rows fit the GPU: far below 2^26
        const uint32_t parts = (__reduce_min_sync(0xffffffffu, min(cost, 0x3FFFFFFu) << 6 | (uint32_t)lane) & 63u) + 1;
        const uint32_t items = (uint32_t)a.nTokens * parts;
        const int perItem = (int)((nPieces + parts - 1) / parts);
        const uint8_t* mine = s_ring + threadIdx.x * 16;            // slot s of this thread: s * kMoeThreads vectors further
        const uint32_t mineAddr = (uint32_t)__cvta_generic_to_shared(mine);
        for (uint32_t it = b + warp * nb; it < items; it += stride) {
            const int t = (int)(it / parts), first = (int)(it - t * parts) * perItem, n = min(perItem, nPieces - first);
            float wk = 0.f;
            unsigned long long srcK = 0;                            // 0: the copy was dropped
            if (lane < a.topk) {
                const uint64_t sm = a.slotMap[(size_t)t * a.topk + lane];
                if (sm != ~0ull && (uint32_t)sm < a.capacity) {
                    wk = a.topkWeight[(size_t)t * a.topk + lane];
                    srcK = reinterpret_cast<unsigned long long>(a.y[sm >> 32] + (size_t)(uint32_t)sm * H);
                }
            }
            const uint32_t have = __ballot_sync(0xffffffffu, srcK != 0);
            auto fetch = [&](int j) {                               // piece j of the item -> ring slots (j % D) * COPIES ..
                const int v = (first + j) * 32 + lane;
#pragma unroll
                for (int k = 0; k < COPIES; ++k) {
                    const uint4* src = reinterpret_cast<const uint4*>(__shfl_sync(0xffffffffu, srcK, k));
                    if (j < n && src != nullptr && v < vecPerRow)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(mineAddr + (uint32_t)((j % D) * COPIES + k) * kMoeThreads * 16), "l"(src + v) : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            for (int j = 0; j < D - 1; ++j) fetch(j);
            for (int j = 0; j < n; ++j) {
                fetch(j + D - 1);                                   // into the slots of piece j - 1, which is summed
                asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
                const int v = (first + j) * 32 + lane;
                float acc[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll
                for (int k = 0; k < COPIES; ++k) {
                    const float w = __shfl_sync(0xffffffffu, wk, k);
                    if (have >> k & 1u) {
                        const uint4 raw = *reinterpret_cast<const uint4*>(mine + (size_t)((j % D) * COPIES + k) * kMoeThreads * 16);
                        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 f = __bfloat1622float2(h[e]);
                            acc[2 * e] += w * f.x;
                            acc[2 * e + 1] += w * f.y;
                        }
                    }
                }
                if (v < vecPerRow) {
                    uint4 o;
                    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                    for (int e = 0; e < 4; ++e) oh[e] = __floats2bfloat162_rn(acc[2 * e], acc[2 * e + 1]);
                    reinterpret_cast<uint4*>(a.out + (size_t)t * H)[v] = o;
                }
            }
        }
    }
    __device__ static void Run(const DevComm& c, const Args& a, int b, int nb)
    {
        OpHead(c, b);
        const uint64_t e0 = LoadEpoch(c, b);
        if (RankBarrier(c, b, 0, e0 + 1, K_MOE_COMBINE)) {          // the peers' expert outputs are final
            if (a.topk > 4) Tokens<8>(a, b, nb);
            else if (a.topk > 2) Tokens<4>(a, b, nb);
            else Tokens<2>(a, b, nb);
        }
        RankBarrier(c, b, 0, e0 + 2, K_MOE_COMBINE);                 // nobody overwrites its outputs while a peer still reads
        StoreEpoch(c, b, e0 + 2);
        OpTail(c, b);
    }
};
static_assert(kMoeMaxTopk == 8, "CombineBody picks its copies by topk");

template <class Body>
HcclResult LaunchMoe(const LaunchTarget& t, const typename Body::Args& a, int nBlocks, size_t smem)
{
    static OncePerDevice allowed;
    if (smem > 0)
        CHK_RET(allowed([&]() -> HcclResult {
            CHK_CUDA(cudaFuncSetAttribute(CollKernel<Body>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            CHK_CUDA(cudaFuncSetAttribute(CollKernelEmu<Body>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            return HCCL_SUCCESS;
        }));
    if (t.emu != nullptr)
        return t.emu->Post(t.emuRank, &a, sizeof(a), nBlocks, Body::kThreads, reinterpret_cast<const void*>(&CollKernelEmu<Body>), t.stream, smem);
    CollKernel<Body><<<nBlocks, Body::kThreads, smem, t.stream>>>(*t.dev, a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { HCCL_ERROR("MoE kernel launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

}  // namespace

HcclResult LaunchMoeCount(const int32_t* topkIdx, int nPairs, int nExperts, uint32_t* counts, uint32_t* pos, cudaStream_t stream)
{
    if (nPairs <= kMoeCountOneBlock) {
        MoeCountOneBlockKernel<<<1, 1024, 0, stream>>>(topkIdx, nPairs, nExperts, counts, pos);
        return cudaGetLastError() == cudaSuccess ? HCCL_SUCCESS : HCCL_E_RUNTIME;
    }
    CHK_CUDA(cudaMemsetAsync(counts, 0, sizeof(uint32_t) * (size_t)nExperts, stream));
    const int blocks = nPairs >= 1 << 16 ? 64 : 16;
    MoeCountKernel<<<blocks, 256, 0, stream>>>(topkIdx, nPairs, nExperts, counts, pos);
    return cudaGetLastError() == cudaSuccess ? HCCL_SUCCESS : HCCL_E_RUNTIME;
}
HcclResult LaunchMoeDispatch(const LaunchTarget& t, const MoeDispatchArgs& a, int nBlocks) { return LaunchMoe<DispatchBody>(t, a, nBlocks, 0); }
HcclResult LaunchMoeCombine(const LaunchTarget& t, const MoeCombineArgs& a, int nBlocks) { return LaunchMoe<CombineBody>(t, a, nBlocks, kCombineSmem); }

}  // namespace hccl

// ------------------------------------------------------------------ expert offsets (local routing helper)
#include "moe_route.cuh"
#include "hccl/hccl_moe.h"

extern "C" HcclResult HcclMoeExpertOffsets(const int32_t* topkIdx, uint64_t nPairs, uint32_t nExperts, uint32_t* offsets, hcclStream_t stream)
{
    using namespace hccl;
    CHK_PTR_NULL(topkIdx);
    CHK_PTR_NULL(offsets);
    if (nExperts == 0 || nExperts > kRouteMaxExperts) { HCCL_ERROR("HcclMoeExpertOffsets: 1..%u experts supported (got %u)", kRouteMaxExperts, nExperts); return HCCL_E_PARA; }
    return LaunchDependent(MoeExpertOffsetsKernel, kRouteCtas, kRouteThreads, 0, (cudaStream_t)stream, 0, topkIdx, nPairs, nExperts, offsets) == cudaSuccess
               ? HCCL_SUCCESS : HCCL_E_RUNTIME;
}
