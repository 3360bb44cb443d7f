// Instantiation, tensor-map encoding and launch of the MC2 kernels (sm_100a).
#include "mc2_launch.h"
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <string>
#include <vector>
#include "../core/comm.h"
#include "../core/cuda_driver.h"
#include "../core/log.h"
#include "../core/per_device.h"
#include "mc2_gemm_2sm_wide.cuh"
#include "mc2_gemm_2sm_split.cuh"

namespace hccl {

using namespace mc2;

Mc2State::~Mc2State()
{
    if (ctl) cudaFree(ctl);
    if (resCtxDev) cudaFree(resCtxDev);
    SymFree(&flags);
    SymFree(&xchg);
}

namespace {

static_assert(kGatherStages * (int)kGatherChunk <= SmemLayout<256>::kTileBytes, "gather ring must fit the GEMM tile ring");

// Tensor map of a row-major bf16 matrix [rows, cols] (cols contiguous) with a box of boxCols x boxRows and the
// 128-byte swizzle the UMMA descriptors assume.
HcclResult MakeMap(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint32_t boxRows, uint32_t boxCols)
{
    const DriverApi* d = GetDriverApi();
    if (!d) return HCCL_E_DRV;
    if ((((uintptr_t)ptr) & 15u) != 0 || (cols * 2) % 16 != 0) {
        HCCL_ERROR("matmul operand %p [%llu x %llu] must be 16-byte aligned with a row pitch that is a multiple of 16 bytes", ptr,
                   (unsigned long long)rows, (unsigned long long)cols);
        return HCCL_E_PARA;
    }
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * 2};
    cuuint32_t box[2] = {boxCols, boxRows};
    cuuint32_t estr[2] = {1, 1};
    auto encode = [&] {
        return d->cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = encode();
    // a thread that has made no runtime call which needs a context (autograd's, when a matmul is its first work) has none yet
    int dev = 0;
    if (r == CUDA_ERROR_INVALID_CONTEXT && cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
    if (r != CUDA_SUCCESS) { HCCL_ERROR("cuTensorMapEncodeTiled failed: %s", DriverErrorString(r)); return HCCL_E_DRV; }
    return HCCL_SUCCESS;
}

// A: logical [M, K].  transA == 0: stored [M, K] (K-major).  transA == 1: stored [K, M] (MN-major).
HcclResult MapA(CUtensorMap* map, const void* a, uint64_t m, uint64_t k, bool mnMajor)
{
    return mnMajor ? MakeMap(map, a, k, m, kBK, 64) : MakeMap(map, a, m, k, kBM, kBK);
}
// B: logical [K, N].  transB == 1: stored [N, K] (K-major).  transB == 0: stored [K, N] (MN-major).
HcclResult MapB(CUtensorMap* map, const void* b, uint64_t n, uint64_t k, bool mnMajor, int bn)
{
    return mnMajor ? MakeMap(map, b, k, n, kBK, 64) : MakeMap(map, b, n, k, (uint32_t)bn, kBK);
}

// Lets `kernel` take `bytes` of dynamic shared memory.  KERNEL: its type does not tell kernels of one signature apart.
template <auto KERNEL> HcclResult AllowSharedMemory(int bytes)
{
    static OncePerDevice once;
    return once([&]() -> HcclResult {
        CHK_CUDA(cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        return HCCL_SUCCESS;
    });
}

template <int BN, bool A_MN, bool B_MN, int MODE>
HcclResult LaunchGemm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, const DevComm& c, int grid, bool cooperative,
                      cudaStream_t stream, const CUtensorMap* taOwn = nullptr)
{
    const CUtensorMap& ta2 = taOwn != nullptr ? *taOwn : ta;      // AG: this rank's own shard, read where it is
    constexpr auto kernel = GemmKernel<BN, A_MN, B_MN, MODE>;
    CHK_RET(AllowSharedMemory<kernel>(SmemLayout<BN>::kTotal));
    if (cooperative) {
        void* args[5] = {(void*)&ta, (void*)&tb, (void*)&ta2, (void*)&g, (void*)&c};
        cudaError_t e = cudaLaunchCooperativeKernel((const void*)kernel, dim3((unsigned)grid), dim3(kThreads), args, SmemLayout<BN>::kTotal, stream);
        if (e != cudaSuccess) { HCCL_ERROR("fused matmul launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
        return HCCL_SUCCESS;
    }
    const cudaError_t e = LaunchDependent(kernel, (unsigned)grid, kThreads, SmemLayout<BN>::kTotal, stream, 0, ta, tb, ta2, g, c);
    if (e != cudaSuccess) { HCCL_ERROR("matmul launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

template <bool A_MN, bool B_MN, int MODE>
HcclResult LaunchGemm2Sm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, const DevComm& c, int grid, bool cooperative,
                         cudaStream_t stream, const CUtensorMap* taOwn = nullptr)
{
    const CUtensorMap& ta2 = taOwn != nullptr ? *taOwn : ta;
    constexpr auto kernel = GemmKernel2Sm<A_MN, B_MN, MODE>;
    CHK_RET(AllowSharedMemory<kernel>(SmemLayout2::kTotal));
    cudaError_t e;
    if (cooperative) {
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = SmemLayout2::kTotal;
        cfg.stream = stream;
        cudaLaunchAttribute attrs[1];
        attrs[0].id = cudaLaunchAttributeCooperative;
        attrs[0].val.cooperative = 1;
        cfg.attrs = attrs;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kernel, ta, tb, ta2, g, c);
    } else {
        e = LaunchDependent(kernel, (unsigned)grid, kThreads, SmemLayout2::kTotal, stream, 0, ta, tb, ta2, g, c);
    }
    if (e != cudaSuccess) { HCCL_ERROR("two-SM matmul launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

template <bool A_MN, bool B_MN>
HcclResult LaunchGemm2SmWide(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, int grid, cudaStream_t stream)
{
    constexpr auto kernel = GemmKernel2SmWide<A_MN, B_MN>;
    CHK_RET(AllowSharedMemory<kernel>(SmemLayoutWide::kTotal));
    const cudaError_t e = LaunchDependent(kernel, (unsigned)grid, kThreads, SmemLayoutWide::kTotal, stream, 0, ta, tb, g);
    if (e != cudaSuccess) { HCCL_ERROR("wide two-SM matmul launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

template <bool W_MN, bool X_MN, int WR, int R>
HcclResult LaunchGemmSplit(const CUtensorMap& tw, const CUtensorMap& tx, const SplitArgs& g, const MatmulPlan& p, cudaStream_t stream)
{
    constexpr auto kernel = GemmSplitKernel<W_MN, X_MN, WR, R>;
    CHK_RET(AllowSharedMemory<kernel>(kSplitMaxSmemBytes));
    const cudaError_t e = LaunchDependent(kernel, (unsigned)p.grid, SplitThreads(std::min(g.M, g.bt), p.split, p.ring), (size_t)SplitSmemBytes(g.barOffset), stream, (unsigned)p.split, tw, tx, g);
    if (e != cudaSuccess) { HCCL_ERROR("split matmul launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}
template <bool W_MN, bool X_MN, int WR>
HcclResult LaunchGemmSplit(const CUtensorMap& tw, const CUtensorMap& tx, const SplitArgs& g, const MatmulPlan& p, cudaStream_t stream)
{
    switch (p.split) {
        case 1: return LaunchGemmSplit<W_MN, X_MN, WR, 1>(tw, tx, g, p, stream);
        case 2: return LaunchGemmSplit<W_MN, X_MN, WR, 2>(tw, tx, g, p, stream);
        case 3:                                                  // tiles of 128 rows only (PlanMatmul)
            if constexpr (WR == 128) return LaunchGemmSplit<W_MN, X_MN, WR, 3>(tw, tx, g, p, stream);
            break;
        case 4: return LaunchGemmSplit<W_MN, X_MN, WR, 4>(tw, tx, g, p, stream);
        case 8: return LaunchGemmSplit<W_MN, X_MN, WR, 8>(tw, tx, g, p, stream);
        default: break;
    }
    return HCCL_E_INTERNAL;                                      // no cut of PlanMatmul
}

template <bool A_MN, bool B_MN>
HcclResult LaunchGemm2SmSplit(const CUtensorMap& ta, const CUtensorMap& tb, const Split2Args& g, int tiles, int split, cudaStream_t stream)
{
    constexpr auto kernel = GemmKernel2SmSplit<A_MN, B_MN>;
    CHK_RET(AllowSharedMemory<kernel>(SmemLayout2Split::kTotal));
    const cudaError_t e = LaunchDependent(kernel, (unsigned)(tiles * split * 2), kSplit2Threads, SmemLayout2Split::kTotal, stream, (unsigned)(2 * split), ta, tb, g);
    if (e != cudaSuccess) { HCCL_ERROR("two-SM split matmul launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}
HcclResult DispatchSplit2(bool aMn, bool bMn, const CUtensorMap& ta, const CUtensorMap& tb, const Split2Args& g, int tiles, int split, cudaStream_t s)
{
    if (!aMn && !bMn) return LaunchGemm2SmSplit<false, false>(ta, tb, g, tiles, split, s);
    if (!aMn && bMn) return LaunchGemm2SmSplit<false, true>(ta, tb, g, tiles, split, s);
    if (aMn && !bMn) return LaunchGemm2SmSplit<true, false>(ta, tb, g, tiles, split, s);
    return LaunchGemm2SmSplit<true, true>(ta, tb, g, tiles, split, s);
}

template <int MODE>
HcclResult DispatchLayout2Sm(bool aMn, bool bMn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, const DevComm& c, int grid,
                             bool coop, cudaStream_t s, const CUtensorMap* taOwn = nullptr)
{
    if (!aMn && !bMn) return LaunchGemm2Sm<false, false, MODE>(ta, tb, g, c, grid, coop, s, taOwn);
    if (!aMn && bMn) return LaunchGemm2Sm<false, true, MODE>(ta, tb, g, c, grid, coop, s, taOwn);
    if (MODE == MODE_PLAIN) {
        if (aMn && !bMn) return LaunchGemm2Sm<true, false, MODE_PLAIN>(ta, tb, g, c, grid, coop, s);
        return LaunchGemm2Sm<true, true, MODE_PLAIN>(ta, tb, g, c, grid, coop, s);
    }
    HCCL_ERROR("fused matmul kernels take A in row-major [M, K] form only");
    return HCCL_E_NOT_SUPPORT;
}

// The two-SM (cta_group::2) kernels are the default for tiles of 256 x 256; HCCL_MC2_2SM=0 keeps the one-SM kernels.
bool Use2Sm()
{
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("HCCL_MC2_2SM");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v == 1;
}

// CTAs of a fused launch that move data instead of computing, taken from the GEMM.  HCCL_MC2_AG_WORKERS /
// HCCL_MC2_RS_WORKERS fix the counts (even, 2 .. 64); otherwise:
int ForcedWorkers(bool gather)
{
    static int forced[2] = {-1, -1};
    int& f = forced[gather ? 1 : 0];
    if (f < 0) {
        f = 0;
        const char* e = getenv(gather ? "HCCL_MC2_AG_WORKERS" : "HCCL_MC2_RS_WORKERS");
        if (e != nullptr) {
            const int n = atoi(e) & ~1;
            if (n >= 2 && n <= 64) f = n;
        }
    }
    return f;
}

// Gather workers of AllGather->Matmul are bound by bytes in flight per SM: measured at 8 ranks, 28 workers beat 20 by
// 11 % although the GEMM then needs one wave more, so they take about one SM in five.
int GatherWorkerCtas(int /*tiles*/, int /*ctasPerTile*/)
{
    if (ForcedWorkers(true) > 0) return ForcedWorkers(true);
    const int sms = SmCount() & ~1;
    return std::max(2, sms / 5) & ~1;
}

// Reduce workers of Matmul->ReduceScatter have to finish an output tile in the time the GEMM produces one for them.
// Measured under the GEMM's memory traffic: about 11.5 us per 128 x 256 tile through the switch, about 4.5 us x (P + 1)
// when the P partials are read from local memory; a wave of 256 x 256 GEMM tiles takes about 5 ns x K.  The count
// minimises max(GEMM time, reduction time) inside SMs/9 .. SMs/3; ties go to the fewer workers.
int ReduceWorkerCtas(int gemmTiles, int ctasPerTile, int localTiles128, int k, int nRanks, bool switchReduce)
{
    if (ForcedWorkers(false) > 0) return ForcedWorkers(false);
    const int sms = SmCount() & ~1;
    const int lo = std::max(2, sms / 9) & ~1, hi = std::max(2, sms / 3) & ~1;
    const double tTile = switchReduce ? 11.5 : 4.5 * (nRanks + 1);
    const double tWave = 5e-3 * k * (ctasPerTile == 2 ? 1.0 : 0.5);
    int best = lo;
    double bestCost = 1e30;
    for (int w = lo; w <= hi; w += 2) {
        const int slots = std::max(1, (sms - w) / ctasPerTile);
        const double gemm = (double)((gemmTiles + slots - 1) / slots) * tWave;
        const double reduce = (double)((localTiles128 + w - 1) / w) * tTile;
        const double cost = std::max(gemm, reduce) + tTile;
        if (cost < bestCost - 1e-9) { bestCost = cost; best = w; }
    }
    return best;
}

template <int BN, int MODE>
HcclResult DispatchLayout(bool aMn, bool bMn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& g, const DevComm& c, int grid,
                          bool coop, cudaStream_t s, const CUtensorMap* taOwn = nullptr)
{
    if (!aMn && !bMn) return LaunchGemm<BN, false, false, MODE>(ta, tb, g, c, grid, coop, s, taOwn);
    if (!aMn && bMn) return LaunchGemm<BN, false, true, MODE>(ta, tb, g, c, grid, coop, s, taOwn);
    if (MODE == MODE_PLAIN) {
        if (aMn && !bMn) return LaunchGemm<BN, true, false, MODE_PLAIN>(ta, tb, g, c, grid, coop, s);
        return LaunchGemm<BN, true, true, MODE_PLAIN>(ta, tb, g, c, grid, coop, s);
    }
    HCCL_ERROR("fused matmul kernels take A in row-major [M, K] form only");
    return HCCL_E_NOT_SUPPORT;
}

// Control block for plain matmuls (no communicator): one per device, zeroed once.  `gaveUp` is a word of host memory that a
// kernel sets when one of its waits ran out (GiveUp).
struct PlainCtl { uint32_t* ctl = nullptr; volatile uint32_t* gaveUp = nullptr; };
HcclResult GetPlainCtl(PlainCtl* out)
{
    static std::mutex mu;
    static std::map<int, PlainCtl> perDev;
    std::lock_guard<std::mutex> lk(mu);
    int dev = 0;
    CHK_CUDA(cudaGetDevice(&dev));
    auto it = perDev.find(dev);
    if (it == perDev.end()) {
        uint32_t *ctl = nullptr, *host = nullptr;
        if (cudaHostAlloc((void**)&host, sizeof(uint32_t), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) return HCCL_E_MEMORY;
        if (cudaMalloc(&ctl, kMc2CtlWords * sizeof(uint32_t)) != cudaSuccess) { cudaFreeHost(host); return HCCL_E_MEMORY; }
        *host = 0;
        std::vector<uint32_t> init(kMc2CtlWords, 0);
        const uint64_t address = (uint64_t)(uintptr_t)host;      // one address space: the device uses the host's pointer
        memcpy(&init[kCtlHostWord], &address, sizeof(address));
        // on every stream the first matmul comes after the block is written
        if (cudaMemcpy(ctl, init.data(), kMc2CtlWords * sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
            cudaFree(ctl);
            cudaFreeHost(host);
            return HCCL_E_RUNTIME;
        }
        it = perDev.emplace(dev, PlainCtl{ctl, host}).first;
    }
    *out = it->second;
    return HCCL_SUCCESS;
}
// An earlier matmul on this device gave up a wait: part of its output was not written, and with the abort word up later ones
// would give up early too.  The call that finds it reports it and starts nothing; the next one runs again.
HcclResult ReportGaveUp(const PlainCtl& p, cudaStream_t stream)
{
    HCCL_ERROR("an earlier matmul on this device gave up a wait; part of its output was not written");
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone) {
        *p.gaveUp = 0;
        CHK_CUDA(cudaMemsetAsync(p.ctl + kCtlAbort, 0, sizeof(uint32_t), stream));
    }
    return HCCL_E_TIMEOUT;
}

// Column tile width of a plain two-SM matmul: the one with the least (waves x time of a tile).  A k-block of a 256 x bn tile
// takes as long as bn + 96 columns of math (the rest is the fill of the 128 rows of A and the turn of the ring; measured per
// wave at K = 8192: 34.5, 36.7, 44.8, 47.5 us for 160, 192, 224, 256).  MN-major B is filled in whole boxes of 64 columns, so
// 160, 192 and 224 bring as many bytes as 256 and two thirds of the difference stay (43.1, 43.7, 46.3, 47.0 us); they pay
// where they save a wave: 4096 x 3584 x 8192 217.7 us with 128, 178.6 with 224, 179.6 with 256; 1024 x 28672 x 8192 464.7 us
// with 128, 334.7 with 224; 8192 x 3584 x 4096 228.5 with 128, 165.8 with 224.
int TwoSmColumnTile(int tilesM2, uint64_t n, int pairs, bool bMn)
{
    int best = 256;
    double bestCost = 1e30;
    for (int cand : {256, 224, 192, 160, 128}) {
        const int loaded = bMn ? 2 * ((cand / 2 + 63) / 64 * 64) : cand;
        const int waves = (tilesM2 * (int)((n + cand - 1) / cand) + pairs - 1) / pairs;
        const double cost = (double)waves * ((cand + 2 * loaded) / 3.0 + 96);
        if (cost < bestCost - 1e-9) { bestCost = cost; best = cand; }
    }
    return best;
}

// CTA pairs per tile of a two-SM split launch.  Clusters of four, six and eight CTAs that fill an SM each fit 33, 22 and 15
// times on a B200 (148 SMs in groups that no cluster crosses); more would run one after the other.
int Split2Pairs(int tiles, int pairs)
{
    if (tiles * 74 <= 15 * pairs) return 4;
    if (tiles * 74 <= 22 * pairs) return 3;
    return tiles * 74 <= 33 * pairs ? 2 : 1;
}

HcclResult CheckShapes(uint64_t m, uint64_t n, uint64_t k)
{
    if (m == 0 || n == 0 || k == 0 || m > (1u << 30) || n > (1u << 30) || k > (1u << 30)) return HCCL_E_PARA;
    if (n % 8 != 0 || k % 8 != 0) { HCCL_ERROR("matmul needs N and K to be multiples of 8 (got N=%llu K=%llu)", (unsigned long long)n, (unsigned long long)k); return HCCL_E_PARA; }
    return HCCL_SUCCESS;
}

void FillPeers(CommImpl* comm, GemmArgs* g)
{
    Mc2State* st = comm->mc2.get();
    for (int q = 0; q < comm->nRanks; ++q) {
        g->xchg[q] = (__nv_bfloat16*)st->xchg.peer[q];
        g->tileFlag[q] = (uint64_t*)st->flags.peer[q];
    }
    g->ctl = st->ctl;
    g->maxTiles = kMc2MaxTiles;
    g->xchgParityElems = st->xchgParityBytes / 2;
    g->rank = comm->rank;
    g->nRanks = comm->nRanks;
}

}  // namespace

#ifdef HCCL_MC2_TRACE
// Trace builds only: one timeline buffer per process, dumped as JSON lines (one per CTA) for the launches
// HCCL_MC2_TRACE_FROM .. +2 of each kind into <HCCL_MC2_TRACE_FILE>.rank<r>.jsonl.
namespace {
uint64_t* TraceBuffer(int grid)
{
    static uint64_t* buf = nullptr;
    static int cap = 0;
    if (grid > cap) {
        if (buf) cudaFree(buf);
        if (cudaMalloc(&buf, (size_t)grid * mc2::kTraceWords * sizeof(uint64_t)) != cudaSuccess) { buf = nullptr; cap = 0; return nullptr; }
        cap = grid;
    }
    cudaMemset(buf, 0, (size_t)grid * mc2::kTraceWords * sizeof(uint64_t));
    return buf;
}
void TraceDump(const char* kind, int which, const GemmArgs& g, int grid, cudaStream_t stream)
{
    static int launches[4] = {0, 0, 0, 0};
    static const int from = [] { const char* e = getenv("HCCL_MC2_TRACE_FROM"); return e ? atoi(e) : 8; }();
    const char* prefix = getenv("HCCL_MC2_TRACE_FILE");
    const int n = launches[which]++;
    if (prefix == nullptr || g.trace == nullptr || n < from || n >= from + 3) return;
    cudaStreamSynchronize(stream);
    std::vector<uint64_t> h((size_t)grid * mc2::kTraceWords);
    cudaMemcpy(h.data(), g.trace, h.size() * sizeof(uint64_t), cudaMemcpyDeviceToHost);
    const std::string path = std::string(prefix) + ".rank" + std::to_string(g.rank) + ".jsonl";
    FILE* f = fopen(path.c_str(), "a");
    if (!f) return;
    for (int c = 0; c < grid; ++c) {
        fprintf(f, "{\"kind\": \"%s\", \"launch\": %d, \"rank\": %d, \"cta\": %d, \"M\": %d, \"N\": %d, \"K\": %d, \"bn\": %d, \"w\": [", kind, n, g.rank, c, g.M, g.N, g.K, g.bn);
        for (int i = 0; i < mc2::kTraceWords; ++i) fprintf(f, "%s%llu", i ? ", " : "", (unsigned long long)h[(size_t)c * mc2::kTraceWords + i]);
        fprintf(f, "]}\n");
    }
    fclose(f);
}
}  // namespace
#define MC2_TRACE_ARM(g, grid) (g).trace = TraceBuffer(grid)
#define MC2_TRACE_DUMP(kind, which, g, grid, stream) TraceDump(kind, which, g, grid, stream)
#else
#define MC2_TRACE_ARM(g, grid)
#define MC2_TRACE_DUMP(kind, which, g, grid, stream)
#endif

HcclResult Mc2EnsureState(CommImpl* comm, uint64_t parityBytes)
{
    if (comm->emulated() || comm->hostComm) return HCCL_E_NOT_SUPPORT;
    if (!comm->mc2) {
        std::shared_ptr<Mc2State> st(new Mc2State());
        CHK_CUDA(cudaMalloc(&st->ctl, kMc2CtlWords * sizeof(uint32_t)));
        CHK_CUDA(cudaMemset(st->ctl, 0, kMc2CtlWords * sizeof(uint32_t)));
        CHK_RET(SymAlloc(*comm->bs, comm->device, ((size_t)comm->nRanks * kMc2MaxTiles + kMc2AgBlocks) * sizeof(uint64_t), false, GetEnvConfig().forceIpc, &st->flags));
        comm->mc2 = std::move(st);
    }
    Mc2State* st = comm->mc2.get();
    if (parityBytes > st->xchgParityBytes) {
        // all ranks call with the same shapes, so they all grow together
        CHK_CUDA(cudaDeviceSynchronize());
        SymFree(&st->xchg);
        const uint64_t rounded = (parityBytes + (2u << 20) - 1) / (2u << 20) * (2u << 20);
        // with a multicast alias when the communicator runs NVLS: Matmul->ReduceScatter then reduces in the switch
        CHK_RET(SymAlloc(*comm->bs, comm->device, (size_t)rounded * 2, comm->nvls(), GetEnvConfig().forceIpc, &st->xchg));
        st->xchgParityBytes = rounded;
    }
    return HCCL_SUCCESS;
}

MatmulSwitches MatmulSwitchesOfEnv()
{
    static const MatmulSwitches s = [] {
        MatmulSwitches v;
        const char* hints = getenv("HCCL_MC2_L2_HINTS");
        const char* wide = getenv("HCCL_MC2_WIDE");
        v.twoSm = Use2Sm();
        v.l2Hints = hints != nullptr && hints[0] == '1';
        // the wide kernel takes no hints: asking for them keeps the narrow tiles unless wide ones are asked for as well
        v.wide = wide == nullptr ? (v.l2Hints ? 0 : -1) : (wide[0] == 'a' ? -1 : (wide[0] == '1' ? 1 : 0));
        return v;
    }();
    return s;
}

namespace {

// Estimated time of a small product on each kernel, in us on a B200.  Up to some 50 us a matmul is bound by what one SM takes in
// (a k-block of a tile comes at 110 .. 145 GB/s from L2), by what a k-block costs at least, by a tile's drain and by whole rounds
// of tiles, so the best kernel and cut are those that balance these four.  Fitted to 16000 timed calls (8 .. 8000 rows, 64 .. 16000
// columns, inner dimensions of 64 .. 16000, back to back in a graph): off by 8 % (two-SM), 12 % (one-SM, pairs) and 15 % (token split) in
// the root mean square; taking the best estimate instead of the best time costs 2-3 %.
struct SmallProduct {
    uint64_t m, n, k;
    int kBlocks, sms;
    bool aMn;
    double a, b;               // rows that lie on 16 bytes only, not on 32, take the copy engine 1.6 times as long
    double hbmUs;              // every operand and the output once at 6.3 TB/s
    SmallProduct(uint64_t m, uint64_t n, uint64_t k, bool aMn, bool bMn, int sms)
        : m(m), n(n), k(k), kBlocks((int)((k + kBK - 1) / kBK)), sms(sms), aMn(aMn), a((aMn ? m : k) % 16 != 0 ? 1.6 : 1.0), b((bMn ? n : k) % 16 != 0 ? 1.6 : 1.0),
          hbmUs(2.0 * ((double)m * k + (double)n * k + (double)m * n) / 6.3e6) {}
};
uint64_t CeilDiv(uint64_t a, uint64_t b) { return (a + b - 1) / b; }
double FourNorm(double a, double b) { return std::sqrt(std::sqrt(a * a * a * a + b * b * b * b)); }
// CTAs of `cluster` that run together, one per SM (clusters stay within groups of SMs: 33 of four, 15 of eight on 148)
double ResidentCtas(int cluster, int sms) { return cluster == 8 ? sms * (120. / 148) : (cluster >= 4 ? sms * (132. / 148) : sms); }

double SplitUs(const SmallProduct& s, int bt, int wr, int split, bool* lone)
{
    // rows of MN-major activations with fewer than 64 tokens come in pieces that all CTAs read from the same few lines
    const double block = 0.134 + (s.aMn && s.m < 64 ? 0.45 * (64 - (double)s.m) / 56 : 0);
    const double ctas = (double)(CeilDiv(s.m, bt) * CeilDiv(s.n, wr) * split), resident = ResidentCtas(split, s.sms);
    *lone = ctas <= resident;                                   // one per SM: the ring may take its whole shared memory
    const double rounds = std::ceil(ctas / (resident * (*lone ? 1 : 2))), perSm = *lone ? 1 : std::min(2.0, std::ceil(ctas / resident));
    const int stages = SplitStages(bt, wr, *lone ? kSplitLoneRingBytes : kSplitRingBytes);
    const double kb = std::ceil((double)s.kBlocks / split), tile = perSm * bt * wr / 16384.;
    const double loads = rounds * kb * std::max({block, perSm * (wr * s.b + bt * s.a) * 128 / 143.6e3, 0.134 * 6 / stages});
    const double hbm = 0.88 * s.hbmUs * std::pow(std::max(1.0, s.sms / std::min(ctas, resident)), 0.6);      // fewer SMs keep fewer bytes on their way
    return 2.2 + (wr == 64 ? 0.7 : 0) + std::max(loads, hbm) + rounds * (1.85 * tile + (split > 1 ? 1.1 + 1.1 * tile : 0));
}
double OneSmUs(const SmallProduct& s, int bn)
{
    const double rounds = (double)CeilDiv(CeilDiv(s.m, kBM) * CeilDiv(s.n, bn), s.sms);
    const double loads = s.kBlocks * (128 * s.a + bn * s.b) * 128 / 138.3e3, drain = 0.77 * bn / 128;
    return 0.87 + std::max(s.hbmUs, rounds * FourNorm(loads, drain)) + drain + 0.71 * rounds;
}
double PairsUs(const SmallProduct& s, int bn, int split)
{
    static const double resident[] = {0, 74, 66, 66, 60};       // CTA pairs
    const double rounds = std::ceil((double)(CeilDiv(s.m, 256) * CeilDiv(s.n, bn) * split) / (resident[split] * s.sms / 148));
    const double loads = std::ceil((double)s.kBlocks / split) * (128 * s.a + bn / 2 * s.b) * 128 / 127.2e3, drain = 3.13 * bn / 128;
    return 0.8 + std::max(rounds * (loads + drain + (split > 1 ? 2.47 : 0)), 3.13 + s.hbmUs);
}
double TwoSmUs(const SmallProduct& s, int bn)
{
    const double rounds = (double)CeilDiv(CeilDiv(s.m, 256) * CeilDiv(s.n, bn), s.sms / 2);
    const double loads = s.kBlocks * (128 * s.a + bn / 2 * s.b) * 128 / 123.6e3, drain = 0.68 * bn / 128;
    return 1.97 + std::max(s.hbmUs, rounds * FourNorm(loads, drain)) + drain + 1.48 * rounds;
}
// Another kernel, or another cut for the same one, is taken where its estimate is lower by more than the two are off against each other.
constexpr double kOtherKernel = 0.87, kOtherCut = 0.9;

// Best cut for the token split, its estimate in *us.
MatmulPlan BestSplit(const SmallProduct& s, double* us)
{
    MatmulPlan best;
    *us = 1e30;
    for (int most : {128, 64, 32}) {
        // equal token tiles of at most `most` (MN-major activations come in boxes of 64)
        const int unit = s.aMn ? 64 : 16, parts = (int)CeilDiv(s.m, most);
        const int bt = (int)(CeilDiv(CeilDiv(s.m, parts), unit) * unit);
        if (bt > most || (parts > 1 && parts == (int)CeilDiv(s.m, 2 * most))) continue;
        // smaller token tiles read the weights more often: from L2, where they fit it; 32 tokens were timed up to 128 rows
        if (parts > (int)CeilDiv(s.m, 128) && s.n * s.k * 2 > (64u << 20)) continue;
        if (most == 32 && s.m > 128) continue;
        for (int wr : {128, 64}) {
            if (wr == 64 && s.aMn) continue;
            for (int split : {1, 2, 4, 8}) {
                if (split > 1 && s.kBlocks < 2 * split) break;
                bool lone;
                const double t = SplitUs(s, bt, wr, split, &lone);
                if (t >= *us) continue;
                *us = t;
                best.route = MatmulRoute::SPLIT;
                best.bt = bt;
                best.bn = wr;
                best.tilesM = (int)CeilDiv(s.m, bt);
                best.tilesN = (int)CeilDiv(s.n, wr);
                best.split = split;
                best.grid = best.tilesM * best.tilesN * split;
                best.ring = lone ? kSplitLoneRingBytes : kSplitRingBytes;
            }
        }
    }
    return best;
}
// 256 x 256 tiles shared by two to four CTA pairs, where that takes less than `most`; no plan otherwise.
MatmulPlan BestPairs256(const SmallProduct& s, double most)
{
    MatmulPlan p;
    for (int split = 2; split <= kSplit2MaxPairs; ++split) {
        const double t = s.kBlocks >= 2 * split ? PairsUs(s, 256, split) : 1e30;
        if (t >= most) continue;
        most = t;
        p.route = MatmulRoute::TWO_SM_SPLIT;
        p.bn = 256;
        p.tilesM = (int)CeilDiv(s.m, 256);
        p.tilesN = (int)CeilDiv(s.n, 256);
        p.split = split;
        p.grid = p.tilesM * p.tilesN * 2 * split;
    }
    return p;
}
MatmulPlan OneSmPlan(uint64_t m, uint64_t n, int bn, int sms)
{
    MatmulPlan p;
    p.route = MatmulRoute::ONE_SM;
    p.bn = bn;
    p.tilesM = (int)CeilDiv(m, kBM);
    p.tilesN = (int)CeilDiv(n, bn);
    p.grid = std::min(sms, p.tilesM * p.tilesN);
    return p;
}

}  // namespace

MatmulPlan PlanMatmul(uint64_t m, uint64_t n, uint64_t k, bool aMn, bool bMn, int sms, const MatmulSwitches& sw, uint32_t outAlign)
{
    MatmulPlan p;
    const int tilesM = (int)((m + kBM - 1) / kBM), tilesM2 = (int)((m + 255) / 256);
    const int pairs = (sms & ~1) / 2;
    // narrow: 256-wide column tiles would leave most SMs idle
    const bool narrow = (uint64_t)tilesM * ((n + 255) / 256) < (uint64_t)sms * 3 / 4;
    // Two-SM tiles: outputs that fill the chip with 256 x 256 tiles, and from 129 rows on those that fill four fifths of the
    // pairs with 256 x 128 ones if the inner dimension is long (us, before on the one-SM kernel -> two-SM: 200 x 10240 x
    // 8192 84.5 -> 45.0, 200 x 57344 x 8192 331.0 -> 199.8, 300 x 8192 x 8192 88.1 -> 49.0, 256 x 8192 x 8192 49.2 -> 40.9,
    // 512 x 4096 x 4096 26.6 -> 23.1, 1000 x 2048 x 2048 16.5 -> 16.1; with fewer tiles the split kernel is ahead: 300 x
    // 2048 x 4096 22.4 against 16.5).
    const bool twoSm = sw.twoSm && ((!narrow && m >= 256) || (m > 128 && k >= 2048 && (uint64_t)tilesM2 * ((n + 127) / 128) * 5 >= (uint64_t)pairs * 4));
    // Two-SM tiles with the inner dimension split over a cluster of CTA pairs (see mc2_gemm_2sm_split.cuh): from 129 rows on, where
    // 256 x 128 tiles do not outnumber the pairs and the inner dimension pays for the sum.  At 129 .. 192 rows a quarter and more
    // of the 256 is padding, and with an inner dimension of 4096 and more the token split keeps them.  Token split and pairs, us,
    // back to back: 129 x 4096 x 4096 13.7 and 13.9, x 8192 20.6 and 21.2, x 14336 31.8 and 32.5, 129 x 7168 x 4096 18.5 and 19.1, 160 x
    // 4096 x 4096 13.7 and 13.9.  The line is not the best one: the pairs are ahead at few columns (129 x 1024 x 8192 15.9 and 14.0,
    // 160 x 2048 x 8192 17.2 and 16.3) and from 176 rows on (176 x 4096 x 4096 14.6 and 13.9, 192 x 1024 x 8192 18.4 and 14.1, 192 x 4096 x
    // 14336 35.3 and 32.4); moving it changes the order in which those products are summed.  The token split stores 8 bytes at a time, all other routes 16: an output that lies on 8 bytes only keeps it.
    const uint64_t tiles128 = (uint64_t)tilesM2 * ((n + 127) / 128);
    if (sw.twoSm && outAlign >= 16 && m > 128 && k >= 2048 && tiles128 <= (uint64_t)pairs && (m > 192 || k < 4096 || twoSm)) {
        p.route = MatmulRoute::TWO_SM_SPLIT;
        p.bn = 128;
        p.tilesM = tilesM2;
        p.tilesN = (int)((n + 127) / 128);
        p.split = Split2Pairs((int)tiles128, pairs);
        p.grid = (int)tiles128 * 2 * p.split;
        // long inner dimensions: 256 x 256 tiles, which bring a third fewer bytes per SM, shared by two to four pairs (255 x 5192 x 9888
        // 37.1 -> 29.3 us, 193 x 5256 x 4216 26.6 -> 20.0)
        const SmallProduct s(m, n, k, aMn, bMn, sms);
        double us = PairsUs(s, 128, p.split);
        const MatmulPlan wide = BestPairs256(s, kOtherKernel * us);
        if (wide.grid > 0) return wide;
        // One or two column tiles (a router's logits): token tiles of 64 and clusters of eight keep more SMs busy (256 x 128 x 8192 11.3 -> 6.4
        // us, 244 x 208 x 10520 18.6 -> 10.6, 637 x 72 x 2784 8.7 -> 5.8).  Neither
        // line is where the two cross.  Columns: the token split is ahead up to some thousand, by less (256 x 1024 x 8192 12.9 and 10.5), and a line
        // further out would change the order of sums of projections, not of routers only.  k-blocks: it is ahead at 2048 as well (512 x 128 x 2048 8.0
        // and 5.0); inner dimensions up to 2248 stay because the tests of the pairs' kernel ask for it there, on products small enough to test.
        if (n > 256 || s.kBlocks <= 36) return p;
        const MatmulPlan split = BestSplit(s, &us);
        return us < kOtherKernel * PairsUs(s, 128, p.split) ? split : p;
    }
    // Inner dimension split over clusters: up to 96 rows always (at 128 rows and 57344 columns the 256-wide one-SM tiles win,
    // 166 against 174 us), beyond that where the output leaves SMs idle; from 129 rows on only if the inner dimension is
    // long (400 x 1024 x 1024: 10.3 us against 9.2 on the one-SM kernel, 300 x 2048 x 4096: 16.5 against 24.7).
    if (!twoSm && (m <= 96 || (narrow && (m <= 128 || k >= 4096)))) {
        p.route = MatmulRoute::SPLIT;
        // token tile: all of them up to 128, else equal tiles of at most 128 (MN-major activations come in 64-column boxes)
        const int unit = aMn ? 64 : 16, parts = (int)((m + kSplitMaxBt - 1) / kSplitMaxBt);
        p.bt = ((int)((m + parts - 1) / parts) + unit - 1) / unit * unit;
        p.bn = 128;
        p.tilesM = (int)((m + p.bt - 1) / p.bt);
        p.tilesN = (int)((n + 127) / 128);
        // Two CTAs per SM, at least four k-blocks each (16 x 8192 x 8192: 34.9, 29.7, 26.7 us with 1, 2, 4 CTAs per tile).  Where that is
        // at most one tile for two SMs, another cut if its estimate is clearly lower, or 128 x 128 tiles where many tokens come with
        // a short inner dimension (128 x 8192 x 256: 4.2 us split, 3.5 on the one-SM kernel).
        const int tiles = p.tilesM * p.tilesN, kBlocks = (int)((k + kBK - 1) / kBK);
        p.split = std::max(1, std::min({4, 2 * sms / tiles, kBlocks / 4}));
        p.grid = tiles * p.split;
        bool lone;
        const SmallProduct s(m, n, k, aMn, bMn, sms);
        double us = SplitUs(s, p.bt, p.bn, p.split, &lone);
        p.ring = lone ? kSplitLoneRingBytes : kSplitRingBytes;
        if (tiles * 2 > sms) return p;
        double bestUs;
        const MatmulPlan best = BestSplit(s, &bestUs);
        if (bestUs < kOtherCut * us) { p = best; us = bestUs; }
        return m > 64 && outAlign >= 16 && OneSmUs(s, 128) < kOtherKernel * us ? OneSmPlan(m, n, 128, sms) : p;
    }
    if (!twoSm) {
        p = OneSmPlan(m, n, narrow ? 128 : 256, sms);
        if (!narrow || outAlign < 16) return p;
        double us;
        const SmallProduct s(m, n, k, aMn, bMn, sms);
        const MatmulPlan split = BestSplit(s, &us);
        const double oneSm = OneSmUs(s, p.bn);
        // outputs of more than one round of one-SM tiles that two-SM tiles cover in one (759 x 3824 x 1552 16.4 -> 11.1 us, 269 x 8056 x 1448
        // 21.5 -> 15.3)
        const int bn2 = TwoSmColumnTile(tilesM2, n, pairs, bMn);
        if (sw.twoSm && m > 128 && TwoSmUs(s, bn2) < std::min(us, kOtherKernel * oneSm)) {
            p = MatmulPlan();
            p.route = MatmulRoute::TWO_SM;
            p.bn = bn2;
            p.tilesM = tilesM;
            p.tilesN = (int)CeilDiv(n, bn2);
            p.grid = std::min(2 * pairs, 2 * tilesM2 * p.tilesN);
            return p;
        }
        return us < kOtherKernel * oneSm ? split : p;
    }
    p.bn = TwoSmColumnTile(tilesM2, n, pairs, bMn);
    p.tilesN = (int)((n + p.bn - 1) / p.bn);
    // Wide tiles (two column tiles per CTA pair, see mc2_gemm_2sm_wide.cuh): where at least two full rounds of them run, so
    // that most of the output gains from the saved L2 traffic, and the inner dimension has 48 k-blocks or more, so that the
    // dozen whose A is loaded twice per tile stay a small part.
    const WideOrder order(tilesM2, p.tilesN, pairs, 8);
    if (sw.wide == 1 ? order.wide > 0 : (sw.wide == -1 && order.wide >= 2 * pairs && k >= 48 * kBK)) {
        p.route = MatmulRoute::WIDE;
        p.grid = 2 * pairs;
        p.wide = order.wide;
        p.singles = order.items - order.wide;
        return p;
    }
    // Short inner dimensions, where the drain of a tile is longer than its math: one-SM tiles, of which twice as many are under way
    // (1000 x 4096 x 256 7.1 -> 4.6 us, 2048 x 8192 x 256 15.6 -> 12.1; outputs of more than 2^24 elements were not timed on
    // both and stay).  Long ones with few tiles: 256 x 256 tiles that pairs share (255 x 5192 x 9888 37.1 -> 29.3 us).
    if (!sw.l2Hints && outAlign >= 16 && sw.wide != 1 && m * n <= (1u << 24)) {
        const SmallProduct s(m, n, k, aMn, bMn, sms);
        double best = kOtherKernel * TwoSmUs(s, p.bn);
        MatmulPlan other;
        for (int bn : {128, 256}) {
            const double us = OneSmUs(s, bn);
            if (us < best) { best = us; other = OneSmPlan(m, n, bn, sms); }
        }
        const MatmulPlan pairs256 = BestPairs256(s, best);
        if (pairs256.grid > 0) return pairs256;
        if (other.grid > 0) return other;
    }
    p.route = MatmulRoute::TWO_SM;
    p.grid = std::min(2 * pairs, 2 * tilesM2 * p.tilesN);
    // Raster and L2 policy (experimental, HCCL_MC2_L2_HINTS=1).  About `pairs` tiles are in flight: r row tiles x c
    // column tiles, walking the columns of a band of r rows.  When one operand is small enough to live in L2 next
    // to the stream of the other, it is loaded "evict last", the streamed one "evict first", and the band covers
    // the whole small operand.  Measured on the decoder's matmuls it did not pay (evict-first lines of the
    // streamed operand leave before the other row tiles of the wave have read them), so it is off by default.
    if (sw.l2Hints) {
        const double bytesA = 2.0 * (double)m * (double)k, bytesB = 2.0 * (double)n * (double)k;
        const double fits = 72.0 * (1 << 20);
        if (bytesA <= fits && bytesB > 1.5 * bytesA) {
            p.l2HintA = 1; p.l2HintB = 2;
            p.rasterGroup = std::min(tilesM2, 32);            // all rows of A in one band: B is read once
        } else if (bytesB <= fits && bytesA > 1.5 * bytesB) {
            p.l2HintA = 2; p.l2HintB = 1;
            p.rasterGroup = std::max(1, std::min(8, pairs / std::max(1, p.tilesN)));   // all columns of B in flight together
        }
    }
    return p;
}

// Bytes that a route stores at a time.
uint32_t MatmulOutAlign(const MatmulPlan& plan) { return plan.route == MatmulRoute::SPLIT ? 8 : 16; }

static uint32_t AlignmentOf(const void* p)           // 2, 4, 8, or 16 for more
{
    const uint32_t low = (uint32_t)((uintptr_t)p & 15u);
    return low == 0 ? 16u : (low & (~low + 1u));
}
static HcclResult RefuseOut(const void* out, uint64_t m, uint64_t n, uint64_t k)
{
    HCCL_ERROR("matmul %llu x %llu x %llu: the output at %p must be 16-byte aligned (8 bytes where the output has few tiles)", (unsigned long long)m,
               (unsigned long long)n, (unsigned long long)k, out);
    return HCCL_E_PARA;
}

// Plans of the sizes that this thread multiplied last: weighing the cuts of a small product takes a microsecond of the host.
static MatmulPlan RecentPlan(uint64_t m, uint64_t n, uint64_t k, bool aMn, bool bMn, uint32_t outAlign)
{
    struct Entry { uint64_t m, n, k; int sms; uint32_t form; MatmulPlan plan; };
    static thread_local Entry recent[64] = {};
    const int sms = SmCount();
    const uint32_t form = (aMn ? 1u : 0u) | (bMn ? 2u : 0u) | outAlign << 2;
    Entry& e = recent[((m * 0x9E3779B97F4A7C15ull) ^ (n * 0xC2B2AE3D27D4EB4Full) ^ (k * 0x165667B19E3779F9ull) ^ form) >> 7 & 63u];
    if (e.m != m || e.n != n || e.k != k || e.sms != sms || e.form != form)
        e = {m, n, k, sms, form, PlanMatmul(m, n, k, aMn, bMn, sms, MatmulSwitchesOfEnv(), outAlign)};
    return e.plan;
}

HcclResult Mc2Matmul(const void* a, const void* b, void* out, uint64_t m, uint64_t n, uint64_t k, int transA, int transB, cudaStream_t stream,
                     const Mc2StalledCta* stalled)
{
    CHK_PTR_NULL(a); CHK_PTR_NULL(b); CHK_PTR_NULL(out);
    CHK_RET(CheckShapes(m, n, k));
    const bool aMn = transA != 0, bMn = transB == 0;
    if (aMn && m % 8 != 0) return HCCL_E_PARA;
    const uint32_t outAlign = AlignmentOf(out);
    if (outAlign < 8) return RefuseOut(out, m, n, k);
    PlainCtl plain;
    CHK_RET(GetPlainCtl(&plain));
    if (*plain.gaveUp != 0) return ReportGaveUp(plain, stream);
    const MatmulPlan plan = RecentPlan(m, n, k, aMn, bMn, outAlign);
    if (outAlign < MatmulOutAlign(plan)) return RefuseOut(out, m, n, k);
    if (plan.route == MatmulRoute::SPLIT) {
        SplitArgs g;
        memset(&g, 0, sizeof(g));
        g.M = (int)m; g.N = (int)n; g.K = (int)k;
        g.out = (__nv_bfloat16*)out;
        g.bt = plan.bt;
        g.tilesM = plan.tilesM;
        // all stages also where a CTA has fewer k-blocks: two CTAs of half a ring each would share an SM while others are idle (5 x 15248 x 248
        // 4.4 us with as many stages as k-blocks, 3.5 with all)
        g.stages = SplitStages(g.bt, plan.bn, plan.ring);
        g.barOffset = SplitBarOffset(g.bt, plan.bn, g.stages, plan.split);
        g.ctl = plain.ctl;
        g.waitLimitNs = stalled != nullptr ? stalled->waitLimitNs : kWaitLimitNs;
        g.stalledCta = stalled != nullptr ? stalled->cta : -1;
        CUtensorMap tw, tx;
        CHK_RET(bMn ? MakeMap(&tw, b, k, n, kBK, 64) : MakeMap(&tw, b, n, k, (uint32_t)plan.bn, kBK));
        CHK_RET(aMn ? MakeMap(&tx, a, k, m, kBK, 64) : MakeMap(&tx, a, m, k, (uint32_t)g.bt, kBK));
        if (plan.bn == 64)                                       // never with MN-major tokens (BestSplit)
            return bMn ? LaunchGemmSplit<true, false, 64>(tw, tx, g, plan, stream) : LaunchGemmSplit<false, false, 64>(tw, tx, g, plan, stream);
        if (!bMn && !aMn) return LaunchGemmSplit<false, false, 128>(tw, tx, g, plan, stream);
        if (!bMn && aMn) return LaunchGemmSplit<false, true, 128>(tw, tx, g, plan, stream);
        if (bMn && !aMn) return LaunchGemmSplit<true, false, 128>(tw, tx, g, plan, stream);
        return LaunchGemmSplit<true, true, 128>(tw, tx, g, plan, stream);
    }
    if (stalled != nullptr && plan.route != MatmulRoute::TWO_SM_SPLIT) return HCCL_E_NOT_SUPPORT;
    CUtensorMap ta, tb;
    CHK_RET(MapA(&ta, a, m, k, aMn));
    // two-SM tiles: B is split between the two CTAs of a pair, each loads half of the B rows of a tile
    CHK_RET(MapB(&tb, b, n, k, bMn, plan.route == MatmulRoute::ONE_SM ? plan.bn : plan.bn / 2));
    if (plan.route == MatmulRoute::TWO_SM_SPLIT) {
        Split2Args split;
        memset(&split, 0, sizeof(split));
        split.M = (int)m; split.N = (int)n; split.K = (int)k;
        split.out = (__nv_bfloat16*)out;
        split.bn = plan.bn;
        split.tilesM2 = plan.tilesM;
        split.tilesN = plan.tilesN;
        split.stages = Split2Stages(plan.bn, bMn);
        split.ctl = plain.ctl;
        split.waitLimitNs = stalled != nullptr ? stalled->waitLimitNs : kWaitLimitNs;
        split.stalledCta = stalled != nullptr ? stalled->cta : -1;
        return DispatchSplit2(aMn, bMn, ta, tb, split, plan.tilesM * plan.tilesN, plan.split, stream);
    }
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    g.M = (int)m; g.N = (int)n; g.K = (int)k;
    g.out = (__nv_bfloat16*)out;
    g.ldc = (int)n;
    g.ctl = plain.ctl;
    g.nRanks = 1;
    g.bn = plan.bn;
    g.tilesM = plan.tilesM;
    g.tilesN = plan.tilesN;
    g.nGemmCtas = plan.grid;
    g.rasterGroup = plan.rasterGroup;
    g.l2HintA = plan.l2HintA;
    g.l2HintB = plan.l2HintB;
    DevComm dummy;
    memset(&dummy, 0, sizeof(dummy));
    if (plan.route == MatmulRoute::WIDE) {
        if (!aMn && !bMn) return LaunchGemm2SmWide<false, false>(ta, tb, g, plan.grid, stream);
        if (!aMn && bMn) return LaunchGemm2SmWide<false, true>(ta, tb, g, plan.grid, stream);
        if (aMn && !bMn) return LaunchGemm2SmWide<true, false>(ta, tb, g, plan.grid, stream);
        return LaunchGemm2SmWide<true, true>(ta, tb, g, plan.grid, stream);
    }
    if (plan.route == MatmulRoute::TWO_SM) return DispatchLayout2Sm<MODE_PLAIN>(aMn, bMn, ta, tb, g, dummy, plan.grid, false, stream);
    if (plan.bn == 128) return DispatchLayout<128, MODE_PLAIN>(aMn, bMn, ta, tb, g, dummy, plan.grid, false, stream);
    return DispatchLayout<256, MODE_PLAIN>(aMn, bMn, ta, tb, g, dummy, plan.grid, false, stream);
}

HcclResult Mc2AllGatherMatmul(CommImpl* comm, const void* aShard, const void* b, void* out, void* gathered, uint64_t mPerRank, uint64_t n,
                              uint64_t k, int transB, cudaStream_t stream)
{
    CHK_PTR_NULL(comm); CHK_PTR_NULL(aShard); CHK_PTR_NULL(b); CHK_PTR_NULL(out); CHK_PTR_NULL(gathered);
    const uint64_t P = (uint64_t)comm->nRanks;
    CHK_RET(CheckShapes(mPerRank * P, n, k));
    if (mPerRank % kBM != 0) { HCCL_ERROR("AllGather->Matmul needs rows per rank to be a multiple of %d (got %llu)", kBM, (unsigned long long)mPerRank); return HCCL_E_PARA; }
    if (P * (mPerRank / kBM) > 8 * 512) return HCCL_E_PARA;
    // Push form when the gathered buffer is symmetric memory (every rank writes its shard into the others' buffers;
    // the shard itself may live anywhere); pull form when only the shard is.  HCCL_MC2_AG_PULL=1 keeps the pull form.
    const char* peers[kMaxDevRanks] = {nullptr};
    const char* gathPeers[kMaxDevRanks] = {nullptr};
    static const bool forcePull = [] { const char* e = getenv("HCCL_MC2_AG_PULL"); return e != nullptr && e[0] == '1'; }();
    const bool push = !forcePull && comm->Lookup(gathered, P * mPerRank * k * 2, gathPeers, nullptr);
    if (!push && !comm->Lookup(aShard, mPerRank * k * 2, peers, nullptr)) {
        HCCL_ERROR("AllGather->Matmul: the gathered buffer or the activation shard must live in symmetric memory (HcclMemAlloc)");
        return HCCL_E_PARA;
    }
    CHK_RET(Mc2EnsureState(comm, 0));
    const bool bMn = transB == 0;
    CUtensorMap ta, tb, taOwn;
    CHK_RET(MapA(&ta, gathered, mPerRank * P, k, false));
    CHK_RET(MapA(&taOwn, aShard, mPerRank, k, false));
    CHK_RET(MapB(&tb, b, n, k, bMn, 256));
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    FillPeers(comm, &g);
    g.M = (int)(mPerRank * P); g.N = (int)n; g.K = (int)k;
    g.out = (__nv_bfloat16*)out;
    g.ldc = (int)n;
    g.tilesM = g.M / kBM;
    g.tilesN = (int)((n + 255) / 256);
    g.mPerRank = (int)mPerRank;
    for (int q = 0; q < comm->nRanks; ++q) g.aPeer[q] = (const __nv_bfloat16*)peers[q];
    g.gathered = (__nv_bfloat16*)gathered;
    if (push) {
        g.agPush = kAgPushWorkers;
        g.aPeer[comm->rank] = (const __nv_bfloat16*)aShard;
        for (int q = 0; q < comm->nRanks; ++q) {
            g.gatheredPeer[q] = (__nv_bfloat16*)gathPeers[q];
            g.agReady[q] = (uint64_t*)comm->mc2->flags.peer[q] + (size_t)comm->nRanks * kMc2MaxTiles;
        }
    }
    const bool twoSm = Use2Sm() && mPerRank % 256 == 0;
    const int grid = SmCount() & ~1;
    // Push form without worker CTAs (the default): every CTA computes, its epilogue warps copy the shard while they
    // wait for accumulators.  HCCL_MC2_AG_WORKERS=<n> keeps n dedicated copy CTAs instead.
    const bool coop = push && ForcedWorkers(true) == 0;
    int workers = 0;
    if (coop) g.agPush = kAgPushCoop;
    else workers = twoSm ? GatherWorkerCtas((g.M / 256) * g.tilesN, 2) : GatherWorkerCtas(g.tilesM * g.tilesN, 1);
    g.nGemmCtas = grid - workers;
    if (twoSm) {
        // column tile width: fewest (waves x (width + 12)); only whole 64-column boxes of MN-major B.  (The plain matmul weighs
        // its widths by measured wave times, TwoSmColumnTile; this kernel's waves also carry the copies and were not timed so.)
        const int pairs = g.nGemmCtas / 2;
        const int tilesM2 = g.M / 256;
        int bestBn = 256;
        double bestCost = 1e30;
        for (int cand : {256, 224, 192, 160, 128}) {
            if (bMn && (cand / 2) % 64 != 0) continue;
            const int tn = (int)((n + cand - 1) / cand);
            const int waves = (tilesM2 * tn + pairs - 1) / pairs;
            const double cost = (double)waves * (cand + 12);
            if (cost < bestCost - 1e-9) { bestCost = cost; bestBn = cand; }
        }
        g.bn = bestBn;
        g.tilesN = (int)((n + bestBn - 1) / bestBn);
        CHK_RET(MapB(&tb, b, n, k, bMn, bestBn / 2));
        MC2_TRACE_ARM(g, grid);
        const HcclResult r = DispatchLayout2Sm<MODE_AG>(false, bMn, ta, tb, g, comm->dev(), grid, true, stream, &taOwn);
        MC2_TRACE_DUMP("ag_matmul", 0, g, grid, stream);
        return r;
    }
    return DispatchLayout<256, MODE_AG>(false, bMn, ta, tb, g, comm->dev(), grid, true, stream, &taOwn);
}

HcclResult Mc2MatmulReduceScatter(CommImpl* comm, const void* a, const void* b, void* out, uint64_t m, uint64_t n, uint64_t k, int transB,
                                  cudaStream_t stream)
{
    CHK_PTR_NULL(comm); CHK_PTR_NULL(a); CHK_PTR_NULL(b); CHK_PTR_NULL(out);
    const uint64_t P = (uint64_t)comm->nRanks;
    CHK_RET(CheckShapes(m, n, k));
    if (m % (P * kBM) != 0) { HCCL_ERROR("Matmul->ReduceScatter needs M to be a multiple of %llu (got %llu)", (unsigned long long)(P * kBM), (unsigned long long)m); return HCCL_E_PARA; }
    const uint64_t mPerRank = m / P;
    const uint64_t tilesN = (n + 255) / 256;
    if ((mPerRank / kBM) * tilesN > (uint64_t)kMc2MaxTiles) return HCCL_E_PARA;
    CHK_RET(Mc2EnsureState(comm, P * mPerRank * n * 2));
    const bool bMn = transB == 0;
    CUtensorMap ta, tb;
    CHK_RET(MapA(&ta, a, m, k, false));
    CHK_RET(MapB(&tb, b, n, k, bMn, 256));
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    FillPeers(comm, &g);
    g.M = (int)m; g.N = (int)n; g.K = (int)k;
    g.out = (__nv_bfloat16*)out;
    g.ldc = (int)n;
    g.tilesM = (int)(m / kBM);
    g.tilesN = (int)tilesN;
    g.mPerRank = (int)mPerRank;
    // switch-reduce form unless determinism is asked for (the switch's summation order is unspecified) or
    // HCCL_MC2_RS_P2P=1 keeps the peer-to-peer form
    static const bool forceP2p = [] { const char* e = getenv("HCCL_MC2_RS_P2P"); return e != nullptr && e[0] == '1'; }();
    // ... or at two ranks, where every rank reduces half of the product and the switch form measured 0.79 ms against
    // 0.51 ms for the peer-to-peer form (HCCL_MC2_RS_P2P=0 asks for the switch form anyway)
    static const bool forceSwitch = [] { const char* e = getenv("HCCL_MC2_RS_P2P"); return e != nullptr && e[0] == '0'; }();
    if (comm->mc2->xchg.mc != nullptr && !forceP2p && comm->cfg.deterministic == Deterministic::OFF && (comm->nRanks > 2 || forceSwitch))
        g.xchgMc = (const __nv_bfloat16*)comm->mc2->xchg.mc;
    const bool twoSm = Use2Sm() && mPerRank % 256 == 0;
    const int localTiles = (int)(mPerRank / kBM) * g.tilesN;
    // No worker CTAs by default: every CTA computes, its epilogue warps reduce the finished tiles of this rank's row
    // block while they wait for accumulators.  HCCL_MC2_RS_WORKERS=<n> keeps n dedicated reduction CTAs instead.
    int workers = 0;
    static const int rsWarps = [] { const char* e = getenv("HCCL_MC2_RS_WARPS"); const int v = e ? atoi(e) : 4; return v < 1 ? 1 : (v > 4 ? 4 : v); }();
    // Every rank count: with the division-free accumulator drain the epilogue warps have the time, and at inner
    // dimensions of ten thousand and more (two-way tensor parallelism) worker CTAs only take SMs from the GEMM
    // (measured at two ranks, 4096 x 8192 x 14336: 0.64 ms against 0.71 ms with workers).
    if (ForcedWorkers(false) == 0) g.rsCoop = rsWarps;
    else workers = twoSm ? ReduceWorkerCtas((g.M / 256) * g.tilesN, 2, localTiles, g.K, g.nRanks, g.xchgMc != nullptr)
                         : ReduceWorkerCtas(g.tilesM * g.tilesN, 1, localTiles, g.K, g.nRanks, g.xchgMc != nullptr);
    const int grid = SmCount() & ~1;
    g.nGemmCtas = grid - workers;
    if (twoSm) {
        g.bn = 256;
        CHK_RET(MapB(&tb, b, n, k, bMn, 128));
        MC2_TRACE_ARM(g, grid);
        const HcclResult r = DispatchLayout2Sm<MODE_RS>(false, bMn, ta, tb, g, comm->dev(), grid, true, stream);
        MC2_TRACE_DUMP("matmul_rs", 1, g, grid, stream);
        return r;
    }
    return DispatchLayout<256, MODE_RS>(false, bMn, ta, tb, g, comm->dev(), grid, true, stream);
}

HcclResult Mc2MatmulAllReduce(CommImpl* comm, const void* a, const void* b, void* out, uint64_t m, uint64_t n, uint64_t k, int transB,
                              cudaStream_t stream)
{
    CHK_PTR_NULL(comm); CHK_PTR_NULL(a); CHK_PTR_NULL(b); CHK_PTR_NULL(out);
    const uint64_t P = (uint64_t)comm->nRanks;
    CHK_RET(CheckShapes(m, n, k));
    if (transB == 0) { HCCL_ERROR("Matmul->AllReduce takes the weight as [N, K]"); return HCCL_E_NOT_SUPPORT; }
    const int tilesM = (int)((m + kBM - 1) / kBM), tilesN = (int)((n + 127) / 128);
    if ((uint64_t)tilesM * tilesN > (uint64_t)kMc2MaxTiles) return HCCL_E_PARA;
    // every tile is reduced by the CTA that computed it, which waits for its peers: all tiles must be resident at once
    if (tilesM * tilesN > SmCount()) { HCCL_ERROR("Matmul->AllReduce handles at most %d output tiles of 128x128 (decode shapes)", SmCount()); return HCCL_E_NOT_SUPPORT; }
    CHK_RET(Mc2EnsureState(comm, P * m * n * 2));
    CUtensorMap ta, tb;
    CHK_RET(MapA(&ta, a, m, k, false));
    CHK_RET(MapB(&tb, b, n, k, false, 128));
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    FillPeers(comm, &g);
    g.M = (int)m; g.N = (int)n; g.K = (int)k;
    g.out = (__nv_bfloat16*)out;
    g.ldc = (int)n;
    g.tilesM = tilesM;
    g.tilesN = tilesN;
    const int grid = tilesM * tilesN;
    g.nGemmCtas = grid;
    return LaunchGemm<128, false, false, MODE_AR>(ta, tb, g, comm->dev(), grid, true, stream);
}

}  // namespace hccl
