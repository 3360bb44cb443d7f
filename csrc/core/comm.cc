#include "comm.h"
#include <algorithm>
#include <chrono>
#include <cstring>
#include "../kernels/dev_types.h"
#include "../select/selector.h"
#include "../topo/topo.h"
#include "log.h"
#include "plan_cache.h"
#include "stuck_detector.h"
#include "../cpu/host_comm.h"

namespace hccl {

// ---------------------------------------------------------------- CtxStore
bool CtxStore::Get(const std::string& tag, std::vector<uint8_t>* out) const
{
    std::lock_guard<std::mutex> lk(mu_);
    auto it = blobs_.find(tag);
    if (it == blobs_.end()) return false;
    if (out) *out = it->second;
    return true;
}
void CtxStore::Put(const std::string& tag, std::vector<uint8_t> blob)
{
    std::lock_guard<std::mutex> lk(mu_);
    blobs_[tag] = std::move(blob);
}
void CtxStore::Erase(const std::string& tag)
{
    std::lock_guard<std::mutex> lk(mu_);
    blobs_.erase(tag);
}
void CtxStore::Clear()
{
    std::lock_guard<std::mutex> lk(mu_);
    blobs_.clear();
}
size_t CtxStore::size() const
{
    std::lock_guard<std::mutex> lk(mu_);
    return blobs_.size();
}

// ---------------------------------------------------------------- CommImpl
CommImpl::CommImpl() : dev_(new DevComm()) { memset(dev_, 0, sizeof(DevComm)); }

CommImpl::~CommImpl()
{
    Destroy();
    delete dev_;
}

StageLayout MakeStageLayout(uint64_t dataBytes, int nRanks)
{
    StageLayout l{};
    l.dataBytes = dataBytes;
    // p2p mailboxes take 1/8 of the slab at most (two halves per sender), at least 64 KiB per half
    uint64_t half = dataBytes / 8 / (2ull * (uint64_t)nRanks);
    half = half > (4ull << 20) ? (4ull << 20) : half;
    half &= ~(uint64_t)4095;
    if (half < 65536) half = 65536;
    const uint64_t mailbox = half * 2 * (uint64_t)nRanks;
    l.mailboxHalf = half;
    l.mailboxOff = (dataBytes - mailbox) & ~(uint64_t)4095;
    const uint64_t rest = l.mailboxOff;
    l.inOff = 0;
    l.inBytes = (rest / 2) & ~(uint64_t)4095;
    l.xchOff = l.inBytes;
    l.xchBytes = (rest - l.inBytes) & ~(uint64_t)4095;
    return l;
}

// The stream of the current device on which its communicators' counters are copied; it goes with the last of them.
static std::shared_ptr<CUstream_st> CountersStream()
{
    static std::mutex mu;
    static std::map<int, std::weak_ptr<CUstream_st>> streams;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(mu);
    if (std::shared_ptr<CUstream_st> there = streams[device].lock()) return there;
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    std::shared_ptr<CUstream_st> made(s, [](cudaStream_t x) { cudaStreamDestroy(x); });
    streams[device] = made;
    return made;
}

HcclResult CommImpl::SetupDeviceState()
{
    CHK_CUDA(cudaMalloc(&dEpochs_, kEpochWords * sizeof(uint64_t)));
    CHK_CUDA(cudaMemset(dEpochs_, 0, kEpochWords * sizeof(uint64_t)));
    CHK_CUDA(cudaMalloc(&dAbort_, 256));
    CHK_CUDA(cudaMemset(dAbort_, 0, 256));
    CHK_CUDA(cudaMalloc(&dP2pSeq_, 2 * kMaxDevRanks * sizeof(uint64_t)));
    CHK_CUDA(cudaMemset(dP2pSeq_, 0, 2 * kMaxDevRanks * sizeof(uint64_t)));
    CHK_CUDA(cudaHostAlloc((void**)&hStatus_, sizeof(DevStatus), cudaHostAllocMapped | cudaHostAllocPortable));
    memset((void*)hStatus_, 0, sizeof(DevStatus));
    CHK_CUDA(cudaHostGetDevicePointer((void**)&dStatus_, (void*)hStatus_, 0));
    countersStream_ = CountersStream();
    if (!countersStream_) return HCCL_E_RUNTIME;
    CHK_CUDA(cudaEventCreateWithFlags(&countersBack_, cudaEventDisableTiming));
    CHK_CUDA(cudaHostAlloc((void**)&hCounters_, 2 * sizeof(uint64_t), cudaHostAllocPortable));
    dev_->rank = rank;
    dev_->nRanks = nRanks;
    for (int q = 0; q < nRanks; ++q) dev_->slab[q] = (char*)slab_.peer[q];
    dev_->slabMc = (char*)slab_.mc;
    dev_->epochs = dEpochs_;
    dev_->abortWord = dAbort_;
    dev_->status = dStatus_;
    dev_->timeoutNs = cfg.execTimeoutNs;
    dev_->stageBytes = slab_.size - kSlabDataOff;
    layout_ = MakeStageLayout(dev_->stageBytes, nRanks);
    CHK_CUDA(cudaDeviceSynchronize());
    selector.reset(new SelectorState());
    plans.reset(new PlanCache());
    return HCCL_SUCCESS;
}

HcclResult CommImpl::Init(const HcclRootInfo& root, int nR, int r, const HcclCommConfig* config)
{
    const EnvConfig& env = GetEnvConfig();
    CHK_RET(MergeConfig(env, config, &cfg));
    rank = r;
    nRanks = nR;
    if (nRanks > kMaxDevRanks) {
        HCCL_ERROR("this build drives one NVSwitch domain of at most %d GPUs (got %d ranks)", kMaxDevRanks, nRanks);
        return HCCL_E_NOT_SUPPORT;
    }
    CHK_CUDA(cudaGetDevice(&device));
    bs.reset(new Bootstrap());
    CHK_RET(bs->Connect(root, rank, nRanks, env.connectTimeoutS));
    char nm[HCCL_COMM_CONFIG_NAME_MAX];
    snprintf(nm, sizeof(nm), "hccl_comm_%016llx", (unsigned long long)bs->uniqueId());
    name = cfg.commName.empty() ? nm : cfg.commName;
    GroupRegister(this);
    const size_t slabBytes = kSlabDataOff + cfg.bufferBytes;
    const bool wantMc = cfg.nvlsEnable != 0 && nRanks > 1;
    CHK_RET(SymAlloc(*bs, device, slabBytes, wantMc, env.forceIpc, &slab_));
    if (cfg.nvlsEnable == 1 && nRanks > 1 && slab_.mc == nullptr)
        HCCL_WARNING("NVLS was requested but the box does not expose multicast: using P2P kernels");
    CHK_RET(SetupDeviceState());
    topo.reset(new TopoInfo());
    CHK_RET(DiscoverTopo(this, topo.get()));
    HCCL_CONFIG_INFO(LOG_MOD_RESOURCE,
                     "comm %s rank %d/%d device %d: slab %zu MiB via %s, NVLS %s, stage-in %llu MiB, exchange %llu MiB, "
                     "mailbox half %llu KiB, wait budget %.1f s",
                     name.c_str(), rank, nRanks, device, slabBytes >> 20,
                     slab_.transport == SymTransport::VMM ? "VMM" : "IPC", slab_.mc ? "on" : "off",
                     (unsigned long long)(layout_.inBytes >> 20), (unsigned long long)(layout_.xchBytes >> 20),
                     (unsigned long long)(layout_.mailboxHalf >> 10), cfg.execTimeoutNs * 1e-9);
    if (env.dfs.stuckDetection) watchdog_ = std::thread([this] { WatchdogLoop(); });
    return bs->Barrier();
}

HcclResult CommImpl::InitEmulated(EmuGroup* group, int nR, int r, const SymSegment& slab, const HcclCommConfig* config)
{
    const EnvConfig& env = GetEnvConfig();
    CHK_RET(MergeConfig(env, config, &cfg));
    rank = r;
    nRanks = nR;
    CHK_CUDA(cudaGetDevice(&device));
    emu_ = group;
    slab_ = slab;
    ownsSlab_ = true;
    char nm[HCCL_COMM_CONFIG_NAME_MAX];
    snprintf(nm, sizeof(nm), "hccl_emu_%p", (void*)group);
    name = cfg.commName.empty() ? nm : cfg.commName;
    GroupRegister(this);
    CHK_RET(SetupDeviceState());
    topo.reset(new TopoInfo());
    CHK_RET(DiscoverTopo(this, topo.get()));
    return HCCL_SUCCESS;
}

namespace {
std::mutex g_groupMu;
std::vector<CommImpl*>& Groups()
{
    static std::vector<CommImpl*> v;
    return v;
}
}  // namespace
void GroupRegister(CommImpl* c)
{
    std::lock_guard<std::mutex> lk(g_groupMu);
    auto& v = Groups();
    if (std::find(v.begin(), v.end(), c) == v.end()) v.push_back(c);
}
void GroupUnregister(CommImpl* c)
{
    std::lock_guard<std::mutex> lk(g_groupMu);
    auto& v = Groups();
    v.erase(std::remove(v.begin(), v.end(), c), v.end());
}
std::vector<CommImpl*> GroupFind(const std::string& name)
{
    std::lock_guard<std::mutex> lk(g_groupMu);
    std::vector<CommImpl*> out;
    for (CommImpl* c : Groups())
        if (c->name == name) out.push_back(c);
    return out;
}

HcclResult CommImpl::Destroy()
{
    if (status_.load() == HCCL_COMM_STATUS_DESTROYED) return HCCL_SUCCESS;
    status_.store(HCCL_COMM_STATUS_DESTROYED);
    GroupUnregister(this);
    watchdogStop_.store(true);
    if (watchdog_.joinable()) watchdog_.join();
    if (hStatus_ || dEpochs_) cudaDeviceSynchronize();
    // Leave together: a peer must not unmap memory another rank's kernel may still touch.
    if (bs) bs->Barrier();
    for (auto& s : userSegs_) SymFree(&s);
    userSegs_.clear();
    if (ownsSlab_) SymFree(&slab_);
    std::lock_guard<std::mutex> counters(countersMu_);
    if (countersBack_) cudaEventDestroy(countersBack_);
    if (hCounters_) cudaFreeHost(hCounters_);
    countersStream_.reset();
    countersBack_ = nullptr; hCounters_ = nullptr; countersAsked_ = false;
    if (dEpochs_) cudaFree(dEpochs_);
    if (dAbort_) cudaFree(dAbort_);
    if (dP2pSeq_) cudaFree(dP2pSeq_);
    if (hStatus_) cudaFreeHost((void*)hStatus_);
    dEpochs_ = nullptr; dAbort_ = nullptr; dP2pSeq_ = nullptr; hStatus_ = nullptr;
    if (bs) bs->Close();
    ctx.Clear();
    if (emu_) emu_->Release(this);
    emu_ = nullptr;
    if (hostComm) HostRankRelease(hostComm);
    hostComm = nullptr;
    return HCCL_SUCCESS;
}

HcclResult CommImpl::CheckReady() const
{
    switch (status_.load()) {
        case HCCL_COMM_STATUS_READY: return HCCL_SUCCESS;
        case HCCL_COMM_STATUS_SUSPENDING: return HCCL_E_SUSPENDING;
        case HCCL_COMM_STATUS_ERROR: return HCCL_E_REMOTE;
        default: return HCCL_E_PARA;
    }
}

std::string CommImpl::DescribeAsyncError() const
{
    if (!hStatus_ || hStatus_->error == DEV_OK) return "";
    char buf[320];
    // The analogue of the reference's exception decode that prints which rank / flag a stuck kernel waited on
    // (hccl_aiv_utils.cc:360-465).
    snprintf(buf, sizeof(buf),
             "comm %s rank %u: kernel family %u, block row %u gave up waiting on flag slot %u for rank %u "
             "(expected >= %llu, last seen %llu) after %.2f s; ops started %llu, finished %llu",
             name.c_str(), hStatus_->rank, hStatus_->kernelId, hStatus_->block, hStatus_->slot, hStatus_->peer,
             (unsigned long long)hStatus_->expected, (unsigned long long)hStatus_->seen, cfg.execTimeoutNs * 1e-9,
             (unsigned long long)hStatus_->head, (unsigned long long)hStatus_->tail);
    return buf;
}

HcclResult CommImpl::PollAsyncError(HcclResult* out)
{
    *out = HCCL_SUCCESS;
    if (!hStatus_) return HCCL_SUCCESS;
    const uint32_t e = hStatus_->error;
    if (e == DEV_OK) return HCCL_SUCCESS;
    *out = (e == DEV_ERR_TIMEOUT) ? HCCL_E_TIMEOUT : HCCL_E_INTERNAL;
    int expect = HCCL_COMM_STATUS_READY;
    if (status_.compare_exchange_strong(expect, HCCL_COMM_STATUS_ERROR)) HCCL_ERROR("%s", DescribeAsyncError().c_str());
    return HCCL_SUCCESS;
}

HcclResult CommImpl::Suspend()
{
    int expect = HCCL_COMM_STATUS_READY;
    status_.compare_exchange_strong(expect, HCCL_COMM_STATUS_SUSPENDING);
    return HCCL_SUCCESS;
}

HcclResult CommImpl::Resume()
{
    if (status_.load() == HCCL_COMM_STATUS_DESTROYED) return HCCL_E_PARA;
    // All ranks arrive with no kernel in flight, clear their flags, epochs, sequence numbers and status, and leave
    // together.  Cached plans and selector state are dropped (reference: state callbacks clearing caches on resume,
    // stuck_detect_counter_helper.h:168-205).
    CHK_CUDA(cudaDeviceSynchronize());
    if (bs) CHK_RET(bs->Barrier());
    CHK_CUDA(cudaMemset(slab_.peer[rank], 0, kSlabDataOff));
    CHK_CUDA(cudaMemset(dEpochs_, 0, kEpochWords * sizeof(uint64_t)));
    CHK_CUDA(cudaMemset(dAbort_, 0, 256));
    CHK_CUDA(cudaMemset(dP2pSeq_, 0, 2 * kMaxDevRanks * sizeof(uint64_t)));
    memset((void*)hStatus_, 0, sizeof(DevStatus));
    CHK_CUDA(cudaDeviceSynchronize());
    if (bs) CHK_RET(bs->Barrier());
    ++generation;
    if (plans) plans->Clear();
    shapeSeen.clear();
    ctx.Clear();
    if (selector) selector.reset(new SelectorState());
    status_.store(HCCL_COMM_STATUS_READY);
    return HCCL_SUCCESS;
}

char* CommImpl::StageBase(int r) const { return (char*)slab_.peer[r] + kSlabDataOff; }
char* CommImpl::StageMcBase() const { return slab_.mc ? (char*)slab_.mc + kSlabDataOff : nullptr; }

LaunchTarget CommImpl::Target(cudaStream_t stream) const
{
    LaunchTarget t;
    t.dev = dev_;
    t.stream = stream;
    t.emu = emu_;
    t.emuRank = rank;
    return t;
}

int CommImpl::MaxBlocks() const
{
    int m = cfg.maxBlocks ? (int)cfg.maxBlocks : 128;
    if (m > kMaxBlocks) m = kMaxBlocks;
    if (emu_) {
        int cap = emu_->maxBlocksPerRank_;
        if (m > cap) m = cap;
    }
    return m;
}

HcclResult CommImpl::MemAlloc(uint64_t size, void** ptr)
{
    CHK_PTR_NULL(ptr);
    if (size == 0) return HCCL_E_PARA;
    SymSegment seg;
    if (emu_) {
        CHK_RET(emu_->MemAlloc(rank, size, &seg));
    } else {
        // the size must agree: a mismatch would map windows of different sizes
        std::vector<uint64_t> sizes((size_t)nRanks);
        CHK_RET(bs->AllGather(&size, sizes.data(), sizeof(size)));
        for (uint64_t s : sizes)
            if (s != size) { HCCL_ERROR("HcclMemAlloc: ranks passed different sizes (%llu vs %llu)", (unsigned long long)size, (unsigned long long)s); return HCCL_E_PARA; }
        CHK_RET(SymAlloc(*bs, device, size, slab_.mc != nullptr, GetEnvConfig().forceIpc, &seg));
    }
    *ptr = seg.peer[rank];
    userSegs_.push_back(seg);
    return HCCL_SUCCESS;
}

HcclResult CommImpl::MemFree(void* ptr)
{
    for (size_t i = 0; i < userSegs_.size(); ++i) {
        if (userSegs_[i].peer[rank] == ptr) {
            CHK_CUDA(cudaDeviceSynchronize());
            if (bs) CHK_RET(bs->Barrier());
            SymFree(&userSegs_[i]);
            userSegs_.erase(userSegs_.begin() + (long)i);
            return HCCL_SUCCESS;
        }
    }
    HCCL_ERROR("HcclMemFree: %p was not returned by HcclMemAlloc on this communicator", ptr);
    return HCCL_E_NOT_FOUND;
}

HcclResult CommImpl::RegisterBuffer(void* ptr, uint64_t size)
{
    CHK_PTR_NULL(ptr);
    if (size == 0) return HCCL_E_PARA;
    if (emu_ || hostComm || nRanks == 1 || bs == nullptr) return HCCL_E_NOT_SUPPORT;
    const char* peers[HCCL_MAX_DEVICE_RANKS];
    if (Lookup(ptr, size, peers, nullptr)) return HCCL_SUCCESS;        // already symmetric (HcclMemAlloc) or registered
    SymSegment seg;
    CHK_RET(SymRegisterUser(*bs, ptr, size, &seg));
    userSegs_.push_back(seg);
    return HCCL_SUCCESS;
}

HcclResult CommImpl::DeregisterBuffer(void* ptr)
{
    for (size_t i = 0; i < userSegs_.size(); ++i) {
        if (userSegs_[i].peer[rank] == ptr && userSegs_[i].transport == SymTransport::USER_IPC) {
            CHK_CUDA(cudaDeviceSynchronize());
            if (bs) CHK_RET(bs->Barrier());       // no peer still reads the buffer
            SymFree(&userSegs_[i]);
            userSegs_.erase(userSegs_.begin() + (long)i);
            return HCCL_SUCCESS;
        }
    }
    HCCL_ERROR("HcclCommDeregister: %p was not registered on this communicator", ptr);
    return HCCL_E_NOT_FOUND;
}

bool CommImpl::Lookup(const void* p, uint64_t bytes, const char* peerPtr[HCCL_MAX_DEVICE_RANKS], const char** mcPtr) const
{
    for (const SymSegment& s : userSegs_) {
        if (!s.ContainsLocal(p, bytes)) continue;
        const size_t off = (size_t)((const char*)p - (const char*)s.peer[rank]);
        for (int q = 0; q < nRanks; ++q) {
            const void* base = s.peer[q];
            if (!base) return false;
            peerPtr[q] = (const char*)base + off;
        }
        if (mcPtr) *mcPtr = s.mc ? (const char*)s.mc + off : nullptr;
        return true;
    }
    return false;
}

HcclResult CommImpl::ReadOpCounters(uint64_t* started, uint64_t* finished, int limitMs, const std::atomic<bool>* stop)
{
    CHK_PTR_NULL(started); CHK_PTR_NULL(finished);
    std::lock_guard<std::mutex> lk(countersMu_);
    if (!dEpochs_ || !countersStream_) return HCCL_E_NOT_SUPPORT;
    // another thread's stream capture is none of this thread's business
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return HCCL_E_RUNTIME;             // the process is on its way out
    const auto until = std::chrono::steady_clock::now() + std::chrono::milliseconds(limitMs);
    bool earlier = countersAsked_;      // the answer on its way is to an earlier call: it frees the buffer, then the device is asked again
    cudaError_t e = cudaSuccess;
    for (;;) {
        if (!countersAsked_) {
            e = cudaMemcpyAsync(hCounters_, dEpochs_ + 2 * kMaxBlocks, 2 * sizeof(uint64_t), cudaMemcpyDeviceToHost, countersStream_.get());
            if (e == cudaSuccess) e = cudaEventRecord(countersBack_, countersStream_.get());
            if (e != cudaSuccess) break;
            countersAsked_ = true;
        }
        e = cudaEventQuery(countersBack_);
        if (e == cudaSuccess) {
            countersAsked_ = false;
            if (!earlier) break;
            earlier = false;
            continue;
        }
        if (e == cudaErrorNotReady) cudaGetLastError();          // no error that the thread's next check should find
        if (e != cudaErrorNotReady || (stop != nullptr && stop->load()) || std::chrono::steady_clock::now() >= until) break;
        std::this_thread::sleep_for(std::chrono::microseconds(200));
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e == cudaErrorNotReady) return HCCL_E_AGAIN;
    if (e != cudaSuccess) return HCCL_E_RUNTIME;
    *started = hCounters_[0];
    *finished = hCounters_[1];
    return HCCL_SUCCESS;
}

HcclResult CommImpl::ReadOpCountersBehind(cudaStream_t stream)
{
    std::lock_guard<std::mutex> lk(countersMu_);
    if (!countersStream_) return HCCL_E_NOT_SUPPORT;
    cudaEvent_t e = nullptr;
    CHK_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    cudaError_t r = cudaEventRecord(e, stream);
    if (r == cudaSuccess) r = cudaStreamWaitEvent(countersStream_.get(), e, 0);
    cudaEventDestroy(e);
    return r == cudaSuccess ? HCCL_SUCCESS : HCCL_E_RUNTIME;
}

void CommImpl::WatchdogLoop()
{
    cudaSetDevice(device);
    StuckDetector detector((double)DeriveTimeouts(cfg.execTimeoutNs).fullNs * 1e-9);
    while (!watchdogStop_.load()) {
        for (int i = 0; i < 10 && !watchdogStop_.load(); ++i) std::this_thread::sleep_for(std::chrono::milliseconds(100));
        uint64_t h = 0, t = 0;
        if (watchdogStop_.load()) break;
        const HcclResult r = ReadOpCounters(&h, &t, 1000, &watchdogStop_);
        if (watchdogStop_.load() || (r != HCCL_SUCCESS && r != HCCL_E_AGAIN)) continue;
        if (detector.Observe(r == HCCL_SUCCESS, h, t, std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count())) {
            stuckReports.fetch_add(1);
            HCCL_ERROR("comm %s rank %d: stuck detection: %llu ops started, %llu finished, no progress for %.0f s%s", name.c_str(), rank,
                       (unsigned long long)detector.started(), (unsigned long long)detector.finished(), detector.idleS(),
                       r == HCCL_SUCCESS ? "" : " (the device does not answer)");
        }
    }
}

// ---------------------------------------------------------------- EmuGroup
HcclResult EmuGroup::Create(int nRanks, const HcclCommConfig* cfg, std::vector<CommImpl*>* comms)
{
    if (nRanks < 1 || nRanks > kMaxDevRanks) return HCCL_E_PARA;
    std::unique_ptr<EmuGroup> g(new EmuGroup());
    g->nRanks_ = nRanks;
    g->alive_ = nRanks;
    g->queues_.resize((size_t)nRanks);
    g->pendingOps.resize((size_t)nRanks);
    EffectiveConfig eff;
    CHK_RET(MergeConfig(GetEnvConfig(), cfg, &eff));
    // emulated ranks share one GPU: keep the per-rank slab modest unless configured
    uint64_t data = (cfg && cfg->hcclBufferSize) || GetEnvConfig().bufferSizeMiB ? eff.bufferBytes : (64ull << 20);
    CHK_RET(SymAllocLocalGroup(nRanks, kSlabDataOff + data, &g->slabs_));
    g->maxBlocksPerRank_ = EmuMaxBlocksPerRank(nRanks);
    CHK_CUDA(cudaMalloc(&g->dComms_, sizeof(DevComm) * (size_t)nRanks));
    comms->clear();
    g->hostComms_.resize((size_t)nRanks);
    for (int r = 0; r < nRanks; ++r) {
        CommImpl* c = new CommImpl();
        HcclResult res = c->InitEmulated(g.get(), nRanks, r, g->slabs_[r], cfg);
        if (res != HCCL_SUCCESS) { delete c; return res; }
        g->hostComms_[r] = c->dev();
        g->members.push_back(c);
        comms->push_back(c);
    }
    CHK_CUDA(cudaMemcpy(g->dComms_, g->hostComms_.data(), sizeof(DevComm) * (size_t)nRanks, cudaMemcpyHostToDevice));
    g.release();
    return HCCL_SUCCESS;
}

EmuGroup::~EmuGroup()
{
    cudaDeviceSynchronize();
    if (dComms_) cudaFree(dComms_);
}

void EmuGroup::Release(CommImpl*)
{
    bool last;
    {
        std::lock_guard<std::mutex> lk(mu_);
        last = (--alive_ == 0);
    }
    if (last) delete this;
}

HcclResult EmuGroup::Post(int rank, const void* args, size_t argBytes, int nBlocks, int threads, const void* kernel,
                          cudaStream_t stream, size_t smem)
{
    std::lock_guard<std::mutex> lk(mu_);
    if (rank < 0 || rank >= nRanks_) return HCCL_E_INTERNAL;
    // One FIFO per rank: a rank may run ahead (an operator that needs several loops posts several launches before
    // the next rank is called); a launch is issued whenever every rank has an entry at the head of its queue.
    PendingPost post;
    post.kernel = kernel; post.nBlocks = nBlocks; post.threads = threads; post.smem = smem;
    post.args.assign((const char*)args, (const char*)args + argBytes);
    queues_[(size_t)rank].push_back(std::move(post));
    for (;;) {
        for (int r = 0; r < nRanks_; ++r)
            if (queues_[(size_t)r].empty()) return HCCL_SUCCESS;
        const PendingPost& first = queues_[0].front();
        for (int r = 1; r < nRanks_; ++r) {
            const PendingPost& o = queues_[(size_t)r].front();
            if (o.kernel != first.kernel || o.nBlocks != first.nBlocks || o.args.size() != first.args.size()) {
                HCCL_ERROR("emulated ranks posted different operations (rank %d differs from rank 0)", r);
                for (auto& q : queues_) q.clear();
                return HCCL_E_PARA;
            }
        }
        const size_t ab = first.args.size();
        int nb = first.nBlocks;
        if (nb > maxBlocksPerRank_) {
            HCCL_ERROR("emulated launch needs %d blocks per rank, only %d fit one cooperative grid", nb, maxBlocksPerRank_);
            for (auto& q : queues_) q.clear();
            return HCCL_E_INTERNAL;
        }
        // the kernel's second parameter: one argument struct per possible rank
        launchArgs_.assign(ab * (size_t)kMaxDevRanks, 0);
        for (int r = 0; r < nRanks_; ++r) memcpy(launchArgs_.data() + (size_t)r * ab, queues_[(size_t)r].front().args.data(), ab);
        const void* fn = first.kernel;
        const int th = first.threads;
        const size_t shared = first.smem;
        for (auto& q : queues_) q.pop_front();
        const DevComm* dc = dComms_;
        void* kargs[3] = {(void*)&dc, (void*)launchArgs_.data(), (void*)&nb};
        cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3((unsigned)(nb * nRanks_)), dim3((unsigned)th), kargs, shared, stream);
        if (e != cudaSuccess) { HCCL_ERROR("cooperative launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    }
}

HcclResult EmuGroup::MemAlloc(int rank, uint64_t size, SymSegment* seg)
{
    std::lock_guard<std::mutex> lk(mu_);
    // Rank r's k-th allocation pairs with every other rank's k-th allocation, whatever the interleaving of the calls.
    // The first rank to reach round k allocates all copies, so that peer pointers are known at once.
    if (allocNext_.empty()) allocNext_.assign((size_t)nRanks_, 0);
    const size_t k = allocNext_[(size_t)rank]++;
    if (k == allocRounds_.size()) {
        allocRounds_.emplace_back();
        CHK_RET(SymAllocLocalGroup(nRanks_, size, &allocRounds_.back()));
    } else if (allocRounds_[k][0].size != size) {
        HCCL_ERROR("HcclMemAlloc: emulated ranks passed different sizes for their allocation number %zu", k);
        return HCCL_E_PARA;
    }
    *seg = allocRounds_[k][(size_t)rank];
    return HCCL_SUCCESS;
}

}  // namespace hccl
