// Host side of the C ABI: sessions (device copies of the index, workspaces, the batch pipeline), the
// stage-level and one-shot operator entry points, training drivers and the synthetic-data entry points.
#include "batch_parts.h"
#include "common.cuh"
#include "kernels.h"
#include "mapped_rows.h"
#include "select.cuh"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstring>
#include <limits>
#include <random>
#include <memory>
#include <new>
#include <numeric>
#include <condition_variable>
#include <deque>
#include <functional>
#include <mutex>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

namespace psb {

// ---- status plumbing ------------------------------------------------------------------------------
std::string& last_error_ref() {
    thread_local std::string e;
    return e;
}
psb_status fail(psb_status code, const std::string& message) {
    last_error_ref() = message;
    return code;
}
psb_status cuda_fail(cudaError_t err, const char* what, const char* file, int line) {
    const char* base = std::strrchr(file, '/');
    last_error_ref() = std::string(cudaGetErrorString(err)) + " in " + what + " (" + (base ? base + 1 : file) + ":" +
                       std::to_string(line) + ")";
    if (err == cudaErrorMemoryAllocation) { cudaGetLastError(); return PSB_OUT_OF_MEMORY; }
    return PSB_CUDA_ERROR;
}
static std::atomic<long long> g_launches{0};
void count_launch(long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launches_total() { return g_launches.load(std::memory_order_relaxed); }

namespace {
// One word per (kernel, device): bit 31 the carve-out is set, the rest the shared memory allowed so far.  Open addressing; a full table
// (never: the library has fewer kernels) just sets the attribute every time.
struct KernelAttr { std::atomic<uintptr_t> key{0}; std::atomic<unsigned> word{0}; };
KernelAttr g_attr[2048];
KernelAttr* kernel_attr(const void* kernel) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    const uintptr_t key = (reinterpret_cast<uintptr_t>(kernel) << 6) ^ (uintptr_t)(dev & 63) ^ ((uintptr_t)1 << 63);
    size_t h = (key * 0x9E3779B97F4A7C15ull) >> 53;
    for (int i = 0; i < 64; ++i, h = (h + 1) & 2047) {
        uintptr_t seen = g_attr[h].key.load(std::memory_order_acquire);
        if (seen == 0 && g_attr[h].key.compare_exchange_strong(seen, key, std::memory_order_acq_rel)) return &g_attr[h];
        if (seen == key) return &g_attr[h];
    }
    return nullptr;
}
}  // namespace
psb_status kernel_shared(const void* kernel, size_t bytes) {
    KernelAttr* a = kernel_attr(kernel);
    const unsigned need = (unsigned)bytes;
    if (a && need <= (a->word.load(std::memory_order_acquire) & 0x7fffffffu)) return PSB_OK;
    static std::mutex mu;   // the attribute only ever grows, whichever threads ask for how much
    std::lock_guard<std::mutex> lk(mu);
    const unsigned have = a ? a->word.load(std::memory_order_relaxed) & 0x7fffffffu : 0;
    if (a && need <= have) return PSB_OK;
    PSB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need));
    if (a) a->word.fetch_add(need - have, std::memory_order_release);
    return PSB_OK;
}
psb_status kernel_carveout_max(const void* kernel) {
    KernelAttr* a = kernel_attr(kernel);
    if (a && (a->word.load(std::memory_order_relaxed) & 0x80000000u)) return PSB_OK;
    PSB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (a) a->word.fetch_or(0x80000000u);
    return PSB_OK;
}

namespace {

// The library's memory pool of each device (work_pool).
struct Pools { std::mutex mu; cudaMemPool_t pool[64] = {}; };
Pools& pools() { static Pools* one = new Pools; return *one; }   // never destroyed: the driver may end first
// What the pool holds and nobody uses goes back to the device.
void trim_pool(int device) {
    if (device < 0 || device >= 64) return;
    std::lock_guard<std::mutex> lk(pools().mu);
    if (pools().pool[device]) cudaMemPoolTrimTo(pools().pool[device], 0);
}

// Device buffer that grows on demand (contents are not preserved).
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    bool part = false;   // a part of a group's allocation
    ~DevBuf() { release(); }
    void release() { if (p && !part) cudaFree(p); p = nullptr; bytes = 0; part = false; }
    psb_status reserve(size_t need) {
        if (need <= bytes) return PSB_OK;
        release();
        cudaError_t e = cudaMalloc(&p, need ? need : 1);
        int device = 0;
        if (e == cudaErrorMemoryAllocation && cudaGetDevice(&device) == cudaSuccess) {   // perhaps the pool holds what is missing
            cudaGetLastError();
            trim_pool(device);
            e = cudaMalloc(&p, need ? need : 1);
        }
        if (e != cudaSuccess) { p = nullptr; return cuda_fail(e, "cudaMalloc", __FILE__, __LINE__); }
        bytes = need;
        return PSB_OK;
    }
    psb_status reserve(size_t need, int, cudaStream_t) { return reserve(need); }   // the signature of PoolBuf
    template <typename T> T* as() const { return static_cast<T*>(p); }
};

// Buffers that a call sizes together, in one allocation: every cudaMalloc above 1 MB takes about 0.35 ms, and a session's first call made
// up to eight of them in a row.  When one has to grow, all are laid out anew (*moved): none shrinks, contents are not preserved.
psb_status reserve_together(DevBuf* whole, std::initializer_list<std::pair<DevBuf*, size_t>> want, int = 0, cudaStream_t = nullptr, bool* moved = nullptr) {
    auto padded = [](size_t n) { return (n + 255) / 256 * 256; };
    bool grow = false;
    for (const auto& w : want) grow = grow || w.second > w.first->bytes;
    if (moved) *moved = grow;
    if (!grow) return PSB_OK;
    std::vector<size_t> sizes;
    size_t total = 0;
    for (const auto& w : want) {
        sizes.push_back(std::max(w.second, w.first->bytes));
        total += padded(sizes.back());
        w.first->release();
    }
    whole->release();
    PSB_TRY(whole->reserve(total));
    unsigned char* at = whole->as<unsigned char>();
    size_t i = 0;
    for (const auto& w : want) {
        const size_t n = sizes[i++];
        if (n == 0) continue;
        w.first->p = at; w.first->bytes = n; w.first->part = true;
        at += padded(n);
    }
    return PSB_OK;
}

// Runs at every operator call.  The full property block (cudaGetDeviceProperties) takes milliseconds on some hosts - 10 of the
// 18 ms of a psb_pq_encode call on 1M rows went there - so two attributes are asked once per device and the SM count is remembered.
psb_status check_device(int device, int* sm_count = nullptr) {
    static std::atomic<int> known_sms[64];
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n <= 0) {
        cudaGetLastError();
        return fail(PSB_NO_DEVICE, "no CUDA device is usable; this library has no CPU path");
    }
    if (device < 0 || device >= n) return fail(PSB_INVALID_ARGUMENT, "device ordinal out of range");
    int sms = device < 64 ? known_sms[device].load(std::memory_order_relaxed) : 0;
    if (sms == 0) {
        int major = 0;
        PSB_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
        PSB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        if (major != 10) return fail(PSB_NO_DEVICE, "device is not sm_100 (kernels are built for sm_100a only)");
        if (device < 64) known_sms[device].store(sms, std::memory_order_relaxed);
    }
    if (sm_count) *sm_count = sms;
    PSB_CUDA(cudaSetDevice(device));
    return PSB_OK;
}

// Work memory of the operators that allocate, run and free within one call (training, one-shot searches): from a memory pool of
// the library per device, stream-ordered, so that a call pays neither cudaMalloc nor the device synchronisation of cudaFree (about
// a third of a small training call).  The pool keeps at most kPoolKeep bytes between calls; what is above goes back to the device at
// the next synchronisation, the rest with the last session of the device or when a session finds no memory.
constexpr unsigned long long kPoolKeep = 1ull << 30;
psb_status work_pool(int device, cudaMemPool_t* out) {
    if (device < 0 || device >= 64) return fail(PSB_UNSUPPORTED_SHAPE, "device ordinal above 63");
    std::lock_guard<std::mutex> lk(pools().mu);
    cudaMemPool_t& known = pools().pool[device];
    if (!known) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t p = nullptr;
        PSB_CUDA(cudaMemPoolCreate(&p, &props));
        unsigned long long keep = kPoolKeep;
        PSB_CUDA(cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep));
        known = p;
    }
    *out = known;
    return PSB_OK;
}

// Stream-ordered buffer from the pool; freed on the same stream, so work queued there before may still use it.
struct PoolBuf {
    void* p = nullptr;
    size_t bytes = 0;
    cudaStream_t st = nullptr;
    PoolBuf() = default;
    PoolBuf(const PoolBuf&) = delete;
    PoolBuf& operator=(const PoolBuf&) = delete;
    ~PoolBuf() { release(); }
    void release() { if (p) cudaFreeAsync(p, st); p = nullptr; bytes = 0; }
    psb_status reserve(size_t need, int device, cudaStream_t stream) {
        if (p && need <= bytes) return PSB_OK;
        release();
        cudaMemPool_t pool;
        PSB_TRY(work_pool(device, &pool));
        PSB_CUDA(cudaMallocFromPoolAsync(&p, need ? need : 1, pool, stream));
        bytes = need; st = stream;
        return PSB_OK;
    }
    template <typename T> T* as() const { return static_cast<T*>(p); }
};

struct HostPages {
    static Mapping map(const void* rows, size_t bytes, int* code) {
        cudaError_t err = cudaHostRegister(const_cast<void*>(rows), bytes, cudaHostRegisterMapped | cudaHostRegisterReadOnly);
        if (err == cudaErrorHostMemoryAlreadyRegistered) { cudaGetLastError(); return Mapping::kOthers; }
        if (err != cudaSuccess) {
            cudaGetLastError();
            err = cudaHostRegister(const_cast<void*>(rows), bytes, cudaHostRegisterMapped);
        }
        if (err == cudaSuccess) return Mapping::kMapped;
        cudaGetLastError();
        *code = (int)err;
        return Mapping::kNot;
    }
    static void unmap(void* rows) { cudaHostUnregister(rows); }
};
MappedRows<HostPages>& mapped_rows() { static auto* one = new MappedRows<HostPages>; return *one; }   // never destroyed: the driver may end first
psb_status map_rows(const void* rows, size_t bytes, bool* counted) {
    int code = 0;
    const Mapping got = mapped_rows().take(rows, bytes, &code);
    *counted = got == Mapping::kMapped;
    if (got == Mapping::kOverlaps) return fail(PSB_CUDA_ERROR, "the exact rows overlap rows another session has mapped; use PSB_EXACT_HOST_STAGED");
    if (got == Mapping::kNot)
        return fail(PSB_CUDA_ERROR, std::string("cannot map the exact rows into the device address space (") + cudaGetErrorString((cudaError_t)code) +
                                        "); use PSB_EXACT_HOST_STAGED");
    return PSB_OK;
}
// The caller's arrays that a call copies to or from the device.  On a way out with an error the copies may still be under way on `st`.
struct HostCopies {
    cudaStream_t st;
    MappedRows<HostPages>::Copies noted;
    bool ended = false;
    HostCopies(cudaStream_t st_, std::initializer_list<std::pair<const void*, size_t>> spans) : st(st_), noted(mapped_rows(), spans) {}
    ~HostCopies() { if (noted.any() && !ended) cudaStreamSynchronize(st); }
};

// Page-locked blocks through which small calls pass, one to a session from its first search to its end, handed on from session to
// session.  A process's first page-locked memory takes 0.8 to 3 ms whatever its size, and again whenever all of it has been given back
// in between: four fifths of the first search of a session that answers single queries.  At most kIdle blocks (2 MiB) stay with the library.
constexpr size_t kSmallIo = 256 * 1024;   // queries and results of a call that passes through the block
constexpr size_t kHostBlock = kSmallIo + 4096;
class HostBlocks {
public:
    static HostBlocks& get() { static HostBlocks* one = new HostBlocks; return *one; }   // never destroyed: the driver may end first
    psb_status take(unsigned char** out) {
        for (;;) {
            unsigned char* p = nullptr;
            { std::lock_guard<std::mutex> lk(mu_); if (!idle_.empty()) { p = idle_.back(); idle_.pop_back(); } }
            if (!p) break;
            cudaPointerAttributes at{};   // a block from before a device reset is no longer the driver's, nor ours to free
            if (cudaPointerGetAttributes(&at, p) == cudaSuccess && at.type == cudaMemoryTypeHost) { *out = p; return PSB_OK; }
            cudaGetLastError();
        }
        PSB_CUDA(cudaHostAlloc(reinterpret_cast<void**>(out), kHostBlock, cudaHostAllocMapped | cudaHostAllocPortable));
        return PSB_OK;
    }
    void give(unsigned char* p) {   // nothing on the device may still use it
        { std::lock_guard<std::mutex> lk(mu_); if (idle_.size() < kIdle) { idle_.push_back(p); return; } }
        cudaFreeHost(p);
    }
private:
    static constexpr size_t kIdle = 8;
    std::mutex mu_;
    std::vector<unsigned char*> idle_;
};

// The pool serves these from what it holds, one by one.
psb_status reserve_together(PoolBuf*, std::initializer_list<std::pair<PoolBuf*, size_t>> want, int device, cudaStream_t st) {
    for (const auto& w : want)
        if (w.second) PSB_TRY(w.first->reserve(w.second, device, st));
    return PSB_OK;
}

// Persistent fork-join pool of host threads for the staged rerank transport (the reference keeps a persistent rerank pool
// too: src/search/ivf_common/ivf_host_rerank.cpp:42-51).  run(job) calls job(t) on every thread t and returns when all are done.
class HostPool {
public:
    explicit HostPool(int n) : n_(n) {
        for (int t = 0; t < n_; ++t) threads_.emplace_back([this, t] { loop(t); });
    }
    ~HostPool() {
        { std::lock_guard<std::mutex> lk(mu_); stop_ = true; ++gen_; }
        cv_.notify_all();
        for (auto& th : threads_) th.join();
    }
    int size() const { return n_; }
    template <typename F>
    void run(F&& job) {
        std::function<void(int)> f = std::forward<F>(job);
        { std::lock_guard<std::mutex> lk(mu_); job_ = &f; pending_ = n_; ++gen_; }
        cv_.notify_all();
        std::unique_lock<std::mutex> lk(mu_);
        done_.wait(lk, [this] { return pending_ == 0; });
        job_ = nullptr;
    }
private:
    void loop(int t) {
        unsigned long long seen = 0;
        for (;;) {
            const std::function<void(int)>* f = nullptr;
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [&] { return gen_ != seen; });
                seen = gen_;
                if (stop_) return;
                f = job_;
            }
            if (f) (*f)(t);
            { std::lock_guard<std::mutex> lk(mu_); if (--pending_ == 0) done_.notify_all(); }
        }
    }
    int n_;
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable cv_, done_;
    const std::function<void(int)>* job_ = nullptr;
    unsigned long long gen_ = 0;
    int pending_ = 0;
    bool stop_ = false;
};

// Timing events of a session, used over and over (creating and destroying the fifteen of a search took longer than recording them).
struct EventPool {
    std::vector<cudaEvent_t> ev;
    size_t used = 0;
    ~EventPool() { for (auto e : ev) cudaEventDestroy(e); }
    psb_status get(cudaEvent_t* out) {
        if (used == ev.size()) {
            cudaEvent_t e;
            PSB_CUDA(cudaEventCreate(&e));
            ev.push_back(e);
        }
        *out = ev[used++];
        return PSB_OK;
    }
};
struct EventTimer {
    EventPool* pool;
    std::vector<cudaEvent_t> ev;
    explicit EventTimer(EventPool* p) : pool(p) {}
    psb_status mark(cudaStream_t s) {
        cudaEvent_t e;
        PSB_TRY(pool->get(&e));
        ev.push_back(e);
        PSB_CUDA(cudaEventRecord(e, s));
        return PSB_OK;
    }
    double ms(size_t a, size_t b) const {
        float t = 0.f;
        if (a < ev.size() && b < ev.size()) cudaEventElapsedTime(&t, ev[a], ev[b]);
        return t;
    }
};

// Centroid-side buffers of the tensor-core coarse filter (built once per index; rebuilt per iteration in training).
template <typename Buf>
struct TcIndexBuffers {
    Buf cb, cn2, cmax, mu;
    bool ready = false;
    // keep_mean: the operands stay centred on the mean of an earlier call (queries prepared then stay valid).
    psb_status prepare(const float* d_centroids, int nlist, int dim, int device, cudaStream_t st, bool keep_mean = false) {
        const int dimp = coarse_tc_padded_dim(dim);
        PSB_TRY(mu.reserve(sizeof(float) * (size_t)dim, device, st));
        PSB_TRY(cb.reserve((size_t)2 * nlist * dimp, device, st));
        PSB_TRY(cn2.reserve(sizeof(float) * (size_t)coarse_tc_tiles(nlist) * 256, device, st));
        PSB_TRY(cmax.reserve(sizeof(float) * 2, device, st));
        if (!keep_mean) PSB_TRY(launch_mean_row(d_centroids, nlist, dim, mu.template as<float>(), st));
        PSB_TRY(launch_tc_prep_centroids(d_centroids, nlist, dim, mu.template as<float>(), cb.p, cn2.template as<float>(), cmax.template as<float>(), st));
        ready = true;
        return PSB_OK;
    }
    CoarseTcIndex view(const float* d_centroids, int nlist, int dim) const {
        CoarseTcIndex ix;
        ix.centroids = d_centroids; ix.cb = cb.p; ix.cn2 = cn2.template as<float>(); ix.mu = mu.template as<float>(); ix.cmax = cmax.template as<float>();
        ix.nlist = nlist; ix.dim = dim;
        return ix;
    }
};

// Per-batch buffers of the tensor-core coarse filter.
template <typename Buf>
struct TcWorkBuffers {
    Buf whole, qb, qnorm, gmin, seltop, selids, cand_cnt, cand, fail_list, scalars, fail_list2, retry_qb, retry_qnorm;
    // own_queries: qb and qnorm are needed (not when the caller keeps prepared rows); bounded: rows come with a previous assignment
    // (launch_coarse_tc_assign), which needs group minima for the rows it searches again only.
    psb_status ensure(int nq, int nlist, int dim, int nprobe, int device, cudaStream_t st, bool own_queries = true, bool bounded = false) {
        const int dimp = coarse_tc_padded_dim(dim);
        const int groups = coarse_tc_tiles(nlist) * (256 / coarse_tc_group(nlist, nprobe));
        const size_t n = (size_t)nq, own = own_queries ? n : 0, retry = bounded ? (size_t)std::min(nq, coarse_tc_retry_rows()) : 0;
        PSB_TRY(reserve_together(&whole, {{&qb, 2 * own * dimp}, {&qnorm, sizeof(float) * 2 * own},
                                          {&gmin, sizeof(float) * (size_t)coarse_tc_pitch(bounded ? (int)retry : nq) * groups},
                                          {&fail_list2, bounded ? sizeof(int) * n : 0}, {&retry_qb, 2 * retry * dimp}, {&retry_qnorm, sizeof(float) * 2 * retry},
                                          {&seltop, sizeof(float) * n * nprobe}, {&selids, nprobe > 1 ? sizeof(int) * n * nprobe : 0}, {&cand_cnt, sizeof(int) * n},
                                          {&cand, sizeof(int) * n * (nprobe == 1 ? coarse_tc_list_cap() : coarse_tc_mask_words(nlist))},
                                          {&fail_list, sizeof(int) * n}}, device, st));
        if (!scalars.p) {
            PSB_TRY(scalars.reserve(sizeof(int) * 8, device, st));
            PSB_CUDA(cudaMemsetAsync(scalars.p, 0, sizeof(int) * 8, st));
        }
        return PSB_OK;
    }
    CoarseTcWorkspace view() const {
        CoarseTcWorkspace w;
        w.qb = qb.p; w.qnorm = qnorm.p; w.gmin = gmin.template as<float>(); w.seltop = seltop.template as<float>();
        w.selids = selids.template as<int>(); w.cand_cnt = cand_cnt.template as<int>(); w.cand = cand.template as<int>();
        w.fail_list = fail_list.template as<int>(); w.n_fail = scalars.template as<int>(); w.status = scalars.template as<int>() + 2;
        w.fail_list2 = fail_list2.template as<int>(); w.n_fail2 = scalars.template as<int>() + 4;
        w.retry_qb = retry_qb.p; w.retry_qnorm = retry_qnorm.p;
        return w;
    }
    // Reads the sticky time-out word (the stream must be idle).
    psb_status check_status() const {
        if (!scalars.p) return PSB_OK;
        int st = 0;
        PSB_CUDA(cudaMemcpy(&st, scalars.template as<int>() + 2, sizeof(int), cudaMemcpyDeviceToHost));
        if (st) return fail(PSB_TIMEOUT, "a bounded wait in the tensor-core coarse kernel gave up");
        return PSB_OK;
    }
};

}  // namespace
}  // namespace psb

using namespace psb;

struct psb_session {
    TcIndexBuffers<DevBuf> tc_index;
    TcWorkBuffers<DevBuf> tc_work;
    int device = 0;
    int sm_count = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    cudaStream_t aux_stream = nullptr;  // second stream of the overlapped pipeline (created on first use)
    cudaStream_t zc_stream = nullptr;   // the gather kernel beside a scan runs here
    cudaEvent_t zc_ev_a = nullptr, zc_ev_b = nullptr;  // stage-level hybrid rerank: fork to and join from zc_stream

    cudaStream_t home_stream = nullptr; // the stream the session was created with (psb_session_set_stream(NULL) returns to it)
    bool background = false;            // stage calls currently run on a caller's second stream: small-grid gather
    psb_options opt{};
    // index shape
    int nlist = 0, dim = 0, m = 0, k = 0;
    long long n_vectors = 0;
    int list_begin = 0, list_end = 0;
    long long row_base = 0, shard_rows = 0;
    // device copies
    DevBuf centroids, offsets, reordered, codes, codebook, cb_maxnorm, global_begin, row_delta, exact_cache, row_aug, row_bias;
    bool striped = false;          // shard holds a slice of every list (options.list_global_begin)
    // exact rows
    int exact_elem = 0;            // 4 = fp32, 1 = u8, 0 = rerank disabled
    const void* exact_host = nullptr;
    const void* exact_dev = nullptr;  // device-visible pointer (mapped host or resident)
    bool mapped = false;           // exact_host is counted in mapped_rows()
    long long exact_count = 0;
    // staged mode
    void* pinned[2] = {nullptr, nullptr};
    size_t pinned_bytes = 0;
    cudaEvent_t pinned_ev[2] = {nullptr, nullptr};
    bool pinned_used[2] = {false, false};  // a copy out of the ring buffer may still be in flight (its event tells)
    int pinned_slot = 0;
    DevBuf opq, q_rot;                     // OPQ rotation [dim][dim] and the rotated queries of the batch in flight
    bool row_bias_is_u16 = false;          // row_bias holds the caller's affine u16 row correction
    bool flat = false;                     // IVF-Flat session: exact rows resident in flat_rows, no PQ parts
    DevBuf flat_rows, flat_norms, flat_whole, flat_slot, flat_again;   // norms: of every row, then the largest of each list
    EventPool timing, timing_aux;          // events of the main stream's marks and of the second stream's (set from one thread each)
    // Host side of a search call: one pinned block through which a small batch's queries and results pass, and the device's counters
    // and status words with the results, so that a call waits for the GPU once.
    unsigned char* h_io = nullptr;         // a block of HostBlocks: kSmallIo bytes, then the tail
    using Tail = CallTail;
    Tail* h_tail = nullptr;
    // Of the call at work (CallMarks): words of `scalars` in which its kernels note the starts of the coarse stage, the scan and the rerank, and
    // the queries, which the first kernel reads from the page-locked block, leaving a copy.  Null: events mark, a copy brings.
    unsigned long long* call_marks = nullptr;
    const float* host_queries = nullptr;
    float* query_copy = nullptr;
    bool one_stream = false;               // the call at work has no second stream: its kernels follow one another (launch_behind)
    static_assert(kSmallIo + sizeof(Tail) <= kHostBlock, "the tail lies behind the block's data");
    bool counters_known = false;           // h_tail->c is what the device's counters hold
    DevBuf row_dist, row_seg, row_runs, row_whole;   // a row of distances per query (IVF-Flat, row form of the ADC scan), the minima of every 32
    std::vector<long long> longest;        // [p] = rows of this shard's p longest lists together
    double own_list_rows = 0.0;            // expected length of the list a random row lies in
    std::unique_ptr<HostPool> host_pool;   // gather threads of the staged transport (created on first use)
    double staged_gather_s = 0.0;          // host time spent gathering rows, and the bytes gathered (reported by the bench)
    long long staged_gather_bytes = 0;
    // Rows of a large batch cross to the device once each: the slot of every row held here, the rows by slot, the number of slots and
    // where each sub-batch's begin (PartMarks).
    DevBuf slot_of, unique, marks, row_bits, row_sums;
    bool slots_dirty = true;             // slot_of is not all -1, or row_bits not as rows_claim expects them (a batch was left half done)
    int bits_turn = 0;                   // the half of row_bits the next claim uses: all 0
    int* h_unique = nullptr;             // pinned: the slots the host threads fill
    size_t h_unique_count = 0;
    size_t slots = 0;                    // of the batch at work, at most
    size_t parts = 0;                    // of the batch at work
    int* h_marks = nullptr;              // pinned
    size_t h_marks_words = 0;
    cudaStream_t list_stream = nullptr;  // brings the slot lists to the host thread beside the row copies
    std::vector<long long> h_global_begin;  // striped shards: host copy of the slices' first rows
    // workspaces
    DevBuf q, q_u8, dist_tile, probes, lut, vis_count, vis_off, vis_cursor, item_off, item_off_tc, visitors, q_rows, thr,
        pool_cnt, pool, fail_list, fallback_partial, scan_whole, call_whole, rows_whole, scalars, lut_h, lut_scale, cand_rows, cand_dist, cand_count, stage, score, out_rows, out_dist, out_ids;
    int ws_scan_queries = 0;        // queries the scan workspace (visitors, pools, cutoffs) currently holds
    long long ws_scan_tables = 0;   // tables the fp16 table buffer currently holds
    int pool_cap = 0;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> scan_events;  // pending (options.time_kernels)
    double scan_ms_total = 0.0;
    long long scan_launches_total = 0;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> gemm_events;  // pending coarse GEMM passes (options.time_kernels)
    double gemm_ms_total = 0.0;
    long long gemm_launches_total = 0;

    bool counted = false;           // among its device's sessions
    static std::atomic<int>& sessions(int device) { static std::atomic<int> n[64]; return n[device & 63]; }
    void count() { counted = true; sessions(device).fetch_add(1); }

    psb_session() = default;
    psb_session(const psb_session&) = delete;
    psb_session& operator=(const psb_session&) = delete;
    // Releases what the session owns; runs for a partially built session too (every failure path of psb_session_create),
    // so the caller's rows never stay pinned after an error.
    ~psb_session() {
        cudaSetDevice(device);
        if (stream) cudaStreamSynchronize(stream);
        if (home_stream) {  // a redirected session: drain and return to the stream it was created with
            cudaStreamSynchronize(home_stream);
            stream = home_stream;
        }
        // A search that returned an error may have left work on its other streams: nothing they use is given back before they have drained.
        for (cudaStream_t other : {list_stream, aux_stream, zc_stream})
            if (other) { cudaStreamSynchronize(other); cudaStreamDestroy(other); }
        collect_scan_events();
        if (mapped) mapped_rows().give(exact_host, (size_t)exact_count * dim * exact_elem);
        for (int i = 0; i < 2; ++i) {
            if (pinned[i]) cudaFreeHost(pinned[i]);
            if (pinned_ev[i]) cudaEventDestroy(pinned_ev[i]);
        }
        if (h_unique) cudaFreeHost(h_unique);
        if (h_marks) cudaFreeHost(h_marks);
        if (h_io) HostBlocks::get().give(h_io);
        if (zc_ev_a) cudaEventDestroy(zc_ev_a);
        if (zc_ev_b) cudaEventDestroy(zc_ev_b);

        if (own_stream && stream) cudaStreamDestroy(stream);
        if (counted && sessions(device).fetch_sub(1) == 1) trim_pool(device);
        cudaGetLastError();
    }

    ScanIndex scan_index() const {
        ScanIndex ix;
        ix.codes = codes.as<uint8_t>(); ix.offsets = offsets.as<long long>(); ix.row_base = row_base;
        ix.nlist = nlist; ix.list_begin = list_begin; ix.list_end = list_end; ix.m = m; ix.k = k;
        ix.row_delta = striped ? row_delta.as<long long>() : nullptr;
        ix.residual = opt.adc_mode == 1;
        ix.centroids = centroids.as<float>(); ix.codebook = codebook.as<float>(); ix.dim = dim; ix.row_aug = row_aug.p; if (row_bias_is_u16) { ix.row_bias_u16 = row_bias.as<uint16_t>(); ix.rc_scale = opt.rc_scale; ix.rc_offset = opt.rc_offset; }
        else ix.row_bias = row_bias.as<float>();
        return ix;
    }
    // Which index-wide rows the exact store and the id table of this session hold.
    RowMap row_map() const {
        RowMap mp;
        if (striped) {
            mp.global_begin = global_begin.as<long long>(); mp.local_offsets = offsets.as<long long>(); mp.nlist = nlist;
        }
        mp.base = 0; mp.count = n_vectors;
        return mp;
    }
    // Reads (and clears) the time-out word of the tensor-core scan; the stream must be idle.
    psb_status check_scan_status() {
        if (!scalars.p) return PSB_OK;
        int st = 0;
        int* word = reinterpret_cast<int*>(scalars.as<unsigned long long>() + 12);
        PSB_CUDA(cudaMemcpy(&st, word, sizeof(int), cudaMemcpyDeviceToHost));
        if (st) {
            PSB_CUDA(cudaMemset(word, 0, sizeof(int)));
            return fail(PSB_TIMEOUT, "a bounded wait in the tensor-core scan kernel gave up");
        }
        return PSB_OK;
    }
    ScanWorkspace scan_ws() const {
        ScanWorkspace w;
        w.vis_count = vis_count.as<int>(); w.vis_off = vis_off.as<int>(); w.vis_cursor = vis_cursor.as<int>();
        w.item_off = item_off.as<long long>(); w.visitors = visitors.as<int>(); w.q_rows = q_rows.as<long long>();
        w.thr = thr.as<float>(); w.pool_cnt = pool_cnt.as<int>(); w.pool = pool.as<uint64_t>();
        w.fail_list = fail_list.as<int>();
        w.fallback_partial = fallback_partial.as<uint64_t>();
        unsigned long long* sc = scalars.as<unsigned long long>();
        w.counters = sc;                                   // [0..7]
        w.work_cursor = sc + 8;
        w.n_fail = reinterpret_cast<int*>(sc + 9);
        w.fail_cursor = reinterpret_cast<int*>(sc + 10);
        w.pool_cap = pool_cap;
        w.lut_h = lut_h.p; w.lut_scale = lut_scale.as<float>(); w.scan_mode = opt.scan_mode;
        w.reserve_ctas = opt.reserve_sms;
        w.seed_sigma = opt.seed_sigma;
        w.item_off_tc = item_off_tc.as<long long>(); w.work_cursor_tc = sc + 11; w.tc_status = reinterpret_cast<int*>(sc + 12);
        w.tc_min_visitors = opt.tc_min_visitors; w.tc_wait_limit = opt.test_wait_limit; w.tc_issue_tiles = opt.test_skip_mma & 1 ? 0 : opt.test_skip_mma & 4 ? 3 : -1;
        w.cap_queries = ws_scan_queries; w.cap_tables = ws_scan_tables;
        return w;
    }
    // Scan workspace with a fresh event pair when kernel timing is on.
    psb_status timed_scan_ws(ScanWorkspace* w) {
        *w = scan_ws();
        if (!opt.time_kernels) return PSB_OK;
        cudaEvent_t a, b;
        PSB_CUDA(cudaEventCreate(&a));
        PSB_CUDA(cudaEventCreate(&b));
        scan_events.emplace_back(a, b);
        w->ev_begin = a; w->ev_end = b;
        return PSB_OK;
    }
    // Folds finished event pairs into the totals (call after a stream synchronisation).
    void collect_scan_events() {
        for (auto& pr : scan_events) {
            float t = 0.f;
            if (cudaEventElapsedTime(&t, pr.first, pr.second) == cudaSuccess) { scan_ms_total += t; ++scan_launches_total; }
            cudaEventDestroy(pr.first); cudaEventDestroy(pr.second);
        }
        scan_events.clear();
        for (auto& pr : gemm_events) {
            float t = 0.f;
            if (cudaEventElapsedTime(&t, pr.first, pr.second) == cudaSuccess) { gemm_ms_total += t; ++gemm_launches_total; }
            cudaEventDestroy(pr.first); cudaEventDestroy(pr.second);
        }
        gemm_events.clear();
        cudaGetLastError();
    }
};

namespace {

// Plain mode: the rerank runs when exact rows exist and n_rerank > topk.  Residual mode: always (the rows are required).
bool rerank_enabled(const psb_session* s, int topk) {
    if (s->opt.adc_mode == 1) return true;
    return s->exact_elem != 0 && s->opt.n_rerank > topk;
}

int stage1_width(const psb_session* s, int topk) {
    if (s->opt.adc_mode == 1)  // src/search/ivfrespq/stage/ivfrespq_cpu_rerank.cpp:623-625
        return std::max(std::max(s->opt.n_rerank, topk), 512);
    if (!rerank_enabled(s, topk)) return topk;
    return (int)std::min<long long>(s->opt.n_rerank, s->n_vectors);
}

// Residual mode without tables: when the tensor-core scan takes every list, nothing reads a materialised per-(query, probe)
// table - the cutoff, the re-scoring selection and the fallback build entries from the query, the centroid and the codebook.
bool residual_table_free(const psb_session* s, int stage1_k) {
    return s->opt.adc_mode == 1 && s->row_aug.p != nullptr && s->row_bias.p != nullptr && (s->opt.scan_mode == 0 || s->opt.scan_mode == 3) &&
           s->opt.tc_min_visitors <= 1 && scan_tc_supported(s->dim, s->m, s->k) &&
           (size_t)pool_capacity(stage1_k) * 8 + (size_t)s->dim * 4 <= (size_t)226 * 1024;
}

// Tables one scan call needs for nq queries.
size_t table_count(const psb_session* s, int nq, int nprobe) {
    return s->opt.adc_mode == 1 ? (size_t)nq * nprobe : (size_t)nq;
}

void note_list_lengths(psb_session* s, const int64_t* offsets) {
    std::vector<long long> len;
    double sq = 0.0;
    for (int l = s->list_begin; l < s->list_end; ++l) { len.push_back(offsets[l + 1] - offsets[l]); sq += (double)len.back() * (double)len.back(); }
    std::sort(len.begin(), len.end(), std::greater<long long>());
    s->longest.assign((size_t)s->nlist + 1, 0);
    for (size_t p = 0; p < (size_t)s->nlist; ++p) s->longest[p + 1] = s->longest[p] + (p < len.size() ? len[p] : 0);
    s->own_list_rows = s->shard_rows > 0 ? sq / (double)s->shard_rows : 0.0;
}

// Words of a session's `scalars`: counters [0..7], work words of the scan and its status [8..12], call marks [13..15], rows fetched.
constexpr size_t kScalars = 24, kRowsFetched = 16;
constexpr long long kRowDistFloats = 1ll << 28;   // distances kept at a time in the row forms: 1 GiB
constexpr long long kPartQueries = 32768;         // queries at a time: they are the grid's second dimension, which ends at 65,535

// Rows a query is expected to scan: its own list's, found in proportion to its length, and those of nprobe - 1 others.
double expected_rows(const psb_session* s, int nprobe) {
    return std::min((double)s->longest[(size_t)std::min(nprobe, s->nlist)], s->own_list_rows + (nprobe - 1) * (double)s->shard_rows / std::max(1, s->nlist));
}

// Whether the ADC scan of nq queries takes its row form (adc_rows.cu).  It starts some 130 us (residual 170) before the list-centric
// scan, a chain of a dozen kernels more, has seen its first row; but its cost per query grows with the visited rows, 4 ns a thousand more
// than the tensor-core filter's and 0.32 ns per sub-space's look-up, and in residual mode with a table per probe, while the
// list-centric scan takes 0.1 us (residual 0.35) a query whatever it visits.  Fitted to both forms at 128 to 4,096 queries over 0.3 to
// 2 million rows, m = 8 to 48, 16 to 64 probes: the line lies where they meet to within 10 % of the time - at 240 queries for 31,000
// rows of m = 48 each, 1,200 for m = 8; lists so short that a query's rows cost less than its fixed share stay with the row form.
// Shapes the filter does not take: in residual mode the row form at any size (0.2 to 0.95 of the list-centric scan's time over twelve
// shapes of dim 60 to 960, m = 8 to 64, at 1 to 6,000 queries; 1.3 at 32 queries of dim 960).  In plain mode the list-centric scan starts
// some 40 us later, 0.1 more for a thousand rows a query visits, and takes 0.29 us more a query, but less a row (a list's visitors share
// its codes) and builds one table per query, where the row form builds one per 4,096 rows or fewer - from codewords of other than 2, 4 or 8
// elements by scalar loads, whose bank conflicts are the common factor of that length and 32.  Fitted to both forms of 29 such shapes
// and 168 drawn batches, 1 to 10,000 queries: the form chosen is on average 0.7 % and at most 21 % slower than the other would have been.
// 10,000 queries of 31,000 rows each: rows 7.8 ms and lists 3.4 for dim 128, m = 8, 13.2 and 4.5 for dim 256, m = 16; of 14,000 rows, dim
// 100, m = 20, 2.9 and 3.3.
// any_probes: the caller's own probes, which may name a list more than once.
long long row_stride(const psb_session* s, int nprobe, bool any_probes) {
    return std::max<long long>(1, any_probes ? s->longest[1] * nprobe : s->longest[(size_t)nprobe]);
}
bool rows_form(const psb_session* s, int nq, int nprobe, bool any_probes = false) {
    if (s->opt.scan_mode != 0 || s->opt.tc_min_visitors > 1 || s->opt.test_wait_limit || s->opt.test_skip_mma || s->longest.empty()) return false;
    const long long stride = row_stride(s, nprobe, any_probes);
    const size_t smem = ((size_t)s->m * s->k + s->dim + nprobe + 1) * 4;
    if (stride > kRowDistFloats || smem > (size_t)220 * 1024) return false;
    const bool residual = s->opt.adc_mode == 1;
    const double visits = expected_rows(s, nprobe);
    if (s->row_aug.p == nullptr) {
        if (residual) return true;
        const int dsub = s->dim / s->m;
        const bool wide = dsub == 2 || dsub == 4 || dsub == 8;
        const double tables = wide ? 0.0 : std::max(1.0, std::ceil(visits / adc_rows_block(nq * visits, s->sm_count)));
        const double table = (double)s->dim * s->k * (8e-7 + 7e-8 * std::gcd(dsub, 32));   // us
        return nq * (visits * (8e-6 - 4e-8 * s->m) + tables * table - 0.29) <= 40.0 + 1e-4 * visits;
    }
    const double per_query = visits * (4e-6 + 3.2e-7 * s->m) + (residual ? nprobe * (0.008 + 2.3e-4 * s->m) - 0.35 : -0.1);   // us
    return nq * per_query <= (residual ? 170.0 : 130.0);
}

// Whether a stage call may leave its tables out, whatever the size of its batch: residual mode where the tensor-core scan takes every list,
// or where the row form takes every batch (shapes without a filter, a shard without rows).
bool tables_optional(const psb_session* s, int nprobe, int stage1_k) {
    return residual_table_free(s, stage1_k) || (s->opt.adc_mode == 1 && s->row_aug.p == nullptr && rows_form(s, 1, nprobe, true));
}

// Queries per sub-batch of the pipeline: a quarter of the batch when the rerank overlaps the scan, and in residual mode
// few enough that the per-(query, probe) tables stay below ~16 GiB.
int sub_batch_rows(const psb_session* s, int n, int nprobe, bool overlap) {
    const int pipeline_parts = s->opt.pipeline_parts >= 2 && s->opt.pipeline_parts <= 32 ? s->opt.pipeline_parts : 4;
    const bool tables = s->opt.adc_mode == 1 && !residual_table_free(s, stage1_width(s, 1)) && !rows_form(s, n, nprobe);
    return part_rows(n, overlap ? pipeline_parts : 1, tables ? (double)nprobe * s->m * s->k * sizeof(float) : 0.0);
}

int host_share(const psb_session* s);
bool device_rows(const psb_session* s);
bool rows_in_place(const psb_session* s, long long requests);
// The staged transport (host gather threads + pinned rings), alone or with the kernel gather beside it.
bool staged_mode(const psb_session* s) { return !device_rows(s) && host_share(s) > 0; }

bool overlap_enabled(const psb_session* s, int n, bool rerank) {
    return rerank && !staged_mode(s) && n >= 2048 && !s->opt.serial_pipeline;
}

bool staged_overlap_enabled(const psb_session* s, int n, bool rerank) { return rerank && staged_mode(s) && n >= 2048 && !s->opt.serial_pipeline; }

// Whether the rows of a whole batch are claimed and fetched once each, sub-batch by sub-batch.
bool rows_shared(const psb_session* s, int n, int stage1_k, bool rerank) {
    return staged_overlap_enabled(s, n, rerank) || (overlap_enabled(s, n, rerank) && !rows_in_place(s, (long long)n * stage1_k));
}

// Sub-batch boundaries of a batch.  Equal cuts, except where rows of host memory are fetched beside the scan.  There the transfer is about as
// long as the scan and costs it little, so the first sub-batch is a small one: the transfer starts early.  Where the kernel fetches, the cuts grow so
// that a sub-batch's scan takes about as long as the transfer of the one before, and the last is small again, for nothing hides its transfer
// (100M x 96, 10,000 queries x 1,000 candidates: 12/18/22/26/22 % 84.3 ms, 10/20/20/25/25 86.1, 10/30/30/30 88.6, seven parts 90.3; no difference
// at 1M to 12M rows).  Host threads are slower than the scan: 10/30/30/30 %.  Where the kernel fetches, a number of sub-batches that the caller gives
// means that many equal ones.
std::vector<int> batch_cuts(const psb_session* s, int n, int nprobe, int stage1_k, bool rerank) {
    const int sb = sub_batch_rows(s, n, nprobe, overlap_enabled(s, n, rerank) || staged_overlap_enabled(s, n, rerank));
    const int plan = s->opt.pipeline_parts != 0 && host_share(s) == 0 ? 1 : s->opt.even_cuts;
    if (rows_shared(s, n, stage1_k, rerank) && (s->opt.adc_mode != 1 || residual_table_free(s, stage1_k)) && sb * 4 >= n && n >= 4096 && plan != 1) {
        if (plan == 2) return {0, (int)(0.32 * n), (int)(0.64 * n), (int)(0.90 * n), n};  // short last sub-batch (scan-bound hosts)
        if (host_share(s) == 0) return {0, (int)(0.12 * n), (int)(0.30 * n), (int)(0.52 * n), (int)(0.78 * n), n};
        return {0, (int)(0.10 * n), (int)(0.40 * n), (int)(0.70 * n), n};
    }
    return even_cuts(n, sb);
}
int longest_cut(const std::vector<int>& cuts) {
    int most = 0;
    for (size_t i = 0; i + 1 < cuts.size(); ++i) most = std::max(most, cuts[i + 1] - cuts[i]);
    return most;
}

psb_status ensure_scalars(psb_session* s, cudaStream_t st) {
    if (s->scalars.p) return PSB_OK;
    PSB_TRY(s->scalars.reserve(sizeof(unsigned long long) * kScalars));
    PSB_CUDA(cudaMemsetAsync(s->scalars.p, 0, sizeof(unsigned long long) * kScalars, st));
    return PSB_OK;
}
// Grows the scan workspace to hold nq queries (never shrinks; a growing buffer is freed first, which waits for the device).
// row_form: the scan's row form takes this call.  It uses the counters alone of all that follows; its distances are run_scan's.
psb_status ensure_scan_ws(psb_session* s, int nq, int nprobe, int stage1_k, bool row_form) {
    PSB_TRY(ensure_scalars(s, s->stream));
    if (row_form) return PSB_OK;
    const size_t tables = table_count(s, nq, nprobe);
    s->ws_scan_queries = 0; s->ws_scan_tables = 0;  // set again below once every buffer has its size
    const int cap = pool_capacity(stage1_k);
    const bool half_tables = s->opt.scan_mode != 1 && !residual_table_free(s, stage1_k);
    const size_t n = (size_t)nq, nl = (size_t)s->nlist;
    PSB_TRY(reserve_together(&s->scan_whole, {{&s->vis_count, sizeof(int) * nl}, {&s->vis_off, sizeof(int) * (nl + 1)}, {&s->vis_cursor, sizeof(int) * nl},
                                              {&s->item_off, sizeof(long long) * (nl + 1)}, {&s->item_off_tc, sizeof(long long) * (nl + 1)},
                                              {&s->visitors, sizeof(int) * n * nprobe}, {&s->q_rows, sizeof(long long) * n}, {&s->thr, sizeof(float) * n},
                                              {&s->pool_cnt, sizeof(int) * n}, {&s->pool, sizeof(uint64_t) * n * cap}, {&s->fail_list, sizeof(int) * n},
                                              {&s->fallback_partial, fallback_partial_bytes(stage1_k)},
                                              {&s->lut_h, half_tables ? sizeof(unsigned short) * tables * s->m * s->k : 0},
                                              {&s->lut_scale, half_tables ? sizeof(float) * tables : 0}}));
    s->pool_cap = cap;
    // what the buffers hold now (reserve() keeps a larger buffer from an earlier call)
    s->ws_scan_queries = (int)std::min<size_t>({s->q_rows.bytes / sizeof(long long), s->thr.bytes / sizeof(float),
                                                s->pool_cnt.bytes / sizeof(int), s->fail_list.bytes / sizeof(int),
                                                s->pool.bytes / (sizeof(uint64_t) * (size_t)cap),
                                                s->visitors.bytes / (sizeof(int) * (size_t)nprobe), (size_t)INT_MAX});
    s->ws_scan_tables = half_tables ? (long long)std::min(s->lut_h.bytes / (sizeof(unsigned short) * (size_t)s->m * s->k),
                                                                    s->lut_scale.bytes / sizeof(float))
                                              : (long long)tables;
    return PSB_OK;
}

// Queries that the row form takes at a time, at most, and its workspace for batches of up to nq.
int row_part(long long stride) { return (int)std::max<long long>(1, std::min(kPartQueries, kRowDistFloats / stride)); }
psb_status ensure_row_ws(psb_session* s, int nq, int nprobe, bool any_probes) {
    const long long stride = row_stride(s, nprobe, any_probes);
    const size_t per = (size_t)std::min(nq, row_part(stride));
    return reserve_together(&s->row_whole, {{&s->row_dist, sizeof(float) * per * stride}, {&s->row_seg, sizeof(int) * per * ((size_t)nprobe + 1)},
                                            {&s->row_runs, sizeof(float) * per * sel::run_count(stride)}});
}

// The ADC scan of one sub-batch.  d_lut may be null in the row form (it then builds its tables in shared memory) and as launch_scan
// allows; tables that are given are what every form scores from.  rows_only: ensure_scan_ws was told of the row form, so nothing else
// has its buffers.
psb_status run_scan(psb_session* s, const ScanWorkspace& ws, bool rows_only, const float* d_queries, const float* d_lut, int nq, const int* d_probes,
                    int nprobe, int stage1_k, int* d_rows, float* d_dist, int* d_count, cudaStream_t st, bool any_probes = false) {
    if (!rows_only && (!d_queries || !rows_form(s, nq, nprobe, any_probes)))
        return launch_scan(s->scan_index(), ws, d_lut, nq, d_probes, nprobe, stage1_k, d_rows, d_dist, d_count, s->sm_count, st, d_queries);
    AdcRows g{};
    g.stride = row_stride(s, nprobe, any_probes);
    const int most = row_part(g.stride), parts = (nq + most - 1) / most, per = (nq + parts - 1) / parts;
    g.run_stride = sel::run_count(g.stride);
    PSB_TRY(ensure_row_ws(s, nq, nprobe, any_probes));
    const ScanIndex ix = s->scan_index();
    g.nprobe = nprobe; g.centroids = ix.centroids; g.codebook = ix.codebook; g.codes = ix.codes; g.offsets = ix.offsets; g.row_base = ix.row_base;
    g.row_delta = ix.row_delta; g.list_begin = ix.list_begin; g.list_end = ix.list_end; g.dim = ix.dim; g.m = ix.m; g.k = ix.k;
    g.residual = ix.residual; g.tree = scan_tree_order(ix); g.stage1_k = stage1_k; g.seg = s->row_seg.as<int>(); g.dist = s->row_dist.as<float>();
    g.expected_rows = expected_rows(s, nprobe); g.longest_list = s->longest[1]; g.counters = ws.counters; g.sm_count = s->sm_count;
    g.mark = s->call_marks ? s->call_marks + 1 : nullptr; g.chained = s->one_stream;
    if (ws.ev_begin) PSB_CUDA(cudaEventRecord(ws.ev_begin, st));
    for (int q0 = 0; q0 < nq; q0 += per) {
        g.queries = d_queries + (size_t)q0 * s->dim; g.probes = d_probes + (size_t)q0 * nprobe;
        g.lut = d_lut ? d_lut + (size_t)q0 * table_count(s, 1, nprobe) * s->m * s->k : nullptr;
        g.out_rows = d_rows + (size_t)q0 * stage1_k; g.out_dist = d_dist ? d_dist + (size_t)q0 * stage1_k : nullptr;
        g.out_count = d_count ? d_count + q0 : nullptr;
        g.runs = !ix.residual && std::min(per, nq - q0) <= sel::kRunQueries ? s->row_runs.as<float>() : nullptr;
        PSB_TRY(launch_adc_rows(g, std::min(per, nq - q0), st));
    }
    if (ws.ev_end) PSB_CUDA(cudaEventRecord(ws.ev_end, st));
    return PSB_OK;
}

psb_status ensure_pipeline_ws(psb_session* s, int nq, int nprobe, int topk, int stage1_k) {
    // For the longest sub-batch: a session's first call lays its workspace out once (for a quarter of the batch where a cut is longer, it was freed and
    // laid out anew within the call, 1.5 ms of 10.1).
    const int sb = longest_cut(batch_cuts(s, nq, nprobe, stage1_k, rerank_enabled(s, topk)));
    const size_t n = (size_t)nq;
    PSB_TRY(reserve_together(&s->call_whole, {{&s->q, sizeof(float) * n * s->dim}, {&s->probes, sizeof(int) * n * nprobe},
                                              {&s->cand_rows, sizeof(int) * n * stage1_k},
                                              {&s->cand_dist, sizeof(float) * n * stage1_k}, {&s->cand_count, sizeof(int) * n},
                                              {&s->out_rows, sizeof(int) * n * topk}, {&s->out_dist, sizeof(float) * n * topk},
                                              {&s->out_ids, sizeof(long long) * n * topk}}));
    if (!residual_table_free(s, stage1_k) && !rows_form(s, sb, nprobe)) PSB_TRY(s->lut.reserve(sizeof(float) * table_count(s, sb, nprobe) * s->m * s->k));
    return ensure_scan_ws(s, sb, nprobe, stage1_k, rows_form(s, sb, nprobe));  // the scan runs one sub-batch at a time
}

bool coarse_by_tc(const psb_session* s, int nq, int nprobe) { return s->tc_index.ready && coarse_tc_supported(nq, s->nlist, s->dim, nprobe); }
// Queries whose distances to all centroids the exact coarse stage keeps at a time, and the bytes they take (0: the tensor cores search).
int exact_coarse_chunk(const psb_session* s, int nq) {
    return std::min(nq, (int)std::max<size_t>(64, ((size_t)1 << 30) / (sizeof(float) * (size_t)s->nlist)));
}
size_t exact_coarse_bytes(const psb_session* s, int nq, int nprobe) {
    return s->opt.coarse_mode != 1 && coarse_by_tc(s, nq, nprobe) ? 0 : sizeof(float) * (size_t)s->nlist * exact_coarse_chunk(s, nq);
}
// Coarse stage on device queries: exact distance tiles + row selection, query-chunked so the distance tile
// stays below ~1 GiB.
psb_status coarse_exact(psb_session* s, const float* d_queries, int nq, int nprobe, int* d_ids, float* d_dist) {
    const int mode = s->opt.coarse_mode;
    const bool tc_ok = coarse_by_tc(s, nq, nprobe);
    if (mode == 2 && !tc_ok) return fail(PSB_UNSUPPORTED_SHAPE, "tensor-core coarse stage does not support this shape");
    if (mode != 1 && tc_ok) {
        PSB_TRY(s->tc_work.ensure(nq, s->nlist, s->dim, nprobe, s->device, s->stream));
        CoarseTcWorkspace tw = s->tc_work.view();
        tw.test_wait_limit = s->opt.test_wait_limit; tw.test_load_tiles = s->opt.test_skip_mma & 2 ? 0 : s->opt.test_skip_mma & 8 ? 3 : -1;
        if (s->opt.time_kernels) {
            for (int i = 0; i < 4; ++i) PSB_CUDA(cudaEventCreate(&tw.ev[i]));
            s->gemm_events.emplace_back(tw.ev[0], tw.ev[1]);
            s->gemm_events.emplace_back(tw.ev[2], tw.ev[3]);
        }
        return launch_coarse_tc(s->tc_index.view(s->centroids.as<float>(), s->nlist, s->dim), tw, d_queries,
                                nq, nprobe, d_ids, d_dist, s->sm_count, s->stream);
    }
    const int chunk = exact_coarse_chunk(s, nq);
    PSB_TRY(s->dist_tile.reserve(sizeof(float) * (size_t)s->nlist * chunk));
    for (int q0 = 0; q0 < nq; q0 += chunk) {
        const int n = std::min(chunk, nq - q0);
        PSB_TRY(launch_coarse_dist_exact(s->host_queries ? s->host_queries : d_queries + (size_t)q0 * s->dim, n, s->centroids.as<float>(), s->nlist, s->dim,
                                         s->dist_tile.as<float>(), s->sm_count, s->stream, q0 == 0 ? s->call_marks : nullptr, s->query_copy));
        PSB_TRY(launch_select_rows(s->dist_tile.as<float>(), n, s->nlist, nprobe, d_ids + (size_t)q0 * nprobe,
                                   d_dist ? d_dist + (size_t)q0 * nprobe : nullptr, s->stream));
    }
    return PSB_OK;
}

psb_status validate_index(const psb_index_view* ix) {
    if (!ix) return fail(PSB_INVALID_ARGUMENT, "index view is null");
    const auto& L = ix->lists;
    if (!L.offsets) return fail(PSB_INVALID_ARGUMENT, "IVF list offsets are null");
    if (L.nlist <= 0 || L.n_vectors < 0) return fail(PSB_INVALID_ARGUMENT, "invalid IVF list layout shape");
    if (L.n_vectors > 0 && !L.reordered_ids) return fail(PSB_INVALID_ARGUMENT, "IVF reordered IDs are null");
    if (L.offsets[0] != 0) return fail(PSB_INVALID_ARGUMENT, "IVF list offsets must start at zero");
    for (int l = 0; l < L.nlist; ++l) {
        const int64_t b = L.offsets[l], e = L.offsets[l + 1];
        if (e < b) return fail(PSB_INVALID_ARGUMENT, "IVF list offsets must be monotonic");
        if (e - b > INT_MAX) return fail(PSB_INVALID_ARGUMENT, "IVF list size exceeds int32 backend limit");
    }
    if (L.offsets[L.nlist] != L.n_vectors) return fail(PSB_INVALID_ARGUMENT, "IVF terminal offset does not match n_vectors");
    if (L.n_vectors > INT_MAX) return fail(PSB_INVALID_ARGUMENT, "n_vectors exceeds int32 row index limit");
    const auto& C = ix->coarse;
    if (!C.centroids || C.nlist != L.nlist || C.dim <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid IVF coarse index view");
    const auto& P = ix->pq;
    if (!P.codes && L.n_vectors > 0) return fail(PSB_INVALID_ARGUMENT, "PQ codes are null");
    if (P.code_storage) return fail(PSB_UNSUPPORTED_SHAPE, "paged CPU code storage is not supported; pass row-major codes");
    if (!P.codebook || P.subvectors <= 0 || C.dim % P.subvectors != 0)
        return fail(PSB_INVALID_ARGUMENT, "PQ subvectors must divide dim");
    if (P.codebook_size <= 0 || P.codebook_size > kMaxCodebook) return fail(PSB_INVALID_ARGUMENT, "PQ codebook_size must be in 1..256");
    const auto& E = ix->exact;
    if (E.fp32 || E.u8) {
        if (E.count != L.n_vectors || E.dim != C.dim) return fail(PSB_INVALID_ARGUMENT, "exact storage shape does not match the index");
        if (E.source_rows) return fail(PSB_UNSUPPORTED_SHAPE, "exact storage with a row permutation is not supported");
    }
    return PSB_OK;
}

psb_status validate_params(const psb_session* s, const psb_query_batch_view* qv, const psb_search_params* p,
                           const psb_search_output_view* out) {
    if (!qv || !p || !out) return fail(PSB_INVALID_ARGUMENT, "null query, params or output view");
    if (qv->count < 0 || qv->dim != s->dim) return fail(PSB_INVALID_ARGUMENT, "query dim does not match the index");
    if (qv->count > 0 && !qv->fp32) return fail(PSB_INVALID_ARGUMENT, "fp32 queries are required");
    if (p->nprobe <= 0 || p->nprobe > s->nlist) return fail(PSB_INVALID_ARGUMENT, "nprobe must be in 1..nlist");
    if (p->topk <= 0) return fail(PSB_INVALID_ARGUMENT, "topk must be positive");
    if (p->batch_size <= 0) return fail(PSB_INVALID_ARGUMENT, "batch_size must be positive");
    if (p->distance != 0) return fail(PSB_UNSUPPORTED_SHAPE, "only squared L2 is supported on this path");
    if (p->nprobe > kMaxProbe) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 is not supported");
    if (p->topk > kMaxTopk) return fail(PSB_UNSUPPORTED_SHAPE, "topk above 2048 is not supported");
    if (qv->count > 0 && (!out->indices || !out->distances)) return fail(PSB_INVALID_ARGUMENT, "output buffers are null");
    if (qv->count > 0 && s->exact_elem == 1 && rerank_enabled(s, p->topk) && !qv->u8) return fail(PSB_INVALID_ARGUMENT, "u8 rerank needs u8 queries");
    return PSB_OK;
}

// Bytes of candidates' rows from which a batch's rows are fetched once each.  Claiming them costs 18 us more of launches and then saves what is
// asked for more than once, and for rows longer than a line the slower reads of scoring in place.  In place against claimed, whole search, us:
// 512-byte rows, 8,000 requests 205 / 209, 16,000 342 / 308, 64,000 1,158 / 856; 256-byte ones, 16,000 217 / 217, 64,000 631 / 521; 128-byte
// ones, 32,000 236 / 246, 64,000 342 / 328, 260,000 1,219 / 898; 32-byte ones, 130,000 313 / 325, 260,000 579 / 485.
// Where a caller has host threads bring a share, handing the work to them costs 2 ms more: that line counts requests.
constexpr long long kClaimBytes = 4500000, kClaimBytesShort = 6500000, kClaimRequestsThreads = 65536;

// Staged rerank transport: host threads gather exact rows into two pinned buffers, and cudaMemcpyAsync moves each filled buffer
// while the other is being filled.  h_rows: the rows of `count` consecutive slots; d_stage: the first slot's place; copies are queued
// on `stream`.
psb_status staged_gather_host(psb_session* s, const int* h_rows, size_t count, void* d_stage, cudaStream_t stream) {
    if (count == 0) return PSB_OK;
    const size_t row_bytes = (size_t)s->dim * s->exact_elem;
    // Sized for the batch, not for the part: growing the buffers from part to part waits for the device every time.  (Buffers of 16 MB, so
    // that a part's first copy starts sooner, cost more in handing out the work: 4,096 queries x 1,000 rows 18.9 -> 25.0 ms.)
    const size_t chunk = std::max<size_t>(1, ((size_t)64 << 20) / std::max<size_t>(1, row_bytes));
    const size_t need = std::min(chunk, std::max<size_t>(std::max(count, s->slots), 4096)) * row_bytes;
    if (s->pinned_bytes < need) {
        for (int i = 0; i < 2; ++i) {
            if (s->pinned_used[i]) PSB_CUDA(cudaEventSynchronize(s->pinned_ev[i]));  // no copy may still read the old buffer
            s->pinned_used[i] = false;
            if (s->pinned[i]) cudaFreeHost(s->pinned[i]);
            s->pinned[i] = nullptr;
            PSB_CUDA(cudaHostAlloc(&s->pinned[i], need, cudaHostAllocDefault));
            if (!s->pinned_ev[i]) PSB_CUDA(cudaEventCreateWithFlags(&s->pinned_ev[i], cudaEventDisableTiming));
        }
        s->pinned_bytes = need;
    }
    if (!s->host_pool) {
        const unsigned hc = s->opt.host_threads > 0 ? (unsigned)s->opt.host_threads : std::max(1u, std::thread::hardware_concurrency());
        s->host_pool.reset(new HostPool((int)std::min<unsigned>(hc, 64)));
    }
    const int nthreads = s->host_pool->size();
    const size_t per = s->pinned_bytes / row_bytes;
    // The ring state outlives the call: the next call may start while this call's last copy is still in flight.
    for (size_t i0 = 0; i0 < count; i0 += per, s->pinned_slot ^= 1) {
        const int slot = s->pinned_slot;
        const size_t total = std::min(per, count - i0);
        if (s->pinned_used[slot]) PSB_CUDA(cudaEventSynchronize(s->pinned_ev[slot]));
        unsigned char* dst = static_cast<unsigned char*>(s->pinned[slot]);
        const unsigned char* src = static_cast<const unsigned char*>(s->exact_host);
        const int* rows = h_rows + i0;
        const auto t_begin = std::chrono::steady_clock::now();
        s->host_pool->run([&](int t) {
            // Rows sit at random places of a host array far larger than the caches: each copy would wait for DRAM.  The row kAhead
            // places on is prefetched while the current one is copied, so a thread keeps several misses in flight.
            constexpr size_t kAhead = 8;
            const size_t b = total * t / nthreads, e = total * (t + 1) / nthreads;
            auto prefetch = [&](size_t i) {
                for (size_t off = 0; off < row_bytes; off += 64) __builtin_prefetch(src + (size_t)rows[i] * row_bytes + off, 0, 0);
            };
            for (size_t i = b; i < std::min(e, b + kAhead); ++i) prefetch(i);
            for (size_t i = b; i < e; ++i) {
                if (i + kAhead < e) prefetch(i + kAhead);
                std::memcpy(dst + i * row_bytes, src + (size_t)rows[i] * row_bytes, row_bytes);
            }
        });
        s->staged_gather_s += std::chrono::duration<double>(std::chrono::steady_clock::now() - t_begin).count();
        s->staged_gather_bytes += (long long)(total * row_bytes);
        PSB_CUDA(cudaMemcpyAsync(static_cast<unsigned char*>(d_stage) + i0 * row_bytes, dst, total * row_bytes, cudaMemcpyHostToDevice, stream));
        PSB_CUDA(cudaEventRecord(s->pinned_ev[slot], stream));
        s->pinned_used[slot] = true;
    }
    return PSB_OK;
}

// The rows of one batch (of one rerank call): claimed part by part, fetched once each, released at the end.  All of a batch's claims,
// fetches and scores are ordered by the caller's streams and events.
psb_status rows_begin(psb_session* s, long long requests, size_t parts, cudaStream_t st) {
    const size_t slots = (size_t)std::max<long long>(1, std::min(requests, s->exact_count));
    s->slots = slots;
    s->parts = parts;
    bool moved = false;
    PSB_TRY(ensure_scalars(s, st));
    PSB_TRY(reserve_together(&s->rows_whole, {{&s->unique, sizeof(int) * slots}, {&s->marks, sizeof(int) * PartMarks::device_words(parts)},
                                              {&s->stage, slots * s->dim * s->exact_elem},
                                              {&s->slot_of, sizeof(int) * (size_t)std::max<long long>(1, s->exact_count)},
                                              {&s->row_bits, sizeof(unsigned) * claim_words(s->exact_count) * 2},
                                              {&s->row_sums, sizeof(int) * claim_sums(s->exact_count)}}, 0, nullptr, &moved));
    if (moved || s->slots_dirty) {
        PSB_CUDA(cudaMemsetAsync(s->slot_of.p, 0xff, s->slot_of.bytes, st));
        PSB_CUDA(cudaMemsetAsync(s->row_bits.p, 0, s->row_bits.bytes, st));
    }
    s->slots_dirty = true;
    PSB_CUDA(cudaMemsetAsync(s->marks.p, 0, sizeof(int) * PartMarks::device_words(parts), st));
    return PSB_OK;
}
int* part_begin(const psb_session* s, int part) { return s->marks.as<int>() + PartMarks::device_begin((size_t)part); }
int* part_end(const psb_session* s, int part) { return part_begin(s, part) + 1; }
psb_status rows_claim(psb_session* s, int part, const int* d_cand, int nq, int width, int stride, const int* d_counts, cudaStream_t st) {
    ClaimBuffers b;
    b.count = s->exact_count; b.slot_of = s->slot_of.as<int>(); b.unique = s->unique.as<int>(); b.sums = s->row_sums.as<int>();
    b.bits = s->row_bits.as<unsigned>() + s->bits_turn * claim_words(s->exact_count);
    b.old_bits = s->row_bits.as<unsigned>() + (s->bits_turn ^ 1) * claim_words(s->exact_count);
    s->bits_turn ^= 1;
    return launch_claim_rows(s->row_map(), d_cand, nq, width, stride, d_counts, b, part_begin(s, part), part_end(s, part), s->marks.as<int>(), st);
}
psb_status rows_end(psb_session* s, cudaStream_t st) {
    PSB_TRY(launch_release_rows(s->unique.as<int>(), s->marks.as<int>(), s->slot_of.as<int>(), s->scalars.as<unsigned long long>() + kRowsFetched, s->sm_count, st));
    s->slots_dirty = false;
    return PSB_OK;
}
// Queues the copy of a part's slot range to the host behind its claim (there once `st` gets to it).
psb_status rows_tell_host(psb_session* s, int part, cudaStream_t st) {
    if (s->h_marks_words < PartMarks::host_words(s->parts)) {   // part 0: the worker of this batch has nothing to read yet
        if (s->h_marks) { PSB_CUDA(cudaDeviceSynchronize()); cudaFreeHost(s->h_marks); }
        s->h_marks = nullptr; s->h_marks_words = 0;
        const size_t words = std::max(PartMarks::host_words(s->parts), (size_t)64);
        PSB_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&s->h_marks), sizeof(int) * words, cudaHostAllocDefault));
        s->h_marks_words = words;
    }
    PSB_CUDA(cudaMemcpyAsync(s->h_marks + PartMarks::host_begin((size_t)part), part_begin(s, part), sizeof(int) * 2, cudaMemcpyDeviceToHost, st));
    return PSB_OK;
}
// The host threads' share of a part whose claim is done: slot list to the host, rows to their slots (copies on `st`).
psb_status rows_from_host(psb_session* s, int part, int host_pct, cudaStream_t st) {
    const int* range = s->h_marks + PartMarks::host_begin((size_t)part);
    const int b = range[0], e = host_share_end(b, range[1], host_pct);
    if (e <= b) return PSB_OK;
    if (!s->list_stream) PSB_CUDA(cudaStreamCreateWithFlags(&s->list_stream, cudaStreamNonBlocking));
    constexpr size_t kListChunk = (size_t)1 << 18;   // ids on the host at a time
    const size_t room = std::min(kListChunk, std::max(s->slots, (size_t)(e - b)));
    if (s->h_unique_count < room) {
        if (s->h_unique) cudaFreeHost(s->h_unique);
        s->h_unique = nullptr; s->h_unique_count = 0;
        PSB_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&s->h_unique), sizeof(int) * room, cudaHostAllocDefault));
        s->h_unique_count = room;
    }
    for (size_t i = b; i < (size_t)e; i += s->h_unique_count) {
        const size_t count = std::min(s->h_unique_count, (size_t)e - i);
        PSB_CUDA(cudaMemcpyAsync(s->h_unique, s->unique.as<int>() + i, sizeof(int) * count, cudaMemcpyDeviceToHost, s->list_stream));
        PSB_CUDA(cudaStreamSynchronize(s->list_stream));
        PSB_TRY(staged_gather_host(s, s->h_unique, count, static_cast<unsigned char*>(s->stage.p) + i * s->dim * s->exact_elem, st));
    }
    return PSB_OK;
}

// The stream of the gather kernel beside a scan.  Highest priority: its few CTAs each need an SM to themselves and must be
// placed before the large grids of the scan stage that become runnable at the same moment.
psb_status ensure_zc_stream(psb_session* s) {
    if (s->zc_stream) return PSB_OK;
    int lo = 0, hi = 0;
    PSB_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    PSB_CUDA(cudaStreamCreateWithPriority(&s->zc_stream, cudaStreamNonBlocking, hi));
    return PSB_OK;
}

// A call's gathers on zc_stream.  Their results are waited for one by one where rows are scored; a call that ends before that, with an error, leaves
// gathers that still read the slot lists and write the slots.  Whatever way the call ends, its stream goes on behind them.
struct Gathers {
    psb_session* s;
    cudaStream_t to;
    bool open = false;   // some may not have been waited for
    ~Gathers() {
        if (!open) return;
        cudaEvent_t e = nullptr;
        const bool joined = cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess && cudaEventRecord(e, s->zc_stream) == cudaSuccess &&
                            cudaStreamWaitEvent(to, e, 0) == cudaSuccess;
        if (e) cudaEventDestroy(e);
        if (!joined) cudaStreamSynchronize(s->zc_stream);
    }
};
// Test hook of that: an error where a call has gathers under way.
psb_status gather_error(const psb_session* s) { return s->opt.test_skip_mma & 16 ? fail(PSB_INTERNAL, "test hook: an error beside a gather") : PSB_OK; }

// SMs of the gather kernel beside a scan: 16 read ascending rows at the link's rate (8: 51.1 GB/s from an array of 0.8 GB but 40.3 from 20 GB, 16
// and 32: 51.0 from either), and the scan's persistent grid leaves them free.
constexpr int kGatherSms = 16;
int gather_sms(const psb_session* s) { return s->opt.gather_ctas > 0 ? 0 : s->opt.reserve_sms > 0 ? s->opt.reserve_sms : kGatherSms; }

// The host threads' share of the rows, in percent.  The kernel reads a part's rows in ascending order at the link's rate, beside a scan
// and alone, and the threads take from the same link: they bring rows only where no kernel can (rows that are not mapped) or where the caller names a share.
int host_share(const psb_session* s) {
    if (s->opt.exact_mode == PSB_EXACT_HOST_STAGED || !s->exact_dev) return 100;
    return s->opt.exact_mode == PSB_EXACT_HOST_HYBRID && s->opt.zero_copy_pct > 0 ? 100 - s->opt.zero_copy_pct : 0;
}
bool device_rows(const psb_session* s) { return s->opt.exact_mode == PSB_EXACT_RESIDENT || s->opt.exact_mode == PSB_EXACT_HOST_CACHED; }
// Rows scored where they lie: in device memory, or so few that fetching each once would not pay for its launches.
bool rows_in_place(const psb_session* s, long long requests) {
    if (device_rows(s)) return true;
    if (!s->exact_dev || s->opt.exact_mode == PSB_EXACT_HOST_STAGED) return false;
    if (host_share(s) > 0) return requests < kClaimRequestsThreads;
    const long long row_bytes = (long long)s->dim * s->exact_elem;
    return requests * row_bytes < (row_bytes <= 128 ? kClaimBytesShort : kClaimBytes);
}

// Scores and selection of one part, the rows being in place or in their slots.  d_ids_out: original ids instead of rows.
psb_status score_and_select(psb_session* s, bool in_place, const void* d_queries, int nq, const int* d_cand, int width, int stride, const int* d_counts,
                            int topk, int* d_out_rows, float* d_out_dist, long long* d_out_ids, float* d_score, cudaStream_t st) {
    PSB_TRY(launch_rerank_score(in_place ? s->exact_dev : s->stage.p, in_place ? nullptr : s->slot_of.as<int>(), s->row_map(), s->dim, s->exact_elem,
                                d_queries, d_cand, nq, width, stride, d_counts, d_score, st, s->call_marks ? s->call_marks + 2 : nullptr, s->one_stream && in_place));
    if (!d_out_rows && !d_out_ids) return PSB_OK;  // partial rerank: the caller combines the scores of all shards
    return launch_topk_select(d_score, d_cand, nq, width, stride, d_counts, topk, d_out_rows, d_out_dist, st, s->reordered.as<long long>(), d_out_ids, s->one_stream);
}

psb_status rerank_impl(psb_session* s, const void* d_queries, int nq, const int* d_cand, int width, int stride,
                       const int* d_counts, int topk, int* d_out_rows, float* d_out_dist, float* d_score = nullptr, long long* d_out_ids = nullptr) {
    if (!s->exact_elem) return fail(PSB_INVALID_ARGUMENT, "session has no exact rows for the rerank");
    if (width <= 0 || stride < width || topk <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid rerank request");
    if (width > kMaxRerankWidth || topk > kMaxTopk) return fail(PSB_UNSUPPORTED_SHAPE, "rerank width above 4096 or topk above 2048");
    if (nq <= 0) return PSB_OK;
    float* score = d_score;
    if (!score) {
        PSB_TRY(s->score.reserve(sizeof(float) * (size_t)nq * width));
        score = s->score.as<float>();
    }
    const bool beside = s->background || (s->aux_stream != nullptr && s->stream == s->aux_stream);
    const bool in_place = rows_in_place(s, (long long)nq * width);
    if (!in_place) {
        PSB_TRY(rows_begin(s, (long long)nq * width, 1, s->stream));
        PSB_TRY(rows_claim(s, 0, d_cand, nq, width, stride, d_counts, s->stream));
        const int host_pct = host_share(s);
        const int row_bytes = s->dim * s->exact_elem;
        // Beside a scan on the other stream the gather kernel runs on SMs of its own: the ones the scan's persistent grid leaves free
        // (reserve_sms), or gather_ctas lean CTAs spread over all SMs when the caller asks for that.
        const int owned = beside ? gather_sms(s) : 0;
        const int lean = beside ? s->opt.gather_ctas : 0;
        if (host_pct == 0) {
            PSB_TRY(launch_gather_unique(s->exact_dev, row_bytes, s->unique.as<int>(), part_begin(s, 0), part_end(s, 0), 0, s->stage.p, s->stream,
                                         s->sm_count, lean, owned));
        } else {
            // This thread and the host pool bring their share while the kernel, on a stream of its own, brings the rest.  The call
            // blocks for the host gather; a caller that overlaps it with a scan queues that scan first.
            PSB_TRY(rows_tell_host(s, 0, s->stream));
            Gathers gathers{s, s->stream};
            if (host_pct < 100) {
                PSB_TRY(ensure_zc_stream(s));
                if (!s->zc_ev_a) PSB_CUDA(cudaEventCreateWithFlags(&s->zc_ev_a, cudaEventDisableTiming));
                if (!s->zc_ev_b) PSB_CUDA(cudaEventCreateWithFlags(&s->zc_ev_b, cudaEventDisableTiming));
                PSB_CUDA(cudaEventRecord(s->zc_ev_a, s->stream));
                PSB_CUDA(cudaStreamWaitEvent(s->zc_stream, s->zc_ev_a, 0));
                gathers.open = true;
                PSB_TRY(launch_gather_unique(s->exact_dev, row_bytes, s->unique.as<int>(), part_begin(s, 0), part_end(s, 0), host_pct, s->stage.p,
                                             s->zc_stream, s->sm_count, 0, owned));
                PSB_CUDA(cudaEventRecord(s->zc_ev_b, s->zc_stream));
            }
            PSB_CUDA(cudaStreamSynchronize(s->stream));
            PSB_TRY(gather_error(s));
            PSB_TRY(rows_from_host(s, 0, host_pct, s->stream));
            if (host_pct < 100) PSB_CUDA(cudaStreamWaitEvent(s->stream, s->zc_ev_b, 0));
            gathers.open = false;
        }
    }
    PSB_TRY(score_and_select(s, in_place, d_queries, nq, d_cand, width, stride, d_counts, topk, d_out_rows, d_out_dist, d_out_ids, score, s->stream));
    return in_place ? PSB_OK : rows_end(s, s->stream);
}

}  // namespace

namespace psb {
SessionShape session_shape(const psb_session* s) {
    SessionShape o;
    o.dim = s->dim; o.m = s->m; o.k = s->k; o.nlist = s->nlist; o.n_rerank = s->opt.n_rerank; o.exact_elem = s->exact_elem;
    o.device = s->device; o.residual = s->opt.adc_mode == 1; o.flat = s->flat; o.stream = s->stream;
    return o;
}
}  // namespace psb

extern "C" {

const char* psb_last_error(void) { return last_error_ref().c_str(); }
const char* psb_version(void) { return kNvtxCompiled ? "paraselect-b200 0.1 (sm_100a, nvtx)" : "paraselect-b200 0.1 (sm_100a)"; }

size_t psb_sizeof(int which) {
    switch (which) {
        case 0: return sizeof(psb_options);
        case 1: return sizeof(psb_stats);
        case 2: return sizeof(psb_index_view);
        case 3: return sizeof(psb_flat_index_view);
        case 4: return sizeof(psb_row_correction_u16_header);
        case 5: return sizeof(psb_search_params);
        default: return 0;
    }
}

int psb_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) { cudaGetLastError(); return 0; }
    int ok = 0;
    for (int i = 0; i < n; ++i) {
        int major = 0;
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, i) == cudaSuccess && major == 10) ++ok;
    }
    return ok;
}

psb_status psb_session_create(const psb_index_view* index, const psb_options* options, psb_session** out) {
    PSB_RANGE("ivfpq_prepare");
    if (!out) return fail(PSB_INVALID_ARGUMENT, "out is null");
    *out = nullptr;
    PSB_TRY(validate_index(index));
    psb_options opt{};
    if (options) opt = *options;
    if (opt.max_batch <= 0) opt.max_batch = 10000;
    if (opt.exact_mode < 0 || opt.exact_mode > PSB_EXACT_HOST_HYBRID) return fail(PSB_INVALID_ARGUMENT, "unknown exact_mode");
    const int nlist = index->lists.nlist;
    int lb = opt.list_begin, le = opt.list_end;
    if (lb == 0 && le == 0) le = nlist;
    if (lb < 0 || le > nlist || lb > le) return fail(PSB_INVALID_ARGUMENT, "invalid list shard range");
    const int64_t* gb = opt.list_global_begin;
    if (gb) {
        if (lb != 0 || le != nlist) return fail(PSB_INVALID_ARGUMENT, "list_global_begin excludes a list range");
        for (int l = 0; l < nlist; ++l) {
            const int64_t len = index->lists.offsets[l + 1] - index->lists.offsets[l];
            if (gb[l] < 0 || gb[l] + len > INT_MAX || (l + 1 < nlist && gb[l] + len > gb[l + 1]))
                return fail(PSB_INVALID_ARGUMENT, "list_global_begin must give disjoint ascending row ranges below 2^31");
        }
    }
    if (opt.n_rerank > kMaxStage1) return fail(PSB_UNSUPPORTED_SHAPE, "n_rerank above 2048 is not supported");
    if (opt.adc_mode != 0 && opt.adc_mode != 1) return fail(PSB_INVALID_ARGUMENT, "unknown adc_mode");
    if (opt.reserve_sms < 0 || opt.reserve_sms > 64) return fail(PSB_INVALID_ARGUMENT, "reserve_sms must be in 0..64");
    if (opt.seed_sigma != 0.f && !(opt.seed_sigma >= 2.f && opt.seed_sigma <= 10.f)) return fail(PSB_INVALID_ARGUMENT, "seed_sigma must be 0 or in 2..10");
    if (opt.pipeline_parts != 0 && (opt.pipeline_parts < 2 || opt.pipeline_parts > 32)) return fail(PSB_INVALID_ARGUMENT, "pipeline_parts must be 0 or in 2..32");
    if (opt.scan_mode < 0 || opt.scan_mode > 3) return fail(PSB_INVALID_ARGUMENT, "scan_mode must be in 0..3");
    if (opt.tc_min_visitors < 0) return fail(PSB_INVALID_ARGUMENT, "tc_min_visitors must not be negative");
    if (opt.zero_copy_pct < 0 || opt.zero_copy_pct > 100) return fail(PSB_INVALID_ARGUMENT, "zero_copy_pct must be in 0..100");
    if (opt.host_threads < 0 || opt.host_threads > 64) return fail(PSB_INVALID_ARGUMENT, "host_threads must be in 0..64");
    // hybrid transport: the gather kernel runs beside the scan on SMs of its own, which the scan's grid has to leave free
    if (opt.exact_mode == PSB_EXACT_HOST_HYBRID && opt.reserve_sms == 0 && opt.gather_ctas == 0) opt.reserve_sms = kGatherSms;
    if (opt.gather_ctas < 0 || opt.gather_ctas > 1024) return fail(PSB_INVALID_ARGUMENT, "gather_ctas must be in 0..1024");
    if (opt.adc_mode == 1 && !index->exact.fp32 && !index->exact.u8)
        return fail(PSB_INVALID_ARGUMENT, "residual mode always reranks: exact rows are required");
    int sms = 0;
    PSB_TRY(check_device(opt.device, &sms));
    std::unique_ptr<psb_session> s(new (std::nothrow) psb_session());
    if (!s) return fail(PSB_OUT_OF_MEMORY, "host allocation failed");
    s->device = opt.device; s->sm_count = sms; s->opt = opt;
    s->nlist = nlist; s->dim = index->coarse.dim; s->m = index->pq.subvectors; s->k = index->pq.codebook_size;
    s->n_vectors = index->lists.n_vectors; s->list_begin = lb; s->list_end = le;
    s->row_base = index->lists.offsets[lb];
    s->shard_rows = index->lists.offsets[le] - s->row_base;
    if (opt.stream) s->stream = static_cast<cudaStream_t>(opt.stream);
    else { PSB_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking)); s->own_stream = true; }
    cudaStream_t st = s->stream;
    const auto& E = index->exact;
    if (E.fp32 || E.u8) {
        s->exact_elem = E.fp32 ? 4 : 1;
        s->exact_host = E.fp32 ? static_cast<const void*>(E.fp32) : static_cast<const void*>(E.u8);
        s->exact_count = E.count;
    }
    const size_t exact_bytes = (size_t)s->exact_count * s->dim * s->exact_elem;
    if ((opt.exact_mode == PSB_EXACT_HOST_MAPPED || opt.exact_mode == PSB_EXACT_HOST_HYBRID) && exact_bytes > 0) {   // before the copies are noted
        PSB_TRY(map_rows(s->exact_host, exact_bytes, &s->mapped));
        void* dp = nullptr;
        PSB_CUDA(cudaHostGetDevicePointer(&dp, const_cast<void*>(s->exact_host), 0));
        s->exact_dev = dp;
    }
    HostCopies copies(st, {{index->coarse.centroids, sizeof(float) * (size_t)nlist * s->dim}, {index->lists.offsets, sizeof(long long) * ((size_t)nlist + 1)},
                           {index->lists.reordered_ids, sizeof(long long) * (size_t)s->n_vectors}, {index->pq.codes, (size_t)s->n_vectors * s->m},
                           {index->pq.codebook, sizeof(float) * (size_t)s->k * s->dim}, {opt.opq_matrix, sizeof(float) * (size_t)s->dim * s->dim},
                           {opt.row_correction_u16, sizeof(uint16_t) * (size_t)s->n_vectors}, {opt.row_correction_fp32, sizeof(float) * (size_t)s->n_vectors},
                           {opt.exact_mode == PSB_EXACT_HOST_CACHED ? s->exact_host : nullptr, exact_bytes}});
    if (gb) {
        s->striped = true;
        s->h_global_begin.assign(gb, gb + nlist);
        std::vector<long long> delta((size_t)nlist);
        for (int l = 0; l < nlist; ++l) delta[(size_t)l] = gb[l] - index->lists.offsets[l];
        PSB_TRY(s->global_begin.reserve(sizeof(long long) * (size_t)nlist));
        PSB_TRY(s->row_delta.reserve(sizeof(long long) * (size_t)nlist));
        PSB_CUDA(cudaMemcpyAsync(s->global_begin.p, s->h_global_begin.data(), sizeof(long long) * (size_t)nlist, cudaMemcpyHostToDevice, st));
        PSB_CUDA(cudaMemcpy(s->row_delta.p, delta.data(), sizeof(long long) * (size_t)nlist, cudaMemcpyHostToDevice));
    }
    PSB_TRY(s->centroids.reserve(sizeof(float) * (size_t)nlist * s->dim));
    PSB_CUDA(cudaMemcpyAsync(s->centroids.p, index->coarse.centroids, sizeof(float) * (size_t)nlist * s->dim, cudaMemcpyHostToDevice, st));
    if (opt.coarse_mode != 1 && nlist >= 1024 && coarse_tc_padded_dim(s->dim) <= 128)
        PSB_TRY(s->tc_index.prepare(s->centroids.as<float>(), nlist, s->dim, s->device, st));
    PSB_TRY(s->offsets.reserve(sizeof(long long) * ((size_t)nlist + 1)));
    PSB_CUDA(cudaMemcpyAsync(s->offsets.p, index->lists.offsets, sizeof(long long) * ((size_t)nlist + 1), cudaMemcpyHostToDevice, st));
    PSB_TRY(s->reordered.reserve(sizeof(long long) * (size_t)std::max<long long>(1, s->n_vectors)));
    if (s->n_vectors > 0)
        PSB_CUDA(cudaMemcpyAsync(s->reordered.p, index->lists.reordered_ids, sizeof(long long) * (size_t)s->n_vectors, cudaMemcpyHostToDevice, st));
    PSB_TRY(s->codes.reserve((size_t)std::max<long long>(1, s->shard_rows) * s->m + 16));
    if (s->shard_rows > 0)
        PSB_CUDA(cudaMemcpyAsync(s->codes.p, index->pq.codes + (size_t)s->row_base * s->m, (size_t)s->shard_rows * s->m, cudaMemcpyHostToDevice, st));
    const size_t cb_bytes = sizeof(float) * (size_t)s->m * s->k * (s->dim / s->m);
    PSB_TRY(s->codebook.reserve(cb_bytes));
    PSB_CUDA(cudaMemcpyAsync(s->codebook.p, index->pq.codebook, cb_bytes, cudaMemcpyHostToDevice, st));
    if (opt.opq_matrix) {
        if (opt.adc_mode == 1) return fail(PSB_INVALID_ARGUMENT, "the OPQ rotation belongs to the plain ADC mode");
        PSB_TRY(s->opq.reserve(sizeof(float) * (size_t)s->dim * s->dim));
        PSB_CUDA(cudaMemcpyAsync(s->opq.p, opt.opq_matrix, sizeof(float) * (size_t)s->dim * s->dim, cudaMemcpyHostToDevice, st));
    }
    // per-row terms of the tensor-core scan (8 bytes per code row), once per index
    if ((opt.scan_mode == 0 || opt.scan_mode == 3) && s->shard_rows > 0 && scan_tc_supported(s->dim, s->m, s->k)) {
        PSB_TRY(s->row_aug.reserve((size_t)s->shard_rows * 8));
        PSB_TRY(launch_row_aug(s->codes.as<uint8_t>(), s->shard_rows, s->dim, s->m, s->k, s->codebook.as<float>(), s->row_aug.p, s->sm_count, st));
        if (opt.adc_mode == 1 && opt.row_correction_u16) {  // the caller's row correction, affine u16
            if (!(opt.rc_scale > 0.f)) return fail(PSB_INVALID_ARGUMENT, "row_correction_u16 needs a positive rc_scale");
            PSB_TRY(s->row_bias.reserve(sizeof(uint16_t) * (size_t)s->shard_rows));
            PSB_CUDA(cudaMemcpyAsync(s->row_bias.p, opt.row_correction_u16 + s->row_base, sizeof(uint16_t) * (size_t)s->shard_rows, cudaMemcpyHostToDevice, st));
            s->row_bias_is_u16 = true;
        } else if (opt.adc_mode == 1 && opt.row_correction_fp32) {
            PSB_TRY(s->row_bias.reserve(sizeof(float) * (size_t)s->shard_rows));
            PSB_CUDA(cudaMemcpyAsync(s->row_bias.p, opt.row_correction_fp32 + s->row_base, sizeof(float) * (size_t)s->shard_rows, cudaMemcpyHostToDevice, st));
        } else if (opt.adc_mode == 1) {  // computed here: the per-row correction of the residual cutoff estimate
            PSB_TRY(s->row_bias.reserve(sizeof(float) * (size_t)s->shard_rows));
            PSB_TRY(launch_row_bias(s->codes.as<uint8_t>(), s->offsets.as<long long>(), s->row_base, lb, le, s->dim, s->m, s->k,
                                    s->codebook.as<float>(), s->centroids.as<float>(), s->row_bias.as<float>(), st));
        }
    }
    {   // per sub-quantiser the largest codeword norm (residual-mode table builder)
        const int dsub = s->dim / s->m;
        std::vector<float> mx((size_t)s->m, 0.0f);
        for (int j = 0; j < s->m; ++j)
            for (int c = 0; c < s->k; ++c) {
                double n2 = 0.0;
                for (int d = 0; d < dsub; ++d) { const double v = index->pq.codebook[((size_t)j * s->k + c) * dsub + d]; n2 += v * v; }
                mx[(size_t)j] = std::max(mx[(size_t)j], (float)(std::sqrt(n2) * 1.0001));
            }
        PSB_TRY(s->cb_maxnorm.reserve(sizeof(float) * (size_t)s->m));
        PSB_CUDA(cudaMemcpy(s->cb_maxnorm.p, mx.data(), sizeof(float) * (size_t)s->m, cudaMemcpyHostToDevice));
    }
    note_list_lengths(s.get(), index->lists.offsets);
    // exact rows
    if (s->exact_host) {
        const size_t bytes = exact_bytes;
        if (opt.exact_mode == PSB_EXACT_RESIDENT) {
            s->exact_dev = s->exact_host;
        } else if (opt.exact_mode == PSB_EXACT_HOST_CACHED && bytes > 0) {
            // the session's own copy of the rows in device memory (a B200 holds 180 GB: C4's 38.4 GB of rows fit beside the index)
            size_t free_b = 0, total_b = 0;
            PSB_CUDA(cudaMemGetInfo(&free_b, &total_b));
            if (bytes + ((size_t)8 << 30) > free_b)
                return fail(PSB_OUT_OF_MEMORY, "the exact rows do not fit in device memory beside the workspaces; use a host mode");
            PSB_TRY(s->exact_cache.reserve(bytes));
            const size_t chunk = (size_t)1 << 30;
            for (size_t off = 0; off < bytes; off += chunk)
                PSB_CUDA(cudaMemcpyAsync(static_cast<unsigned char*>(s->exact_cache.p) + off,
                                         static_cast<const unsigned char*>(s->exact_host) + off, std::min(chunk, bytes - off),
                                         cudaMemcpyHostToDevice, st));
            s->exact_dev = s->exact_cache.p;
        }
    }
    PSB_CUDA(cudaStreamSynchronize(st));
    copies.ended = true;
    s->count();
    *out = s.release();
    return PSB_OK;
}

psb_status psb_session_destroy(psb_session* s) {
    delete s;  // the destructor releases everything the session owns (also a partially built one)
    return PSB_OK;
}

psb_status psb_session_sync(psb_session* s) {
    if (!s) return fail(PSB_INVALID_ARGUMENT, "session is null");
    PSB_CUDA(cudaStreamSynchronize(s->stream));
    PSB_TRY(s->tc_work.check_status());
    return s->check_scan_status();
}

psb_status psb_session_set_stream(psb_session* s, void* stream, int background) {
    if (!s) return fail(PSB_INVALID_ARGUMENT, "session is null");
    if (!s->home_stream) s->home_stream = s->stream;
    s->stream = stream ? static_cast<cudaStream_t>(stream) : s->home_stream;
    s->background = stream != nullptr && background != 0;
    return PSB_OK;
}

psb_status psb_stage_coarse(psb_session* s, const float* d_queries, int nq, int nprobe, int* d_ids, float* d_dist) {
    PSB_RANGE("coarse_search");
    if (!s || !d_queries || !d_ids) return fail(PSB_INVALID_ARGUMENT, "null argument");
    if (nprobe <= 0 || nprobe > s->nlist) return fail(PSB_INVALID_ARGUMENT, "nprobe must be in 1..nlist");
    if (nprobe > kMaxProbe) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 is not supported");
    PSB_CUDA(cudaSetDevice(s->device));
    return coarse_exact(s, d_queries, nq, nprobe, d_ids, d_dist);
}

psb_status psb_rotate_rows(const float* d_in, const float* d_matrix, int64_t n, int dim, float* d_out, int device, void* stream) {
    if (!d_in || !d_matrix || !d_out || n < 0 || dim <= 0 || d_in == d_out) return fail(PSB_INVALID_ARGUMENT, "invalid rotation request");
    PSB_TRY(check_device(device));
    return launch_rotate_rows(d_in, d_matrix, n, dim, d_out, static_cast<cudaStream_t>(stream));
}

int psb_sign_padded_dim(int dim) { return sign_padded_dim(dim); }

psb_status psb_sign_rotation_scale(int padded_dim, float* h_scale, int device, void* stream) {
    if (!h_scale || sign_padded_dim(padded_dim) != padded_dim) return fail(PSB_INVALID_ARGUMENT, "padded_dim must be 32, 64, 128 or 256");
    PSB_TRY(check_device(device));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* d = nullptr;
    PSB_CUDA(cudaMalloc(reinterpret_cast<void**>(&d), sizeof(float)));
    psb_status rc = launch_sign_scale(padded_dim, d, st);
    cudaError_t e = rc == PSB_OK ? cudaMemcpyAsync(h_scale, d, sizeof(float), cudaMemcpyDeviceToHost, st) : cudaSuccess;
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (rc == PSB_OK && e != cudaSuccess) rc = cuda_fail(e, "psb_sign_rotation_scale", __FILE__, __LINE__);
    return rc;
}

psb_status psb_sign_rotate(const float* d_rows, int64_t n, int dim, int padded_dim, uint32_t seed, float* d_rotated,
                           uint32_t* d_codes, float* d_norms, float* d_norm_sq, int device, void* stream) {
    if (!d_rows || n < 0 || (!d_rotated && !d_codes && !d_norms && !d_norm_sq)) return fail(PSB_INVALID_ARGUMENT, "invalid sign rotation request");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    return launch_sign_rotate(d_rows, n, dim, padded_dim, seed, d_rotated, d_codes, d_norms, d_norm_sq, sms,
                              static_cast<cudaStream_t>(stream));
}

psb_status psb_sign_encode_database(const void* d_rows, int elem_bytes, int64_t n, const float* d_centroids,
                                    const int64_t* d_list_offsets, int nlist, int dim, int padded_dim, uint32_t seed,
                                    int64_t row_offset, uint32_t* d_codes, float* d_scales, int device, void* stream) {
    if (!d_rows || !d_centroids || !d_list_offsets || !d_codes || n < 0 || nlist <= 0 || row_offset < 0)
        return fail(PSB_INVALID_ARGUMENT, "invalid sign database encoding request");
    if (elem_bytes != 1 && elem_bytes != 4) return fail(PSB_INVALID_ARGUMENT, "rows must be u8 (1) or fp32 (4)");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    return launch_sign_encode_database(d_rows, elem_bytes, n, d_centroids, reinterpret_cast<const long long*>(d_list_offsets), nlist,
                                       dim, padded_dim, seed, row_offset, d_codes, d_scales, sms,
                                       static_cast<cudaStream_t>(stream));
}

psb_status psb_sign_encode_queries(const float* d_queries, const float* d_centroids, const int* d_probes, int nq, int nprobe,
                                   int nlist, int dim, int padded_dim, uint32_t seed, float* d_states, float* d_norm_sq,
                                   uint32_t* d_state_codes, float* d_norms, int device, void* stream) {
    if (!d_queries || !d_centroids || !d_probes || nq < 0 || nprobe <= 0 || nlist <= 0 || (!d_states && !d_state_codes))
        return fail(PSB_INVALID_ARGUMENT, "invalid sign query encoding request");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    return launch_sign_encode_queries(d_queries, d_centroids, d_probes, nq, nprobe, nlist, dim, padded_dim, seed, d_states, d_norm_sq,
                                      d_state_codes, d_norms, sms, static_cast<cudaStream_t>(stream));
}

psb_status psb_sign_search_candidates(int mode, const float* d_states, const float* d_norm_sq, const uint32_t* d_state_codes,
                                      const float* d_norms, const uint32_t* d_codes, const float* d_row_params,
                                      const int64_t* d_list_offsets, int nlist, const int* d_probes, int nq, int nprobe,
                                      int padded_dim, int candidate_count, int* d_rows_out, float* d_dist_out, int device,
                                      void* stream) {
    PSB_RANGE("sign_candidates");
    if (mode != PSB_SIGN_FLOAT_STATES && mode != PSB_SIGN_CODED_STATES) return fail(PSB_INVALID_ARGUMENT, "unknown sign score mode");
    if (mode == PSB_SIGN_FLOAT_STATES ? (!d_states || !d_norm_sq) : (!d_state_codes || !d_norms))
        return fail(PSB_INVALID_ARGUMENT, "the states of the chosen score mode are missing");
    if (!d_codes || !d_row_params || !d_list_offsets || !d_probes || !d_rows_out || nq < 0 || nprobe <= 0 || nlist <= 0)
        return fail(PSB_INVALID_ARGUMENT, "invalid sign candidate search request");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    PoolBuf partial;   // the slices of queries whose probes go to several CTAs
    const size_t bytes = sign_partial_bytes(nq, nprobe, candidate_count, sms);
    if (bytes) PSB_TRY(partial.reserve(bytes, device, static_cast<cudaStream_t>(stream)));
    return launch_sign_candidates(mode, d_states, d_norm_sq, d_state_codes, d_norms, d_codes, d_row_params,
                                  reinterpret_cast<const long long*>(d_list_offsets), nlist, d_probes, nq, nprobe, padded_dim,
                                  candidate_count, d_rows_out, d_dist_out, partial.p, sms, static_cast<cudaStream_t>(stream));
}

psb_status psb_stage_rotate_queries(psb_session* s, const float* d_queries, int nq, float* d_rotated) {
    if (!s || !d_queries || !d_rotated || nq < 0 || d_queries == d_rotated) return fail(PSB_INVALID_ARGUMENT, "invalid rotation request");
    if (!s->opq.p) return fail(PSB_INVALID_ARGUMENT, "the session has no OPQ rotation");
    PSB_CUDA(cudaSetDevice(s->device));
    return launch_rotate_rows(d_queries, s->opq.as<float>(), nq, s->dim, d_rotated, s->stream);
}

psb_status psb_stage_build_lut(psb_session* s, const float* d_queries, int nq, float* d_lut) {
    PSB_RANGE("pq_lut_build");
    if (!s || !d_queries || !d_lut) return fail(PSB_INVALID_ARGUMENT, "null argument");
    PSB_CUDA(cudaSetDevice(s->device));
    return launch_build_lut(d_queries, nq, s->dim, s->codebook.as<float>(), s->m, s->k, d_lut, s->stream);
}

psb_status psb_stage_build_lut_residual(psb_session* s, const float* d_queries, int nq, const int* d_probes, int nprobe,
                                        float* d_lut) {
    PSB_RANGE("pq_lut_build");
    if (!s || !d_queries || !d_probes || !d_lut) return fail(PSB_INVALID_ARGUMENT, "null argument");
    if (nprobe <= 0 || nprobe > kMaxProbe) return fail(PSB_INVALID_ARGUMENT, "nprobe must be in 1..4096");
    PSB_CUDA(cudaSetDevice(s->device));
    return launch_build_lut_residual(d_queries, nq, s->dim, d_probes, nprobe, s->centroids.as<float>(), s->nlist,
                                     s->codebook.as<float>(), s->m, s->k, d_lut, s->stream);
}

psb_status psb_stage_quantize_lut_u8(psb_session* s, const float* d_lut, int64_t tables, uint8_t* d_q8, float* d_scales,
                                     float* d_lo_sum, float* d_inflation) {
    if (!s || !d_lut || !d_q8 || !d_scales || !d_lo_sum || !d_inflation || tables < 0) return fail(PSB_INVALID_ARGUMENT, "null argument");
    PSB_CUDA(cudaSetDevice(s->device));
    return launch_lut_to_u8(d_lut, tables, s->m, s->k, s->opt.adc_mode == 1 ? 1 : 0, d_q8, d_scales, d_lo_sum, d_inflation, s->stream);
}

psb_status psb_stage_scan(psb_session* s, const float* d_lut, int nq, const int* d_probes, int nprobe,
                          int stage1_k, int* d_rows, float* d_dist, int* d_count) {
    return psb_stage_scan_queries(s, nullptr, d_lut, nq, d_probes, nprobe, stage1_k, d_rows, d_dist, d_count);
}

psb_status psb_stage_scan_queries(psb_session* s, const float* d_queries, const float* d_lut, int nq, const int* d_probes,
                                  int nprobe, int stage1_k, int* d_rows, float* d_dist, int* d_count) {
    PSB_RANGE("pq_adc_scan");
    if (!s || !d_probes || !d_rows) return fail(PSB_INVALID_ARGUMENT, "null argument");
    if (nq < 0 || nprobe <= 0 || stage1_k <= 0) return fail(PSB_INVALID_ARGUMENT, "nprobe and stage1_k must be positive, nq not negative");
    if (nprobe > kMaxProbe || stage1_k > kMaxStage1) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 or stage1_k above 2048");
    if (nq == 0) return PSB_OK;
    if (!d_lut && !(d_queries && tables_optional(s, nprobe, stage1_k)))
        return fail(PSB_INVALID_ARGUMENT, "the scan needs the lookup tables (they may be left out only in residual mode, with the queries at hand)");
    s->counters_known = false;
    PSB_CUDA(cudaSetDevice(s->device));
    const bool rows_only = d_queries != nullptr && rows_form(s, nq, nprobe, true);
    PSB_TRY(ensure_scan_ws(s, nq, nprobe, stage1_k, rows_only));
    ScanWorkspace ws;
    PSB_TRY(s->timed_scan_ws(&ws));
    return run_scan(s, ws, rows_only, d_queries, d_lut, nq, d_probes, nprobe, stage1_k, d_rows, d_dist, d_count, s->stream, true);
}

int psb_scan_sample_words(const psb_session* s, int stage1_k) {
    if (!s || stage1_k <= 0) return 0;
    return seed_record_keys(stage1_k, s->opt.seed_sigma) + kSeedTail;
}

namespace {
psb_status check_scan_stage(psb_session* s, const int* d_probes, int nprobe, int stage1_k) {
    if (!s || !d_probes) return fail(PSB_INVALID_ARGUMENT, "null argument");
    if (nprobe <= 0 || stage1_k <= 0) return fail(PSB_INVALID_ARGUMENT, "nprobe and stage1_k must be positive");
    if (nprobe > kMaxProbe || stage1_k > kMaxStage1) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 or stage1_k above 2048");
    return PSB_OK;
}
}  // namespace

psb_status psb_stage_scan_sample(psb_session* s, const float* d_queries, const float* d_lut, int nq, const int* d_probes,
                                 int nprobe, int stage1_k, uint32_t* d_samples) {
    PSB_RANGE("pq_adc_scan_sample");
    PSB_TRY(check_scan_stage(s, d_probes, nprobe, stage1_k));
    if (!d_samples) return fail(PSB_INVALID_ARGUMENT, "null argument");
    s->counters_known = false;
    PSB_CUDA(cudaSetDevice(s->device));
    PSB_TRY(ensure_scan_ws(s, nq, nprobe, stage1_k, false));
    ScanWorkspace ws;
    PSB_TRY(s->timed_scan_ws(&ws));
    ws.phase = 1; ws.seed_export = d_samples; ws.seed_keys = seed_record_keys(stage1_k, s->opt.seed_sigma);
    return launch_scan(s->scan_index(), ws, d_lut, nq, d_probes, nprobe, stage1_k, nullptr, nullptr, nullptr, s->sm_count, s->stream, d_queries);
}

psb_status psb_stage_scan_shared(psb_session* s, const float* d_queries, const float* d_lut, int nq, const int* d_probes,
                                 int nprobe, int stage1_k, const uint32_t* d_all_samples, int shards, int* d_rows, float* d_dist,
                                 int* d_count, float* d_cutoff, int64_t* d_rows_scanned) {
    PSB_RANGE("pq_adc_scan");
    PSB_TRY(check_scan_stage(s, d_probes, nprobe, stage1_k));
    if (!d_all_samples || !d_rows || shards <= 0) return fail(PSB_INVALID_ARGUMENT, "null argument or no shards");
    s->counters_known = false;
    PSB_CUDA(cudaSetDevice(s->device));
    if (nq > s->ws_scan_queries) return fail(PSB_INVALID_ARGUMENT, "psb_stage_scan_shared follows psb_stage_scan_sample of the same queries");
    ScanWorkspace ws;
    PSB_TRY(s->timed_scan_ws(&ws));
    ws.phase = 2; ws.seed_all = d_all_samples; ws.seed_shards = shards; ws.seed_keys = seed_record_keys(stage1_k, s->opt.seed_sigma);
    ws.rows_global = reinterpret_cast<long long*>(d_rows_scanned);
    PSB_TRY(launch_scan(s->scan_index(), ws, d_lut, nq, d_probes, nprobe, stage1_k, d_rows, d_dist, d_count, s->sm_count, s->stream, d_queries));
    if (d_cutoff) PSB_CUDA(cudaMemcpyAsync(d_cutoff, ws.thr, sizeof(float) * (size_t)nq, cudaMemcpyDeviceToDevice, s->stream));
    return PSB_OK;
}

psb_status psb_stage_rerank(psb_session* s, const float* d_queries, int nq, const int* d_candidates,
                            int candidate_count, int candidate_stride, const int* d_counts, int topk,
                            int* d_out_rows, float* d_out_dist) {
    PSB_RANGE("pq_rerank");
    if (!s || !d_queries || !d_candidates || !d_out_rows || !d_out_dist) return fail(PSB_INVALID_ARGUMENT, "null argument");
    PSB_CUDA(cudaSetDevice(s->device));
    return rerank_impl(s, d_queries, nq, d_candidates, candidate_count, candidate_stride, d_counts, topk, d_out_rows, d_out_dist);
}

psb_status psb_stage_rerank_partial(psb_session* s, const float* d_queries, int nq, const int* d_candidates,
                                    int candidate_count, int candidate_stride, const int* d_counts, float* d_dist) {
    PSB_RANGE("pq_rerank");
    if (!s || !d_queries || !d_candidates || !d_dist) return fail(PSB_INVALID_ARGUMENT, "null argument");
    PSB_CUDA(cudaSetDevice(s->device));
    return rerank_impl(s, d_queries, nq, d_candidates, candidate_count, candidate_stride, d_counts, 1, nullptr, nullptr, d_dist);
}

psb_status psb_stage_select_topk(psb_session* s, const float* d_dist, const int* d_candidates, int nq,
                                 int candidate_count, int candidate_stride, const int* d_counts, int topk,
                                 int* d_out_rows, float* d_out_dist) {
    if (!s || !d_dist || !d_candidates || !d_out_rows || !d_out_dist) return fail(PSB_INVALID_ARGUMENT, "null argument");
    if (candidate_count <= 0 || candidate_stride < candidate_count || topk <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid selection request");
    if (topk > kMaxTopk) return fail(PSB_UNSUPPORTED_SHAPE, "topk above 2048 is not supported");
    PSB_CUDA(cudaSetDevice(s->device));
    return launch_topk_select(d_dist, d_candidates, nq, candidate_count, candidate_stride, d_counts, topk, d_out_rows,
                              d_out_dist, s->stream);
}

psb_status psb_stage_map_ids(psb_session* s, const int* d_rows, int64_t n, int64_t* d_indices) {
    PSB_RANGE("pq_map_ids");
    if (!s || !d_rows || !d_indices) return fail(PSB_INVALID_ARGUMENT, "null argument");
    PSB_CUDA(cudaSetDevice(s->device));
    return launch_map_ids(d_rows, n, s->reordered.as<long long>(), s->row_map(), reinterpret_cast<long long*>(d_indices), s->stream);
}

psb_status psb_stage_merge(psb_session* s, const int* d_rows, const float* d_dist, int parts, int nq, int k,
                           int* d_out_rows, float* d_out_dist) {
    if (!s || !d_rows || !d_dist || !d_out_rows || !d_out_dist || parts <= 0 || k <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid merge request");
    PSB_CUDA(cudaSetDevice(s->device));
    return launch_merge(d_rows, d_dist, parts, nq, k, d_out_rows, d_out_dist, s->stream);
}

psb_status psb_session_counters(psb_session* s, psb_stats* stats, int reset) {
    if (!s || !stats) return fail(PSB_INVALID_ARGUMENT, "null argument");
    s->counters_known = false;
    PSB_CUDA(cudaSetDevice(s->device));
    unsigned long long h[kScalars] = {};
    if (s->scalars.p) {
        PSB_CUDA(cudaMemcpyAsync(h, s->scalars.p, sizeof(h), cudaMemcpyDeviceToHost, s->stream));
        if (reset) {
            PSB_CUDA(cudaMemsetAsync(s->scalars.p, 0, sizeof(unsigned long long) * 8, s->stream));
            PSB_CUDA(cudaMemsetAsync(s->scalars.as<unsigned long long>() + kRowsFetched, 0, sizeof(unsigned long long), s->stream));
        }
        PSB_CUDA(cudaStreamSynchronize(s->stream));
    }
    stats->pq_scanned_codes = (long long)h[0];
    stats->pq_adc_lookups = (long long)h[0] * s->m;
    stats->threshold_candidates = (long long)h[1];
    stats->fallback_queries = (long long)h[2];
    stats->prefilter_survivors = (long long)h[3];
    stats->tc_wait_item_cycles = (long long)h[4]; stats->tc_wait_rows_cycles = (long long)h[5];
    stats->tc_wait_acc_cycles = (long long)h[6]; stats->tc_tiles = (long long)h[7];
    stats->rerank_rows_fetched = (long long)h[kRowsFetched];
    stats->staged_gather_ms = s->staged_gather_s * 1e3; stats->staged_gather_bytes = s->staged_gather_bytes;
    if (reset) { s->staged_gather_s = 0.0; s->staged_gather_bytes = 0; }
    stats->kernel_launches = launches_total();
    if (!s->scalars.p) PSB_CUDA(cudaStreamSynchronize(s->stream));
    s->collect_scan_events();
    stats->scan_kernel_ms = s->scan_ms_total;
    stats->scan_kernel_launches = s->scan_launches_total;
    stats->coarse_gemm_ms = s->gemm_ms_total;
    stats->coarse_gemm_launches = s->gemm_launches_total;
    if (reset) { s->gemm_ms_total = 0.0; s->gemm_launches_total = 0; }
    stats->coarse_fallback_queries = 0;
    if (s->tc_work.scalars.p) {
        int v = 0;
        PSB_CUDA(cudaMemcpy(&v, s->tc_work.scalars.as<int>() + 3, sizeof(int), cudaMemcpyDeviceToHost));
        stats->coarse_fallback_queries = v;
        if (reset) PSB_CUDA(cudaMemset(s->tc_work.scalars.as<int>() + 3, 0, sizeof(int)));
    }
    if (reset) { s->scan_ms_total = 0.0; s->scan_launches_total = 0; }
    return PSB_OK;
}

namespace {

// Stage times of one search call: spans between events, read once the stream has drained.  A recorded time costs the GPU about five
// microseconds between two kernels, so stages that follow one another on a stream share the event between them.
struct StageTimes {
    enum Stage { kCoarse, kLut, kScan, kRerank, kMap, kStages };
    double ms[kStages] = {0, 0, 0, 0, 0};
    EventTimer tm_s, tm_x;
    struct Span { Stage stage; cudaEvent_t a, b; };
    std::vector<Span> spans, spans_x;   // of the main thread, of the thread that drives the second stream
    cudaEvent_t last = nullptr;         // the main stream's latest mark; null once something else may have been queued behind it
    explicit StageTimes(psb_session* s) : tm_s(&s->timing), tm_x(&s->timing_aux) {}
    psb_status mark(cudaStream_t st) { PSB_TRY(tm_s.mark(st)); last = tm_s.ev.back(); return PSB_OK; }
    psb_status begin(cudaStream_t st) { return last ? PSB_OK : mark(st); }
    psb_status end(Stage stage, cudaStream_t st) {   // of a stage that began at `last`
        const cudaEvent_t from = last;
        PSB_TRY(mark(st));
        spans.push_back({stage, from, last});
        return PSB_OK;
    }
    psb_status mark_x(cudaStream_t st, cudaEvent_t* e) { PSB_TRY(tm_x.mark(st)); *e = tm_x.ev.back(); return PSB_OK; }
    void collect() {
        for (const auto* v : {&spans, &spans_x})
            for (const Span& sp : *v) { float t = 0.f; cudaEventElapsedTime(&t, sp.a, sp.b); ms[sp.stage] += t; }
        spans.clear(); spans_x.clear();
        tm_s.ev.clear(); tm_x.ev.clear();
        tm_s.pool->used = 0; tm_x.pool->used = 0;
        last = nullptr;
    }
};

// The session's page-locked block.
psb_status ensure_host_io(psb_session* s) {
    if (s->h_io) return PSB_OK;
    PSB_TRY(HostBlocks::get().take(&s->h_io));
    s->h_tail = reinterpret_cast<psb_session::Tail*>(s->h_io + kSmallIo);
    std::memset(s->h_tail, 0, sizeof(*s->h_tail));
    return PSB_OK;
}
// Queues the device's counters and status words behind the work on `st`.
psb_status queue_tail(psb_session* s, cudaStream_t st) {
    return launch_call_tail(s->scalars.as<unsigned long long>(), s->tc_work.scalars.as<int>(), s->h_tail, st, s->call_marks != nullptr);
}
// Small calls on one stream: the kernels note their starts themselves and the first reads the queries where they are.  A recorded event costs the
// GPU five microseconds between two kernels and the host two, and a small copy to the device as much again.
// The whole call then, with its transfers, which have no times of their own, is what passes on the host's clock from the first copy to the last.
using HostClock = std::chrono::steady_clock;
double ms_since(HostClock::time_point t) { return std::chrono::duration<double, std::milli>(HostClock::now() - t).count(); }
struct CallMarks {
    psb_session* s;
    bool on;
    CallMarks(psb_session* s_, bool on_, const float* h_queries, int n) : s(s_), on(on_) {
        if (!on) return;
        s->call_marks = s->scalars.as<unsigned long long>() + 13;
        // every 64 centroids are behind a read of the queries over PCIe: up to 64 KB of reads
        if (coarse_few(n, s->nlist, s->dim) && (size_t)n * s->dim * sizeof(float) * ((s->nlist + kCoarseFewBlock - 1) / kCoarseFewBlock) <= 65536) {
            s->host_queries = h_queries;
            s->query_copy = s->q.as<float>();
        }
    }
    ~CallMarks() { s->call_marks = nullptr; s->host_queries = nullptr; s->query_copy = nullptr; }
    double ms(int from, int to) const {   // 0: coarse stage, 1: scan, 2: rerank, 3: end
        const psb_session::Tail& t = *s->h_tail;
        const unsigned long long a = t.c[13 + from], b = to == 3 ? t.end : t.c[13 + to];
        return b > a ? (double)(b - a) * 1e-6 : 0.0;
    }
};
// The counters as they are before a call: what the last call left, unless others have run in between.
psb_status counters_before(psb_session* s, cudaStream_t st, unsigned long long (&c)[4]) {
    if (!s->counters_known) {
        PSB_TRY(queue_tail(s, st));
        PSB_CUDA(cudaStreamSynchronize(st));
    }
    std::memcpy(c, s->h_tail->c, sizeof(c));
    return PSB_OK;
}
// Once the stream has drained: the status words the tail brought.
psb_status check_tail(psb_session* s) {
    s->counters_known = true;
    if (s->h_tail->tc[2]) return fail(PSB_TIMEOUT, "a bounded wait in the tensor-core coarse kernel gave up");
    if ((int)s->h_tail->c[12]) {
        s->counters_known = false;
        return s->check_scan_status();
    }
    return PSB_OK;
}

// One batch, device in / device out.  With a rerank from mapped or resident exact rows the batch is cut into
// sub-batches: coarse + LUT + scan of sub-batch i run on the session's stream while the PCIe gather, exact scoring,
// selection and id map of sub-batch i-1 run on a second stream, so the transfer hides behind the scan.
psb_status search_device(psb_session* s, const float* dq, const void* dq_exact, int n, int nprobe, int topk, int stage1_k,
                         bool rerank, long long* d_ids, float* d_dist, int* d_probes, StageTimes* times) {
    PSB_RANGE("ivfpq_batch");
    cudaStream_t st = s->stream;
    const bool overlap = overlap_enabled(s, n, rerank);
    // Staged transport, overlapped: a host worker thread takes each sub-batch's candidates as soon as its scan has finished,
    // gathers the rows with the host cores into the pinned rings and queues copies + exact scoring on the second stream,
    // while this thread goes on queueing the next sub-batch's scan.  No SM is spent on the transfer.
    const bool staged_overlap = staged_overlap_enabled(s, n, rerank);
    const bool residual = s->opt.adc_mode == 1;
    // The rows of the whole batch are claimed and fetched once each, sub-batch by sub-batch (a row an earlier sub-batch has fetched is
    // in its slot already), unless they are scored in place.
    const int host_pct = host_share(s);
    const bool shared_rows = rows_shared(s, n, stage1_k, rerank);
    const bool kernel_gather = shared_rows && host_pct < 100;   // on a stream of its own
    const std::vector<int> cuts = batch_cuts(s, n, nprobe, stage1_k, rerank);
    const int sb_max = longest_cut(cuts);
    // The sub-batch size depends on this batch's own n (a short tail batch may run in one piece where the full batch ran
    // in four), so the tables and the scan workspace are sized here, for the largest sub-batch of THIS batch.
    const bool rows_only = rows_form(s, sb_max, nprobe), table_free = residual_table_free(s, stage1_k) || rows_only;
    if (!table_free) PSB_TRY(s->lut.reserve(sizeof(float) * table_count(s, sb_max, nprobe) * s->m * s->k));
    PSB_TRY(ensure_scan_ws(s, sb_max, nprobe, stage1_k, rows_only));
    // The row form's too: sub-batches that grow laid it out anew, one after the other (5,611 queries, first call of a session 5.5 -> 3.1 ms).
    int row_queries = 0;
    for (size_t i = 0; i + 1 < cuts.size(); ++i)
        if (rows_only || rows_form(s, cuts[i + 1] - cuts[i], nprobe)) row_queries = std::max(row_queries, cuts[i + 1] - cuts[i]);
    if (row_queries > 0) PSB_TRY(ensure_row_ws(s, row_queries, nprobe, false));
    if ((overlap || staged_overlap) && !s->aux_stream) {
        int lo = 0, hi = 0;  // lowest priority: the scan's CTAs get the SMs first, the transfer fills the gaps
        PSB_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
        PSB_CUDA(cudaStreamCreateWithPriority(&s->aux_stream, cudaStreamNonBlocking, lo));
    }
    cudaStream_t sx = (overlap || staged_overlap) ? s->aux_stream : st;
    struct OneStream {
        psb_session* s;
        OneStream(psb_session* s_, bool one) : s(s_) { s->one_stream = one; }
        ~OneStream() { s->one_stream = false; }
    } one_stream(s, !overlap && !staged_overlap);
    struct EventList {  // destroyed on every way out of this function (an event may be destroyed once the waits on it are queued)
        std::vector<cudaEvent_t> v;
        ~EventList() { for (auto e : v) cudaEventDestroy(e); }
        void push_back(cudaEvent_t e) { v.push_back(e); }
    } deps;
    if (overlap || staged_overlap) {  // the second stream starts after everything already queued on the main stream
        cudaEvent_t e0;
        PSB_CUDA(cudaEventCreateWithFlags(&e0, cudaEventDisableTiming));
        deps.push_back(e0);
        PSB_CUDA(cudaEventRecord(e0, st));
        PSB_CUDA(cudaStreamWaitEvent(sx, e0, 0));
    }
    psb_status rc = PSB_OK;
    Gathers gathers{s, st};
    struct Job { int part, p0, m; cudaEvent_t ready; cudaEvent_t gathered; };
    std::mutex mu;
    std::condition_variable cv;
    std::deque<Job> jobs;
    bool done = false;
    psb_status worker_rc = PSB_OK;
    std::string worker_msg;
    std::thread worker;
    const int row_bytes = s->dim * s->exact_elem;
    if (kernel_gather) PSB_TRY(ensure_zc_stream(s));
    if (shared_rows) {
        PSB_TRY(s->score.reserve(sizeof(float) * (size_t)sb_max * stage1_k));
        PSB_TRY(rows_begin(s, (long long)n * stage1_k, cuts.size() - 1, st));
        cudaEvent_t e0;
        PSB_CUDA(cudaEventCreateWithFlags(&e0, cudaEventDisableTiming));
        deps.push_back(e0);
        PSB_CUDA(cudaEventRecord(e0, st));
        PSB_CUDA(cudaStreamWaitEvent(sx, e0, 0));
    }
    auto score_part = [&](int p0, int m) {
        const unsigned char* qe = static_cast<const unsigned char*>(dq_exact) + (size_t)p0 * row_bytes;
        return score_and_select(s, false, qe, m, s->cand_rows.as<int>() + (size_t)p0 * stage1_k, stage1_k, stage1_k, s->cand_count.as<int>() + p0, topk,
                                s->striped ? s->out_rows.as<int>() + (size_t)p0 * topk : nullptr, d_dist + (size_t)p0 * topk,
                                s->striped ? nullptr : d_ids + (size_t)p0 * topk, s->score.as<float>(), sx);
    };
    if (staged_overlap) {
        worker = std::thread([&]() {
            cudaSetDevice(s->device);
            auto process = [&](const Job& j) -> psb_status {
                PSB_RANGE("pq_rerank");
                PSB_CUDA(cudaEventSynchronize(j.ready));
                cudaEvent_t t0 = nullptr, t1 = nullptr;
                if (times) PSB_TRY(times->mark_x(sx, &t0));
                // Hybrid transport: the kernel's share of the slots comes through the gather kernel, which the main thread queued right
                // behind this sub-batch's claim (j.gathered marks its end); the host threads and the copy engine bring the others; the
                // scoring waits for both.
                PSB_TRY(gather_error(s));
                PSB_TRY(rows_from_host(s, j.part, host_pct, sx));
                if (j.gathered) PSB_CUDA(cudaStreamWaitEvent(sx, j.gathered, 0));
                PSB_TRY(score_part(j.p0, j.m));
                if (times) { PSB_TRY(times->mark_x(sx, &t1)); times->spans_x.push_back({StageTimes::kRerank, t0, t1}); }
                if (s->striped) {
                    PSB_TRY(launch_map_ids(s->out_rows.as<int>() + (size_t)j.p0 * topk, (long long)j.m * topk, s->reordered.as<long long>(), s->row_map(),
                                           d_ids + (size_t)j.p0 * topk, sx));
                    if (times) { PSB_TRY(times->mark_x(sx, &t0)); times->spans_x.push_back({StageTimes::kMap, t1, t0}); }
                }
                return PSB_OK;
            };
            for (;;) {
                Job j;
                {
                    std::unique_lock<std::mutex> lk(mu);
                    cv.wait(lk, [&] { return !jobs.empty() || done; });
                    if (jobs.empty()) return;
                    j = jobs.front();
                    jobs.pop_front();
                }
                if (worker_rc != PSB_OK) continue;  // drain
                const psb_status r = process(j);
                if (r != PSB_OK) { worker_rc = r; worker_msg = psb_last_error(); }
            }
        });
    }
    auto finish_worker = [&]() {
        if (!worker.joinable()) return;
        { std::lock_guard<std::mutex> lk(mu); done = true; }
        cv.notify_all();
        worker.join();
    };
    // Coarse stage for the whole batch first: one large GEMM is more efficient than four small ones, and the tensor-core
    // kernel (a full SM's shared and tensor memory per CTA) then never has to share SMs with the transfer stream.
    if (times) rc = times->begin(st);
    if (rc == PSB_OK) { PSB_RANGE("coarse_search"); rc = coarse_exact(s, dq, n, nprobe, d_probes, nullptr); }
    // OPQ index: the PQ side works on the rotated queries (counted with the coarse stage's time)
    const float* dq_pq = dq;
    if (rc == PSB_OK && s->opq.p) {
        rc = s->q_rot.reserve(sizeof(float) * (size_t)n * s->dim);
        if (rc == PSB_OK) rc = launch_rotate_rows(dq, s->opq.as<float>(), n, s->dim, s->q_rot.as<float>(), st);
        dq_pq = s->q_rot.as<float>();
    }
    if (rc == PSB_OK && times) rc = times->end(StageTimes::kCoarse, st);
    for (size_t ci = 0; ci + 1 < cuts.size() && rc == PSB_OK; ++ci) {
        const int p0 = cuts[ci];
        const int m = cuts[ci + 1] - p0;
        const float* q = dq_pq + (size_t)p0 * s->dim;
        int* probes = d_probes + (size_t)p0 * nprobe;
        int* rows_out = rerank ? s->cand_rows.as<int>() + (size_t)p0 * stage1_k : s->out_rows.as<int>() + (size_t)p0 * topk;
        float* dist_out = rerank ? s->cand_dist.as<float>() + (size_t)p0 * stage1_k : d_dist + (size_t)p0 * topk;
        int* cnt_out = s->cand_count.as<int>() + p0;
        if (times) rc = times->begin(st);
        ScanWorkspace sws;
        if (rc == PSB_OK) rc = s->timed_scan_ws(&sws);
        if (kernel_gather) sws.reserve_ctas = std::max(sws.reserve_ctas, gather_sms(s));   // the gather kernel gets SMs of its own
        if (rc == PSB_OK && !table_free) {
            PSB_RANGE("pq_lut_build");
            if (residual && residual_tables_fused(sws, s->m, s->k)) {  // fp32 and fp16 tables in one kernel
                rc = launch_build_tables_residual(q, m, s->dim, probes, nprobe, s->centroids.as<float>(), s->nlist,
                                                  s->codebook.as<float>(), s->m, s->k, s->cb_maxnorm.as<float>(), s->lut.as<float>(),
                                                  sws, st);
                sws.half_tables_ready = true;
            } else if (residual) {
                rc = launch_build_lut_residual(q, m, s->dim, probes, nprobe, s->centroids.as<float>(), s->nlist,
                                               s->codebook.as<float>(), s->m, s->k, s->lut.as<float>(), st);
            } else {
                rc = launch_build_lut(q, m, s->dim, s->codebook.as<float>(), s->m, s->k, s->lut.as<float>(), st);
            }
        }
        if (rc == PSB_OK && times && !table_free) rc = times->end(StageTimes::kLut, st);
        if (rc == PSB_OK) {
            PSB_RANGE("pq_adc_scan");
            rc = run_scan(s, sws, rows_only, q, table_free ? nullptr : s->lut.as<float>(), m, probes, nprobe, stage1_k, rows_out, dist_out, cnt_out, st);
        }
        if (rc == PSB_OK && times) rc = times->end(StageTimes::kScan, st);
        if (rc != PSB_OK) break;
        cudaEvent_t ready = nullptr, gathered = nullptr;
        auto event = [&](cudaEvent_t* e) -> psb_status {
            if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return fail(PSB_CUDA_ERROR, "event creation failed");
            deps.push_back(*e);
            return PSB_OK;
        };
        if (shared_rows) {
            rc = rows_claim(s, (int)ci, rows_out, m, stage1_k, stage1_k, cnt_out, st);
            if (rc == PSB_OK && staged_overlap) rc = rows_tell_host(s, (int)ci, st);
            if (rc != PSB_OK) break;
        }
        if (shared_rows || overlap) {
            if ((rc = event(&ready)) != PSB_OK) break;
            cudaEventRecord(ready, st);
        }
        if (kernel_gather) {   // queued now: the transfer starts the moment the rows are claimed
            if ((rc = event(&gathered)) != PSB_OK) break;
            cudaStreamWaitEvent(s->zc_stream, ready, 0);
            gathers.open = true;
            rc = launch_gather_unique(s->exact_dev, row_bytes, s->unique.as<int>(), part_begin(s, (int)ci), part_end(s, (int)ci), host_pct, s->stage.p,
                                      s->zc_stream, s->sm_count, s->opt.gather_ctas, gather_sms(s));
            if (rc != PSB_OK) break;
            cudaEventRecord(gathered, s->zc_stream);
            if (!staged_overlap && (rc = gather_error(s)) != PSB_OK) break;
        }
        if (staged_overlap) {  // the worker takes over: the event marks the slot range ready
            { std::lock_guard<std::mutex> lk(mu); jobs.push_back(Job{(int)ci, p0, m, ready, gathered}); }
            cv.notify_all();
            continue;
        }
        if (overlap) cudaStreamWaitEvent(sx, ready, 0);
        // second half of the sub-batch (on the second stream when overlapping)
        cudaStream_t keep = s->stream;
        s->stream = sx;  // rerank_impl and the launchers below run on s->stream
        cudaEvent_t t0 = nullptr, t1 = nullptr;   // second stream
        if (times && overlap) rc = times->mark_x(sx, &t0);
        bool mapped_ids = false;
        if (rc == PSB_OK && rerank) {
            PSB_RANGE("pq_rerank");
            mapped_ids = !s->striped;
            if (shared_rows) {
                cudaStreamWaitEvent(sx, gathered, 0);
                rc = score_part(p0, m);
            } else {
                const unsigned char* qe = static_cast<const unsigned char*>(dq_exact) + (size_t)p0 * row_bytes;
                rc = rerank_impl(s, qe, m, rows_out, stage1_k, stage1_k, cnt_out, topk, mapped_ids ? nullptr : s->out_rows.as<int>() + (size_t)p0 * topk,
                                 d_dist + (size_t)p0 * topk, nullptr, mapped_ids ? d_ids + (size_t)p0 * topk : nullptr);
            }
        }
        if (rc == PSB_OK && times && rerank && !overlap) rc = times->end(StageTimes::kRerank, st);
        if (rc == PSB_OK && times && overlap) { rc = times->mark_x(sx, &t1); times->spans_x.push_back({StageTimes::kRerank, t0, t1}); }
        if (rc == PSB_OK && !mapped_ids) {
            PSB_RANGE("pq_map_ids");
            rc = launch_map_ids(s->out_rows.as<int>() + (size_t)p0 * topk, (long long)m * topk, s->reordered.as<long long>(),
                                s->row_map(), d_ids + (size_t)p0 * topk, sx);
        }
        if (rc == PSB_OK && times && !overlap && !mapped_ids) rc = times->end(StageTimes::kMap, st);
        if (rc == PSB_OK && times && overlap && !mapped_ids) { rc = times->mark_x(sx, &t0); times->spans_x.push_back({StageTimes::kMap, t1, t0}); }
        s->stream = keep;
    }
    finish_worker();
    if (worker_rc != PSB_OK && rc == PSB_OK) rc = fail(worker_rc, "rerank worker: " + worker_msg);
    if (rc == PSB_OK) gathers.open = false;   // the second stream has waited for each, and the main stream waits for that below
    if (shared_rows && rc == PSB_OK) rc = rows_end(s, sx);
    if (times && (overlap || staged_overlap)) times->last = nullptr;
    if (overlap || staged_overlap) {  // the main stream continues only after the second stream has finished this batch
        cudaEvent_t e;
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess) {
            deps.push_back(e);
            cudaEventRecord(e, sx);
            cudaStreamWaitEvent(st, e, 0);
        } else if (rc == PSB_OK) rc = fail(PSB_CUDA_ERROR, "event creation failed");
    }
    return rc;
}

}  // namespace

psb_status psb_session_search_device(psb_session* s, const float* d_queries, const uint8_t* d_queries_u8, int nq,
                                     const psb_search_params* params, int64_t* d_indices, float* d_distances,
                                     int* d_coarse_ids) {
    if (!s || !params || !d_queries || !d_indices || !d_distances) return fail(PSB_INVALID_ARGUMENT, "null argument");
    if (nq < 0 || nq > s->opt.max_batch) return fail(PSB_INVALID_ARGUMENT, "nq must be in 0..max_batch");
    if (params->nprobe <= 0 || params->nprobe > s->nlist || params->topk <= 0) return fail(PSB_INVALID_ARGUMENT, "nprobe must be in 1..nlist and topk positive");
    if (params->nprobe > kMaxProbe || params->topk > kMaxTopk) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 or topk above 2048");
    if (params->distance != 0) return fail(PSB_UNSUPPORTED_SHAPE, "only squared L2 is supported on this path");
    if (nq == 0) return PSB_OK;
    s->counters_known = false;
    PSB_CUDA(cudaSetDevice(s->device));
    const int topk = params->topk;
    const int stage1_k = stage1_width(s, topk);
    const bool rerank = rerank_enabled(s, topk);
    if (stage1_k > kMaxStage1) return fail(PSB_UNSUPPORTED_SHAPE, "candidate width above 2048 is not supported");
    if (rerank && s->exact_elem == 1 && !d_queries_u8) return fail(PSB_INVALID_ARGUMENT, "u8 rerank needs u8 queries");
    PSB_TRY(ensure_pipeline_ws(s, nq, params->nprobe, topk, stage1_k));
    int* probes = d_coarse_ids ? d_coarse_ids : s->probes.as<int>();
    const void* qe = s->exact_elem == 1 ? static_cast<const void*>(d_queries_u8) : static_cast<const void*>(d_queries);
    return search_device(s, d_queries, qe, nq, params->nprobe, topk, stage1_k, rerank, reinterpret_cast<long long*>(d_indices),
                         d_distances, probes, nullptr);
}

psb_status psb_session_search(psb_session* s, const psb_query_batch_view* queries, const psb_search_params* params,
                              const psb_search_output_view* output, psb_stats* stats) {
    PSB_RANGE("ivfpq_search");
    if (!s) return fail(PSB_INVALID_ARGUMENT, "session is null");
    PSB_TRY(validate_params(s, queries, params, output));
    PSB_CUDA(cudaSetDevice(s->device));
    if (stats) std::memset(stats, 0, sizeof(*stats));
    const int total = queries->count;
    if (total == 0) return PSB_OK;
    const int nprobe = params->nprobe, topk = params->topk;
    const int batch = std::min(std::min(params->batch_size, s->opt.max_batch), total);
    const int stage1_k = stage1_width(s, topk);
    const bool rerank = rerank_enabled(s, topk);
    if (stage1_k > kMaxStage1) return fail(PSB_UNSUPPORTED_SHAPE, "candidate width above 2048 is not supported");
    PSB_TRY(ensure_pipeline_ws(s, batch, nprobe, topk, stage1_k));
    const bool u8 = rerank && s->exact_elem == 1;
    if (u8) PSB_TRY(s->q_u8.reserve((size_t)batch * s->dim));
    cudaStream_t st = s->stream;
    // A small call's queries go to the device from the pinned block, and its results are written there by the kernels themselves.
    const size_t b_q = (sizeof(float) * (size_t)total * s->dim + 255) / 256 * 256, b_u8 = u8 ? ((size_t)total * s->dim + 255) / 256 * 256 : 0,
                 b_ids = sizeof(long long) * (size_t)total * topk, b_dist = sizeof(float) * (size_t)total * topk;
    const bool small = batch == total && b_q + b_u8 + b_ids + b_dist <= kSmallIo;
    PSB_TRY(ensure_host_io(s));
    HostCopies copies(st, {{small ? nullptr : queries->fp32, sizeof(float) * (size_t)total * s->dim}, {small || !u8 ? nullptr : queries->u8, (size_t)total * s->dim},
                           {small ? nullptr : output->indices, b_ids}, {small ? nullptr : output->distances, b_dist}, {output->coarse_ids, sizeof(int) * (size_t)total * nprobe}});
    const bool one_stream = total < 2048 && sub_batch_rows(s, total, nprobe, false) >= total;
    CallMarks marks(s, small && one_stream && rows_form(s, total, nprobe) && !coarse_by_tc(s, total, nprobe) &&
                           (!rerank || rows_in_place(s, (long long)total * stage1_k)), reinterpret_cast<const float*>(s->h_io), total);
    const bool timed = stats && !marks.on;   // by events
    const long long launches0 = launches_total();
    unsigned long long c0[4] = {0, 0, 0, 0};
    if (stats) PSB_TRY(counters_before(s, st, c0));
    s->counters_known = false;
    s->collect_scan_events();
    const double scan_ms0 = s->scan_ms_total;
    const long long scan_n0 = s->scan_launches_total;
    s->timing.used = s->timing_aux.used = 0;
    StageTimes times(s);
    double t_h2d = 0, t_d2h = 0, t_total = 0;
    long long h2d = 0, d2h = 0;
    int nb = 0;
    const auto began = HostClock::now();
    for (int q0 = 0; q0 < total; q0 += batch, ++nb) {
        const int n = std::min(batch, total - q0);
        cudaEvent_t t_begin = nullptr, t_in = nullptr, t_done = nullptr;
        if (timed) { PSB_TRY(times.mark(st)); t_begin = times.last; }
        const void* from = queries->fp32 + (size_t)q0 * s->dim;
        const void* from_u8 = u8 ? queries->u8 + (size_t)q0 * s->dim : nullptr;
        if (small) {
            std::memcpy(s->h_io, from, sizeof(float) * (size_t)n * s->dim);
            from = s->h_io;
            if (u8) { std::memcpy(s->h_io + b_q, from_u8, (size_t)n * s->dim); from_u8 = s->h_io + b_q; }
        }
        if (!s->host_queries) PSB_CUDA(cudaMemcpyAsync(s->q.p, from, sizeof(float) * (size_t)n * s->dim, cudaMemcpyHostToDevice, st));
        h2d += (long long)sizeof(float) * n * s->dim;
        if (u8) {
            PSB_CUDA(cudaMemcpyAsync(s->q_u8.p, from_u8, (size_t)n * s->dim, cudaMemcpyHostToDevice, st));
            h2d += (long long)n * s->dim;
        }
        if (timed) { PSB_TRY(times.mark(st)); t_in = times.last; }
        const void* qe = s->exact_elem == 1 ? s->q_u8.p : s->q.p;
        long long* ids = small ? reinterpret_cast<long long*>(s->h_io + b_q + b_u8) : s->out_ids.as<long long>();
        float* dist = small ? reinterpret_cast<float*>(s->h_io + b_q + b_u8 + b_ids) : s->out_dist.as<float>();
        PSB_TRY(search_device(s, s->q.as<float>(), qe, n, nprobe, topk, stage1_k, rerank, ids, dist, s->probes.as<int>(), timed ? &times : nullptr));
        if (timed) { PSB_TRY(times.begin(st)); t_done = times.last; }
        if (!small) {
            PSB_CUDA(cudaMemcpyAsync(output->indices + (size_t)q0 * topk, ids, sizeof(long long) * (size_t)n * topk, cudaMemcpyDeviceToHost, st));
            PSB_CUDA(cudaMemcpyAsync(output->distances + (size_t)q0 * topk, dist, sizeof(float) * (size_t)n * topk, cudaMemcpyDeviceToHost, st));
        }
        d2h += (long long)(sizeof(long long) + sizeof(float)) * n * topk;
        if (output->coarse_ids) {
            PSB_CUDA(cudaMemcpyAsync(output->coarse_ids + (size_t)q0 * nprobe, s->probes.p, sizeof(int) * (size_t)n * nprobe, cudaMemcpyDeviceToHost, st));
            d2h += (long long)sizeof(int) * n * nprobe;
        }
        if (q0 + batch >= total) PSB_TRY(queue_tail(s, st));
        if (timed) PSB_TRY(times.mark(st));
        PSB_CUDA(cudaStreamSynchronize(st));
        if (small) {
            std::memcpy(output->indices, ids, b_ids);
            std::memcpy(output->distances, dist, b_dist);
        }
        if (timed) {
            auto span = [](cudaEvent_t a, cudaEvent_t b) { float t = 0.f; cudaEventElapsedTime(&t, a, b); return (double)t; };
            t_h2d += span(t_begin, t_in); t_d2h += span(t_done, times.last); t_total += span(t_begin, times.last);
            times.collect();
        }
    }
    copies.ended = true;
    const double call_ms = ms_since(began);
    PSB_TRY(check_tail(s));
    if (stats && marks.on) {
        times.ms[StageTimes::kCoarse] = marks.ms(0, 1);
        times.ms[StageTimes::kScan] = marks.ms(1, rerank ? 2 : 3);
        if (rerank) times.ms[StageTimes::kRerank] = marks.ms(2, 3);
        t_total = call_ms;
    }
    if (stats) {
        const unsigned long long* c1 = s->h_tail->c;
        stats->h2d_ms = t_h2d; stats->coarse_search_ms = times.ms[StageTimes::kCoarse]; stats->pq_lut_build_ms = times.ms[StageTimes::kLut];
        stats->pq_adc_scan_ms = times.ms[StageTimes::kScan]; stats->pq_rerank_ms = times.ms[StageTimes::kRerank];
        stats->pq_map_ids_ms = times.ms[StageTimes::kMap]; stats->d2h_ms = t_d2h;
        stats->total_ms = t_total;  // stage times can overlap: their sum may exceed the total
        stats->pq_scanned_codes = (long long)(c1[0] - c0[0]);
        stats->pq_adc_lookups = stats->pq_scanned_codes * s->m;
        stats->threshold_candidates = (long long)(c1[1] - c0[1]);
        stats->fallback_queries = (long long)(c1[2] - c0[2]);
        stats->prefilter_survivors = (long long)(c1[3] - c0[3]);
        stats->h2d_bytes = h2d; stats->d2h_bytes = d2h;
        stats->kernel_launches = launches_total() - launches0;
        s->collect_scan_events();
        stats->scan_kernel_ms = s->scan_ms_total - scan_ms0;
        stats->scan_kernel_launches = s->scan_launches_total - scan_n0;
        stats->batches = nb;
    }
    return PSB_OK;
}

// ---- IVF-Flat ----------------------------------------------------------------------------------------------------

psb_status psb_flat_session_create(const psb_flat_index_view* index, const psb_options* options, psb_flat_session** out) {
    if (!out) return fail(PSB_INVALID_ARGUMENT, "out is null");
    *out = nullptr;
    if (!index) return fail(PSB_INVALID_ARGUMENT, "index view is null");
    {   // the list layout rules of the PQ index (src/search/ivf_common/ivf_list_layout.h:19-45)
        psb_index_view probe{};
        probe.coarse = index->coarse; probe.lists = index->lists;
        static const float one_codeword = 0.0f;
        static const uint8_t no_codes = 0;
        probe.pq.codes = &no_codes; probe.pq.codebook = &one_codeword; probe.pq.subvectors = 1; probe.pq.codebook_size = 1;
        if (index->coarse.dim <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid IVF coarse index view");
        PSB_TRY(validate_index(&probe));
    }
    if (!index->rowmajor_fp32 && index->lists.n_vectors > 0) return fail(PSB_INVALID_ARGUMENT, "IVF-Flat rows are null");
    psb_options opt{};
    if (options) opt = *options;
    if (opt.max_batch <= 0) opt.max_batch = 10000;
    int sms = 0;
    PSB_TRY(check_device(opt.device, &sms));
    std::unique_ptr<psb_session> s(new (std::nothrow) psb_session());
    if (!s) return fail(PSB_OUT_OF_MEMORY, "host allocation failed");
    s->flat = true;
    s->device = opt.device; s->sm_count = sms; s->opt = opt;
    s->nlist = index->lists.nlist; s->dim = index->coarse.dim; s->n_vectors = index->lists.n_vectors;
    s->list_begin = 0; s->list_end = s->nlist; s->row_base = 0; s->shard_rows = s->n_vectors;
    if (opt.stream) s->stream = static_cast<cudaStream_t>(opt.stream);
    else { PSB_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking)); s->own_stream = true; }
    cudaStream_t st = s->stream;
    const size_t nl = (size_t)s->nlist, n = (size_t)std::max<long long>(1, s->n_vectors);
    HostCopies copies(st, {{index->coarse.centroids, sizeof(float) * nl * s->dim}, {index->lists.offsets, sizeof(long long) * (nl + 1)},
                           {index->lists.reordered_ids, sizeof(long long) * (size_t)s->n_vectors}, {index->rowmajor_fp32, sizeof(float) * (size_t)s->n_vectors * s->dim}});
    PSB_TRY(s->centroids.reserve(sizeof(float) * nl * s->dim));
    PSB_CUDA(cudaMemcpyAsync(s->centroids.p, index->coarse.centroids, sizeof(float) * nl * s->dim, cudaMemcpyHostToDevice, st));
    if (opt.coarse_mode != 1 && s->nlist >= 1024 && coarse_tc_padded_dim(s->dim) <= 128)
        PSB_TRY(s->tc_index.prepare(s->centroids.as<float>(), s->nlist, s->dim, s->device, st));
    PSB_TRY(s->offsets.reserve(sizeof(long long) * (nl + 1)));
    PSB_CUDA(cudaMemcpyAsync(s->offsets.p, index->lists.offsets, sizeof(long long) * (nl + 1), cudaMemcpyHostToDevice, st));
    PSB_TRY(s->reordered.reserve(sizeof(long long) * n));
    // One allocation: the norms of their own took the room in a block of the driver's that the first call's workspace then lacked (21 queries x 7 lists
    // of 1,000 rows, first call 85 -> 480 us).
    PSB_TRY(reserve_together(&s->flat_whole, {{&s->flat_rows, sizeof(float) * n * s->dim}, {&s->flat_norms, sizeof(float) * (n + nl)}}));
    if (s->n_vectors > 0) {
        PSB_CUDA(cudaMemcpyAsync(s->reordered.p, index->lists.reordered_ids, sizeof(long long) * n, cudaMemcpyHostToDevice, st));
        PSB_CUDA(cudaMemcpyAsync(s->flat_rows.p, index->rowmajor_fp32, sizeof(float) * n * s->dim, cudaMemcpyHostToDevice, st));
    }
    note_list_lengths(s.get(), index->lists.offsets);
    PSB_TRY(launch_flat_norms(s->flat_rows.as<float>(), s->n_vectors, s->dim, s->offsets.as<long long>(), s->nlist, s->flat_norms.as<float>(),
                              s->flat_norms.as<unsigned>() + n, st));
    PSB_TRY(ensure_scalars(s.get(), st));
    PSB_CUDA(cudaStreamSynchronize(st));
    copies.ended = true;
    s->count();
    *out = s.release();
    return PSB_OK;
}

psb_status psb_flat_session_destroy(psb_flat_session* s) {
    delete s;
    return PSB_OK;
}

namespace {
psb_status flat_search_device(psb_session* s, const float* dq, int n, int nprobe, int topk, long long* d_ids, float* d_dist) {
    // A row of distances per query, as long as the nprobe longest lists; queries in parts of at most 1 GiB of them.
    FlatScan f{};
    f.stride = std::max<long long>(1, s->longest[(size_t)nprobe]);
    const long long most = std::max<long long>(1, std::min(kPartQueries, kRowDistFloats / f.stride));
    const int parts = (int)((n + most - 1) / most), per = (n + parts - 1) / parts;
    f.run_stride = sel::run_count(f.stride);
    // All that the call needs in one allocation, before anything is queued (a first call of 1,000 queries x 16 lists of 390 rows x 128: 900 -> 543 us).
    const bool lists = flat_list_form(per, nprobe, s->nlist, s->n_vectors, s->dim);
    const size_t pairs = lists ? (size_t)per * nprobe : 0, nl = lists ? (size_t)s->nlist + 1 : 0;
    PSB_TRY(reserve_together(&s->row_whole, {{&s->probes, sizeof(int) * (size_t)n * nprobe}, {&s->dist_tile, exact_coarse_bytes(s, n, nprobe)},
                                             {&s->row_dist, sizeof(float) * (size_t)per * f.stride}, {&s->row_seg, sizeof(int) * (size_t)per * ((size_t)nprobe + 1)},
                                             {&s->row_runs, sizeof(float) * (size_t)per * f.run_stride},
                                             {&s->vis_count, sizeof(int) * nl}, {&s->vis_off, sizeof(int) * nl}, {&s->item_off, sizeof(long long) * nl},
                                             {&s->visitors, sizeof(int) * pairs}, {&s->flat_slot, sizeof(int) * pairs},
                                             {&s->flat_again, lists ? sizeof(int) * (size_t)per : 0}}));
    PSB_TRY(coarse_exact(s, dq, n, nprobe, s->probes.as<int>(), nullptr));
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    if (s->opt.time_kernels) {  // bracket the fine scan (read back by psb_session_counters)
        PSB_CUDA(cudaEventCreate(&ev0));
        PSB_CUDA(cudaEventCreate(&ev1));
        s->scan_events.emplace_back(ev0, ev1);
        PSB_CUDA(cudaEventRecord(ev0, s->stream));
    }
    f.dim = s->dim; f.nprobe = nprobe; f.offsets = s->offsets.as<long long>(); f.nlist = s->nlist; f.n_rows = s->n_vectors; f.rows = s->flat_rows.as<float>();
    f.norms = s->flat_norms.as<float>(); f.most = s->flat_norms.as<unsigned>() + std::max<long long>(1, s->n_vectors);
    f.ids = s->reordered.as<long long>(); f.topk = topk; f.form = s->opt.scan_mode; f.dist = s->row_dist.as<float>(); f.seg = s->row_seg.as<int>();
    f.vis_count = s->vis_count.as<int>(); f.slot = s->flat_slot.as<int>(); f.vis_off = s->vis_off.as<int>(); f.item_off = s->item_off.as<long long>();
    f.visitors = s->visitors.as<int>(); f.again = s->flat_again.as<int>(); f.counters = s->scalars.as<unsigned long long>(); f.sm_count = s->sm_count;
    for (int q0 = 0; q0 < n; q0 += per) {
        f.queries = dq + (size_t)q0 * s->dim; f.probes = s->probes.as<int>() + (size_t)q0 * nprobe;
        f.out_ids = d_ids + (size_t)q0 * topk; f.out_dist = d_dist + (size_t)q0 * topk;
        f.runs = std::min(per, n - q0) <= sel::kRunQueries ? s->row_runs.as<float>() : nullptr;
        PSB_TRY(launch_flat_scan(f, std::min(per, n - q0), s->stream));
    }
    if (ev1) PSB_CUDA(cudaEventRecord(ev1, s->stream));
    return PSB_OK;
}
psb_status flat_check(const psb_session* s, const psb_search_params* p) {
    if (!s || !s->flat) return fail(PSB_INVALID_ARGUMENT, "not an IVF-Flat session");
    if (!p) return fail(PSB_INVALID_ARGUMENT, "params are null");
    if (p->nprobe <= 0 || p->nprobe > s->nlist) return fail(PSB_INVALID_ARGUMENT, "nprobe must be in 1..nlist");
    if (p->topk <= 0) return fail(PSB_INVALID_ARGUMENT, "topk must be positive");
    if (p->batch_size <= 0) return fail(PSB_INVALID_ARGUMENT, "batch_size must be positive");
    if (p->distance != 0) return fail(PSB_UNSUPPORTED_SHAPE, "only squared L2 is supported on this path");
    if (p->nprobe > kMaxProbe || p->topk > kMaxTopk) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 or topk above 2048");
    return PSB_OK;
}
}  // namespace

psb_status psb_flat_session_search_device(psb_flat_session* s, const float* d_queries, int nq, const psb_search_params* params,
                                          int64_t* d_indices, float* d_distances) {
    PSB_TRY(flat_check(s, params));
    if (!d_queries || !d_indices || !d_distances) return fail(PSB_INVALID_ARGUMENT, "null argument");
    if (nq < 0 || nq > s->opt.max_batch) return fail(PSB_INVALID_ARGUMENT, "nq must be in 0..max_batch");
    if (nq == 0) return PSB_OK;
    s->counters_known = false;
    PSB_CUDA(cudaSetDevice(s->device));
    return flat_search_device(s, d_queries, nq, params->nprobe, params->topk, reinterpret_cast<long long*>(d_indices), d_distances);
}

psb_status psb_flat_session_search(psb_flat_session* s, const psb_query_batch_view* queries, const psb_search_params* params,
                                   const psb_search_output_view* output, psb_stats* stats) {
    PSB_RANGE("ivfflat_search");
    PSB_TRY(flat_check(s, params));
    if (!queries || !output) return fail(PSB_INVALID_ARGUMENT, "null query or output view");
    if (queries->count < 0 || queries->dim != s->dim) return fail(PSB_INVALID_ARGUMENT, "query dim does not match the index");
    if (queries->count > 0 && (!queries->fp32 || !output->indices || !output->distances)) return fail(PSB_INVALID_ARGUMENT, "null query or output buffers");
    PSB_CUDA(cudaSetDevice(s->device));
    if (stats) std::memset(stats, 0, sizeof(*stats));
    const int total = queries->count, nprobe = params->nprobe, topk = params->topk;
    if (total == 0) return PSB_OK;
    const int batch = std::min(std::min(params->batch_size, s->opt.max_batch), total);
    cudaStream_t st = s->stream;
    PSB_TRY(reserve_together(&s->call_whole, {{&s->q, sizeof(float) * (size_t)batch * s->dim}, {&s->out_ids, sizeof(long long) * (size_t)batch * topk},
                                              {&s->out_dist, sizeof(float) * (size_t)batch * topk}}));
    const size_t b_q = (sizeof(float) * (size_t)total * s->dim + 255) / 256 * 256, b_ids = sizeof(long long) * (size_t)total * topk,
                 b_dist = sizeof(float) * (size_t)total * topk;
    const bool small = batch == total && b_q + b_ids + b_dist <= kSmallIo;   // through the pinned block, as psb_session_search
    PSB_TRY(ensure_host_io(s));
    HostCopies copies(st, {{small ? nullptr : queries->fp32, sizeof(float) * (size_t)total * s->dim}, {small ? nullptr : output->indices, b_ids},
                           {small ? nullptr : output->distances, b_dist}, {output->coarse_ids, sizeof(int) * (size_t)total * nprobe}});
    CallMarks marks(s, small && !coarse_by_tc(s, total, nprobe), reinterpret_cast<const float*>(s->h_io), total);
    const bool timed = stats && !marks.on;   // by events
    const long long launches0 = launches_total();
    unsigned long long c0[4] = {0, 0, 0, 0};
    if (stats) PSB_TRY(counters_before(s, st, c0));
    s->counters_known = false;
    s->timing.used = 0;
    EventTimer tm(&s->timing);
    if (timed) PSB_TRY(tm.mark(st));
    int nb = 0;
    const auto began = HostClock::now();
    for (int q0 = 0; q0 < total; q0 += batch, ++nb) {
        const int n = std::min(batch, total - q0);
        const void* from = queries->fp32 + (size_t)q0 * s->dim;
        if (small) { std::memcpy(s->h_io, from, sizeof(float) * (size_t)n * s->dim); from = s->h_io; }
        if (!s->host_queries) PSB_CUDA(cudaMemcpyAsync(s->q.p, from, sizeof(float) * (size_t)n * s->dim, cudaMemcpyHostToDevice, st));
        long long* ids = small ? reinterpret_cast<long long*>(s->h_io + b_q) : s->out_ids.as<long long>();
        float* dist = small ? reinterpret_cast<float*>(s->h_io + b_q + b_ids) : s->out_dist.as<float>();
        PSB_TRY(flat_search_device(s, s->q.as<float>(), n, nprobe, topk, ids, dist));
        if (!small) {
            PSB_CUDA(cudaMemcpyAsync(output->indices + (size_t)q0 * topk, ids, sizeof(long long) * (size_t)n * topk, cudaMemcpyDeviceToHost, st));
            PSB_CUDA(cudaMemcpyAsync(output->distances + (size_t)q0 * topk, dist, sizeof(float) * (size_t)n * topk, cudaMemcpyDeviceToHost, st));
        }
        if (output->coarse_ids)
            PSB_CUDA(cudaMemcpyAsync(output->coarse_ids + (size_t)q0 * nprobe, s->probes.p, sizeof(int) * (size_t)n * nprobe, cudaMemcpyDeviceToHost, st));
        if (q0 + batch >= total) {
            PSB_TRY(queue_tail(s, st));
            if (timed) PSB_TRY(tm.mark(st));
        }
        PSB_CUDA(cudaStreamSynchronize(st));  // the batch buffers are reused
        if (small) {
            std::memcpy(output->indices, ids, b_ids);
            std::memcpy(output->distances, dist, b_dist);
        }
    }
    copies.ended = true;
    const double call_ms = ms_since(began);
    PSB_TRY(check_tail(s));
    if (stats) {
        stats->total_ms = timed ? tm.ms(0, 1) : call_ms;
        stats->pq_scanned_codes = (long long)(s->h_tail->c[0] - c0[0]);  // rows scanned
        stats->h2d_bytes = (long long)sizeof(float) * total * s->dim;
        stats->d2h_bytes = (long long)(sizeof(long long) + sizeof(float)) * total * topk;
        stats->kernel_launches = launches_total() - launches0;
        stats->batches = nb;
    }
    return PSB_OK;
}

// ---- one-shot operators on host arrays ------------------------------------------------------------------

psb_status psb_rerank_host(const psb_host_storage_view* storage, const uint8_t* h_queries_u8,
                           const float* h_queries_fp32, const int* h_candidates, int batch_n,
                           int candidate_count, int candidate_stride, int topk, int* h_output_ids,
                           float* h_output_distances, const int* h_candidate_counts, int device) {
    if (!storage || !h_candidates || !h_output_ids || !h_output_distances || batch_n <= 0 || candidate_count <= 0 ||
        candidate_stride < candidate_count || topk <= 0 || storage->count <= 0 || storage->dim <= 0)
        return fail(PSB_INVALID_ARGUMENT, "invalid host IVF rerank request");
    const bool use_float = storage->fp32 != nullptr;
    if ((use_float && !h_queries_fp32) || (!use_float && (!storage->u8 || !h_queries_u8)))
        return fail(PSB_INVALID_ARGUMENT, "host IVF rerank dtype does not match storage");
    if (storage->source_rows) return fail(PSB_UNSUPPORTED_SHAPE, "exact storage with a row permutation is not supported");
    if (h_candidate_counts)
        for (int q = 0; q < batch_n; ++q)
            if (h_candidate_counts[q] < 0 || h_candidate_counts[q] > candidate_count)
                return fail(PSB_INVALID_ARGUMENT, "host rerank candidate count exceeds row width");
    if (candidate_count > kMaxRerankWidth || topk > kMaxTopk) return fail(PSB_UNSUPPORTED_SHAPE, "rerank width above 4096 or topk above 2048");
    PSB_TRY(check_device(device));
    const int elem = use_float ? 4 : 1;
    const int dim = storage->dim;
    const size_t base_bytes = (size_t)storage->count * dim * elem;
    DevBuf base, q, cand, counts, out_rows, out_dist;
    PSB_TRY(base.reserve(base_bytes)); PSB_TRY(q.reserve((size_t)batch_n * dim * elem));
    PSB_TRY(cand.reserve(sizeof(int) * (size_t)batch_n * candidate_stride));
    PSB_TRY(out_rows.reserve(sizeof(int) * (size_t)batch_n * topk)); PSB_TRY(out_dist.reserve(sizeof(float) * (size_t)batch_n * topk));
    cudaStream_t st = nullptr;
    HostCopies copies(st, {{use_float ? (const void*)storage->fp32 : (const void*)storage->u8, base_bytes},
                           {use_float ? (const void*)h_queries_fp32 : (const void*)h_queries_u8, (size_t)batch_n * dim * elem},
                           {h_candidates, sizeof(int) * (size_t)batch_n * candidate_stride}, {h_candidate_counts, sizeof(int) * (size_t)batch_n},
                           {h_output_ids, sizeof(int) * (size_t)batch_n * topk}, {h_output_distances, sizeof(float) * (size_t)batch_n * topk}});
    PSB_CUDA(cudaMemcpy(base.p, use_float ? (const void*)storage->fp32 : (const void*)storage->u8, base_bytes, cudaMemcpyHostToDevice));
    PSB_CUDA(cudaMemcpy(q.p, use_float ? (const void*)h_queries_fp32 : (const void*)h_queries_u8, (size_t)batch_n * dim * elem, cudaMemcpyHostToDevice));
    PSB_CUDA(cudaMemcpy(cand.p, h_candidates, sizeof(int) * (size_t)batch_n * candidate_stride, cudaMemcpyHostToDevice));
    const int* d_counts = nullptr;
    if (h_candidate_counts) {
        PSB_TRY(counts.reserve(sizeof(int) * (size_t)batch_n));
        PSB_CUDA(cudaMemcpy(counts.p, h_candidate_counts, sizeof(int) * (size_t)batch_n, cudaMemcpyHostToDevice));
        d_counts = counts.as<int>();
    }
    RowMap mp;
    mp.count = storage->count;
    DevBuf score;
    PSB_TRY(score.reserve(sizeof(float) * (size_t)batch_n * candidate_count));
    PSB_TRY(launch_rerank_score(base.p, nullptr, mp, dim, elem, q.p, cand.as<int>(), batch_n, candidate_count, candidate_stride,
                                d_counts, score.as<float>(), st));
    PSB_TRY(launch_topk_select(score.as<float>(), cand.as<int>(), batch_n, candidate_count, candidate_stride, d_counts,
                               topk, out_rows.as<int>(), out_dist.as<float>(), st));
    PSB_CUDA(cudaMemcpy(h_output_ids, out_rows.p, sizeof(int) * (size_t)batch_n * topk, cudaMemcpyDeviceToHost));
    PSB_CUDA(cudaMemcpy(h_output_distances, out_dist.p, sizeof(float) * (size_t)batch_n * topk, cudaMemcpyDeviceToHost));
    return PSB_OK;
}

psb_status psb_coarse_host(const float* h_queries, int nq, const float* h_centroids, int nlist, int dim,
                           int nprobe, int coarse_mode, int64_t* h_ids, float* h_dist, int device) {
    if (!h_queries || !h_centroids || !h_ids || nq < 0 || nlist <= 0 || dim <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid coarse request");
    if (nprobe <= 0 || nprobe > nlist) return fail(PSB_INVALID_ARGUMENT, "nprobe must be in 1..nlist");
    if (nprobe > kMaxProbe) return fail(PSB_UNSUPPORTED_SHAPE, "nprobe above 4096 is not supported");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    if (nq == 0) return PSB_OK;
    DevBuf q, c, tile, ids, ids64, dist;
    PSB_TRY(q.reserve(sizeof(float) * (size_t)nq * dim)); PSB_TRY(c.reserve(sizeof(float) * (size_t)nlist * dim));
    PSB_TRY(ids.reserve(sizeof(int) * (size_t)nq * nprobe)); PSB_TRY(ids64.reserve(sizeof(long long) * (size_t)nq * nprobe));
    PSB_TRY(dist.reserve(sizeof(float) * (size_t)nq * nprobe));
    HostCopies copies(nullptr, {{h_queries, sizeof(float) * (size_t)nq * dim}, {h_centroids, sizeof(float) * (size_t)nlist * dim},
                                {h_ids, sizeof(long long) * (size_t)nq * nprobe}, {h_dist, sizeof(float) * (size_t)nq * nprobe}});
    PSB_CUDA(cudaMemcpy(q.p, h_queries, sizeof(float) * (size_t)nq * dim, cudaMemcpyHostToDevice));
    PSB_CUDA(cudaMemcpy(c.p, h_centroids, sizeof(float) * (size_t)nlist * dim, cudaMemcpyHostToDevice));
    const bool tc_ok = coarse_tc_supported(nq, nlist, dim, nprobe);
    if (coarse_mode == 2 && !tc_ok) return fail(PSB_UNSUPPORTED_SHAPE, "tensor-core coarse stage does not support this shape");
    if (coarse_mode != 1 && tc_ok) {
        TcIndexBuffers<PoolBuf> tix;
        TcWorkBuffers<PoolBuf> twk;
        PSB_TRY(tix.prepare(c.as<float>(), nlist, dim, device, nullptr));
        PSB_TRY(twk.ensure(nq, nlist, dim, nprobe, device, nullptr));
        PSB_TRY(launch_coarse_tc(tix.view(c.as<float>(), nlist, dim), twk.view(), q.as<float>(), nq, nprobe, ids.as<int>(),
                                 dist.as<float>(), sms, nullptr));
        PSB_CUDA(cudaDeviceSynchronize());
        PSB_TRY(twk.check_status());
    } else {
        const size_t row_bytes = sizeof(float) * (size_t)nlist;
        int chunk = (int)std::max<size_t>(64, ((size_t)1 << 30) / row_bytes);
        chunk = std::min(chunk, nq);
        PSB_TRY(tile.reserve(row_bytes * (size_t)chunk));
        for (int q0 = 0; q0 < nq; q0 += chunk) {
            const int n = std::min(chunk, nq - q0);
            PSB_TRY(launch_coarse_dist_exact(q.as<float>() + (size_t)q0 * dim, n, c.as<float>(), nlist, dim, tile.as<float>(), sms, nullptr));
            PSB_TRY(launch_select_rows(tile.as<float>(), n, nlist, nprobe, ids.as<int>() + (size_t)q0 * nprobe,
                                       dist.as<float>() + (size_t)q0 * nprobe, nullptr));
        }
    }
    PSB_TRY(launch_widen_ids(ids.as<int>(), (long long)nq * nprobe, ids64.as<long long>(), nullptr));
    PSB_CUDA(cudaMemcpy(h_ids, ids64.p, sizeof(long long) * (size_t)nq * nprobe, cudaMemcpyDeviceToHost));
    if (h_dist) PSB_CUDA(cudaMemcpy(h_dist, dist.p, sizeof(float) * (size_t)nq * nprobe, cudaMemcpyDeviceToHost));
    return PSB_OK;
}

psb_status psb_knn_exact(const float* d_queries, int nq, const float* d_base, int64_t n, int dim, int k,
                         int* d_rows, float* d_dist, int device, void* stream) {
    if (!d_queries || !d_base || !d_rows || !d_dist || nq <= 0 || n <= 0 || dim <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid knn request");
    if (k <= 0 || k > n) return fail(PSB_INVALID_ARGUMENT, "k must be in 1..n");
    if (k > kMaxProbe) return fail(PSB_UNSUPPORTED_SHAPE, "k above 4096 is not supported");
    if (n > INT_MAX) return fail(PSB_UNSUPPORTED_SHAPE, "more than 2^31-1 base rows");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // tiles of base rows, each at most 1 GiB of distances, then a merge of the per-tile winners.  A last tile with fewer
    // than k rows is folded into the tile before it, so every tile selects exactly k rows.
    long long tile = std::max<long long>(std::max<long long>(4096, k), ((long long)1 << 28) / nq);
    tile = std::min<long long>(tile, n);
    std::vector<std::pair<long long, int>> spans;  // (first row, rows)
    for (long long r0 = 0; r0 < n;) {
        long long rows = std::min<long long>(tile, n - r0);
        const long long rest = n - (r0 + rows);
        if (rest > 0 && rest < k) rows += rest;
        spans.emplace_back(r0, (int)rows);
        r0 += rows;
    }
    const int tiles = (int)spans.size();
    if ((long long)tiles * k > 16384) return fail(PSB_UNSUPPORTED_SHAPE, "knn: too many tiles for the merge; pass fewer base rows per call");
    DevBuf dist, trows, tdist;
    PSB_TRY(dist.reserve(sizeof(float) * (size_t)nq * (size_t)(tile + k)));
    PSB_TRY(trows.reserve(sizeof(int) * (size_t)tiles * nq * k));
    PSB_TRY(tdist.reserve(sizeof(float) * (size_t)tiles * nq * k));
    for (int t = 0; t < tiles; ++t) {
        const long long r0 = spans[(size_t)t].first;
        const int rows = spans[(size_t)t].second;  // >= k: k <= n, and no span is shorter than k unless it is the only one
        PSB_TRY(launch_coarse_dist_exact(d_queries, nq, d_base + (size_t)r0 * dim, rows, dim, dist.as<float>(), sms, st));
        PSB_TRY(launch_select_rows(dist.as<float>(), nq, rows, k, trows.as<int>() + (size_t)t * nq * k,
                                   tdist.as<float>() + (size_t)t * nq * k, st));
        PSB_TRY(launch_offset_rows(trows.as<int>() + (size_t)t * nq * k, (long long)nq * k, (int)r0, st));
    }
    PSB_TRY(launch_merge(trows.as<int>(), tdist.as<float>(), tiles, nq, k, d_rows, d_dist, st));
    PSB_CUDA(cudaStreamSynchronize(st));
    return PSB_OK;
}

// ---- training ---------------------------------------------------------------------------------------------

namespace {
// Nearest-centroid assignment of n device rows: the coarse stage with nprobe 1.  Large problems take the tensor-core filter with
// exact refinement (identical assignments and distances: ties go to the lower centroid id on both paths), others the exact kernels.
// One object serves all iterations of a training: the rows' bf16 operand is made once (centred on the first iteration's mean
// centroid - any point will do) and kept when it takes at most kKeepRows bytes, and nothing is copied to the host in between.
class Assigner {
public:
    // form: 0 = the rule below, 1 = without the filter, 2 = with it (filter_takes)
    Assigner(const float* d_data, int64_t n, int dim, int k, int device, int sms, cudaStream_t st, int form = 0)
        : data_(d_data), n_(n), dim_(dim), k_(k), device_(device), sms_(sms), st_(st) {
        // The filter costs about 2 ns a row whatever the number of centroids, and its launches more than the row kernel's; that takes 1.2e-4 ns for
        // each dimension of a pair and as much as 20 of them besides.  Trainings of three iterations, rows / filter, us: 20,000 x 64, 256 centroids 548 / 631, 400 654 / 572; 20,000 x
        // 128, 128 613 / 756, 200 749 / 673; 100,000 x 96, 128 1,218 / 1,239, 1,000 5,020 / 1,200; 400,000 x 100, 128 4,031 / 3,216, 1,000 19,369 / 3,233; 100,000 x 3, 600
        // 784 / 827, 3,000 2,516 / 1,270; 10,000 x 16, 3,000 552 / 512.  Of 200 trainings (700 to 300,000 rows of 3 to 128 dimensions) the form taken is on average 0.5 % slower than the other.
        tc_ = form == 2 || (form == 0 && filter_takes(n, dim, k) && (!nearest_rows_fit(dim) || (double)k * (dim + 20) >= 8000.0 + 3.0e8 / (double)n));
    }
    static bool filter_takes(int64_t n, int dim, int k) { return n >= 64 && k >= 128 && coarse_tc_padded_dim(dim) <= 128; }
    // d_assign [n], d_best [n] out; bounded: d_assign holds an assignment on entry, whose distances bound the nearest ones (one
    // filter pass instead of two).
    psb_status run(const float* d_centroids, int* d_assign, float* d_best, bool bounded) {
        if (!tc_) return exact(d_centroids, d_assign, d_best);
        PSB_TRY(index_.prepare(d_centroids, k_, dim_, device_, st_, index_.ready));
        const CoarseTcIndex ix = index_.view(d_centroids, k_, dim_);
        const int dimp = coarse_tc_padded_dim(dim_);
        const bool keep = (size_t)n_ * dimp * 2 <= kKeepRows;
        if (keep && !rows_.p) {
            PSB_TRY(rows_.reserve((size_t)n_ * dimp * 2, device_, st_));
            PSB_TRY(norms_.reserve((size_t)n_ * 8, device_, st_));
            PSB_TRY(launch_tc_prep_queries(ix, data_, n_, rows_.p, norms_.p, st_));
        }
        // Rows per launch: the group minima of a first pass (k / 32 floats a row) or the candidate lists (32 ids a row) bound it;
        // equal parts, so that no part falls below the filter's smallest batch.
        const int64_t most = bounded ? 2097152 : 262144;
        const int64_t parts = (n_ + most - 1) / most;
        const int64_t chunk = ((n_ + parts - 1) / parts + 127) / 128 * 128;
        for (int64_t r0 = 0; r0 < n_; r0 += chunk) {
            const int nn = (int)std::min<int64_t>(chunk, n_ - r0);
            PSB_TRY(work_.ensure((int)std::min<int64_t>(chunk, n_), k_, dim_, 1, device_, st_, !keep, bounded));
            CoarseTcWorkspace w = work_.view();
            if (keep) {
                w.qb = rows_.as<unsigned char>() + (size_t)r0 * dimp * 2;
                w.qnorm = norms_.as<unsigned char>() + (size_t)r0 * 8;
                w.queries_ready = true;
            }
            const float* rows = data_ + (size_t)r0 * dim_;
            if (bounded) PSB_TRY(launch_coarse_tc_assign(ix, w, rows, nn, d_assign + r0, d_assign + r0, d_best + r0, sms_, st_));
            else PSB_TRY(launch_coarse_tc(ix, w, rows, nn, 1, d_assign + r0, d_best + r0, sms_, st_));
        }
        if (!bounded) work_.gmin.release();
        return PSB_OK;
    }
    psb_status check_status() const { return tc_ ? work_.check_status() : PSB_OK; }
private:
    static constexpr size_t kKeepRows = (size_t)4 << 30;
    psb_status exact(const float* d_centroids, int* d_assign, float* d_best) {
        if (nearest_rows_pays((int)std::min<int64_t>(n_, INT_MAX), k_, dim_)) {
            for (int64_t r0 = 0; r0 < n_; r0 += 1 << 30) {
                const int nn = (int)std::min<int64_t>(1 << 30, n_ - r0), range = nearest_rows_range(nn, k_, dim_, sms_);
                if (range < k_) PSB_TRY(keys_.reserve(sizeof(unsigned long long) * (size_t)nn, device_, st_));
                PSB_TRY(launch_nearest_rows(data_ + (size_t)r0 * dim_, nn, d_centroids, k_, dim_, range, keys_.as<unsigned long long>(), d_assign + r0, d_best + r0, st_));
            }
            return PSB_OK;
        }
        const size_t row_bytes = sizeof(float) * (size_t)k_;
        const int64_t chunk = std::min<int64_t>((int64_t)std::max<size_t>(64, ((size_t)1 << 30) / row_bytes), n_);
        PSB_TRY(tile_.reserve(row_bytes * (size_t)chunk, device_, st_));
        for (int64_t r0 = 0; r0 < n_; r0 += chunk) {
            const int nn = (int)std::min<int64_t>(chunk, n_ - r0);
            PSB_TRY(launch_coarse_dist_exact(data_ + (size_t)r0 * dim_, nn, d_centroids, k_, dim_, tile_.as<float>(), sms_, st_));
            PSB_TRY(launch_select_rows(tile_.as<float>(), nn, k_, 1, d_assign + r0, d_best + r0, st_));
        }
        return PSB_OK;
    }
    const float* data_;
    int64_t n_;
    int dim_, k_, device_, sms_;
    cudaStream_t st_;
    bool tc_;
    TcIndexBuffers<PoolBuf> index_;
    TcWorkBuffers<PoolBuf> work_;
    PoolBuf rows_, norms_, tile_, keys_;
};
}  // namespace

psb_status psb_kmeans_train(const float* d_data, int64_t n, int dim, float* d_centroids, int k, int iters,
                            int* d_assign, double* h_objective, int device, void* stream) {
    if (!d_data || !d_centroids || n <= 0 || dim <= 0 || k <= 0 || iters < 0) return fail(PSB_INVALID_ARGUMENT, "invalid k-means request");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    PoolBuf assign, best, sums, counts, obj, acc_order, acc_offsets, acc_cursor;   // the last three: rows grouped by centroid
    PSB_TRY(best.reserve(sizeof(float) * (size_t)n, device, st));
    int* d_as = d_assign;
    if (!d_as) { PSB_TRY(assign.reserve(sizeof(int) * (size_t)n, device, st)); d_as = assign.as<int>(); }
    PSB_TRY(sums.reserve(sizeof(double) * (size_t)k * dim, device, st)); PSB_TRY(counts.reserve(sizeof(int) * (size_t)k, device, st));
    PSB_TRY(obj.reserve(sizeof(double) * ((size_t)iters + 1), device, st));
    PSB_TRY(acc_order.reserve(sizeof(int) * (size_t)n, device, st));
    PSB_TRY(acc_offsets.reserve(sizeof(int) * ((size_t)k + 1), device, st));
    PSB_TRY(acc_cursor.reserve(sizeof(int) * (size_t)k, device, st));
    KmeansAccumWs acc_ws;
    acc_ws.order = acc_order.as<int>(); acc_ws.offsets = acc_offsets.as<int>(); acc_ws.cursor = acc_cursor.as<int>();
    PSB_CUDA(cudaMemsetAsync(obj.p, 0, sizeof(double) * ((size_t)iters + 1), st));
    Assigner assigner(d_data, n, dim, k, device, sms, st);
    for (int it = 0; it <= iters; ++it) {
        // After the first iteration every row brings a bound along - its distance to the centroid it had, where that centroid
        // is now - and the filter GEMM runs once instead of twice.
        PSB_TRY(assigner.run(d_centroids, d_as, best.as<float>(), it > 0));
        PSB_CUDA(cudaMemsetAsync(counts.p, 0, sizeof(int) * (size_t)k, st));
        PSB_TRY(launch_kmeans_accumulate(d_data, n, dim, d_as, best.as<float>(), k, sums.as<double>(), counts.as<int>(),
                                         obj.as<double>() + it, acc_ws, st));
        if (it < iters) PSB_TRY(launch_kmeans_update(sums.as<double>(), counts.as<int>(), k, dim, d_centroids, st));
    }
    HostCopies copies(st, {{h_objective, sizeof(double) * ((size_t)iters + 1)}});
    if (h_objective) PSB_CUDA(cudaMemcpyAsync(h_objective, obj.p, sizeof(double) * ((size_t)iters + 1), cudaMemcpyDeviceToHost, st));
    PSB_CUDA(cudaStreamSynchronize(st));
    return assigner.check_status();
}

// ---- one Lloyd iteration in three calls (data-parallel training: the caller all-reduces sums and counts in between) ----

psb_status psb_kmeans_assign(const float* d_data, int64_t n, int dim, const float* d_centroids, int k, int* d_assign,
                             float* d_best, int device, void* stream) {
    return psb_kmeans_assign_bounded(d_data, n, dim, d_centroids, k, d_assign, d_best, 0, device, stream);
}

psb_status psb_kmeans_assign_bounded(const float* d_data, int64_t n, int dim, const float* d_centroids, int k, int* d_assign,
                                     float* d_best, int have_previous, int device, void* stream) {
    return psb_kmeans_assign_form(d_data, n, dim, d_centroids, k, d_assign, d_best, have_previous, 0, device, stream);
}

psb_status psb_kmeans_assign_form(const float* d_data, int64_t n, int dim, const float* d_centroids, int k, int* d_assign,
                                  float* d_best, int have_previous, int form, int device, void* stream) {
    if (!d_data || !d_centroids || !d_assign || !d_best || n <= 0 || dim <= 0 || k <= 0 || form < 0 || form > 2)
        return fail(PSB_INVALID_ARGUMENT, "invalid k-means assignment request");
    if (form == 2 && !Assigner::filter_takes(n, dim, k)) return fail(PSB_UNSUPPORTED_SHAPE, "the tensor-core filter does not take this shape");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Assigner assigner(d_data, n, dim, k, device, sms, st, form);
    PSB_TRY(assigner.run(d_centroids, d_assign, d_best, have_previous != 0));
    PSB_CUDA(cudaStreamSynchronize(st));
    return assigner.check_status();
}

psb_status psb_kmeans_accumulate(const float* d_data, int64_t n, int dim, const int* d_assign, const float* d_best, int k,
                                 double* d_sums, int* d_counts, double* d_objective, int device, void* stream) {
    if (!d_data || !d_assign || !d_best || !d_sums || !d_counts || !d_objective || n < 0 || dim <= 0 || k <= 0)
        return fail(PSB_INVALID_ARGUMENT, "invalid k-means accumulation request");
    PSB_TRY(check_device(device));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    PSB_CUDA(cudaMemsetAsync(d_counts, 0, sizeof(int) * (size_t)k, st));
    PSB_CUDA(cudaMemsetAsync(d_objective, 0, sizeof(double), st));
    PoolBuf order, offsets, cursor;   // rows grouped by centroid
    PSB_TRY(order.reserve(sizeof(int) * (size_t)std::max<int64_t>(n, 1), device, st));
    PSB_TRY(offsets.reserve(sizeof(int) * ((size_t)k + 1), device, st));
    PSB_TRY(cursor.reserve(sizeof(int) * (size_t)k, device, st));
    KmeansAccumWs ws;
    ws.order = order.as<int>(); ws.offsets = offsets.as<int>(); ws.cursor = cursor.as<int>();
    PSB_TRY(launch_kmeans_accumulate(d_data, n, dim, d_assign, d_best, k, d_sums, d_counts, d_objective, ws, st));
    PSB_CUDA(cudaStreamSynchronize(st));
    return PSB_OK;
}

psb_status psb_kmeans_update(const double* d_sums, const int* d_counts, int k, int dim, float* d_centroids, int device,
                             void* stream) {
    if (!d_sums || !d_counts || !d_centroids || k <= 0 || dim <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid k-means update request");
    PSB_TRY(check_device(device));
    return launch_kmeans_update(d_sums, d_counts, k, dim, d_centroids, static_cast<cudaStream_t>(stream));
}

psb_status psb_residual_rows(const float* d_data, int64_t n, int dim, const float* d_centroids, const int* d_assign,
                             float* d_out, int device, void* stream) {
    if (!d_data || !d_centroids || !d_assign || !d_out || n < 0 || dim <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid residual request");
    if ((long long)n * dim > 0x7fffffffLL * 256) return fail(PSB_UNSUPPORTED_SHAPE, "too many elements for one call");
    PSB_TRY(check_device(device));
    return launch_residual_rows(d_data, n, dim, d_centroids, d_assign, d_out, static_cast<cudaStream_t>(stream));
}

}  // extern "C"

namespace {

// The reference's choice of initial centroids (init_centroids_by_sampling, src/clustering/kmeans/kmeans.cu:716-862), as the
// data rows it picks: std::mt19937(seed); below n * k = 2e7 (policy 0) k-means++ seeding - first row uniform, every further
// row with probability proportional to its squared distance from the nearest row picked so far (fp32 sequential sums,
// fp64 running total) - above it k distinct rows by a partial Fisher-Yates shuffle.  The standard library's engine and
// distributions make the draws the same as the reference's, draw for draw.  row(i) must return row i's `dim` values.
template <typename RowFn>
void kmeans_init_rows(long long n, int dim, int k, int seed, int policy, RowFn row, std::vector<long long>& picked) {
    picked.assign((size_t)k, 0);
    if (n <= 0 || k <= 0) return;
    const int ni = (int)n;
    const int k_eff = std::min<long long>(k, n);
    std::mt19937 rng((unsigned)seed);
    const bool plusplus = policy == 2 || (policy == 0 && (long long)ni * k_eff <= 20000000LL);
    if (!plusplus) {
        // the identity permutation is kept implicit: only the places the shuffle has touched are stored
        std::unordered_map<int, int> moved;
        auto at = [&](int i) { const auto it = moved.find(i); return it == moved.end() ? i : it->second; };
        for (int i = 0; i < k_eff; ++i) {
            std::uniform_int_distribution<int> dist(i, ni - 1);
            const int j = dist(rng), x = at(i), y = at(j);
            moved[j] = x;
            moved[i] = y;
        }
        for (int c = 0; c < k; ++c) picked[(size_t)c] = at(c < k_eff ? c : 0);
        return;
    }
    auto dist2 = [&](const float* x, const float* c) {
        float acc = 0.0f;
        for (int d = 0; d < dim; ++d) { const float diff = x[d] - c[d]; acc = acc + diff * diff; }
        return acc;
    };
    std::uniform_int_distribution<int> uni(0, ni - 1);
    picked[0] = uni(rng);
    std::vector<float> best((size_t)ni);
    for (int i = 0; i < ni; ++i) best[(size_t)i] = dist2(row(i), row(picked[0]));
    for (int c = 1; c < k_eff; ++c) {
        double total = 0.0;
        for (int i = 0; i < ni; ++i) total += (double)best[(size_t)i];
        int next = -1;
        if (total <= 0.0) {
            next = uni(rng);
        } else {
            std::uniform_real_distribution<double> urd(0.0, total);
            const double r = urd(rng);
            double cum = 0.0;
            for (int i = 0; i < ni; ++i) {
                cum += (double)best[(size_t)i];
                if (cum >= r) { next = i; break; }
            }
            if (next < 0) next = ni - 1;
        }
        picked[(size_t)c] = next;
        const float* cc = row(next);
        for (int i = 0; i < ni; ++i) {
            const float d2 = dist2(row(i), cc);
            if (d2 < best[(size_t)i]) best[(size_t)i] = d2;
        }
    }
    for (int c = k_eff; c < k; ++c) picked[(size_t)c] = picked[0];
}

}  // namespace

extern "C" {

psb_status psb_kmeans_init(const float* h_data, int64_t n, int dim, int k, int seed, int policy, float* h_centroids, int64_t* h_rows) {
    if (!h_data || !h_centroids || n <= 0 || n > INT_MAX || dim <= 0 || k <= 0 || policy < 0 || policy > 2)
        return fail(PSB_INVALID_ARGUMENT, "invalid k-means initialisation request");
    std::vector<long long> picked;
    kmeans_init_rows(n, dim, k, seed, policy, [&](long long i) { return h_data + (size_t)i * dim; }, picked);
    for (int c = 0; c < k; ++c) {
        std::memcpy(h_centroids + (size_t)c * dim, h_data + (size_t)picked[(size_t)c] * dim, sizeof(float) * (size_t)dim);
        if (h_rows) h_rows[c] = picked[(size_t)c];
    }
    return PSB_OK;
}

psb_status psb_pq_train(const float* d_data, int64_t n, int dim, int subvectors, int codebook_size, int iters,
                        uint64_t seed, float* d_codebook, int device, void* stream) {
    if (!d_data || !d_codebook || n <= 0 || dim <= 0 || subvectors <= 0 || dim % subvectors || codebook_size <= 0 ||
        codebook_size > kMaxCodebook || iters < 0)
        return fail(PSB_INVALID_ARGUMENT, "invalid PQ training request");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    if (n > INT_MAX) return fail(PSB_UNSUPPORTED_SHAPE, "PQ training on more than 2^31-1 rows");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int dsub = dim / subvectors, words = subvectors * codebook_size;
    // One block: codes, sums, counts (with the seeding's status words behind them), rows, draws, first rows.
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t b_codes = up((size_t)n * subvectors), b_sums = up(sizeof(double) * (size_t)words * dsub),
                 b_counts = up(sizeof(int) * ((size_t)words + subvectors)), b_rows = up(sizeof(long long) * (size_t)words),
                 b_draws = up(sizeof(double) * (size_t)words), b_first = up(sizeof(int) * (size_t)subvectors);
    PoolBuf block;
    PSB_TRY(block.reserve(b_codes + b_sums + b_counts + b_rows + b_draws + b_first, device, st));
    uint8_t* codes = block.as<uint8_t>();
    double* sums = reinterpret_cast<double*>(codes + b_codes);
    int* counts = reinterpret_cast<int*>(codes + b_codes + b_sums);
    int* status = counts + words;
    long long* d_rows = reinterpret_cast<long long*>(codes + b_codes + b_sums + b_counts);
    double* d_draws = reinterpret_cast<double*>(codes + b_codes + b_sums + b_counts + b_rows);
    int* d_first = reinterpret_cast<int*>(codes + b_codes + b_sums + b_counts + b_rows + b_draws);
    PSB_CUDA(cudaMemsetAsync(sums, 0, b_sums + b_counts, st));
    // Initial codewords as the reference's GPU trainer picks them (src/quantization/pq/pq_trainer.cu:30-95): subspace `sub`
    // runs the k-means initialisation with seed + sub * 104729 on its own sub-vectors.  The random-rows policy needs no data;
    // the k-means++ policy (small training sets only: n * K <= 2e7) runs on the device with the draws made here.
    const bool plusplus = (long long)n * std::min<long long>(codebook_size, n) <= 20000000LL;
    const bool on_device = plusplus && pq_seed_fits(n);
    auto sub_seed = [&](int sub) { return (int)((unsigned)seed + (unsigned)sub * 104729u); };
    std::vector<long long> rows((size_t)words), picked;
    std::vector<double> draws;
    std::vector<int> first, to_host((size_t)subvectors, plusplus ? 1 : 0);
    if (on_device) {
        draws.assign((size_t)words, 0.0);
        first.resize((size_t)subvectors);
        const int keff = (int)std::min<long long>(codebook_size, n);
        for (int sub = 0; sub < subvectors; ++sub) {
            std::mt19937 rng((unsigned)sub_seed(sub));
            first[(size_t)sub] = std::uniform_int_distribution<int>(0, (int)n - 1)(rng);
            for (int c = 1; c < keff; ++c)
                draws[(size_t)sub * (codebook_size - 1) + (c - 1)] = std::generate_canonical<double, std::numeric_limits<double>::digits>(rng);
        }
        PSB_CUDA(cudaMemcpyAsync(d_draws, draws.data(), sizeof(double) * draws.size(), cudaMemcpyHostToDevice, st));
        PSB_CUDA(cudaMemcpyAsync(d_first, first.data(), sizeof(int) * first.size(), cudaMemcpyHostToDevice, st));
        PSB_TRY(launch_pq_seed(d_data, (int)n, dim, subvectors, codebook_size, d_draws, d_first, d_rows, status, st));
        PSB_CUDA(cudaMemcpyAsync(to_host.data(), status, sizeof(int) * to_host.size(), cudaMemcpyDeviceToHost, st));
        PSB_CUDA(cudaStreamSynchronize(st));
    }
    {
        std::vector<float> sub_host;
        for (int sub = 0; sub < subvectors; ++sub) {
            if (on_device && !to_host[(size_t)sub]) continue;
            if (plusplus) {
                sub_host.resize((size_t)n * dsub);
                PSB_CUDA(cudaMemcpy2DAsync(sub_host.data(), sizeof(float) * (size_t)dsub, d_data + (size_t)sub * dsub, sizeof(float) * (size_t)dim,
                                           sizeof(float) * (size_t)dsub, (size_t)n, cudaMemcpyDeviceToHost, st));
                PSB_CUDA(cudaStreamSynchronize(st));
            }
            kmeans_init_rows(n, dsub, codebook_size, sub_seed(sub), 0, [&](long long i) { return sub_host.data() + (size_t)i * dsub; }, picked);
            std::copy(picked.begin(), picked.end(), rows.begin() + (size_t)sub * codebook_size);
            PSB_CUDA(cudaMemcpyAsync(d_rows + (size_t)sub * codebook_size, rows.data() + (size_t)sub * codebook_size, sizeof(long long) * (size_t)codebook_size,
                                     cudaMemcpyHostToDevice, st));
        }
    }
    PSB_TRY(launch_pq_init_rows(d_data, dim, subvectors, codebook_size, d_rows, d_codebook, st));
    for (int it = 0; it < iters; ++it) {
        PSB_TRY(launch_pq_assign_train(d_data, n, dim, d_codebook, subvectors, codebook_size, codes, sms, st));
        PSB_TRY(launch_pq_accumulate(d_data, n, dim, codes, subvectors, codebook_size, sums, counts, st));
        PSB_TRY(launch_pq_update(sums, counts, subvectors, codebook_size, dsub, d_codebook, st));
    }
    PSB_CUDA(cudaStreamSynchronize(st));
    return PSB_OK;
}

psb_status psb_pq_encode(const float* d_data, int64_t n, int dim, const float* d_codebook, int subvectors,
                         int codebook_size, uint8_t* d_codes, int device, void* stream) {
    if (!d_data || !d_codebook || !d_codes || n < 0 || dim <= 0 || subvectors <= 0 || dim % subvectors ||
        codebook_size <= 0 || codebook_size > kMaxCodebook)
        return fail(PSB_INVALID_ARGUMENT, "invalid PQ encode request");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    return launch_pq_encode(d_data, n, dim, d_codebook, subvectors, codebook_size, d_codes, sms, static_cast<cudaStream_t>(stream));
}

psb_status psb_pq_encode_limited(const float* d_data, int64_t n, int dim, const float* d_codebook, int subvectors, int codebook_size,
                                 uint8_t* d_codes, int64_t items, int* d_gave_up, int device, void* stream) {
    if (!d_data || !d_codebook || !d_codes || n < 0 || dim <= 0 || subvectors <= 0 || dim % subvectors ||
        codebook_size <= 0 || codebook_size > kMaxCodebook)
        return fail(PSB_INVALID_ARGUMENT, "invalid PQ encode request");
    if (!pq_nearest_supported(dim / subvectors, codebook_size, false)) return fail(PSB_UNSUPPORTED_SHAPE, "no filter takes codewords of this shape");
    int sms = 0;
    PSB_TRY(check_device(device, &sms));
    NearTest test;
    test.items = items; test.gave_up = d_gave_up;
    return launch_pq_nearest(d_data, n, dim, d_codebook, subvectors, codebook_size, false, d_codes, sms, static_cast<cudaStream_t>(stream), test);
}

// ---- index-build glue (host) ---------------------------------------------------------------------------------

psb_status psb_ivf_layout_from_assignment(const int* h_assign, int64_t n, int nlist, int64_t* h_offsets, int64_t* h_reordered_ids) {
    if (!h_assign || !h_offsets || !h_reordered_ids || n < 0 || nlist <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid layout request");
    std::fill(h_offsets, h_offsets + nlist + 1, (int64_t)0);
    for (int64_t i = 0; i < n; ++i) {
        const int l = h_assign[i];
        if (l < 0 || l >= nlist) return fail(PSB_INVALID_ARGUMENT, "list assignment outside 0..nlist-1 at row " + std::to_string(i));
        ++h_offsets[l + 1];
    }
    for (int l = 0; l < nlist; ++l) h_offsets[l + 1] += h_offsets[l];
    std::vector<int64_t> cursor(h_offsets, h_offsets + nlist);
    for (int64_t i = 0; i < n; ++i) h_reordered_ids[cursor[(size_t)h_assign[i]]++] = i;  // stable: ascending id within a list
    return PSB_OK;
}

psb_status psb_reorder_rows(const void* h_src, int64_t n, size_t row_bytes, const int64_t* h_reordered_ids, void* h_dst) {
    if (!h_src || !h_dst || !h_reordered_ids || n < 0 || row_bytes == 0) return fail(PSB_INVALID_ARGUMENT, "invalid reorder request");
    std::vector<bool> seen((size_t)n, false);
    for (int64_t local = 0; local < n; ++local) {
        const int64_t id = h_reordered_ids[local];
        if (id < 0 || id >= n || seen[(size_t)id]) return fail(PSB_INVALID_ARGUMENT, "invalid IVF reordered IDs");
        seen[(size_t)id] = true;
    }
    const unsigned char* src = static_cast<const unsigned char*>(h_src);
    unsigned char* dst = static_cast<unsigned char*>(h_dst);
    const int threads = (int)std::min<unsigned>(std::max(1u, std::thread::hardware_concurrency()), 32u);
    std::vector<std::thread> pool;
    for (int t = 0; t < threads; ++t)
        pool.emplace_back([=]() {
            for (int64_t local = n * t / threads; local < n * (t + 1) / threads; ++local)
                std::memcpy(dst + (size_t)local * row_bytes, src + (size_t)h_reordered_ids[local] * row_bytes, row_bytes);
        });
    for (auto& th : pool) th.join();
    return PSB_OK;
}

// ---- per-row correction of residual-PQ indices (host) ---------------------------------------------------------------

psb_status psb_row_correction_compute(const float* h_centroids, const int64_t* h_offsets, int nlist, int dim, const uint8_t* h_codes,
                                      const float* h_codebook, int m, int k, float* h_values) {
    if (!h_centroids || !h_offsets || !h_codes || !h_codebook || !h_values || nlist <= 0 || dim <= 0 || m <= 0 || k <= 0 || dim % m)
        return fail(PSB_INVALID_ARGUMENT, "row-correction builder input is incomplete");
    for (int l = 0; l < nlist; ++l)
        if (h_offsets[l] < 0 || h_offsets[l + 1] < h_offsets[l]) return fail(PSB_INVALID_ARGUMENT, "row-correction cluster offsets are invalid");
    const int dsub = dim / m;
    const int threads = (int)std::min<unsigned>(std::max(1u, std::thread::hardware_concurrency()), 64u);
    std::vector<std::thread> pool;
    for (int t = 0; t < threads; ++t)
        pool.emplace_back([=]() {
            for (int l = t; l < nlist; l += threads) {
                const float* cen = h_centroids + (size_t)l * dim;
                for (int64_t row = h_offsets[l]; row < h_offsets[l + 1]; ++row) {
                    const uint8_t* code = h_codes + (size_t)row * m;
                    double corr = 0.0;
                    for (int sub = 0; sub < m; ++sub) {
                        const float* cw = h_codebook + ((size_t)sub * k + code[sub]) * dsub;
                        const float* cs = cen + sub * dsub;
                        for (int d = 0; d < dsub; ++d) corr += (double)cw[d] * cw[d] + 2.0 * (double)cs[d] * cw[d];
                    }
                    h_values[row] = (float)corr;
                }
            }
        });
    for (auto& th : pool) th.join();
    return PSB_OK;
}

psb_status psb_row_correction_quantize_u16(const float* h_values, int64_t n, psb_row_correction_u16_header* header, uint16_t* h_u16) {
    if (!h_values || !header || !h_u16 || n <= 0) return fail(PSB_INVALID_ARGUMENT, "invalid row-correction quantisation request");
    float lo = h_values[0], hi = h_values[0];
    for (int64_t i = 0; i < n; ++i) {
        if (!std::isfinite(h_values[i])) return fail(PSB_INVALID_ARGUMENT, "row-correction values contain non-finite data");
        lo = std::min(lo, h_values[i]); hi = std::max(hi, h_values[i]);
    }
    const float offset = std::floor(lo);
    const float range = hi - offset;
    const float scale = range > 0.0f ? std::nextafter(range / 65534.0f, std::numeric_limits<float>::infinity()) : 1.0f;
    if (!(scale > 0.0f) || !std::isfinite(scale)) return fail(PSB_INVALID_ARGUMENT, "row-correction range cannot be quantized");
    for (int64_t i = 0; i < n; ++i) {
        const double qv = std::ceil(((double)h_values[i] - offset) / scale);
        if (qv < 0.0 || qv > 65534.0) return fail(PSB_INTERNAL, "row-correction quantization overflow");
        h_u16[i] = (uint16_t)qv;
    }
    std::memset(header, 0, sizeof(*header));
    static const char magic[8] = {0x49, 0x53, 0x52, 0x43, 0x31, 0x36, 0x00, 0x00};
    std::memcpy(header->magic, magic, 8);
    header->version = 2; header->header_bytes = 32; header->count = (uint64_t)n; header->scale = scale; header->offset = offset;
    return PSB_OK;
}

psb_status psb_row_correction_model_u16(const float* h_centroids, int nlist, const float* h_codebook, int m, int k, int dsub,
                                        float* scale, float* offset) {
    if (!h_centroids || !h_codebook || !scale || !offset || nlist <= 0 || m <= 0 || k <= 0 || k > 256 || dsub <= 0)
        return fail(PSB_INVALID_ARGUMENT, "row correction: invalid PQ model");
    const int64_t dim = (int64_t)m * dsub;
    // slack for an fp32 producer's 2 dim + 8 roundings, relative to the magnitude, plus an absolute term for underflow
    const long double ops = 2.L * dim + 8;
    const long double err = ops * std::numeric_limits<float>::epsilon();
    if (err >= 0.25L) return fail(PSB_INVALID_ARGUMENT, "row correction: PQ dimension exceeds the error-bound contract");
    const long double gamma = err / (1 - err);
    const long double inf_ld = std::numeric_limits<long double>::infinity();
    long double lower = inf_ld, upper = -inf_ld;
    for (int c = 0; c < nlist; ++c) {
        long double lo = 0, hi = 0, mag = 0;
        for (int sub = 0; sub < m; ++sub) {
            long double s_lo = inf_ld, s_hi = -inf_ld, s_abs = 0;
            for (int code = 0; code < k; ++code) {
                long double score = 0, absolute = 0;
                for (int j = 0; j < dsub; ++j) {
                    const long double w = h_codebook[((size_t)sub * k + code) * dsub + j];
                    const long double cv = h_centroids[(size_t)c * dim + sub * dsub + j];
                    if (!std::isfinite(w) || !std::isfinite(cv)) return fail(PSB_INVALID_ARGUMENT, "row correction: non-finite PQ model");
                    score += w * w + 2 * cv * w;
                    absolute += w * w + 2 * std::abs(cv * w);
                }
                s_lo = std::min(s_lo, score); s_hi = std::max(s_hi, score); s_abs = std::max(s_abs, absolute);
            }
            lo += s_lo; hi += s_hi; mag += s_abs;
        }
        if (mag * (1 + gamma) >= std::numeric_limits<float>::max()) return fail(PSB_INVALID_ARGUMENT, "row correction: the model can overflow an fp32 producer");
        const long double pad = gamma * mag + ops * std::numeric_limits<float>::min();
        lower = std::min(lower, lo - pad); upper = std::max(upper, hi + pad);
    }
    const float inf = std::numeric_limits<float>::infinity();
    const float off = std::nextafter((float)lower, -inf);
    const float high = std::nextafter((float)upper, inf);
    const float sc = std::nextafter((float)(((double)high - off) / 65534.), inf);
    if (!std::isfinite(off) || !std::isfinite(high) || !std::isfinite(sc) || !(sc > 0.f) || !std::isfinite(std::fma(sc, 65534.f, off)))
        return fail(PSB_INVALID_ARGUMENT, "row correction: the model has no finite u16 encoding");
    *scale = sc; *offset = off;
    return PSB_OK;
}

psb_status psb_row_correction_encode_u16(const float* h_values, int64_t n, float scale, float offset, uint16_t* h_u16) {
    if (!h_values || !h_u16 || n < 0 || !(scale > 0.f) || !std::isfinite(scale) || !std::isfinite(offset))
        return fail(PSB_INVALID_ARGUMENT, "row correction: invalid u16 scale or offset");
    for (int64_t i = 0; i < n; ++i) {
        const float v = h_values[i];
        if (!std::isfinite(v)) return fail(PSB_INVALID_ARGUMENT, "row correction: non-finite value");
        const double code = std::ceil(((double)v - (double)offset) / (double)scale);
        if (v < offset || !(code >= 0 && code <= 65534)) return fail(PSB_INVALID_ARGUMENT, "row correction: value outside the fixed u16 range");
        h_u16[i] = (uint16_t)code;
    }
    return PSB_OK;
}

psb_status psb_row_correction_write_u16(const char* path, const psb_row_correction_u16_header* header, const uint16_t* h_u16) {
    if (!path || !header || !h_u16) return fail(PSB_INVALID_ARGUMENT, "null argument");
    FILE* f = std::fopen(path, "wb");
    if (!f) return fail(PSB_INVALID_ARGUMENT, std::string("failed to create row-correction payload ") + path);
    const bool ok = std::fwrite(header, sizeof(*header), 1, f) == 1 &&
                    std::fwrite(h_u16, sizeof(uint16_t), (size_t)header->count, f) == (size_t)header->count;
    if (std::fclose(f) != 0 || !ok) return fail(PSB_INTERNAL, "failed to write row-correction payload");
    return PSB_OK;
}

psb_status psb_row_correction_read_u16(const char* path, psb_row_correction_u16_header* header, uint16_t* h_u16, int64_t capacity) {
    if (!path || !header) return fail(PSB_INVALID_ARGUMENT, "null argument");
    FILE* f = std::fopen(path, "rb");
    if (!f) return fail(PSB_INVALID_ARGUMENT, std::string("cannot open row-correction payload ") + path);
    psb_status st = PSB_OK;
    static const char magic[8] = {0x49, 0x53, 0x52, 0x43, 0x31, 0x36, 0x00, 0x00};
    if (std::fread(header, sizeof(*header), 1, f) != 1 || std::memcmp(header->magic, magic, 8) != 0 || header->version != 2 ||
        header->header_bytes != 32 || !std::isfinite(header->scale) || !(header->scale > 0.0f) || !std::isfinite(header->offset))
        st = fail(PSB_INVALID_ARGUMENT, "not a row-correction u16 payload (magic, version, header size, scale or offset)");
    else if (h_u16) {
        if ((int64_t)header->count > capacity) st = fail(PSB_INVALID_ARGUMENT, "row-correction payload holds more rows than the buffer");
        else if (std::fread(h_u16, sizeof(uint16_t), (size_t)header->count, f) != (size_t)header->count)
            st = fail(PSB_INVALID_ARGUMENT, "row-correction payload is truncated");
    }
    std::fclose(f);
    return st;
}

// ---- synthetic data -------------------------------------------------------------------------------------------

psb_status psb_gen_mixture_rows(const float* d_centres, const int64_t* d_offsets, int ncomp, int dim,
                                float sigma, uint64_t seed, int64_t row_begin, int64_t n, float* d_out,
                                int device, void* stream) {
    if (!d_centres || !d_offsets || !d_out || ncomp <= 0 || dim <= 0 || n < 0) return fail(PSB_INVALID_ARGUMENT, "invalid generator request");
    PSB_TRY(check_device(device));
    const long long step = ((long long)1 << 31) / dim;  // rows per launch
    for (long long r = 0; r < n; r += step)
        PSB_TRY(launch_gen_mixture(d_centres, reinterpret_cast<const long long*>(d_offsets), ncomp, dim, sigma, seed,
                                   row_begin + r, std::min<long long>(step, n - r), d_out + (size_t)r * dim,
                                   static_cast<cudaStream_t>(stream)));
    return PSB_OK;
}

psb_status psb_gen_normal(uint64_t seed, int64_t first_elem, int64_t n_elems, float scale, float* d_out,
                          int device, void* stream) {
    if (!d_out || n_elems < 0) return fail(PSB_INVALID_ARGUMENT, "invalid generator request");
    PSB_TRY(check_device(device));
    const long long step = (long long)1 << 31;
    for (long long r = 0; r < n_elems; r += step)
        PSB_TRY(launch_gen_normal(seed, first_elem + r, std::min<long long>(step, n_elems - r), scale, d_out + r,
                                  static_cast<cudaStream_t>(stream)));
    return PSB_OK;
}

}  // extern "C"
