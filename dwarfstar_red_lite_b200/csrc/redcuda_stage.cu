// See redcuda_stage.cuh.
//
// Measured (16-core host): matvec of an 8192 x 2048 Q4_K matrix for 4 tokens (9.4 MB of pageable rows) 2180 -> 370 us a call, the
// upload itself 290 (one thread copies those bytes in 540, the link moves them in 180); matvec 64 x 256 of Q8_0 700 -> 34;
// dequantisation of 8192 x 4096 values 39 -> 8.5 ms (bound by the page faults of the 134 MB it returns).
#include "redcuda_stage.cuh"
#include "../../include/redcuda.h"

#include <string.h>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif
#include <algorithm>
#include <condition_variable>
#include <deque>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace rc {

// ---- threads that copy between pageable and pinned memory ----
// One core moves about 10 GB/s, the link 50: large arrays are cut into pieces that several threads copy while the copy
// engine moves the pieces already done. The threads are started at the first large array and live as long as the process.
namespace {
constexpr size_t PIECE = 512u << 10;             // a piece takes a core about 50 us and the link 10
constexpr size_t INLINE_MAX = 256u << 10;        // below this waking a thread costs more than it saves
constexpr size_t PINNED_MAX = 32u << 20;         // pinned bytes of a lease; larger arrays go through it in rounds
constexpr size_t KEEP_DEVICE = 256u << 20;       // device bytes that the idle leases of a device keep together
constexpr size_t KEEP_PINNED = 64u << 20;        // pinned bytes that they keep together
constexpr size_t KEEP_LEASES = 4;                // idle leases per device

inline void cpu_relax() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}

// Host memory to the pinned buffer. Stores that bypass the caches: a DMA read of lines that still sit modified in a core's cache
// has to fetch them from there, which held the copy engine to 8 GB/s (9.4 MB in pieces: 1130 us until the last was on the device, 290 with these stores).
inline void copy_streaming(uint8_t *dst, const uint8_t *src, size_t n) {
#if defined(__x86_64__)
    size_t i = 0;
    if (((uintptr_t)dst & 15u) == 0) {
        for (; i + 64 <= n; i += 64) {
            const __m128i a = _mm_loadu_si128((const __m128i *)(src + i)), b = _mm_loadu_si128((const __m128i *)(src + i + 16)),
                          c = _mm_loadu_si128((const __m128i *)(src + i + 32)), d = _mm_loadu_si128((const __m128i *)(src + i + 48));
            _mm_stream_si128((__m128i *)(dst + i), a); _mm_stream_si128((__m128i *)(dst + i + 16), b);
            _mm_stream_si128((__m128i *)(dst + i + 32), c); _mm_stream_si128((__m128i *)(dst + i + 48), d);
        }
        _mm_sfence();
    }
    memcpy(dst + i, src + i, n - i);
#else
    memcpy(dst, src, n);
#endif
}

// One array cut into pieces. Threads claim them in order; piece i may be claimed once `avail` > i (the pieces of a download arrive one
// after the other, and nobody waits for one with a claim on it) and done[i] is set when it has been copied.
struct CopyBatch {
    uint8_t *dst; const uint8_t *src;
    size_t bytes, n;
    std::atomic<size_t> next{0}, avail{0};
    std::vector<std::atomic<int>> done;
    CopyBatch(uint8_t *d, const uint8_t *s, size_t b) : dst(d), src(s), bytes(b), n((b + PIECE - 1) / PIECE), done(n) {}
    size_t piece(size_t i) const { return std::min(PIECE, bytes - i * PIECE); }
    bool exhausted() const { return next.load(std::memory_order_relaxed) >= n; }
    bool claimable() const { return next.load(std::memory_order_relaxed) < std::min(n, avail.load()); }
    // claims and copies one piece; false when none can be claimed now
    bool step() {
        size_t i = next.load(std::memory_order_relaxed);
        do {
            if (i >= n || i >= avail.load(std::memory_order_acquire)) return false;
        } while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
        copy_streaming(dst + i * PIECE, src + i * PIECE, piece(i));
        done[i].store(1, std::memory_order_release);
        return true;
    }
    // until piece i, claimed by another thread, has been copied: that thread may need this core to finish
    void wait(size_t i) const {
        for (int k = 0; !done[i].load(std::memory_order_acquire); ++k) { if (k < 4000) cpu_relax(); else std::this_thread::yield(); }
    }
    // no further claims; returns when nobody copies any more
    void stop() { for (size_t i = 0, c = std::min(n, next.exchange(n)); i < c; ++i) wait(i); }
};

struct CopyPool {
    std::mutex mu;
    std::condition_variable cv;
    std::deque<std::shared_ptr<CopyBatch>> batches;
    std::atomic<uint32_t> posted{0}, asleep{0};
    bool started = false;

    void start() {         // mu held
        if (started) return;
        started = true;
        const unsigned hw = std::thread::hardware_concurrency(), n = std::min(7u, hw > 1u ? hw / 2u : 0u);
        for (unsigned i = 0; i < n; ++i) {
            try { std::thread([this] { work(); }).detach(); } catch (...) { break; }      // fewer helpers: the caller copies what is left itself
        }
    }
    // a batch with a piece to claim
    std::shared_ptr<CopyBatch> pick() {         // mu held
        for (auto it = batches.begin(); it != batches.end();) {
            if ((*it)->exhausted()) { it = batches.erase(it); continue; }
            if ((*it)->claimable()) return *it;
            ++it;
        }
        return nullptr;
    }
    void work() {
        std::unique_lock<std::mutex> lk(mu);
        for (;;) {
            std::shared_ptr<CopyBatch> b = pick();
            if (!b) {
                asleep.fetch_add(1);
                b = pick();             // what became claimable before wake() could see this thread asleep
                if (!b) cv.wait(lk);
                asleep.fetch_sub(1);
            }
            if (!b) continue;
            lk.unlock();
            while (b->step()) {}
            b.reset();
            // pieces and calls follow one another closely: look for the next for about as long as a wake-up takes before going to sleep
            const uint32_t seen = posted.load(std::memory_order_relaxed);
            for (int i = 0; i < 1500 && posted.load(std::memory_order_relaxed) == seen; ++i) cpu_relax();
            lk.lock();
        }
    }
    // pieces became claimable
    void wake() {
        posted.fetch_add(1);
        if (!asleep.load()) return;
        { std::lock_guard<std::mutex> lk(mu); }         // a thread counted asleep holds mu until it waits
        cv.notify_all();
    }
    void post(const std::shared_ptr<CopyBatch> &b) {
        { std::lock_guard<std::mutex> lk(mu); start(); batches.push_back(b); }
        wake();
    }
};
CopyPool &copy_pool() { static CopyPool *p = new CopyPool(); return *p; }      // never destroyed: its threads outlive static destructors
}  // namespace

struct StageLease {
    int device = 0;
    cudaStream_t s = nullptr;
    uint8_t *dev = nullptr, *pin = nullptr;
    size_t dev_bytes = 0, pin_bytes = 0;
    std::vector<cudaEvent_t> events;
    cudaEvent_t behind = nullptr;      // Stage::follow_default_stream
    ~StageLease() {
        for (cudaEvent_t e : events) cudaEventDestroy(e);
        if (behind) cudaEventDestroy(behind);
        if (dev) cudaFree(dev);
        if (pin) cudaFreeHost(pin);
        if (s) cudaStreamDestroy(s);
    }
};

// The entry points have C linkage: what the containers above and below throw (a host without memory) ends a call with an error.
template <class F>
static int no_throw(F f) {
    try { return f(); } catch (const std::exception &e) { set_error("host-buffer call: %s", e.what()); return 0; }
}

static std::mutex g_stage_mu;
static std::vector<StageLease *> &stage_idle() { static std::vector<StageLease *> *v = new std::vector<StageLease *>(); return *v; }

void stage_trim() {
    std::vector<StageLease *> drop;
    if (!no_throw([&] { std::lock_guard<std::mutex> lk(g_stage_mu); drop.swap(stage_idle()); return 1; })) return;
    if (drop.empty()) return;              // nothing kept: no device is touched (there may be none)
    int cur = 0;
    cudaGetDevice(&cur);
    for (StageLease *l : drop) { cudaSetDevice(l->device); delete l; }
    cudaSetDevice(cur);
}

int Stage::open(size_t device_bytes) { return no_throw([&] { return open_or_throw(device_bytes); }); }
int Stage::upload(void *dst_dev, const void *src_host, size_t bytes) { return no_throw([&] { return upload_or_throw(dst_dev, src_host, bytes); }); }
int Stage::download(void *dst_host, const void *src_dev, size_t bytes) { return no_throw([&] { return download_or_throw(dst_host, src_dev, bytes); }); }

int Stage::open_or_throw(size_t device_bytes) {
    int dev = 0;
    RC_CUDA(cudaGetDevice(&dev));
    const bool own = device_bytes > KEEP_DEVICE;
    {
        std::lock_guard<std::mutex> lk(g_stage_mu);
        auto &v = stage_idle();
        // the smallest idle lease that is large enough, else the largest (it grows); a call whose area is not kept brings its own
        // and takes the smallest, so that it uses up no warm one
        const size_t want = own ? 0u : device_bytes;
        size_t best = v.size();
        for (size_t i = 0; i < v.size(); ++i) {
            if (v[i]->device != dev) continue;
            if (best == v.size()) { best = i; continue; }
            const bool fits = v[i]->dev_bytes >= want, best_fits = v[best]->dev_bytes >= want;
            if (fits != best_fits ? fits : fits ? v[i]->dev_bytes < v[best]->dev_bytes : v[i]->dev_bytes > v[best]->dev_bytes) best = i;
        }
        if (best < v.size()) { lease_ = v[best]; v.erase(v.begin() + best); }
    }
    if (!lease_) {
        lease_ = new StageLease();
        lease_->device = dev;
        RC_CUDA(cudaStreamCreateWithFlags(&lease_->s, cudaStreamNonBlocking));
    }
    if (own) {
        if (!own_.alloc(device_bytes)) {             // the lease's area may be what is missing
            if (!lease_->dev) return 0;
            cudaFree(lease_->dev); lease_->dev = nullptr; lease_->dev_bytes = 0;
            if (!own_.alloc(device_bytes)) return 0;
        }
    } else if (lease_->dev_bytes < device_bytes) {
        if (lease_->dev) { cudaFree(lease_->dev); lease_->dev = nullptr; lease_->dev_bytes = 0; }
        size_t want = 1u << 20;
        while (want < device_bytes) want <<= 1;      // powers of two: a few growths, then none
        DevMem m;
        if (!m.alloc(want)) return 0;
        lease_->dev = m.as<uint8_t>(); lease_->dev_bytes = want;
        m.p = nullptr; m.bytes = 0;
    }
    dev_ = own ? own_.as<uint8_t>() : lease_->dev; used_ = 0; pinned_used_ = 0; followed_ = false;
    return 1;
}

// The copy engine reads and writes such arrays by itself, and the caller may have copies of its own under way on them: one
// that still fills an input, or one that still reads what is about to be overwritten. A call on such an array therefore starts
// behind the default stream (and, with it, behind every stream that synchronises with it), as it did when it ran there.
int Stage::follow_default_stream() {
    if (followed_) return 1;
    if (!lease_->behind) RC_CUDA(cudaEventCreateWithFlags(&lease_->behind, cudaEventDisableTiming));
    RC_CUDA(cudaEventRecord(lease_->behind, cudaStreamLegacy));
    RC_CUDA(cudaStreamWaitEvent(lease_->s, lease_->behind, 0));
    followed_ = true;
    return 1;
}

Stage::~Stage() {
    if (!lease_) return;
    cudaStreamSynchronize(lease_->s);        // after an error a copy may still be in flight
    own_.release();
    uint8_t *dev = nullptr, *pin = nullptr;  // what the idle leases may not keep
    bool keep = lease_->s != nullptr;
    if (keep && no_throw([] { stage_idle(); return 1; })) {
        std::lock_guard<std::mutex> lk(g_stage_mu);
        auto &v = stage_idle();
        size_t same = 0, dev_sum = lease_->dev_bytes, pin_sum = lease_->pin_bytes;
        for (StageLease *l : v) if (l->device == lease_->device) { ++same; dev_sum += l->dev_bytes; pin_sum += l->pin_bytes; }
        keep = same < KEEP_LEASES;
        if (keep) {
            if (dev_sum > KEEP_DEVICE) { dev = lease_->dev; lease_->dev = nullptr; lease_->dev_bytes = 0; }
            if (pin_sum > KEEP_PINNED) { pin = lease_->pin; lease_->pin = nullptr; lease_->pin_bytes = 0; }
            keep = no_throw([&] { v.push_back(lease_); return 1; }) != 0;
        }
    }
    if (!keep) delete lease_;
    if (dev) cudaFree(dev);
    if (pin) cudaFreeHost(pin);
}

cudaStream_t Stage::stream() const { return lease_->s; }

// Makes the pinned buffer at least `want` bytes large (PINNED_MAX at most). A host that has no pinned memory left is no error: the
// lease is left without a buffer, and the caller leaves the array to the driver's own copy of pageable memory.
static int stage_pinned(StageLease *l, size_t want) {
    want = std::min(PINNED_MAX, std::max<size_t>(want, 1u << 20));
    if (l->pin_bytes >= want) return 1;
    size_t p = 1u << 20;
    while (p < want) p <<= 1;
    RC_CUDA(cudaStreamSynchronize(l->s));
    if (l->pin) { cudaFreeHost(l->pin); l->pin = nullptr; l->pin_bytes = 0; }
    if (cudaMallocHost((void **)&l->pin, p) != cudaSuccess) {
        cudaGetLastError();
        l->pin = nullptr;
        stage_trim();                  // what idle leases keep may be what is missing
        if (cudaMallocHost((void **)&l->pin, p) != cudaSuccess) { cudaGetLastError(); l->pin = nullptr; return 1; }
    }
    l->pin_bytes = p;
    return 1;
}
// memory the copy engine can reach by itself: pinned, managed, and device memory (a caller may hand in either kind of pointer)
static bool dma_reaches(const void *p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type != cudaMemoryTypeUnregistered;
}

int Stage::drain_pinned() { RC_CUDA(cudaStreamSynchronize(lease_->s)); pinned_used_ = 0; return 1; }

int Stage::upload_or_throw(void *dst_dev, const void *src_host, size_t bytes) {
    if (!bytes) return 1;
    cudaStream_t s = lease_->s;
    if (dma_reaches(src_host)) {
        if (!follow_default_stream()) return 0;
        RC_CUDA(cudaMemcpyAsync(dst_dev, src_host, bytes, cudaMemcpyDefault, s));
        return 1;
    }
    const uint8_t *src = static_cast<const uint8_t *>(src_host);
    uint8_t *dst = static_cast<uint8_t *>(dst_dev);
    if (lease_->pin_bytes - pinned_used_ < bytes && lease_->pin_bytes < PINNED_MAX) {
        const size_t want = pinned_used_ + bytes;
        if (!drain_pinned() || !stage_pinned(lease_, want)) return 0;
    }
    if (!lease_->pin) { RC_CUDA(cudaMemcpyAsync(dst_dev, src_host, bytes, cudaMemcpyHostToDevice, s)); return 1; }
    for (size_t at = 0; at < bytes;) {
        if (pinned_used_ == lease_->pin_bytes && !drain_pinned()) return 0;
        const size_t n = std::min(bytes - at, lease_->pin_bytes - pinned_used_);
        uint8_t *pin = lease_->pin + pinned_used_;
        if (n <= INLINE_MAX) {
            copy_streaming(pin, src + at, n);
            RC_CUDA(cudaMemcpyAsync(dst + at, pin, n, cudaMemcpyHostToDevice, s));
        } else {
            auto b = std::make_shared<CopyBatch>(pin, src + at, n);
            b->avail.store(b->n);
            copy_pool().post(b);
            cudaError_t err = cudaSuccess;
            for (size_t i = 0; i < b->n; ++i) {          // every piece is waited for, also after an error: the source is the caller's
                while (!b->done[i].load(std::memory_order_acquire)) if (!b->step()) { b->wait(i); break; }
                if (err == cudaSuccess) err = cudaMemcpyAsync(dst + at + i * PIECE, pin + i * PIECE, b->piece(i), cudaMemcpyHostToDevice, s);
            }
            RC_CUDA(err);
        }
        pinned_used_ = std::min(lease_->pin_bytes, pad(pinned_used_ + n));
        at += n;
    }
    return 1;
}

// Returns with the bytes in dst_host (pageable memory) or with the copy queued (pinned memory)
int Stage::download_or_throw(void *dst_host, const void *src_dev, size_t bytes) {
    if (!bytes) return 1;
    cudaStream_t s = lease_->s;
    if (dma_reaches(dst_host)) {
        if (!follow_default_stream()) return 0;
        RC_CUDA(cudaMemcpyAsync(dst_host, src_dev, bytes, cudaMemcpyDefault, s));
        return 1;
    }
    uint8_t *dst = static_cast<uint8_t *>(dst_host);
    const uint8_t *src = static_cast<const uint8_t *>(src_dev);
    if (bytes > INLINE_MAX && lease_->pin_bytes < std::min(bytes, PINNED_MAX) && !stage_pinned(lease_, bytes)) return 0;
    if (!lease_->pin && !stage_pinned(lease_, bytes)) return 0;
    if (!lease_->pin) {
        RC_CUDA(cudaMemcpyAsync(dst_host, src_dev, bytes, cudaMemcpyDeviceToHost, s));
        RC_CUDA(cudaStreamSynchronize(s));
        pinned_used_ = 0;
        return 1;
    }
    for (size_t at = 0; at < bytes;) {
        const size_t n = std::min(bytes - at, lease_->pin_bytes), np = (n + PIECE - 1) / PIECE;
        // the device's copies are queued behind the uploads that still read the pinned buffer, so its start can be reused
        while (lease_->events.size() < np) {
            cudaEvent_t e = nullptr;
            RC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            lease_->events.push_back(e);
        }
        for (size_t i = 0; i < np; ++i) {
            RC_CUDA(cudaMemcpyAsync(lease_->pin + i * PIECE, src + at + i * PIECE, std::min(PIECE, n - i * PIECE), cudaMemcpyDeviceToHost, s));
            RC_CUDA(cudaEventRecord(lease_->events[i], s));
        }
        if (np == 1) {
            RC_CUDA(cudaEventSynchronize(lease_->events[0]));
            memcpy(dst + at, lease_->pin, n);
            at += n;
            continue;
        }
        // the helpers are called when the first piece is there (until then they would have nothing to do but wait for the GPU)
        auto b = std::make_shared<CopyBatch>(dst + at, lease_->pin, n);
        cudaError_t err = cudaSuccess;
        for (size_t i = 0; i < np && err == cudaSuccess; ++i) {
            err = cudaEventSynchronize(lease_->events[i]);
            if (err != cudaSuccess) break;
            b->avail.store(i + 1);
            if (i == 0) copy_pool().post(b); else copy_pool().wake();
        }
        if (err == cudaSuccess) while (b->step()) {}
        b->stop();
        RC_CUDA(err);
        at += n;
    }
    pinned_used_ = 0;
    return 1;
}

int Stage::finish() { RC_CUDA(cudaStreamSynchronize(lease_->s)); pinned_used_ = 0; return 1; }

}  // namespace rc

extern "C" int redcuda_trim(void) { rc::stage_trim(); return 1; }
