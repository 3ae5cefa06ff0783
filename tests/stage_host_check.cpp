// The host-buffer staging (csrc/redcuda_stage.cu) against a fake CUDA runtime: copies are queued and carried out when something waits
// for them, after a delay that stands for the GPU's work, and allocations fail on demand. Driven by test_stage_host.py.
#include "../dwarfstar_red_lite_b200/csrc/redcuda_stage.cuh"

#include <chrono>
#include <mutex>
#include <deque>
#include <map>
#include <new>
#include <string.h>
#include <stdlib.h>
#include <thread>
#include <time.h>
#include <vector>

namespace {
struct Op { void *dst; const void *src; size_t n; uint64_t event; };
struct FakeStream { std::deque<Op> q; };
std::mutex g_mu;
uint64_t g_next_event = 1;
std::map<void *, FakeStream *> g_event_stream;
std::map<void *, uint64_t> g_event_id;
int g_delay_ms = 0;
size_t g_dev_bytes = 0, g_pin_bytes = 0;
std::map<void *, size_t> g_dev, g_pin;
int g_dev_allocs = 0, g_pin_allocs = 0, g_pin_fail = 0;
std::string g_error;

void run_until(FakeStream *s, uint64_t event) {         // event 0: everything
    if (!s) return;
    if (g_delay_ms && !s->q.empty()) { std::this_thread::sleep_for(std::chrono::milliseconds(g_delay_ms)); g_delay_ms = 0; }
    std::lock_guard<std::mutex> lk(g_mu);
    while (!s->q.empty()) {
        Op o = s->q.front();
        s->q.pop_front();
        if (o.event) { if (o.event == event) return; continue; }
        memcpy(o.dst, o.src, o.n);
    }
}
}  // namespace

// C++ allocations of this library: the k-th one of the marked thread fails
static thread_local int t_fail_in = -1;
void *operator new(size_t n) {
    if (t_fail_in >= 0 && t_fail_in-- == 0) throw std::bad_alloc();
    if (void *p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
struct NoFail { int keep = t_fail_in; NoFail() { t_fail_in = -1; } ~NoFail() { t_fail_in = keep; } };      // the fake runtime's own allocations

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
static int g_set_device = 0;
cudaError_t cudaSetDevice(int) { ++g_set_device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { NoFail nf; *s = (cudaStream_t) new FakeStream(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete (FakeStream *)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { run_until((FakeStream *)s, 0); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    NoFail nf;
    std::lock_guard<std::mutex> lk(g_mu);
    g_event_stream[e] = (FakeStream *)s; g_event_id[e] = g_next_event;
    ((FakeStream *)s)->q.push_back(Op{nullptr, nullptr, 0, g_next_event++});
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    // a link of about 25 GB/s
    std::this_thread::sleep_for(std::chrono::microseconds(20));
    FakeStream *s; uint64_t id; bool queued = false;
    { std::lock_guard<std::mutex> lk(g_mu); s = g_event_stream[e]; id = g_event_id[e]; for (auto &o : s->q) queued = queued || o.event == id; }
    if (queued) run_until(s, id);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    NoFail nf;
    std::lock_guard<std::mutex> lk(g_mu);
    ((FakeStream *)s)->q.push_back(Op{dst, src, n, 0});
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { NoFail nf; *p = malloc(n); std::lock_guard<std::mutex> lk(g_mu); g_dev[*p] = n; g_dev_bytes += n; ++g_dev_allocs; return cudaSuccess; }
cudaError_t cudaFree(void *p) { { std::lock_guard<std::mutex> lk(g_mu); g_dev_bytes -= g_dev[p]; g_dev.erase(p); } free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) {
    NoFail nf;
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_pin_fail) return cudaErrorMemoryAllocation;
    *p = malloc(n); g_pin[*p] = n; g_pin_bytes += n; ++g_pin_allocs;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { { std::lock_guard<std::mutex> lk(g_mu); g_pin_bytes -= g_pin[p]; g_pin.erase(p); } free(p); return cudaSuccess; }
}

namespace rc {
void set_error(const char *fmt, ...) { NoFail nf; char b[512]; va_list ap; va_start(ap, fmt); vsnprintf(b, sizeof(b), fmt, ap); va_end(ap); g_error = b; }
std::atomic<uint64_t> g_launches{0};
int DevMem::alloc(size_t n) { release(); if (cudaMalloc(&p, n) != cudaSuccess) return 0; bytes = n; return 1; }
void DevMem::release() { if (p) { cudaFree(p); p = nullptr; bytes = 0; } }
}  // namespace rc

static double cpu_seconds() { timespec t; clock_gettime(CLOCK_PROCESS_CPUTIME_ID, &t); return t.tv_sec + 1e-9 * t.tv_nsec; }

extern "C" {
// host -> "device" -> host of n bytes; 1 when the bytes came back
int check_roundtrip(const uint8_t *src, uint8_t *dst, size_t n) {
    rc::Stage st;
    if (!st.open(rc::Stage::pad(n))) return 0;
    uint8_t *d = st.take(n);
    return st.upload(d, src, n) && st.download(dst, d, n) && st.finish() && memcmp(src, dst, n) == 0;
}
// CPU seconds that a download of n bytes takes when the GPU's work before it takes delay_ms
double check_download_cpu(const uint8_t *src, uint8_t *dst, size_t n, int delay_ms) {
    rc::Stage st;
    if (!st.open(rc::Stage::pad(n))) return -1.0;
    uint8_t *d = st.take(n);
    memcpy(d, src, n);
    g_delay_ms = delay_ms;
    const double t = cpu_seconds();
    if (!st.download(dst, d, n) || !st.finish() || memcmp(src, dst, n)) return -1.0;
    return cpu_seconds() - t;
}
// work areas of several calls open at once, each of n bytes; then all of them end
int check_open_many(size_t n, int calls) {
    std::vector<rc::Stage *> v;
    int ok = 1;
    for (int i = 0; i < calls; ++i) { v.push_back(new rc::Stage()); ok &= v.back()->open(n); }
    for (rc::Stage *s : v) delete s;
    return ok;
}
// the same with the k-th C++ allocation of this thread failing; -1: none was left to fail
int check_roundtrip_failing(const uint8_t *src, uint8_t *dst, size_t n, int k) {
    t_fail_in = k;
    const int ok = check_roundtrip(src, dst, n);
    const bool failed = t_fail_in < 0;
    t_fail_in = -1;
    return failed ? ok : -1;
}
void check_pinned_fails(int on) { g_pin_fail = on; }
int check_set_device_calls() { return g_set_device; }
size_t check_device_bytes() { return g_dev_bytes; }
size_t check_pinned_bytes() { return g_pin_bytes; }
int check_device_allocs() { return g_dev_allocs; }
int check_pinned_allocs() { return g_pin_allocs; }
const char *check_error() { return g_error.c_str(); }
}
