// The functions of the CUDA runtime that batch.cpp and hostblock.h call; see
// fake_cuda.h.  Device 0 .. DEVICES - 1; a graph replays nothing.
#include "fake_cuda.h"

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <vector>

struct CUstream_st {
    std::deque<std::function<void()>> ops;
    long long queued = 0, run = 0;
};
struct CUevent_st {
    CUstream_st *stream = nullptr;
    long long at = 0;
};
struct CUgraph_st {};
struct CUgraphExec_st {};

namespace {
std::recursive_mutex mu;
CUstream_st legacy;
std::set<CUstream_st *> streams;   // destroyed ones too: their queued work still runs
thread_local int device = 0;
std::atomic<int> host_alloc_device{-1};

CUstream_st *of(cudaStream_t s) {
    return s == nullptr || s == cudaStreamLegacy ? &legacy : reinterpret_cast<CUstream_st *>(s);
}
void run_until(CUstream_st *s, long long at) {
    while (s->run < at && !s->ops.empty()) {
        auto op = std::move(s->ops.front());
        s->ops.pop_front();
        ++s->run;
        op();
    }
}
}  // namespace

namespace fake {
void enqueue(cudaStream_t s, std::function<void()> op) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    of(s)->ops.push_back(std::move(op));
    ++of(s)->queued;
}
void drain_all() {
    std::lock_guard<std::recursive_mutex> lk(mu);
    run_until(&legacy, legacy.queued);
    for (CUstream_st *s : streams) run_until(s, s->queued);
}
int current_device() { return device; }
int last_host_alloc_device() { return host_alloc_device; }
}  // namespace fake

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { *n = fake::DEVICES; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d >= fake::DEVICES) return cudaErrorInvalidDevice;
    device = d;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { fake::drain_all(); return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { fake::drain_all(); std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) {
    host_alloc_device = device;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) {
    fake::enqueue(s, [=] { std::free(p); });
    return cudaSuccess;
}

// pageable to device: staged at once, on the device when the legacy stream gets there
cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, cudaMemcpyKind) {
    fake::drain_all();
    auto stage = std::make_shared<std::vector<char>>((const char *)src, (const char *)src + n);
    fake::enqueue(nullptr, [=] { std::memcpy(dst, stage->data(), stage->size()); });
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    fake::enqueue(nullptr, [=] { std::memset(p, v, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    fake::enqueue(s, [=] { std::memcpy(dst, src, n); });
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
    fake::enqueue(s, [=] { std::memset(p, v, n); });
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    auto *n = new CUstream_st;   // kept to the end of the process
    streams.insert(n);
    *s = n;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    run_until(of(s), of(s)->queued);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = new CUgraph_st; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    *e = new CUgraphExec_st;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete e; return cudaSuccess; }

cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = new CUevent_st; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    e->stream = of(s);
    e->at = of(s)->queued;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (e->stream) run_until(e->stream, e->at);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaEventQuery(e); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
}
