// The CUDA runtime calls of the library's host code on host memory, for tests
// of that code without a GPU. All streams are one queue, and queued work runs
// when somebody waits for it (as on a GPU that is slower than its host).
// Test-only; included by one translation unit of a test program.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <vector>

namespace fake {

using Op = std::function<void()>;
inline std::deque<Op> queue;
inline unsigned long long queued = 0, done = 0;  // operations so far
inline std::vector<Op>* capture = nullptr;
inline size_t room = size_t(1) << 40, used = 0;  // device memory
inline std::map<void*, size_t> sizes;
inline std::map<cudaStream_t, unsigned long long> waited;  // operations queued at a stream's last synchronisation
inline double now_ms = 0.0;  // device clock, advanced by the work

inline void run_until(unsigned long long n) {
    while (done < n && !queue.empty()) {
        Op op = std::move(queue.front());
        queue.pop_front();
        ++done;
        op();
    }
}
inline void run_all() { run_until(queued); }
inline void enqueue(Op op) {
    if (capture) {
        capture->push_back(std::move(op));
    } else {
        queue.push_back(std::move(op));
        ++queued;
    }
}

struct Event {
    unsigned long long at = 0;
    double ms = 0.0;
};
struct Graph {
    std::vector<Op> ops;
};

}  // namespace fake

extern "C" {

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 10;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    p->major = 10;
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* total) {
    *f = fake::room - fake::used;
    *total = fake::room;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = nullptr;
    if (n > fake::room - fake::used) return cudaErrorMemoryAllocation;
    *p = std::calloc(n ? n : 1, 1);
    fake::sizes[*p] = n;
    fake::used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    fake::run_all();
    const auto it = fake::sizes.find(p);
    if (it == fake::sizes.end()) return cudaSuccess;
    fake::used -= it->second;
    fake::sizes.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    fake::run_all();
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    fake::enqueue([=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    fake::run_all();
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    fake::enqueue([=] { std::memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { fake::run_all(); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    fake::waited[s] = fake::queued;
    fake::run_all();
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(new int);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete reinterpret_cast<int*>(s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(new fake::Event);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<fake::Event*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    auto* ev = reinterpret_cast<fake::Event*>(e);
    fake::enqueue([ev] { ev->ms = fake::now_ms; });
    if (!fake::capture) ev->at = fake::queued;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    fake::run_until(reinterpret_cast<fake::Event*>(e)->at);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
    *ms = static_cast<float>(reinterpret_cast<fake::Event*>(b)->ms - reinterpret_cast<fake::Event*>(a)->ms);
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    fake::capture = new std::vector<fake::Op>;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    auto* graph = new fake::Graph{std::move(*fake::capture)};
    delete fake::capture;
    fake::capture = nullptr;
    *g = reinterpret_cast<cudaGraph_t>(graph);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* ge, cudaGraph_t g, unsigned long long) {
    *ge = reinterpret_cast<cudaGraphExec_t>(new fake::Graph(*reinterpret_cast<fake::Graph*>(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<fake::Graph*>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { delete reinterpret_cast<fake::Graph*>(g); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t) {
    for (const auto& op : reinterpret_cast<fake::Graph*>(g)->ops) fake::enqueue(op);
    return cudaSuccess;
}

}  // extern "C"
