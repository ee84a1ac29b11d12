// fake_cuda.hpp -- the host side of the library on the CPU: idb_api.cu compiled by
// g++ against this stand-in for the CUDA runtime and for the kernel launchers.
//
// Device memory is host memory.  Everything asynchronous is queued in issue order
// and runs at the next synchronisation, the latest point the runtime's contract
// allows: a copy reads its source only then, so a source that was freed or
// changed before is seen (freed: by the address sanitizer).  Captured work is
// recorded and queued again by each graph launch.  Allocations fail when `fail_alloc`
// says so.  The launchers log themselves and set the counters the test scripts.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace fake {

using Op = std::function<void()>;

struct State {
    std::vector<Op> queue;
    std::vector<Op> *capture = nullptr;
    std::map<void *, size_t> dev;               // device allocations
    size_t dev_bytes = 0;
    std::function<bool(size_t)> fail_alloc;     // of the bytes asked for
    cudaError_t last = cudaSuccess;             // what cudaGetLastError returns once
    std::vector<std::string> log;               // launches, in order
    int syncs = 0;
};
inline State &st() {
    static State s;
    return s;
}
inline void push(Op f) { (st().capture ? *st().capture : st().queue).push_back(std::move(f)); }
inline void drain() {
    std::vector<Op> q;
    q.swap(st().queue);
    for (auto &f : q) f();
}
struct Graph {
    std::vector<Op> ops;
};

}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    auto &s = fake::st();
    *p = nullptr;
    if (s.fail_alloc && s.fail_alloc(n)) return s.last = cudaErrorMemoryAllocation;
    *p = std::calloc(1, n);
    s.dev[*p] = n;
    s.dev_bytes += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {   // waits for the device
    auto &s = fake::st();
    fake::drain();
    auto it = s.dev.find(p);
    if (it != s.dev.end()) {
        s.dev_bytes -= it->second;
        s.dev.erase(it);
        std::free(p);
    }
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { fake::drain(); std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    fake::push([=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    fake::drain();
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    fake::push([=] { std::memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { ++fake::st().syncs; fake::drain(); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { fake::drain(); return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = fake::st().last; fake::st().last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    fake::st().capture = &(new fake::Graph)->ops;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    *g = reinterpret_cast<cudaGraph_t>(fake::st().capture);   // ops is the graph's only member
    fake::st().capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    for (auto &f : *reinterpret_cast<std::vector<fake::Op> *>(e)) fake::push(f);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<fake::Graph *>(g); return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t *, size_t *n) { *n = 0; return cudaSuccess; }
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType *) { return cudaSuccess; }
}  // extern "C"
