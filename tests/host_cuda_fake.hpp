// CUDA runtime calls of the host code under test, answered on the CPU: device memory is host memory, streams
// and events are numbers, and a chosen call fails.  For checks of error paths without a GPU.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

namespace fake {
inline std::map<std::string, int> calls;  // how often each entry was called
inline std::string fail_call;             // this entry fails ...
inline int fail_at = -1;                  // ... at its n-th call (from 0)
inline std::set<void*> device, streams, events;
inline int capturing = 0;                 // streams in capture mode
inline cudaError_t last = cudaSuccess;

inline void reset() {
    calls.clear();
    fail_call.clear();
    fail_at = -1;
    capturing = 0;
    last = cudaSuccess;
    for (auto* s : {&device, &streams, &events}) {
        for (void* p : *s) std::free(p);
        s->clear();
    }
}
inline cudaError_t enter(const char* name) {
    const int n = calls[name]++;
    return fail_call == name && n == fail_at ? cudaErrorUnknown : cudaSuccess;
}
inline void* make(std::set<void*>& s, size_t bytes = 8) {
    void* p = std::malloc(bytes ? bytes : 1);
    s.insert(p);
    return p;
}
inline cudaError_t drop(std::set<void*>& s, void* p) {
    if (p && s.erase(p)) std::free(p);
    return cudaSuccess;
}
}  // namespace fake

#define FAKE(name) \
    if (cudaError_t e_ = fake::enter(#name)) return e_

extern "C" {
inline const char* fake_message() { return "a fake error"; }
const char* cudaGetErrorString(cudaError_t) { return fake_message(); }
cudaError_t cudaGetLastError(void) {
    FAKE(cudaGetLastError);
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
cudaError_t cudaGetDevice(int* d) { FAKE(cudaGetDevice); *d = 0; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { FAKE(cudaMalloc); *p = fake::make(fake::device, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { FAKE(cudaFree); return fake::drop(fake::device, p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    FAKE(cudaMallocFromPoolAsync);
    *p = fake::make(fake::device, n);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { FAKE(cudaFreeAsync); return fake::drop(fake::device, p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { FAKE(cudaHostAlloc); *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { FAKE(cudaFreeHost); std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    FAKE(cudaMemcpyAsync);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    FAKE(cudaMemPoolCreate);
    *p = (cudaMemPool_t)8;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { FAKE(cudaMemPoolSetAttribute); return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { FAKE(cudaMemPoolTrimTo); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) { FAKE(cudaGetSymbolAddress); *p = const_cast<void*>(sym); return cudaSuccess; }
cudaError_t cudaStreamGetPriority(cudaStream_t, int* p) { FAKE(cudaStreamGetPriority); *p = 0; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) {
    FAKE(cudaStreamCreateWithPriority);
    *s = (cudaStream_t)fake::make(fake::streams);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { FAKE(cudaStreamDestroy); return fake::drop(fake::streams, s); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    FAKE(cudaEventCreateWithFlags);
    *e = (cudaEvent_t)fake::make(fake::events);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { FAKE(cudaEventDestroy); return fake::drop(fake::events, e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { FAKE(cudaEventRecord); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { FAKE(cudaStreamWaitEvent); return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    FAKE(cudaStreamBeginCapture);
    if (fake::capturing) return cudaErrorIllegalState;
    fake::capturing = 1;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    FAKE(cudaStreamEndCapture);
    *g = (cudaGraph_t)fake::make(fake::device);
    fake::capturing = 0;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { FAKE(cudaGraphDestroy); return fake::drop(fake::device, g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    FAKE(cudaGraphInstantiate);
    *x = (cudaGraphExec_t)fake::make(fake::device);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { FAKE(cudaGraphExecDestroy); return fake::drop(fake::device, x); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { FAKE(cudaGraphLaunch); return fake::capturing ? cudaErrorIllegalState : cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { FAKE(cudaStreamSynchronize); return cudaSuccess; }
}
