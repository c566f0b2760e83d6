// fake_cudart.cpp - the CUDA runtime calls the library makes, answered on the host: device memory is host memory,
// kernels do nothing, every call that matters is written to a log, a chosen allocation can be made to fail and a stream
// can be marked as being captured. Linked with the library's own objects in place of the CUDA runtime, so that the
// order of its calls, its clean-up after a failing call and what it does under stream capture can be tested without a
// GPU (and without a fault on one).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>

namespace {

// host stub -> mangled device name (filled while the objects' own static initialisers run)
std::map<const void*, std::string>& kernels() {
    static std::map<const void*, std::string> k;
    return k;
}
std::mutex mu;
std::set<void*> live;                         // pool allocations not freed yet
std::set<const void*> capturing;              // streams being captured
std::string text, last_kernel;
long long fail_in = -1;                       // pool allocations until one fails (-1: none does)
bool failed = false;                          // ... and whether one has
thread_local cudaError_t last = cudaSuccess;
thread_local struct { dim3 grid, block; size_t smem; cudaStream_t st; } config;

cudaError_t err(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
bool captured(cudaStream_t st) { return capturing.count(st) != 0; }
void note(const std::string& what, cudaStream_t st) { text += what + (captured(st) ? " captured\n" : "\n"); }

}  // namespace

extern "C" {

// ---- what the tests use ----
void fake_reset() { std::lock_guard<std::mutex> l(mu); text.clear(); fail_in = -1; capturing.clear(); last = cudaSuccess; }
void fake_fail_in(long long k) { std::lock_guard<std::mutex> l(mu); fail_in = k; failed = false; }
int fake_failed() { std::lock_guard<std::mutex> l(mu); return failed; }
long long fake_live() { std::lock_guard<std::mutex> l(mu); return (long long)live.size(); }
void fake_capture(void* st, int on) {
    std::lock_guard<std::mutex> l(mu);
    if (on) capturing.insert(st); else capturing.erase(st);
}
const char* fake_log() { std::lock_guard<std::mutex> l(mu); return text.c_str(); }

// ---- module registration and launches ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels()[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st* st) {
    config = {g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    *g = config.grid; *b = config.block; *smem = config.smem; *(cudaStream_t*)st = config.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    last_kernel = kernels()[f];
    note("launch " + last_kernel, st);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return cudaLaunchKernel(f, c->gridDim, c->blockDim, nullptr, 0, c->stream);
}

// ---- memory ----
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    if (fail_in >= 0 && fail_in-- == 0) {
        failed = true;
        return err(cudaErrorMemoryAllocation);
    }
    note("alloc", st);
    *p = std::calloc(n ? n : 1, 1);
    live.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    std::lock_guard<std::mutex> l(mu);
    if (!live.erase(p)) return err(cudaErrorInvalidValue);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    note("copy", st);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    note("memset " + std::to_string((unsigned long long)d) + " " + std::to_string(n), st);
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    *a = {};
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = (cudaMemPool_t)&mu; return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) { *(size_t*)v = 0; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return err(cudaErrorInvalidSymbol); }

// ---- streams, events, capture ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) { *st = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t st) { std::free(st); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    if (captured(st)) return err(cudaErrorStreamCaptureUnsupported);
    note("sync", st);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus* s) {
    std::lock_guard<std::mutex> l(mu);
    *s = captured(st) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t, unsigned) {
    std::lock_guard<std::mutex> l(mu);
    note("wait", st);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    note("record", st);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {   // the one-thread-per-edge form counts fastest
    std::lock_guard<std::mutex> l(mu);
    *ms = last_kernel.find("k_tc_octs") != std::string::npos ? 0.5f : 1.0f;
    return cudaSuccess;
}

// ---- graphs ----
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) { *g = (cudaGraph_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { std::free(g); return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
    *h = 1;
    return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
    static cudaGraph_t body = (cudaGraph_t)std::malloc(1);
    *n = nullptr;
    p->conditional.phGraph_out = &body;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t st, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                          size_t, cudaStreamCaptureMode) {
    fake_capture(st, 1);
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t*) { fake_capture(st, 0); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = (cudaGraphExec_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
    std::lock_guard<std::mutex> l(mu);
    note("graph launch", st);
    return cudaSuccess;
}

// ---- device, functions, errors ----
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {
    std::lock_guard<std::mutex> l(mu);
    *a = {};
    text += "load " + kernels()[f] + "\n";
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) { return err(cudaErrorNotSupported); }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }

}  // extern "C"
