// fake_cudart.cpp -- the CUDA runtime calls libfemstep's host code makes, for a machine
// without a GPU.  Device memory is host memory and no kernel runs; what is modelled is
// when work is complete:
//   * a copy from pageable memory and a memset on the legacy stream stay pending until
//     something waits for that stream (both may return before the device is done);
//   * a launch on another stream is counted as unordered while any of them is pending,
//     and as in flight until its stream is waited for.
// The test (test_host_order.py) links it with the library's own objects.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>

namespace {

cudaError_t g_last = cudaSuccess;
int g_pending = 0;               // legacy-stream work not known to be complete
int g_in_flight = 0;             // launches on the handles' streams not waited for
int g_unordered = 0;             // launches while legacy-stream work was pending
int g_freed_in_flight = 0;       // device memory freed on the legacy stream with launches in flight
int g_refuse_clusters = 0;       // cudaLaunchKernelExC refuses cluster launches
int g_malloc_fails_at = 0;       // the n-th allocation on a handle's own stream from now fails
bool g_capturing = false;
bool g_after_graph = false;      // the stream's last work is a graph launch
int g_early_after_graph = 0;     // programmatic launches right after one
int g_calls = 0;                 // launches, allocations, copies, memsets and waits

cudaError_t result(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}

void launched(bool early) {
    ++g_calls;
    if (g_capturing) return;
    if (g_pending) ++g_unordered;
    if (g_after_graph && early) ++g_early_after_graph;
    g_after_graph = false;
    ++g_in_flight;
}

}  // namespace

extern "C" {

int fake_pending() { return g_pending; }
int fake_unordered() { return g_unordered; }
int fake_freed_in_flight() { return g_freed_in_flight; }
int fake_early_after_graph() { return g_early_after_graph; }
int fake_calls() { return g_calls; }
int fake_last_error() { return (int)g_last; }
void fake_set_last_error(int e) { g_last = (cudaError_t)e; }
void fake_refuse_clusters(int on) { g_refuse_clusters = on; }
void fake_fail_malloc(int n) { g_malloc_fails_at = n; }
void fake_reset() {
    g_last = cudaSuccess;
    g_pending = g_in_flight = g_unordered = g_freed_in_flight = g_refuse_clusters = g_malloc_fails_at = 0;
    g_early_after_graph = g_calls = 0;
    g_capturing = g_after_graph = false;
}

// ---- registration and launches ----
void** __cudaRegisterFatBinary(void*) {
    static void* handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = *block = dim3(1);
    *smem = 0;
    *static_cast<cudaStream_t*>(stream) = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
    launched(false);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void*, void**) {
    bool early = false;
    for (unsigned i = 0; i < cfg->numAttrs; ++i) {
        if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension && g_refuse_clusters)
            return result(cudaErrorInvalidConfiguration);
        if (cfg->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
            early = early || cfg->attrs[i].val.programmaticStreamSerializationAllowed != 0;
    }
    launched(early);
    return cudaSuccess;
}

// ---- memory ----
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t stream) {
    ++g_calls;
    if (stream != cudaStreamLegacy && g_malloc_fails_at && --g_malloc_fails_at == 0) return result(cudaErrorMemoryAllocation);
    *p = std::aligned_alloc(256, (bytes + 255) / 256 * 256 + 256);
    std::memset(*p, 0, (bytes + 255) / 256 * 256 + 256);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t stream) {
    ++g_calls;
    if (stream == cudaStreamLegacy && g_in_flight) ++g_freed_in_flight;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    *p = std::malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
    ++g_calls;
    std::memcpy(dst, src, bytes);
    g_pending = kind == cudaMemcpyHostToDevice ? g_pending + 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaMemset(void* dst, int value, size_t bytes) {
    ++g_calls;
    std::memset(dst, value, bytes);
    ++g_pending;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    ++g_calls;
    std::memcpy(dst, src, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* dst, int value, size_t bytes, cudaStream_t) {
    ++g_calls;
    std::memset(dst, value, bytes);
    return cudaSuccess;
}

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(std::malloc(16));
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    ++g_calls;
    (s == cudaStreamLegacy ? g_pending : g_in_flight) = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    g_pending = g_in_flight = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    g_capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    g_capturing = false;
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* exec, cudaGraph_t, unsigned long long) {
    *exec = reinterpret_cast<cudaGraphExec_t>(std::malloc(16));
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    launched(false);
    g_after_graph = true;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t exec) {
    std::free(exec);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(16));
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    g_in_flight = 0;
    g_after_graph = false;
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.0f;
    return cudaSuccess;
}

// ---- device and kernel properties ----
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    switch (a) {
        case cudaDevAttrMultiProcessorCount: *v = 148; break;
        case cudaDevAttrComputeCapabilityMajor: *v = 10; break;
        case cudaDevAttrMaxGridDimX: *v = 0x7fffffff; break;  // (a scan's launches step by it)
        default: *v = 0;
    }
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    std::strcpy(p->name, "fake");
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    *p = nullptr;
    return cudaErrorInvalidSymbol;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult*) {
    *p = nullptr;
    return cudaErrorNotSupported;
}

// ---- errors ----
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "an error"; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }

}  // extern "C"
