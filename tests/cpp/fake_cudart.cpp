// A CUDA runtime without a GPU, for tests of the library's host code: memory is
// host memory, a launch only notes the kernel's name, streams and events are
// what the test says they are.  Linked with the library's own object files.
#include <cuda_runtime_api.h>

#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <thread>

namespace {
// never destroyed: the library may be called while the program exits
auto& g_names = *new std::map<const void*, std::string>;  // host stub -> mangled kernel name
auto& g_recorded = *new std::map<cudaEvent_t, cudaStream_t>;
auto& g_busy = *new std::set<cudaStream_t>;
auto& g_capturing = *new std::set<cudaStream_t>;
std::atomic<void*> g_full{nullptr};                      // a stream that takes no more work
std::atomic<int> g_blocked{0};                           // records that wait for it
std::string g_launch;                                    // last kernel launched
int g_cluster = 0, g_launches = 0, g_frees = 0, g_mallocs = 0, g_records = 0, g_occupancy = 0;
int g_device = 0, g_fail_malloc = -1;
bool g_relaxed = false;
cudaStream_t g_config = nullptr;
const void* g_node = nullptr;  // the kernel of the last graph made or changed
long g_unfinished = 0;  // bytes that pageable copies may still have on the way
long g_uploaded = 0;    // bytes copied to the device
int g_early = 0;        // launches that are not ordered after them
cudaError_t g_last = cudaSuccess;

cudaError_t note(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}
void launched(const void* f, int cluster, cudaStream_t s) {
    if (g_unfinished && s != nullptr && s != cudaStreamLegacy) g_early++;
    g_launch = g_names.count(f) ? g_names[f] : "?";
    g_cluster = cluster;
    g_launches++;
}
}  // namespace

extern "C" {
// ---- what the tests set and read ----
void fake_reset() {
    g_busy.clear();
    g_capturing.clear();
    g_launch.clear();
    g_early = g_cluster = g_launches = g_frees = g_mallocs = g_records = g_occupancy = 0;
    g_fail_malloc = -1;
    g_unfinished = g_uploaded = 0;
    g_last = cudaSuccess;
}
void fake_stream_busy(void* s, int busy) {
    const cudaStream_t st = static_cast<cudaStream_t>(s);
    if (busy) g_busy.insert(st);
    else g_busy.erase(st);
}
void fake_stream_capturing(void* s, int on) {
    const cudaStream_t st = static_cast<cudaStream_t>(s);
    if (on) g_capturing.insert(st);
    else g_capturing.erase(st);
}
void fake_stream_full(void* s) { g_full = s; }
int fake_blocked() { return g_blocked; }
void fake_fail_malloc(int after) { g_fail_malloc = after; }
void fake_set_error(int e) { g_last = static_cast<cudaError_t>(e); }
int fake_peek_error() { return g_last; }
const char* fake_last_launch() { return g_launch.c_str(); }
int fake_last_cluster() { return g_cluster; }
int fake_launches() { return g_launches; }
int fake_frees() { return g_frees; }
int fake_mallocs() { return g_mallocs; }
int fake_records() { return g_records; }
int fake_occupancy_queries() { return g_occupancy; }
long fake_unfinished() { return g_unfinished; }
long fake_uploaded() { return g_uploaded; }
int fake_early_launches() { return g_early; }

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) {
    g_mallocs++;
    if (g_fail_malloc == 0) return note(cudaErrorMemoryAllocation);
    if (g_fail_malloc > 0) g_fail_malloc--;
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    return *p ? cudaSuccess : note(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) {
    if (p) g_frees++;
    std::free(p);
    return cudaSuccess;
}
// A copy from pageable memory may return before its data has reached the device.
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
    std::memcpy(d, s, n);
    if (k == cudaMemcpyHostToDevice) {
        g_unfinished += static_cast<long>(n);
        g_uploaded += static_cast<long>(n);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
    std::memset(p, v, n);
    g_unfinished += static_cast<long>(n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return note(cudaErrorInvalidSymbol); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {  // every buffer is pinned host memory
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeHost;
    a->devicePointer = a->hostPointer = const_cast<void*>(p);
    return cudaSuccess;
}

// ---- devices: two of 152 SMs ----
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = g_device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    g_device = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    p->multiProcessorCount = 152;
    p->sharedMemPerBlockOptin = 232448;
    p->sharedMemPerMultiprocessor = 233472;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    g_unfinished = 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (g_capturing.count(s)) return note(cudaErrorStreamCaptureUnsupported);
    if (s == nullptr || s == cudaStreamLegacy) g_unfinished = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = g_capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
    const bool was = g_relaxed;
    g_relaxed = *m == cudaStreamCaptureModeRelaxed;
    *m = was ? cudaStreamCaptureModeRelaxed : cudaStreamCaptureModeGlobal;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    g_recorded.erase(e);
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (s && g_full == s) {
        g_blocked++;
        for (int i = 0; i < 3000 && g_full == s; i++) std::this_thread::sleep_for(std::chrono::milliseconds(1));
        g_blocked--;
    }
    g_recorded[e] = s;
    g_records++;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (g_recorded.count(e) && (g_recorded[e] == nullptr || g_recorded[e] == cudaStreamLegacy)) g_unfinished = 0;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    return g_recorded.count(e) && g_busy.count(g_recorded[e]) ? note(cudaErrorNotReady) : cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphAddMemsetNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t,
                                   const cudaMemsetParams*) {
    return cudaSuccess;
}
cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t,
                                   const cudaKernelNodeParams* p) {
    g_node = p->func;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaGraphExecKernelNodeSetParams(cudaGraphExec_t, cudaGraphNode_t, const cudaKernelNodeParams* p) {
    g_node = p->func;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
    if (g_capturing.count(s)) return note(cudaErrorStreamCaptureUnsupported);
    launched(g_node, 0, s);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
    std::free(e);
    return cudaSuccess;
}

// ---- kernels ----
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int threads, size_t smem) {
    const int by_smem = static_cast<int>(233472 / (smem + 1024)), by_regs = 65536 / (80 * threads);
    *n = by_smem < by_regs ? by_smem : by_regs;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
    static const int room[17] = {0, 152, 76, 46, 36, 28, 23, 0, 0, 0, 13, 0, 0, 0, 0, 0, 7};  // one CTA per SM
    g_occupancy++;
    *n = room[c->attrs[0].val.clusterDim.x];
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) {
    launched(f, 0, s);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    launched(f, c->numAttrs ? static_cast<int>(c->attrs[0].val.clusterDim.x) : 0, c->stream);
    return cudaSuccess;
}
// What nvcc's host code calls to register and launch kernels.
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, void*, void*, void*, void*, int*) {
    g_names[stub] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void* s) {
    g_config = static_cast<cudaStream_t>(s);
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void* s) {
    *static_cast<cudaStream_t*>(s) = g_config;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t s) {
    launched(reinterpret_cast<const void*>(k), 0, s);
    return cudaSuccess;
}
}  // extern "C"
