// A CUDA runtime without a GPU: what the library's host code calls, as far as the tests need it. Linked with the library's own
// objects into a second library whose copies are plain memcpy calls and whose launches are only written down. Test infrastructure.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <unistd.h>
#include <vector>

namespace {
std::mutex g_mutex;
std::map<const void *, std::string> g_kernels;       // host stub -> mangled device name
std::string g_log;                                   // one line per launch / copy
std::map<const void *, int> g_configured;            // cudaFuncSetAttribute calls per kernel
std::set<const void *> g_pinned;
std::set<std::pair<pthread_t, cudaStream_t>> g_users;   // streams that copies and events were enqueued on, per thread
std::atomic<int> g_capture{0}, g_violations{0}, g_slow{0}, g_fail_new{-1}, g_set_device{0};
CUcontext g_primary = (CUcontext)0x100, g_other = (CUcontext)0x200;
thread_local CUcontext t_context = nullptr;
thread_local cudaStreamCaptureMode t_mode = cudaStreamCaptureModeGlobal;
thread_local int t_device = 0;
thread_local bool t_count_new = false;

CUcontext current() { return t_context ? t_context : (t_context = g_primary); }
cudaError_t unsafe() {   // a call that another thread's capture in global mode forbids
    if (g_capture && t_mode == cudaStreamCaptureModeGlobal) {
        ++g_violations;
        return cudaErrorStreamCaptureUnsupported;
    }
    return cudaSuccess;
}
void used(cudaStream_t s) {
    std::lock_guard<std::mutex> l(g_mutex);
    g_users.insert({pthread_self(), s});
}
CUresult ctx_get_current(CUcontext *c) { *c = t_context; return CUDA_SUCCESS; }
CUresult ctx_set_current(CUcontext c) { t_context = c; return CUDA_SUCCESS; }
CUresult stream_get_ctx(CUstream s, CUcontext *c) { *c = s == (CUstream)0x300 ? g_other : current(); return CUDA_SUCCESS; }
CUresult encode_tiled(...) { return CUDA_SUCCESS; }
}  // namespace

// ---- what the tests set and read ------------------------------------------------------------------------------------------
extern "C" {
void fake_capture(int on) { g_capture = on; g_violations = 0; }
int fake_violations() { return g_violations; }
void fake_slow_us(int us) { g_slow = us; }
void fake_context(int other) { t_context = other ? g_other : g_primary; }
int fake_context_is_other() { return t_context == g_other; }
int fake_set_device_calls() { return g_set_device; }
void fake_fail_new(int n) { t_count_new = n >= 0; g_fail_new = n; }   // the n-th allocation by operator new on this thread fails
void fake_reset_device() { std::lock_guard<std::mutex> l(g_mutex); g_pinned.clear(); }
int fake_most_configured() {
    std::lock_guard<std::mutex> l(g_mutex);
    int m = 0;
    for (auto &k : g_configured) m = k.second > m ? k.second : m;
    return m;
}
int fake_stream_users() { std::lock_guard<std::mutex> l(g_mutex); const int n = (int)g_users.size(); g_users.clear(); return n; }
int fake_pinned() { std::lock_guard<std::mutex> l(g_mutex); return (int)g_pinned.size(); }
const char *fake_log() { static std::string s; std::lock_guard<std::mutex> l(g_mutex); s.swap(g_log); g_log.clear(); return s.c_str(); }

// ---- registration and launches ----------------------------------------------------------------------------------------------
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *stub, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) { g_kernels[stub] = name; }
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **, size_t, cudaStream_t) {
    std::lock_guard<std::mutex> l(g_mutex);
    g_log += g_kernels[f] + "\n";
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *f, void **) {
    std::lock_guard<std::mutex> l(g_mutex);
    g_log += g_kernels[f] + "\n";
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int) {
    { std::lock_guard<std::mutex> l(g_mutex); ++g_configured[f]; }
    usleep(g_slow);
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *c) {
    usleep(g_slow);
    *n = (int)(c->gridDim.x / c->attrs[0].val.clusterDim.x);
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **fn, unsigned long long, cudaDriverEntryPointQueryResult *r) {
    const std::string s = name;
    *fn = s == "cuCtxGetCurrent" ? (void *)ctx_get_current : s == "cuCtxSetCurrent" ? (void *)ctx_set_current : s == "cuStreamGetCtx" ? (void *)stream_get_ctx
                                                                                                                                    : (void *)encode_tiled;
    if (r) *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) { static int word; *p = &word; return cudaSuccess; }

// ---- devices, contexts, capture ---------------------------------------------------------------------------------------------
cudaError_t cudaGetDevice(int *d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; t_context = g_primary; ++g_set_device; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { current(); *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) { std::swap(t_mode, *m); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }

// ---- memory, events, copies -------------------------------------------------------------------------------------------------
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    if (cudaError_t e = unsafe()) return e;
    *p = malloc(n);
    std::lock_guard<std::mutex> l(g_mutex);
    g_pinned.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void *) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *a, size_t *b) { *a = *b = size_t(1) << 37; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::lock_guard<std::mutex> l(g_mutex);
    a->type = g_pinned.count(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    used(st);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)0x1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) {   // stream 0x300 belongs to the other context, every event to the current one
    used(s);
    return s == (cudaStream_t)0x300 && current() != g_other ? cudaErrorInvalidResourceHandle : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return unsafe(); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return unsafe(); }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t *, void *) { return cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void **, cudaIpcMemHandle_t, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void *) { return cudaErrorNotSupported; }
}

// ---- allocations that fail on demand -----------------------------------------------------------------------------------------
void *operator new(size_t n) {
    if (t_count_new && g_fail_new >= 0 && g_fail_new-- == 0) throw std::bad_alloc();
    if (void *p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
