// Large copies between device memory and pageable host memory.
//
// The runtime takes pageable memory through its staging buffer on the calling thread: one core copies and - towards the host, into
// fresh memory - takes the page faults. Here several threads move chunks between the caller's memory and pinned buffers of their
// own while the copy engine moves the neighbouring chunks, so the caller's pages are touched by all of them at once: a [4096,
// 4096] fp32 tensor to packed tiles on the device and back, 64 MiB each way, 36.9 ms before, 8.4 ms now. Either way a large copy
// to the device returns after the work ahead of it on the stream.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>

#include <cuda.h>

#include "common.cuh"

namespace ttb {
namespace {

constexpr size_t kChunk = 1 << 20;
constexpr int kThreads = 8, kSlots = 2;          // threads, pinned chunks of each
// Below these starting threads costs more than it gives (us, the runtime's copy / this one: 4 MiB to the device 341 / 382, 5 MiB 426 /
// 372; 4 MiB to the host 410 / 355, into fresh memory 1790 / 1010).
constexpr size_t kMinToDevice = 5 << 20, kMinToHost = 4 << 20;

// 16 MiB of pinned memory, allocated by the first large copy and kept for the next ones; one copy at a time uses it.
struct Staging {
    std::mutex mutex;
    uint8_t *base = nullptr;
    ~Staging() {
        if (base) cudaFreeHost(base);
    }
};
Staging g_staging;

bool memory_is(const void *p, cudaMemoryType type) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return a.type == type;
}

// The driver's view of contexts, through the runtime's entry points (no link against the driver library).
struct Contexts {
    CUresult (*get_current)(CUcontext *) = nullptr;
    CUresult (*set_current)(CUcontext) = nullptr;
    CUresult (*of_stream)(CUstream, CUcontext *) = nullptr;
    bool ok = false;
    Contexts() {
        auto find = [](const char *name, void **fn) {
            cudaDriverEntryPointQueryResult r;
            return cudaGetDriverEntryPoint(name, fn, cudaEnableDefault, &r) == cudaSuccess && r == cudaDriverEntryPointSuccess && *fn;
        };
        ok = find("cuCtxGetCurrent", reinterpret_cast<void **>(&get_current)) && find("cuCtxSetCurrent", reinterpret_cast<void **>(&set_current)) &&
             find("cuStreamGetCtx", reinterpret_cast<void **>(&of_stream));
        if (!ok) (void)cudaGetLastError();
    }
};
const Contexts &contexts() {
    static const Contexts c;
    return c;
}

// While some thread captures in global mode, the others' allocations and waits are forbidden unless they declare themselves
// relaxed, and end that thread's capture. Nothing here belongs to a capture.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Chunks t, t + threads, ... of the copy, alternating between this thread's two pinned buffers.
cudaError_t copy_chunks(int t, int threads, uint8_t *dev, uint8_t *host, size_t bytes, bool to_device, uint8_t *pinned, cudaStream_t stream) {
    cudaEvent_t done[kSlots] = {};
    uint8_t *target[kSlots] = {};    // towards the host: where the chunk in flight in a buffer belongs, and its size
    size_t size[kSlots] = {};
    const RelaxedCapture relaxed;
    cudaError_t e = cudaSuccess;
    for (int s = 0; s < kSlots && e == cudaSuccess; ++s) e = cudaEventCreateWithFlags(&done[s], cudaEventDisableTiming);
    auto drain = [&](int s) {        // the buffer's previous chunk has been moved on
        if (e == cudaSuccess && size[s]) {
            e = cudaEventSynchronize(done[s]);
            if (e == cudaSuccess && !to_device) std::memcpy(target[s], pinned + s * kChunk, size[s]);
            size[s] = 0;
        }
    };
    int s = 0;
    for (size_t off = t * kChunk; off < bytes && e == cudaSuccess; off += threads * kChunk, s ^= 1) {
        drain(s);
        if (e != cudaSuccess) break;
        const size_t n = std::min(kChunk, bytes - off);
        uint8_t *const buf = pinned + s * kChunk;
        if (to_device) std::memcpy(buf, host + off, n);
        e = to_device ? cudaMemcpyAsync(dev + off, buf, n, cudaMemcpyHostToDevice, stream) : cudaMemcpyAsync(buf, dev + off, n, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaEventRecord(done[s], stream);
        target[s] = host + off;
        size[s] = n;
    }
    for (int i = 0; i < kSlots; ++i, s ^= 1) drain(s);
    if (e != cudaSuccess) cudaStreamSynchronize(stream);   // nothing of this thread's uses the buffers any more
    for (int i = 0; i < kSlots; ++i)
        if (done[i]) cudaEventDestroy(done[i]);
    return e;
}

}  // namespace

// Copies through the pinned buffers if that is the better way, complete on return; false: the caller copies as usual. What
// belongs to a capture, small or already pinned is left alone, and so is a copy that meets another one at work. The handle of
// the per-thread default stream names another stream on each of the threads here, none of them ordered after the caller's work.
// The helper threads work in the caller's context (which need not be its device's primary one); a stream of another context, whose
// work the events here could not mark, is left alone too.
bool copy_staged(void *dev, void *host, size_t bytes, bool to_device, cudaStream_t stream, cudaError_t &error) {
    if (bytes < (to_device ? kMinToDevice : kMinToHost) || stream == cudaStreamPerThread || !memory_is(host, cudaMemoryTypeUnregistered)) return false;
    cudaStreamCaptureStatus capturing;
    if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return false;
    }
    CUcontext context = nullptr, owner = nullptr;
    if (!contexts().ok || contexts().get_current(&context) != CUDA_SUCCESS || !context || contexts().of_stream(stream, &owner) != CUDA_SUCCESS ||
        owner != context)
        return false;
    std::unique_lock<std::mutex> lock(g_staging.mutex, std::try_to_lock);
    if (!lock.owns_lock()) return false;
    const RelaxedCapture relaxed;
    if (g_staging.base && !memory_is(g_staging.base, cudaMemoryTypeHost)) g_staging.base = nullptr;   // went with its context (cudaDeviceReset)
    if (!g_staging.base) {
        void *p = nullptr;
        if (cudaHostAlloc(&p, kChunk * kThreads * kSlots, cudaHostAllocPortable) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        g_staging.base = (uint8_t *)p;
    }
    const int threads = (int)std::min<size_t>({(size_t)kThreads, bytes / (2 * kChunk), std::max<size_t>(1, std::thread::hardware_concurrency())});
    cudaError_t results[kThreads] = {};
    auto work = [&](int t) {
        results[t] = copy_chunks(t, threads, (uint8_t *)dev, (uint8_t *)host, bytes, to_device, g_staging.base + t * kSlots * kChunk, stream);
    };
    std::thread pool[kThreads];
    int started = 1;
    try {
        for (; started < threads; ++started)
            pool[started] = std::thread([&, t = started] {
                if (contexts().set_current(context) == CUDA_SUCCESS)
                    work(t);
                else
                    results[t] = cudaErrorInvalidValue;
            });
    } catch (...) {   // no more threads, or no memory for one: this one takes their chunks as well
    }
    work(0);
    for (int t = started; t < threads; ++t) work(t);
    for (int t = 1; t < started; ++t) pool[t].join();
    error = cudaSuccess;
    for (int t = 0; t < threads; ++t)
        if (error == cudaSuccess) error = results[t];
    return true;
}

}  // namespace ttb
