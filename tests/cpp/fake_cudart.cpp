#include "fake_cudart.hpp"

#include <cuda_runtime_api.h>
#include <malloc.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <vector>

// Freed memory does not keep its contents.
void operator delete(void *p) noexcept {
    if (p) std::memset(p, 0xDD, malloc_usable_size(p));
    std::free(p);
}
void operator delete(void *p, std::size_t) noexcept { operator delete(p); }
void *operator new(std::size_t n) {
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}

namespace {

std::recursive_mutex mutex;
std::vector<std::function<void()>> queue;
long long stale = 0, launched = 0, fail_in = 0;
unsigned long long largest_allocation = ~0ull;

using Lock = std::lock_guard<std::recursive_mutex>;

void enqueue(std::function<void()> work) {
    Lock lock(mutex);
    queue.push_back(std::move(work));
}

std::uint64_t digest(const void *p, std::size_t n) {
    std::uint64_t h = 1469598103934665603ull;
    for (std::size_t i = 0; i < n; ++i) h = (h ^ static_cast<const unsigned char *>(p)[i]) * 1099511628211ull;
    return h;
}

cudaError_t launch() {
    Lock lock(mutex);
    ++launched;
    return fail_in > 0 && --fail_in == 0 ? cudaErrorLaunchOutOfResources : cudaSuccess;
}

cudaError_t handle(void *out) {
    static std::uintptr_t next = 0;
    Lock lock(mutex);
    next += 16;
    *static_cast<std::uintptr_t *>(out) = next;
    return cudaSuccess;
}

cudaError_t last = cudaSuccess;

}  // namespace

namespace fake {

void run_queued() {
    Lock lock(mutex);
    for (auto &work : queue) work();
    queue.clear();
}
long long stale_sources() { return stale; }
void fail_launch(long long n) { fail_in = n; }
long long launches() { return launched; }
void limit_allocations(unsigned long long bytes) { largest_allocation = bytes; }

}  // namespace fake

extern "C" {

void **__cudaRegisterFatBinary(void *) {
    static void *h = nullptr;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = *block = dim3{1, 1, 1};
    *smem = 0;
    *static_cast<cudaStream_t *>(stream) = nullptr;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *kernel, const void *f) {
    *kernel = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t) { return last = launch(); }
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return launch(); }

cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "an error of the stand-in"; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceGetPCIBusId(char *s, int n, int) {
    std::strncpy(s, "0", std::size_t(n));
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof *p);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    return *n = 2, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    static unsigned long long scratch[1024];
    return *p = scratch, cudaSuccess;
}

cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = std::calloc(n ? n : 1, 1), cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) {
    if (n > largest_allocation) return last = cudaErrorMemoryAllocation;
    return cudaHostAlloc(p, n, 0);
}
// memory that queued work may still name is not handed out again
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaFreeHost(void *) { return cudaSuccess; }

cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    const std::uint64_t before = kind == cudaMemcpyHostToDevice ? digest(from, n) : 0;
    enqueue([=] {
        if (kind == cudaMemcpyHostToDevice && digest(from, n) != before) ++stale;
        std::memcpy(to, from, n);
    });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *to, const void *from, size_t n, cudaMemcpyKind) {
    fake::run_queued();
    std::memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
    enqueue([=] { std::memset(p, v, n); });
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    fake::run_queued();
    std::memset(p, v, n);
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return fake::run_queued(), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return fake::run_queued(), cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }

// no graphs
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"
