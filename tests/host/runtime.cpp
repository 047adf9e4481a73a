#include "runtime.h"

#include <cstdlib>
#include <cstring>

namespace fake {
long allocations = 0, fail_at = -1, fail_on = 0, syncs = 0;
std::map<void*, size_t> live;

static cudaError_t take(void** p, size_t bytes) {
    const long k = allocations++;
    if (fail_at >= 0 && (k == fail_at || (fail_on && k > fail_at))) return cudaErrorMemoryAllocation;
    *p = std::aligned_alloc(256, (bytes + 511) & ~(size_t)255);
    for (size_t i = 0; i < bytes / 4 + 1; ++i) static_cast<uint32_t*>(*p)[i] = 1u;
    live[*p] = bytes;
    return cudaSuccess;
}
static cudaError_t give(void* p) {
    if (!p) return cudaSuccess;
    if (!live.erase(p)) std::abort();
    std::free(p);
    return cudaSuccess;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake::take(p, n); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return fake::take(p, n); }
cudaError_t cudaFree(void* p) { return fake::give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return fake::give(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = std::calloc(1, n);
    fake::live[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return fake::give(p); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    ++fake::syncs;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1 << 16;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
const char* cudaGetErrorName(cudaError_t) { return "refused"; }
}
