// A stand-in for the CUDA runtime, preloaded in front of libcudart so that the library's host code
// runs without a GPU: device memory is host memory, launches do nothing, and the calls that a
// test names return an error. Only the calls that librtc8_gb300.so makes are here.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

namespace {
std::mutex g_mutex;
std::map<void*, size_t> g_live;  // device allocations
size_t g_bytes = 0, g_limit = static_cast<size_t>(1) << 40;
int g_fail[5] = {0, 0, 0, 0, 0};  // calls of a kind until they fail, 0 = none fails
int g_calls[5] = {0, 0, 0, 0, 0};
cudaError_t g_last = cudaSuccess;  // what cudaGetLastError reports once

bool fails(int kind) {
    std::lock_guard<std::mutex> lock(g_mutex);
    ++g_calls[kind];
    if (g_fail[kind] > 1) --g_fail[kind];
    else return g_fail[kind] == 1;
    return false;
}
cudaError_t take(void** p, size_t bytes) {
    if (fails(0)) return g_last = cudaErrorMemoryAllocation;
    std::lock_guard<std::mutex> lock(g_mutex);
    if (g_bytes + bytes > g_limit) return g_last = cudaErrorMemoryAllocation;
    *p = std::calloc(1, bytes ? bytes : 1);
    g_live[*p] = bytes;
    g_bytes += bytes;
    return cudaSuccess;
}
cudaError_t give(void* p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> lock(g_mutex);
    auto it = g_live.find(p);
    if (it == g_live.end()) return cudaErrorInvalidValue;
    g_bytes -= it->second;
    g_live.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t launch() {
    return fails(3) ? g_last = cudaErrorLaunchOutOfResources : cudaSuccess;
}
}  // namespace

extern "C" {
// What a test sets and reads. Kinds: 0 allocation, 1 copy, 2 free-memory query, 3 launch, 4 memset. The
// nth call of a kind from now and all after it fail until nth = 0 is set.
void fake_fail(int kind, int nth) { g_fail[kind] = nth; }
int fake_calls(int kind) { return g_calls[kind]; }
void fake_limit(size_t bytes) { g_limit = bytes; }
size_t fake_bytes() { return g_bytes; }

cudaError_t cudaMalloc(void** p, size_t bytes) { return take(p, bytes); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaMallocHost(void** p, size_t bytes) {
    *p = std::calloc(1, bytes ? bytes : 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*) {
    *pool = reinterpret_cast<cudaMemPool_t>(&g_live);
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t bytes, cudaMemPool_t, cudaStream_t) { return take(p, bytes); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) {
    if (fails(2)) return g_last = cudaErrorInvalidValue;
    *free_bytes = g_limit > g_bytes ? g_limit - g_bytes : 0;
    *total = g_limit;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t bytes, cudaMemcpyKind) {
    if (fails(1)) return g_last = cudaErrorInvalidValue;
    std::memcpy(dst, src, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t) {
    return cudaMemcpy(dst, src, bytes, kind);
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void* p, int value, size_t bytes) {
    if (fails(4)) return g_last = cudaErrorInvalidValue;
    std::memset(p, value, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int value, size_t bytes, cudaStream_t) { return cudaMemset(p, value, bytes); }

cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return launch(); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return launch(); }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return launch(); }
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void* entry) {
    *kernel = reinterpret_cast<cudaKernel_t>(const_cast<void*>(entry));
    return cudaSuccess;
}

cudaError_t cudaGetDevice(int* device) {
    *device = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr, int) {
    *value = 4;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* status) {
    *status = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* blocks, const void*, int, size_t) {
    *blocks = 1;
    return cudaSuccess;
}
}
