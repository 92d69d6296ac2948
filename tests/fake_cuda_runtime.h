// Stand-in for the few CUDA runtime calls of csrc/hostcopy.cuh, for
// tests/hostcopy_check.cpp (included there as <cuda_runtime.h>): "device"
// memory is host memory, copies happen at once, waits and the order of calls
// are counted.
#pragma once
#include <atomic>
#include <cstdlib>
#include <cstring>

enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyDeviceToHost = 2 };
typedef int* cudaStream_t;
typedef int* cudaEvent_t;
constexpr unsigned cudaEventDisableTiming = 2;

namespace fake {
inline std::atomic<int> waits{0}, copies{0}, copies_before_wait{0};
inline bool no_pinned = false;
inline long fail_copy = -1;  // index of the copy that fails
inline void reset() {
    waits = copies = copies_before_wait = 0;
    no_pinned = false;
    fail_copy = -1;
}
}  // namespace fake

inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaMallocHost(void** p, size_t n) {
    if (fake::no_pinned) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
inline cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = static_cast<int*>(std::malloc(sizeof(int)));
    return *e ? cudaSuccess : cudaErrorMemoryAllocation;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) {
    ++fake::waits;
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fake::waits == 0) ++fake::copies_before_wait;
    if (fake::copies++ == fake::fail_copy) return cudaErrorUnknown;
    std::memcpy(dst, src, n);
    return cudaSuccess;
}
