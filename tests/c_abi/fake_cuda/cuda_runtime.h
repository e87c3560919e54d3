/* The part of the CUDA runtime that host_stage.cuh uses, on host memory: copies are memcpy, and the one that `fake_fail_at` counts
 * down to fails. */
#pragma once
#include <cstdlib>
#include <cstring>

typedef void* cudaStream_t;
typedef void* cudaEvent_t;
enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 999, cudaErrorNotReady = 600 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1 };
constexpr unsigned cudaHostAllocDefault = 0, cudaEventDisableTiming = 2;
inline int fake_fail_at = -1;

inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::aligned_alloc(4096, n); return *p ? cudaSuccess : cudaErrorUnknown; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = e; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fake_fail_at >= 0 && fake_fail_at-- == 0) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
