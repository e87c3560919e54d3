/* The part of the CUDA runtime that host_stage.cuh uses, on host memory: copies are memcpy, and the one that `fake_fail_at` counts
 * down to fails.  Streams are any handles; a use of one that has been destroyed is counted and fails. */
#pragma once
#include <cstdlib>
#include <cstring>
#include <set>

typedef void* cudaStream_t;
typedef void* cudaEvent_t;
enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 999, cudaErrorNotReady = 600 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1 };
constexpr unsigned cudaHostAllocDefault = 0, cudaEventDisableTiming = 2;
inline int fake_fail_at = -1, fake_dead_uses = 0;
inline std::set<cudaStream_t> fake_dead;
inline cudaError_t fake_stream(cudaStream_t s) { return fake_dead.count(s) ? (++fake_dead_uses, cudaErrorUnknown) : cudaSuccess; }

inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::aligned_alloc(4096, n); return *p ? cudaSuccess : cudaErrorUnknown; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = e; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { return fake_stream(s); }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { const cudaError_t e = fake_stream(s); fake_dead.insert(s); return e; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) { return fake_stream(s); }
inline cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t stream) {
    if (fake_stream(stream) != cudaSuccess) return cudaErrorUnknown;
    if (fake_fail_at >= 0 && fake_fail_at-- == 0) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
