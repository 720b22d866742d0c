// The few runtime calls host_copy.h makes, on host memory: copies are complete on
// return, every pointer is pageable, no stream is captured.
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone = 0, cudaStreamCaptureStatusActive = 1 };
struct cudaPointerAttributes { cudaMemoryType type; };
using cudaStream_t = void *;
using cudaEvent_t = void *;
constexpr unsigned cudaEventDisableTiming = 2, cudaHostAllocPortable = 1;

inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s)
{
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    *p = std::malloc(n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
inline cudaError_t cudaFreeHost(void *p)
{
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    *e = std::malloc(1);
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    std::free(e);
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
