// The few CUDA runtime calls of csrc/dsmc_hostlink.h on the host, counted, for
// a CPU test of it: copies are done when they are issued, page-locking
// changes nothing, and can be made to fail.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <cstring>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
typedef struct FakeStream* cudaStream_t;
typedef struct FakeEvent* cudaEvent_t;
enum { cudaHostRegisterDefault = 0, cudaEventDisableTiming = 2 };

namespace fake {
inline bool failRegister = false;
inline int registered = 0;
inline size_t registeredBytes = 0;
inline std::atomic<int> events{0};
inline cudaError_t lastError = cudaSuccess;
}  // namespace fake

inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError()
{
    const cudaError_t e = fake::lastError;
    fake::lastError = cudaSuccess;
    return e;
}
inline cudaError_t cudaHostRegister(void* p, size_t n, unsigned)
{
    if (fake::failRegister || !p || !n) return fake::lastError = cudaErrorMemoryAllocation;
    ++fake::registered;
    fake::registeredBytes += n;
    return cudaSuccess;
}
inline cudaError_t cudaHostUnregister(void* p)
{
    --fake::registered;
    return p ? cudaSuccess : cudaErrorInvalidValue;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    ++fake::events;
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    std::free(e);
    --fake::events;
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e ? cudaSuccess : cudaErrorInvalidValue; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) { return e ? cudaSuccess : cudaErrorInvalidValue; }
