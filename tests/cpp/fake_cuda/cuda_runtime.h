// Stand-in for the parts of the CUDA runtime that csrc/pt_hostcopy.cuh uses, on
// the host: copies are done at once, and the calls that matter are counted.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <cstring>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2 };
using cudaStream_t = struct FakeStream*;
using cudaEvent_t = struct FakeEvent*;
inline const cudaStream_t cudaStreamPerThread = reinterpret_cast<cudaStream_t>(2);
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
struct cudaPointerAttributes {
    cudaMemoryType type;
};
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone = 0, cudaStreamCaptureStatusActive = 1 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
constexpr unsigned int cudaHostAllocDefault = 0, cudaEventDisableTiming = 2;

namespace fake {
inline std::atomic<int> hostAllocs{0}, hostFrees{0}, copies{0};
inline std::atomic<int> failCopyAt{-1}; // the copy with this number fails
inline std::atomic<bool> hostAllocFails{false}, capturing{false};
inline const void* pinned = nullptr; // start of a host array that counts as pinned
} // namespace fake

inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    a->type = p == fake::pinned && p != nullptr ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s)
{
    *s = fake::capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (fake::copies++ == fake::failCopyAt) {
        return cudaErrorInvalidValue;
    }
    std::memcpy(to, from, n);
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int)
{
    ++fake::hostAllocs;
    *p = fake::hostAllocFails ? nullptr : std::malloc(n);
    return *p != nullptr ? cudaSuccess : cudaErrorMemoryAllocation;
}
inline cudaError_t cudaFreeHost(void* p)
{
    ++fake::hostFrees;
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int)
{
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
