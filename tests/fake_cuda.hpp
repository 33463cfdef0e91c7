// fake_cuda.hpp -- the CUDA runtime calls that common.cu makes, on host memory,
// for tests of its host logic without a GPU.  "Device" memory is malloc'd;
// copies run at once.  A null pointer given to cudaFreeAsync is an error, as
// only cudaFree documents it as nothing to do.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace fake {

inline thread_local int device = 0;              // cudaSetDevice's
inline size_t room = (size_t)-1;                 // device bytes left for cudaMallocAsync
inline std::atomic<int> null_frees{0};           // cudaFreeAsync(nullptr)
inline thread_local cudaError_t last = cudaSuccess;  // cudaGetLastError's
inline std::mutex mu;

// Sizes of the live allocations, kept before each block.
inline void* alloc(size_t bytes) {
    char* p = static_cast<char*>(std::malloc(bytes + 16));
    std::memcpy(p, &bytes, sizeof bytes);
    return p + 16;
}
inline void release(void* q) {
    char* p = static_cast<char*>(q) - 16;
    size_t bytes;
    std::memcpy(&bytes, p, sizeof bytes);
    room += bytes;
    std::free(p);
}

}  // namespace fake

extern "C" {

cudaError_t cudaGetDevice(int* d) { return *d = fake::device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return fake::device = d, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
const char* cudaGetErrorName(cudaError_t) { return "cudaErrorFake"; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) {
    std::lock_guard<std::mutex> lock(fake::mu);
    if (bytes > fake::room) return fake::last = cudaErrorMemoryAllocation;
    fake::room -= bytes;
    return *p = fake::alloc(bytes), cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    std::lock_guard<std::mutex> lock(fake::mu);
    if (!p) return fake::null_frees++, fake::last = cudaErrorInvalidValue;
    return fake::release(p), cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lock(fake::mu);
    if (p) fake::release(p);
    return cudaSuccess;
}

// Defined by the tests of downloads.
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p);
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned flags);
cudaError_t cudaFreeHost(void* p);
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned flags);
cudaError_t cudaEventDestroy(cudaEvent_t e);
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s);
cudaError_t cudaEventSynchronize(cudaEvent_t e);
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t s);

}  // extern "C"
