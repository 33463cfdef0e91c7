// fake_cuda.hpp -- the CUDA runtime calls that common.cu makes, on host memory,
// for tests of its host logic without a GPU, on as many devices as a test names.
// "Device" memory is malloc'd; copies run at once.  A null pointer given to
// cudaFreeAsync is an error, as only cudaFree documents it as nothing to do.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#define EXPECT(x) \
    if (!(x)) return std::printf("line %d: %s\n", __LINE__, #x), 1

namespace fake {

inline thread_local int device = 0;                  // cudaSetDevice's
inline thread_local cudaError_t last = cudaSuccess;  // cudaGetLastError's
inline size_t room = (size_t)-1;                     // device bytes left for cudaMallocAsync
inline std::atomic<int> null_frees{0}, streams{0}, events{0}, pinned{0};  // the last three: alive
inline void (*on_copy)(void* dst, size_t bytes) = nullptr;
inline void (*on_event_wait)() = nullptr;
inline void (*on_host_alloc)() = nullptr;
inline std::mutex mu;
struct Block {
    size_t bytes;
    int dev;
};
inline std::map<void*, Block> blocks;  // live device memory, by its start

inline cudaError_t failed(cudaError_t e) { return last = e; }

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

cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) {
    std::lock_guard<std::mutex> lock(fake::mu);
    if (bytes > fake::room) return fake::failed(cudaErrorMemoryAllocation);
    fake::room -= bytes;
    *p = std::malloc(bytes);
    fake::blocks[*p] = {bytes, fake::device};
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lock(fake::mu);
    if (!p) return cudaSuccess;
    fake::room += fake::blocks.at(p).bytes;
    fake::blocks.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    if (!p) return fake::null_frees++, fake::failed(cudaErrorInvalidValue);
    return cudaFree(p);
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    fake::streams++;
    return *s = reinterpret_cast<cudaStream_t>(std::malloc(1)), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return fake::streams--, std::free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }

// An event holds the device it was made on, the only one it can be recorded on.
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    fake::events++;
    return *e = reinterpret_cast<cudaEvent_t>(new int(fake::device)), cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { return fake::events--, delete reinterpret_cast<int*>(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    return *reinterpret_cast<int*>(e) == fake::device ? cudaSuccess : fake::failed(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    if (fake::on_event_wait) fake::on_event_wait();
    return cudaSuccess;
}

cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    if (fake::on_host_alloc) fake::on_host_alloc();
    return fake::pinned++, *p = std::malloc(bytes), cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return fake::pinned--, std::free(p), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> lock(fake::mu);
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    auto b = fake::blocks.upper_bound(const_cast<void*>(p));
    if (b != fake::blocks.begin() && static_cast<const char*>((--b)->first) + b->second.bytes > p) {
        a->type = cudaMemoryTypeDevice;
        a->device = b->second.dev;
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    if (fake::on_copy) fake::on_copy(dst, bytes);
    return std::memcpy(dst, src, bytes), cudaSuccess;
}

}  // extern "C"
