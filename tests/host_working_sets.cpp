// The working sets' cache (StreamCache) on the fake runtime: a request that
// finds no room for a larger buffer fails and leaves nothing behind: the next
// ones work, and no later check finds its error.
#include "fake_cuda.hpp"

#include "common.cuh"

int main() {
    imops::StreamCache cache("test");
    const cudaStream_t s = reinterpret_cast<cudaStream_t>(0x10);
    void* p = nullptr;
    fake::room = 1000;
    EXPECT(cache.get(s, 100, &p) == IMOPS_OK && p);
    EXPECT(cache.get(s, 2000, &p) == IMOPS_ERR_OUT_OF_MEMORY);  // the larger form of a call
    EXPECT(cudaGetLastError() == cudaSuccess);
    EXPECT(cache.get(s, 800, &p) == IMOPS_OK && p);             // and its form with less
    EXPECT(cache.get(s, 100, &p) == IMOPS_OK && p);
    EXPECT(fake::room == 200 && fake::null_frees == 0);
    EXPECT(cache.get(s, 2000, &p) == IMOPS_ERR_OUT_OF_MEMORY);
    EXPECT(cache.get(s, 3000, &p) == IMOPS_ERR_OUT_OF_MEMORY);  // twice in a row
    cache.release_device(0);
    EXPECT(fake::room == 1000 && fake::null_frees == 0);
    EXPECT(cache.get(s, 500, &p) == IMOPS_OK && p);
    return 0;
}
