// The few runtime calls of device/arena.hpp on host memory, counted, with a
// limit on what may be allocated (for tests that run without a GPU).
#pragma once
#include <cstddef>
#include <cstdlib>
#include <map>

enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };

struct FakeMemory {
    std::map<void *, size_t> live;
    size_t bytes = 0, limit = ~size_t(0);
    int mallocs = 0, frees = 0, errors_cleared = 0;
};
inline FakeMemory fake;

inline cudaError_t cudaMalloc(void **p, size_t n) {
    if (fake.bytes + n > fake.limit) return cudaErrorMemoryAllocation;
    *p = std::malloc(64);                       // the address only
    fake.live[*p] = n;
    fake.bytes += n;
    ++fake.mallocs;
    return cudaSuccess;
}

inline cudaError_t cudaFree(void *p) {
    auto it = fake.live.find(p);
    if (it == fake.live.end()) std::abort();    // freed twice, or never allocated
    fake.bytes -= it->second;
    std::free(p);
    fake.live.erase(it);
    ++fake.frees;
    return cudaSuccess;
}

inline cudaError_t cudaGetLastError() {
    ++fake.errors_cleared;
    return cudaSuccess;
}
