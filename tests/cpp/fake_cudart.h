// A stand-in for the CUDA runtime calls that the host code's buffers and tables use, for tests without a GPU.
// "Device" memory is host memory.  A copy from pageable memory takes its source at the call and arrives
// only when its own stream (or the device) is synchronised, as CUDA allows: cudaMemcpy uses the legacy
// stream, which the program's streams do not wait for.  Failures are injected by call; a failed call
// leaves its error for cudaGetLastError, which clears it.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>
#include <vector>

#include "engine.h"

namespace fake {
struct Copy
{
    char* dst;
    std::vector<char> data;
};
inline std::map<cudaStream_t, std::vector<Copy>> pending;
inline std::map<void*, size_t> device;  // allocations
inline size_t largest = ~size_t(0);     // larger allocations fail
inline int failCopies = 0, failAllocs = 0;
inline cudaError_t last = cudaSuccess;

inline cudaError_t done(cudaError_t e)
{
    if (e != cudaSuccess) last = e;
    return e;
}
inline cudaError_t alloc(void** p, size_t n)
{
    if (n > largest || failAllocs > 0)
    {
        if (failAllocs > 0) --failAllocs;
        return done(cudaErrorMemoryAllocation);
    }
    *p = std::malloc(n ? n : 1);
    std::memset(*p, 0xa5, n);
    device[*p] = n;
    return cudaSuccess;
}
inline cudaError_t release(void* p)
{
    device.erase(p);
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t copy(void* dst, const void* src, size_t n, cudaStream_t s)
{
    if (failCopies > 0)
    {
        --failCopies;
        return done(cudaErrorInvalidValue);
    }
    const char* c = static_cast<const char*>(src);
    pending[s].push_back(Copy{static_cast<char*>(dst), std::vector<char>(c, c + n)});
    return cudaSuccess;
}
inline void arrive(cudaStream_t s)
{
    for (const Copy& c : pending[s]) std::memcpy(c.dst, c.data.data(), c.data.size());
    pending[s].clear();
}
inline bool inFlight()
{
    for (const auto& kv : pending)
        if (!kv.second.empty()) return true;
    return false;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return fake::alloc(p, n); }
cudaError_t cudaFree(void* p) { return fake::release(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return fake::release(p); }
cudaError_t cudaMallocHost(void** p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return fake::release(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return fake::copy(d, s, n, nullptr); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    return fake::copy(d, s, n, st);
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return fake::arrive(s), cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return std::exchange(fake::last, cudaSuccess); }
const char* cudaGetErrorString(cudaError_t) { return "injected"; }
}

namespace cf {
Slot::~Slot() {}
Context::~Context() {}
}  // namespace cf
