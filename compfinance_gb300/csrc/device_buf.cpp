// Device and pinned host buffers, and the thread's last error.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "engine.h"

namespace cf {

thread_local std::string g_lastError;

int fail(int code, const std::string& msg)
{
    g_lastError = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* what)
{
    return fail(e == cudaErrorMemoryAllocation ? CF_E_NOMEM : CF_E_CUDA,
                std::string(what) + ": " + cudaGetErrorString(e));
}

std::atomic<unsigned long long> DevBuf::growths{0};

// A failed allocation as a status.  The runtime also keeps it as the thread's last error, which would be taken
// for a failure of the next kernel launch that asks for one: callers may go on with a smaller form.
static int alloc_fail(cudaError_t e, const char* what)
{
    cudaGetLastError();
    return cuda_fail(e, what);
}

int DevBuf::ensure(size_t n, cudaStream_t stream)
{
    if (n <= bytes) return CF_OK;
    ++growths;
    const size_t want = n + n / 4;
    cudaError_t e;
    if (stream)
    {
        // the old buffer is freed after the stream's earlier work, the new one is ready for its later work
        if (ptr) cudaFreeAsync(ptr, stream);
        ptr = nullptr;
        bytes = 0;
        e = cudaMallocAsync(&ptr, want, stream);
    }
    else
    {
        release();
        e = cudaMalloc(&ptr, want);
    }
    if (e != cudaSuccess)
    {
        ptr = nullptr;
        bytes = 0;
        return alloc_fail(e, "cudaMalloc");
    }
    bytes = want;
    return CF_OK;
}

int DevBuf::upload(const void* src, size_t n, cudaStream_t stream, size_t at)
{
    if (!n) return CF_OK;
    cudaError_t e = cudaMemcpyAsync(static_cast<char*>(ptr) + at, src, n, cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e == cudaSuccess ? CF_OK : cuda_fail(e, "table upload");
}

void DevBuf::release()
{
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
}

int PinnedBuf::ensure(size_t n)
{
    if (n <= bytes) return CF_OK;
    release();
    // at least 16 MB (the finished risks of a 200-payoff portfolio on a 120x60 grid are 11.5 MB):
    // freeing pinned memory waits for the device, so a serving slot should not regrow it
    const size_t want = std::max(n + n / 4, size_t(16) << 20);
    cudaError_t e = cudaMallocHost(&ptr, want);
    if (e != cudaSuccess)
    {
        ptr = nullptr;
        bytes = 0;
        return alloc_fail(e, "cudaMallocHost");
    }
    bytes = want;
    return CF_OK;
}

void PinnedBuf::release()
{
    if (ptr) cudaFreeHost(ptr);
    ptr = nullptr;
    bytes = 0;
}

}  // namespace cf
