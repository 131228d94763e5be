// Allocation of the device buffers of a context.
//
// dev_malloc is cudaMalloc, except that the environment variable
// TJ_FAIL_ALLOC=n makes the n-th call from the time the variable got that value
// (n+: and every later one) return cudaErrorMemoryAllocation without allocating:
// the error paths are tested without filling a GPU's memory. A failure leaves no
// pending runtime error, so a caller that has a smaller way may go on.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <mutex>
#include <string>

namespace tj {

inline bool alloc_fails_by_request()
{
    const char* v = std::getenv("TJ_FAIL_ALLOC");
    if (!v || !*v) return false;
    static std::mutex m;
    static std::string seen;
    static long calls = 0;
    std::lock_guard<std::mutex> lock(m);
    if (seen != v) {
        seen = v;
        calls = 0;
    }
    char* end = nullptr;
    const long n = std::strtol(v, &end, 10);
    return ++calls == n || (*end == '+' && calls > n);
}

template <class T>
inline cudaError_t dev_malloc(T** p, size_t bytes)
{
    if (alloc_fails_by_request()) return cudaErrorMemoryAllocation;
    const cudaError_t e = cudaMalloc(reinterpret_cast<void**>(p), bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace tj
