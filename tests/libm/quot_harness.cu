// Test harness (not part of the library): the integer-pipe binary64 division
// and square root of tenjin_gb300/csrc/tj_quot.h beside the language's own, on
// the host (any C++ compiler; the seeds moved by `ulps`) or on the GPU (nvcc).
#ifndef __CUDACC__
#define TJQ_TEST_SEED
#endif
#include "tj_quot.h"

#ifndef __CUDACC__
namespace tj {
int tjq_seed_ulps = 0;
}

extern "C" int tjq_eval(const double* a, const double* b, int n, int ulps, double* q, double* q0, double* r, double* r0)
{
    tj::tjq_seed_ulps = ulps;
    for (int i = 0; i < n; ++i) {
        q[i] = tj::tjq_div(a[i], b[i]);
        q0[i] = a[i] / b[i];
        r[i] = tj::tjq_sqrt(a[i]);
        r0[i] = std::sqrt(a[i]);
    }
    return 0;
}
extern "C" int tjq_convert(const double* a, int n, float* f, float* f0, double* w, double* w0)
{
    for (int i = 0; i < n; ++i) {
        f[i] = tj::narrow(a[i]);
        f0[i] = (float)a[i];
        w[i] = tj::widen(f0[i]);
        w0[i] = (double)f0[i];
    }
    return 0;
}
#else
__global__ void k_convert(const double* a, int n, float* f, double* w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    f[i] = tj::narrow(a[i]);
    f[n + i] = (float)a[i];
    w[i] = tj::widen(f[n + i]);
    w[n + i] = (double)f[n + i];
}

extern "C" int tjq_convert(const double* a, int n, float* f, float* f0, double* w, double* w0)
{
    double* d = nullptr;
    const size_t m = (size_t)n;
    if (cudaMalloc(&d, sizeof(double) * 4 * m) != cudaSuccess) return -1;
    float* df = reinterpret_cast<float*>(d + 3 * m);
    cudaMemcpy(d, a, sizeof(double) * m, cudaMemcpyHostToDevice);
    k_convert<<<(n + 255) / 256, 256>>>(d, n, df, d + m);
    cudaMemcpy(f, df, sizeof(float) * m, cudaMemcpyDeviceToHost);
    cudaMemcpy(f0, df + m, sizeof(float) * m, cudaMemcpyDeviceToHost);
    cudaMemcpy(w, d + m, sizeof(double) * m, cudaMemcpyDeviceToHost);
    cudaMemcpy(w0, d + 2 * m, sizeof(double) * m, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaFree(d);
    return e == cudaSuccess ? 0 : -2;
}

__global__ void k_eval(const double* a, const double* b, int n, double* o)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = tj::tjq_div(a[i], b[i]);
    o[n + i] = a[i] / b[i];
    o[2 * (size_t)n + i] = tj::tjq_sqrt(a[i]);
    o[3 * (size_t)n + i] = sqrt(a[i]);
}

extern "C" int tjq_eval(const double* a, const double* b, int n, int, double* q, double* q0, double* r, double* r0)
{
    double* d = nullptr;
    const size_t m = (size_t)n, bytes = sizeof(double) * m;
    if (cudaMalloc(&d, 6 * bytes) != cudaSuccess) return -1;
    cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(d + m, b, bytes, cudaMemcpyHostToDevice);
    k_eval<<<(n + 255) / 256, 256>>>(d, d + m, n, d + 2 * m);
    double* out[4] = {q, q0, r, r0};
    for (int k = 0; k < 4; ++k) cudaMemcpy(out[k], d + (2 + k) * m, bytes, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaFree(d);
    return e == cudaSuccess ? 0 : -2;
}
#endif
