// Arithmetic diagnostics.  Peak microbenchmarks: the roofline denominators for the FP64 / FP32 SIMT
// kernels; each thread runs 8 independent FMA chains; the grid fills every SM several times.
// And the accuracy of the reciprocals of recip.cuh.
#include <cuda_runtime.h>

#include <cmath>

#include "../../../include/gfnff_b200.h"
#include "recip.cuh"

namespace {

template <class T>
__global__ void k_fma_peak(T* out, int iters, T a, T b)
{
    T x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
    for (int k = 0; k < iters; ++k) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
            x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
        }
    }
    const T s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
    if (s == (T)1234.5678) out[0] = s;   // keeps the chains alive
}

template <class T>
double run(int device)
{
    if (cudaSetDevice(device) != cudaSuccess) return -1.0;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    T* out = nullptr;
    if (cudaMalloc(&out, sizeof(T)) != cudaSuccess) return -1.0;
    const int threads = 256, blocks = sms * 8, iters = 2048;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 0.0;
    for (int rep = 0; rep < 4; ++rep) {
        cudaEventRecord(e0);
        k_fma_peak<T><<<blocks, threads>>>(out, iters, (T)0.999999, (T)1e-7);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double flops = 2.0 * 8.0 * 16.0 * iters * (double)threads * blocks;
        if (rep > 0 && ms > 0.f) best = fmax(best, flops / (ms * 1e-3) / 1e12);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    return cudaGetLastError() == cudaSuccess ? best : -1.0;
}

// largest difference from the library function over n arguments, spread evenly over log [lo, hi] with
// their low bits mixed, in units in the last place of the library's result
__global__ void k_recip_ulps(int root, double loglo, double step, long n, double* worst)
{
    double m = 0.0;
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        unsigned h = (unsigned)k * 2654435761u;
        h ^= h >> 15;
        const double x0 = exp(loglo + step * (double)k);
        const double x = __hiloint2double(__double2hiint(x0), (int)(h * 2246822519u));
        const double ref = root ? rsqrt(x) : 1.0 / x, got = root ? rsqrt_pos(x) : rcp_pos(x);
        const double ulp = scalbn(1.0, ilogb(ref) - 52);
        const double d = fabs(got - ref) / ulp;
        m = d > m || !(d == d) ? d : m;
        if (!(d == d)) break;
    }
    // non-negative doubles (and NaN, above them) order like their bits
    atomicMax(reinterpret_cast<unsigned long long*>(worst), (unsigned long long)__double_as_longlong(m) & 0x7fffffffffffffffull);
}

}  // namespace

extern "C" double gfnff_reciprocal_ulps(int device, int root, double lo, double hi, long n)
{
    if (!(lo > 0.0) || !(hi >= lo) || n < 2 || cudaSetDevice(device) != cudaSuccess) return -1.0;
    double *d = nullptr, h = -1.0;
    if (cudaMalloc(&d, sizeof(double)) != cudaSuccess) return -1.0;
    cudaMemset(d, 0, sizeof(double));
    k_recip_ulps<<<1184, 256>>>(root, std::log(lo), (std::log(hi) - std::log(lo)) / (double)(n - 1), n, d);
    if (cudaMemcpy(&h, d, sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) h = -1.0;
    cudaFree(d);
    return h;
}

extern "C" double gfnff_fma_peak_tflops(int device, int fp64)
{
    return fp64 ? run<double>(device) : run<float>(device);
}
