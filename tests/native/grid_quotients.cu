// Test harness: the 3D resistive EMF and Div::quot_grid in FP32, built with the
// flags of the FP32 kernels, beside the same expressions written as divisions,
// for tests/test_gpu_grid_quotients.py.  All arrays are host memory of n floats.
#include <cuda_runtime.h>

#include "mhd3d_kernels.cuh"

using namespace ccb;

namespace {
__host__ __device__ float by_grid(float a, float b, float y) {
    return divided<float>([&](auto& d) { return d.quot_grid(a, b, y); });
}

__global__ void grid_quotients_kernel(const float* d1, const float* d2, long n, float h1, float h2, float i1, float i2, float eta,
                                      float* out) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    M3Const<float> c{};
    c.eta = eta;
    out[i] = by_grid(d1[i], h1, i1);
    out[n + i] = d1[i] / h1;
    out[2 * n + i] = m3_resistive_emf(c, d1[i], h1, i1, d2[i], h2, i2);
    const float a = d1[i] / h1, b = d2[i] / h2;
    out[3 * n + i] = eta * (a - b);
    out[4 * n + i] = d1[i] * i1;
}
}  // namespace

// out: quot_grid, the division, the EMF, the EMF by divisions, the product with the reciprocal.  0, or a cudaError_t.
extern "C" int grid_quotients(const float* d1, const float* d2, long n, const double* h, double eta, float* out) {
    if (n < 1 || n > (1L << 24)) return (int)cudaErrorInvalidValue;
    const size_t bytes = sizeof(float) * (size_t)n;
    float* d = nullptr;
    cudaError_t e = cudaMalloc(&d, 7 * bytes);
    if (e == cudaSuccess) e = cudaMemcpy(d, d1, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, d2, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        grid_quotients_kernel<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, n, (float)h[0], (float)h[1], (float)(1.0 / h[0]),
                                                                    (float)(1.0 / h[1]), (float)eta, d + 2 * n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, 5 * bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
