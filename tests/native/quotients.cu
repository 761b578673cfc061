// Test harness: the branch-free FP64 reciprocals and quotients of cc_device.cuh
// on arrays of operands, one thread an operand pair, for
// tests/test_gpu_quotient_bits.py.  All arrays are host memory of n doubles.
#include <cuda_runtime.h>

#include "cc_device.cuh"

using namespace ccb;

namespace {
struct Out { double *start, *recip, *fast, *quot, *div, *by; unsigned char* inside; };

__host__ __device__ double by_div(double a, double b) {
    return divided<double>([&](auto& d) { return d.div(a, b); });
}
__host__ __device__ double by_quot_by(double a, double b, double y) {
    return divided<double>([&](auto& d) { return d.quot_by(a, b, y); });
}

__global__ void quotients_kernel(const double* a, const double* b, long n, Out o) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double y = recip_fast(b[i]);
    o.start[i] = recip_start(b[i]);
    o.recip[i] = y;
    o.fast[i] = quotient_fast(a[i], b[i], y);
    o.quot[i] = quotient(a[i], b[i], 1.0 / b[i]);
    o.div[i] = by_div(a[i], b[i]);
    o.by[i] = by_quot_by(a[i], b[i], 1.0 / b[i]);
    o.inside[i] = (unsigned char)((divisor_inside(b[i]) ? 1 : 0) | (quotient_inside(a[i]) ? 2 : 0));
}
}  // namespace

// out: start, recip, fast, quot, div, by.  0, or a cudaError_t.
extern "C" int quotients(const double* a, const double* b, long n, double* const* out, unsigned char* inside) {
    if (n < 1 || n > (1L << 24)) return (int)cudaErrorInvalidValue;
    const size_t bytes = sizeof(double) * (size_t)n;
    double* d = nullptr;
    unsigned char* m = nullptr;
    cudaError_t e = cudaMalloc(&d, 8 * bytes);
    if (e == cudaSuccess) e = cudaMalloc(&m, (size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        quotients_kernel<<<(unsigned)((n + 255) / 256), 256>>>(
            d, d + n, n, Out{d + 2 * n, d + 3 * n, d + 4 * n, d + 5 * n, d + 6 * n, d + 7 * n, m});
        e = cudaGetLastError();
    }
    for (int k = 0; k < 6 && e == cudaSuccess; k++) e = cudaMemcpy(out[k], d + (2 + k) * n, bytes, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(inside, m, (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(m);
    return (int)e;
}
