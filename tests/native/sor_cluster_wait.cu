// Test harness: sor_cluster_kernel<2> with a given limit on its waits, for
// tests/test_gpu_sor_cluster_wait.py.  rhs and phi are host memory of nx*ny doubles.
#include <cuda_runtime.h>

#include "poisson_kernels.cuh"

using namespace ccb;

// err: the kernel's error flag; iters: its sweeps.  0, or a cudaError_t.
extern "C" int sor_cluster_wait(int nx, int ny, int max_iter, double tol, int max_polls, const double* rhs, double* phi, int* err,
                                int* iters) {
    const int half = (nx + 1) / 2, M = half * ny, S = 2 * SOR_CL_NT, nb = (M + 1023) / 1024, nc = (M + S - 1) / S;
    if (nx < 4 || ny < 4 || (nx & 1) || (ny & 1) || half > S || nc > SOR_CL_MAXC) return (int)cudaErrorInvalidValue;
    const size_t n = (size_t)nx * ny, smem = sor_cluster_smem(S, half, nb);
    if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
    double* d = nullptr;
    int* fl = nullptr;
    cudaError_t e = cudaMalloc(&d, (2 * n + 1) * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&fl, 2 * sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(d, rhs, n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(fl, 0, 2 * sizeof(int));
    const void* fn = (const void*)sor_cluster_kernel<2>;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) {
        SorArgs a{};
        a.nx = nx; a.ny = ny;
        a.ax = AxisMap{nx, 1}; a.ay = AxisMap{ny, 1};
        a.idx2 = a.idy2 = 1.0; a.denom = 4.0; a.omega = 1.7; a.tol = tol;
        a.max_iter = max_iter;
        a.rhs = d; a.phi = d + n; a.res_out = d + 2 * n;
        a.bar.err = fl; a.iters_out = fl + 1;
        a.max_polls = max_polls;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = nc; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(nc); cfg.blockDim = dim3(SOR_CL_NT); cfg.dynamicSmemBytes = smem;
        cfg.attrs = at; cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, sor_cluster_kernel<2>, a);
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    int f[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpy(f, fl, sizeof(f), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(phi, d + n, n * sizeof(double), cudaMemcpyDeviceToHost);
    *err = f[0];
    *iters = f[1];
    cudaFree(d);
    cudaFree(fl);
    return (int)e;
}
