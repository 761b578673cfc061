// Precision-independent kernels and launchers: dt finalisation, the device
// clock, and the cooperative red-black SOR.  Built with -fmad=false (FP64
// arithmetic that must round like the reference).
#include "mhd2d_launch.h"

namespace ccb {

__global__ void m2_dt_finalize_kernel(const double* __restrict__ spd_part, int nparts, DtSpec d,
                                      double* __restrict__ dt_out, const double* __restrict__ t_now,
                                      int* __restrict__ active) {
    if (threadIdx.x >= 32 || blockIdx.x != 0) return;
    // one warp: each lane folds a strided share of the partials into the seed
    // (a NaN partial never wins), then the lanes' maxima are combined; max is
    // exact, so the order does not matter
    double maxs = d.seed;
    for (int b = threadIdx.x; b < nparts; b += 32) maxs = vmax(maxs, spd_part[b]);
    for (int o = 16; o > 0; o >>= 1) maxs = vmax(maxs, __shfl_xor_sync(0xffffffffu, maxs, o));
    if (threadIdx.x != 0) return;
    const double dt_h = d.cfl * d.hmin / maxs;
    double dt = dt_h;
    if (d.cap) {
        double dt_r = 1e100;
        if (d.eta > 0.0) dt_r = 0.25 * d.hmin * d.hmin / d.eta;
        dt = vmin(dt_h, dt_r);
    }
    if (d.clamp_to_end) {
        const double t = *t_now;
        if (!(t < d.t_end - d.end_eps)) { active[0] = 0; *dt_out = 0.0; return; }
        if (d.check && !(isfinite(dt) && dt > 0.0)) { active[0] = 0; active[3] = 1; *dt_out = 0.0; return; }
        if (t + dt > d.t_end) dt = d.t_end - t;
    }
    active[0] = 1;
    *dt_out = dt;
}

__global__ void m2_clock_kernel(double* __restrict__ t, const double* __restrict__ dt, const int* __restrict__ active,
                                long long* __restrict__ steps) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && *active) { *t = *t + *dt; *steps = *steps + 1; }
}

__global__ void set_scalar_kernel(double* p, double v) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *p = v;
}

cudaError_t launch_dt_finalize(const double* spd_part, DtSpec d, double* dt_out, const double* t_now, int* active,
                               cudaStream_t s) {
    m2_dt_finalize_kernel<<<1, 32, 0, s>>>(spd_part, RED_BLOCKS, d, dt_out, t_now, active);
    return cudaGetLastError();
}

cudaError_t launch_clock(double* t, const double* dt, const int* active, long long* steps, cudaStream_t s) {
    m2_clock_kernel<<<1, 32, 0, s>>>(t, dt, active, steps);
    return cudaGetLastError();
}

cudaError_t launch_set_scalar(double* p, double v, cudaStream_t s) {
    set_scalar_kernel<<<1, 32, 0, s>>>(p, v);
    return cudaGetLastError();
}

constexpr int SOR_NT = 1024;

// The cluster kernel's shape for a grid, or V = 0 where sor_rb_kernel solves it:
// the grid has to fit 16 CTAs of SOR_CL_MAXV pairs a thread (about 360^2,
// beyond which the whole chip is as fast), a row the pairs of a CTA, and the
// pairs the blocks of sor_rb_kernel one to a thread (an odd nx can exceed them
// by a few), whose sums it repeats.
constexpr size_t SOR_CL_MAX_SMEM = 224 * 1024;
struct SorClusterPlan { int V, nc; size_t smem; };
static SorClusterPlan sor_cluster_plan(const SorArgs& a) {
    SorClusterPlan p{0, 0, 0};
    if (a.nx < 1 || a.ny < 1 || (long long)a.nx * a.ny > 2LL * SOR_CL_NT * SOR_CL_MAXV * SOR_CL_MAXC) return p;
    if ((a.ax.periodic && (a.nx & 1)) || (a.ay.periodic && (a.ny & 1))) return p;
    const int half = (a.nx + 1) / 2, M = half * a.ny;
    const int nb = (M + SOR_NT - 1) / SOR_NT;
    if (M > (a.nx * a.ny / 2 + SOR_NT - 1) / SOR_NT * SOR_NT) return p;
    const int S = (nb + SOR_CL_MAXC - 1) / SOR_CL_MAXC * SOR_NT, V = S / SOR_CL_NT;
    const size_t smem = sor_cluster_smem(S, half, nb);
    if (V > SOR_CL_MAXV || half > S || smem > SOR_CL_MAX_SMEM) return p;
    p.V = V; p.nc = (M + S - 1) / S; p.smem = smem;
    return p;
}

template <int V> static cudaError_t launch_sor_cluster(const SorArgs& a, const SorClusterPlan& p, cudaStream_t s, bool* done) {
    const void* fn = (const void*)sor_cluster_kernel<V>;
    // the limit is the device's, for every handle and captured graph: what the largest grid may take, not this one
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOR_CL_MAX_SMEM);
    if (e == cudaSuccess && p.nc > 8) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.nc; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.nc); cfg.blockDim = dim3(SOR_CL_NT); cfg.dynamicSmemBytes = p.smem; cfg.stream = s;
    cfg.attrs = at; cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg);
    if (e != cudaSuccess || clusters < 1) { cudaGetLastError(); return cudaSuccess; }   // no room for such a cluster here
    *done = true;
    return cudaLaunchKernelEx(&cfg, sor_cluster_kernel<V>, a);
}

cudaError_t launch_sor(const SorArgs& a, int* nblocks_out, cudaStream_t s) {
    const SorClusterPlan plan = sor_cluster_plan(a);
    if (plan.V > 0) {
        bool done = false;
        cudaError_t ec = cudaSuccess;
        switch (plan.V) {
            case 2: ec = launch_sor_cluster<2>(a, plan, s, &done); break;
            case 4: ec = launch_sor_cluster<4>(a, plan, s, &done); break;
            case 6: ec = launch_sor_cluster<6>(a, plan, s, &done); break;
            default: ec = launch_sor_cluster<8>(a, plan, s, &done); break;
        }
        if (ec != cudaSuccess || done) { if (nblocks_out) *nblocks_out = plan.nc; return ec; }
    }
    int dev = 0, nsm = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sor_rb_kernel<SOR_NT>, SOR_NT, 0)) != cudaSuccess)
        return e;
    if (per_sm < 1) return cudaErrorLaunchOutOfResources;
    // enough blocks to cover half the grid per colour, at most one wave
    const int ncell = a.nx * a.ny;
    int want = (ncell / 2 + SOR_NT - 1) / SOR_NT;
    if (want < 1) want = 1;
    int cap = nsm;   // one 1024-thread CTA per SM: the sweeps are grid-barrier bound, and fewer, larger CTAs arrive faster
    int nb = want < cap ? want : cap;
    if (nblocks_out) *nblocks_out = nb;
    SorArgs args = a;
    void* params[] = {&args};
    return cudaLaunchCooperativeKernel((const void*)sor_rb_kernel<SOR_NT>, dim3(nb), dim3(SOR_NT), params, 0, s);
}

constexpr int SOR_LEX_NT = 1024;

template <class T>
cudaError_t launch_sor_lex(const SorLexArgs& a, const T* rho, cudaStream_t s) {
    sor_lex_kernel<T, SOR_LEX_NT><<<1, SOR_LEX_NT, 0, s>>>(a, rho);
    return cudaGetLastError();
}
template cudaError_t launch_sor_lex<float>(const SorLexArgs&, const float*, cudaStream_t);
template cudaError_t launch_sor_lex<double>(const SorLexArgs&, const double*, cudaStream_t);

}  // namespace ccb
