// Direct Poisson solve for the batched ensemble, in the state precision T
// (FP64 instances: FP64 throughout, bitwise reproducible on the CPU; FP32
// instances: the same operations in FP32).
//
// It solves the discrete problem the reference's SOR iterates towards
// (mhd2d_resistive_hlld_ct_gravity.cpp:207-223: 5-point Laplacian, clamp or
// wrap neighbours, zero-mean potential) exactly instead of iterating:
//   1. U = R * Tx^T     R = 4 pi G (rho - mean), Tx rows = orthonormal
//                       eigenvectors of the x second difference (DCT-II for
//                       clamp, Hartley for periodic)        -- dp_gemm, MODE 0
//   2. per x wavenumber k: (Dyy + lam_x[k]) u_k = U[:, k] along y: Thomas,
//      cyclic Thomas (Sherman-Morrison), or for k = 0 the cumulative-flux
//      solution with its mean removed                        -- dp_ysolve
//   3. phi = U * Tx                                          -- dp_gemm, MODE 1
// The translation unit is compiled with -fmad=false and every multiply-add is
// an explicit fma() in a fixed order, so the CPU restatement (std::fma in the
// same order) reproduces the result bit for bit.
//
// Work-lists: GEMM tiles {instance, (tm << 16) | tn} of TM x TM outputs (TM 64,
// or 32 when 64-tiles would leave SMs idle: same per-output k order, same bits);
// y-solve items {instance, -1} (the singular wavenumber 0) and {instance,
// column block} of DPC wavenumbers 1 + DPC cb + lane, one thread per column.
#pragma once
#include <type_traits>

#include "batch_kernels.cuh"

namespace ccb {

constexpr int DPK = 16, DPNT = 256;   // GEMM K chunk and threads; tiles TM x TM, TM/16 x TM/16 outputs per thread
constexpr int DPC = 32;                                    // y-solve columns per block

// Software-pipelined tile loop: the next K chunk is loaded into registers
// while the current one is multiplied from shared memory; raw values are
// converted (MODE 0: 4 pi G (rho - mean)) only when they are stored, so no
// instruction waits on a load in flight during the multiply.
template <class T, int MODE, int TM>
__global__ void __launch_bounds__(DPNT)
dp_gemm_kernel(const BatchInst<T>* __restrict__ inst, const int2* __restrict__ gwork, int ngwork, int src,
               const double* __restrict__ rho_mean, const int* __restrict__ active) {
    constexpr int RPT = TM / 16;            // outputs per thread per dimension
    constexpr int LQ = TM * DPK / DPNT;     // tile elements each thread loads per K chunk
    __shared__ T As[DPK][TM + 1];           // k-major A tile
    __shared__ T Bs[DPK][TM];
    const int tr = threadIdx.x / 16, tc = threadIdx.x % 16;
    for (int w = blockIdx.x; w < ngwork; w += gridDim.x) {
        const int2 it = gwork[w];
        if (active[it.x] == 0) continue;   // uniform over the block
        const BatchInst<T>& I = inst[it.x];
        const int nx = I.c.nx, ny = I.c.ny, P = I.c.pitch;
        const int m0 = (it.y >> 16) * TM, n0 = (it.y & 0xffff) * TM;
        const T* __restrict__ B = (MODE == 0) ? I.txt : I.tx;   // K x N row-major, K = N = nx
        const T* __restrict__ rho = I.buf[src].rho;
        const T* __restrict__ ah = I.ah;
        const T mean = (MODE == 0) ? (T)rho_mean[it.x] : T(0);
        const T fpg = (T)I.fourpiG;
        T ra[LQ];
        T rb[LQ];
        auto gload = [&](int k0) {
#pragma unroll
            for (int q = 0; q < LQ; q++) {
                const int e = threadIdx.x + q * DPNT;
                const int gm = m0 + e / DPK, gk = k0 + e % DPK;
                ra[q] = T(0);
                if (gm < ny && gk < nx) {
                    if (MODE == 0) ra[q] = rho[(size_t)gm * P + gk];
                    else ra[q] = ah[(size_t)gm * nx + gk];
                }
                const int gkb = k0 + e / TM, gn = n0 + e % TM;
                rb[q] = (gkb < nx && gn < nx) ? B[(size_t)gkb * nx + gn] : T(0);
            }
        };
        T acc[RPT][RPT];
#pragma unroll
        for (int r = 0; r < RPT; r++)
#pragma unroll
            for (int c = 0; c < RPT; c++) acc[r][c] = T(0);
        gload(0);
        for (int k0 = 0; k0 < nx; k0 += DPK) {
#pragma unroll
            for (int q = 0; q < LQ; q++) {
                const int e = threadIdx.x + q * DPNT;
                const int m = e / DPK, kk = e % DPK;
                T v = ra[q];
                if (MODE == 0) v = (m0 + m < ny && k0 + kk < nx) ? fpg * (v - mean) : T(0);
                As[kk][m] = v;
                Bs[e / TM][e % TM] = rb[q];
            }
            __syncthreads();
            if (k0 + DPK < nx) gload(k0 + DPK);
            const int kend = min(DPK, nx - k0);
            for (int kk = 0; kk < kend; kk++) {
                T a[RPT], b[RPT];
#pragma unroll
                for (int r = 0; r < RPT; r++) a[r] = As[kk][tr + 16 * r];
#pragma unroll
                for (int c = 0; c < RPT; c++) b[c] = Bs[kk][tc + 16 * c];
#pragma unroll
                for (int r = 0; r < RPT; r++)
#pragma unroll
                    for (int c = 0; c < RPT; c++) acc[r][c] = fma(a[r], b[c], acc[r][c]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < RPT; r++) {
            const int gm = m0 + tr + 16 * r;
            if (gm >= ny) continue;
#pragma unroll
            for (int c = 0; c < RPT; c++) {
                const int gn = n0 + tc + 16 * c;
                if (gn >= nx) continue;
                if (MODE == 0) I.ah[(size_t)gm * nx + gn] = acc[r][c];
                else I.phi[(size_t)gm * P + gn] = acc[r][c];
            }
        }
    }
}

// y solves: one thread per x wavenumber k >= 1 (a warp covers 32 adjacent
// wavenumbers, so every row access is one coalesced 256-byte line), the
// singular k = 0 on a CTA of its own.  Each sweep is a chain of fma's whose
// loads do not depend on the chain, and a grid has few of these warps, so a sweep
// takes its chain only if its rows are under way long before: column and factors
// by cp.async in a ring of shared memory, YB rows to a group, YD - 1 groups ahead
// of the group being computed (registers that hold rows under way cannot be passed
// on from group to group without waiting for them: one group ahead is all they
// give).  The arithmetic and its order are those of the CPU restatement (bitwise).
// One clamped 512^2 in FP64: 93 -> 41 us; 128 FP32 instances of 64 to 256 cells a
// side: 52 -> 26.
constexpr int YB = 8, YD = 8;
template <class T> using YRing = T[2][YD][YB][DPC];

template <class S_> __device__ __forceinline__ void y_fetch(S_* smem, const S_* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g),
                 "n"(sizeof(S_)) : "memory");
}

// u_i <- f(u_i, w_i) for the rows i < n in turn, row i at u + i St, w + i St
template <class S_, class F>
__device__ __forceinline__ void ysweep(S_* u, const S_* w, YRing<S_>& ring, ptrdiff_t St, int n, F f) {
    const int lane = threadIdx.x;
    __threadfence_block();   // the sweep before wrote the rows that the copies read
    auto fetch = [&](int g) {
        const S_* pu = u + (ptrdiff_t)g * YB * St;
        const S_* pw = w + (ptrdiff_t)g * YB * St;
#pragma unroll
        for (int t = 0; t < YB; t++) {
            if (g * YB + t < n) {
                y_fetch(&ring[0][g % YD][t][lane], pu);
                y_fetch(&ring[1][g % YD][t][lane], pw);
            }
            pu += St; pw += St;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int g = 0; g < YD - 1; g++) fetch(g);
    for (int g = 0; g * YB < n; g++) {
        fetch(g + YD - 1);   // into the slots of group g - 1
        asm volatile("cp.async.wait_group %0;" ::"n"(YD - 1) : "memory");   // group g is there
        S_ uv[YB], wv[YB];
#pragma unroll
        for (int t = 0; t < YB; t++) { uv[t] = ring[0][g % YD][t][lane]; wv[t] = ring[1][g % YD][t][lane]; }
        S_* p = u + (ptrdiff_t)g * YB * St;
#pragma unroll
        for (int t = 0; t < YB; t++) {
            if (g * YB + t < n) *p = f(uv[t], wv[t]);
            p += St;
        }
    }
}

// The singular k = 0 by a warp: flux G_j = a (u_{j+1} - u_j) = G_{j-1} + r_j, then
// the mean removed.  A lane loads and stores a row of 32; every lane runs the
// chain, on rows handed round by shuffles.
template <class T> __device__ __forceinline__ void ysolve_singular(T* u, size_t S, int n, bool py, T dy2) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x;
    auto row = [&](int j) { return j < n ? u[j * S] : T(0); };
    T g0 = T(0);
    if (py) {
        T Sr = T(0), SS = T(0), v = row(lane);
        for (int j = 0; j < n; j += 32) {
            const T nv = row(j + 32 + lane);
#pragma unroll
            for (int t = 0; t < 32; t++) {
                const T r = __shfl_sync(ALL, v, t);
                if (j + t < n) { Sr = Sr + r; SS = SS + Sr; }
            }
            v = nv;
        }
        g0 = -(SS / (T)n);
    }
    T G = g0, prev = T(0), m = T(0), v = row(lane);
    for (int j = 0; j < n; j += 32) {
        const T nv = row(j + 32 + lane);
        T mine = T(0);
#pragma unroll
        for (int t = 0; t < 32; t++) {
            const T r = __shfl_sync(ALL, v, t);
            if (lane == t) mine = prev;
            if (j + t < n) {
                m = m + prev;
                G = G + r;
                prev = fma(dy2, G, prev);
            }
        }
        if (j + lane < n) u[(j + lane) * S] = mine;
        v = nv;
    }
    m = m / (T)n;
    for (int j = lane; j < n; j += 32 * 8) {
        T q[8];
#pragma unroll
        for (int t = 0; t < 8; t++) q[t] = row(j + 32 * t);
#pragma unroll
        for (int t = 0; t < 8; t++)
            if (j + 32 * t < n) u[(j + 32 * t) * S] = q[t] - m;
    }
}

template <class T>
__global__ void __launch_bounds__(DPC)
dp_ysolve_kernel(const BatchInst<T>* __restrict__ inst, const int2* __restrict__ ywork, int nywork,
                 const int* __restrict__ active) {
    __shared__ YRing<T> ring;
    for (int w = blockIdx.x; w < nywork; w += gridDim.x) {
        const int2 it = ywork[w];
        if (active[it.x] == 0) continue;
        const BatchInst<T>& I = inst[it.x];
        const int nx = I.c.nx, n = I.c.ny;
        const ptrdiff_t S = nx;
        const bool py = I.c.ay.periodic != 0;
        const T a = (T)I.ay;
        if (it.y < 0) {
            ysolve_singular(I.ah, (size_t)nx, n, py, (T)I.dy2);
            continue;
        }
        const int col = 1 + it.y * DPC + threadIdx.x;
        if (col >= nx) continue;
        T* u = I.ah + col;
        // forward: d_0 = u_0 inv_0, d_j = (u_j - a d_{j-1}) inv_j, u_j <- d_j
        T d = u[0] * I.yinv[col];
        u[0] = d;
        ysweep(u + S, I.yinv + col + S, ring, S, n - 1, [&](T uj, T inv) { return d = fma(-a, d, uj) * inv; });
        // backward: x_{n-1} = d_{n-1}, x_j = d_j - cp_j x_{j+1}, u_j <- x_j
        T x = d;
        ysweep(u + (n - 2) * S, I.ycp + col + (n - 2) * S, ring, -S, n - 1, [&](T uj, T cp) { return x = fma(-cp, x, uj); });
        if (!py) continue;
        const T gam = -fma(T(-2), a, I.lamx[col]);
        const T fac = fma(a / gam, d, x) * I.yfden[col];   // d = x_{n-1}, x = x_0
        ysweep(u, I.yz + col, ring, S, n, [&](T uj, T z) { return fma(-fac, z, uj); });
    }
}

}  // namespace ccb
