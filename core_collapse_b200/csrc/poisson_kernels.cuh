// Self-gravity Poisson solves (templated on T; instantiated per precision).
//
// Spectral periodic solve (navier_stokes_2d_hllc_poisson.cpp:285-328), three
// passes over a complex work array A (nx*ny, row-major):
//   1. rows:    A = FFT_x(rho - mean)                      (fft_rows_fwd)
//   2. columns: A = IFFT_y( K(k) * FFT_y(A) ),  K = -4 pi G / |k|^2, K(0)=0
//   3. rows:    phi = Re IFFT_x(A)
// Every 1D transform is the reference's radix-2 decimation-in-time FFT
// (NS:152-177): bit-reversed load, log2(n) butterfly passes with twiddles built
// on the host by the reference's recurrence w *= wlen, inverse scaled by 1/n.
// The reference runs the inverse as rows-then-columns; here it is
// columns-then-rows so that the column inverse fuses with the spectral
// multiply (rounding differs at the 1e-16 level; stated in the tests).
//
// Red-black SOR (the GPU ordering of M2:207-223 / EH:335-368): grids up to about
// 360^2 inside one thread-block cluster (sor_cluster_kernel), larger ones in a
// persistent cooperative kernel with one grid barrier per colour (sor_rb_kernel);
// deterministic FP64 mean removal after each sweep (applied lazily), optional
// residual test.
#pragma once
#include <cooperative_groups.h>
#include <type_traits>

#include "cc_device.cuh"

namespace ccb {

template <class T> struct Cplx { T re, im; };

// the reference's complex product (x.re*w.re - x.im*w.im, x.re*w.im + x.im*w.re)
template <class T> __device__ __forceinline__ Cplx<T> cmul(Cplx<T> x, Cplx<T> w) {
    Cplx<T> r;
    r.re = x.re * w.re - x.im * w.im;
    r.im = x.re * w.im + x.im * w.re;
    return r;
}

__device__ __forceinline__ int bitrev(int i, int logn) { return (int)(__brev((unsigned)i) >> (32 - logn)); }

// Shared-memory slot of element i of a transform line: a spare slot after every
// 16 and another after every 128, so that both the strided accesses of the
// grouped passes below and the bit-reversed scatter of the first pass hit
// distinct banks.  A line of n elements takes fft_line_slots(n) slots.
__host__ __device__ constexpr int fft_line_slots(int n) { return n + (n >> 4) + (n >> 7); }
__device__ __forceinline__ int fpad(int i) { return i + (i >> 4) + (i >> 7); }

// The transforms run R consecutive radix-2 stages of the reference's DIT
// transform at a time (half-lengths h0, 2 h0, ..., 2^(R-1) h0): a thread takes
// the 2^R elements base + m h0 (m < 2^R) of one group, which only exchange
// data among themselves in these stages, and runs the stages in registers.
// Every butterfly u = a[p], v = a[p+h] * tw[h-1 + (p mod h)], a[p] = u + v,
// a[p+h] = u - v is the reference's, with the same operands and twiddle, so the
// result is the same bit for bit as one stage per pass.
//
// These kernels are bound by latency (a line of 1024 points is three passes),
// so a CTA has the threads that its groups need and no more: eight CTAs of 64
// threads to an SM at n = 1024 where 512 threads, 448 of them waiting, held it
// alone.  The first pass takes its elements from the loads (the group of
// thread g after bit reversal is elements g, g + n/2^R, ...: coalesced), the
// last one hands its results to the stores, and between the forward and the
// inverse column transform they stay in registers: four trips through shared
// memory to a column instead of nine.  FP64 solve (rows, columns, inverse
// rows), before -> now: 128^2 20.7 -> 14.2 us, 512^2 49 -> 20, 1024^2 148 ->
// 49, 2048^2 403 -> 188.
template <class T, int R>
__device__ __forceinline__ void fft_stages(Cplx<T> (&x)[1 << R], int h0, int o, const Cplx<T>* __restrict__ tw) {
    constexpr int M = 1 << R;
#pragma unroll
    for (int st = 0; st < R; st++) {
        const int hs = 1 << st, h = h0 << st;
#pragma unroll
        for (int m = 0; m < M; m++) {
            if (m & hs) continue;
            const Cplx<T> w = tw[h - 1 + o + (m & (hs - 1)) * h0];   // p mod h = o + (m mod hs) h0
            const Cplx<T> u = x[m];
            const Cplx<T> v = cmul(x[m + hs], w);
            x[m].re = u.re + v.re; x[m].im = u.im + v.im;
            x[m + hs].re = u.re - v.re; x[m + hs].im = u.im - v.im;
        }
    }
}

// m with its R bits reversed
template <int R> __host__ __device__ constexpr int rev_bits(int m) {
    int r = 0;
    for (int b = 0; b < R; b++) r |= ((m >> b) & 1) << (R - 1 - b);
    return r;
}

// work item g of `lines` lines with gpl groups each: line l, group q.  IL: the
// lines interleaved (adjacent columns in adjacent threads).
template <bool IL> __device__ __forceinline__ void fft_item(int g, int lines, int gpl, int& l, int& q) {
    if (IL) { l = g % lines; q = g / lines; }
    else { l = g / gpl; q = g - l * gpl; }
}

// First stages (h0 = 1): elements from ld(line, natural index), results to the
// lines in shared memory, or to st(line, index, x) where n = 2^R (LAST).
template <class T, int R, bool IL, bool LAST, class LD, class ST>
__device__ __forceinline__ void fft_first(Cplx<T>* a, int LS, int n, int logn, int lines, const Cplx<T>* __restrict__ tw, LD ld,
                                          ST st) {
    constexpr int M = 1 << R;
    const int gpl = n >> R;
    for (int g = threadIdx.x; g < lines * gpl; g += blockDim.x) {
        int l, q;
        fft_item<IL>(g, lines, gpl, l, q);
        Cplx<T> x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = ld(l, rev_bits<R>(m) * gpl + q);
        fft_stages<T, R>(x, 1, 0, tw);
        const int base = (LAST ? 0 : bitrev(q, logn - R)) * M;
#pragma unroll
        for (int m = 0; m < M; m++) {
            if (LAST) st(l, base + m, x[m]);
            else a[l * LS + fpad(base + m)] = x[m];
        }
    }
    __syncthreads();
}

// R stages from h0 on within shared memory, or out of it through st(line, index, x) (LAST, 2^R h0 = n).
template <class T, int R, bool IL, bool LAST, class ST>
__device__ __forceinline__ void fft_next(Cplx<T>* a, int LS, int n, int lines, int h0, const Cplx<T>* __restrict__ tw, ST st) {
    constexpr int M = 1 << R;
    const int gpl = n >> R;
    for (int g = threadIdx.x; g < lines * gpl; g += blockDim.x) {
        int l, q;
        fft_item<IL>(g, lines, gpl, l, q);
        const int o = q & (h0 - 1), base = (q / h0) * (M * h0) + o;
        Cplx<T>* line = a + l * LS;
        Cplx<T> x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = line[fpad(base + m * h0)];
        fft_stages<T, R>(x, h0, o, tw);
#pragma unroll
        for (int m = 0; m < M; m++) {
            if (LAST) st(l, base + m * h0, x[m]);
            else line[fpad(base + m * h0)] = x[m];
        }
    }
    __syncthreads();
}

// f(std::integral_constant<int, r>) for 1 <= r <= RB
template <int RB, class F> __device__ __forceinline__ void with_radix(int r, F f) {
    if constexpr (RB >= 4)
        if (r == 4) { f(std::integral_constant<int, 4>()); return; }
    if constexpr (RB >= 3)
        if (r == 3) { f(std::integral_constant<int, 3>()); return; }
    if (r == 2) f(std::integral_constant<int, 2>());
    else f(std::integral_constant<int, 1>());
}

// A whole transform of `lines` lines, RB stages a pass; the first pass takes what logn leaves over.
// tw: twiddles of all stages, half-length h at tw[h-1 .. 2h-2].
template <class T, int RB, bool IL, class LD, class ST>
__device__ __forceinline__ void fft_lines(Cplx<T>* a, int LS, int n, int logn, int lines, const Cplx<T>* __restrict__ tw,
                                          LD ld, ST st) {
    const int r = (logn - 1) % RB + 1;
    if (r == logn) {
        with_radix<RB>(r, [&](auto R) { fft_first<T, decltype(R)::value, IL, true>(a, LS, n, logn, lines, tw, ld, st); });
        return;
    }
    with_radix<RB>(r, [&](auto R) { fft_first<T, decltype(R)::value, IL, false>(a, LS, n, logn, lines, tw, ld, st); });
    int h0 = 1 << r;
    for (; (h0 << RB) < n; h0 <<= RB) fft_next<T, RB, IL, false>(a, LS, n, lines, h0, tw, st);
    fft_next<T, RB, IL, true>(a, LS, n, lines, h0, tw, st);
}

// the kernels below run on at most FFT_NT threads; the column pass takes FFT_CW columns (32 bytes of a row) a CTA
constexpr int FFT_NT = 512, FFT_CW = 2;

// lines of an n-point transform to a CTA (of `total`), and its threads: one per group of 2^RB
__host__ __device__ inline int fft_lines_per_cta(int n, int total) {
    const int l = n >= 512 ? 1 : 512 / n;
    return l < total ? l : total;
}
__host__ __device__ inline int fft_threads(int n, int lines, int RB) {
    const int t = ((lines * n >> RB) + 31) / 32 * 32;
    return t < 32 ? 32 : (t > FFT_NT ? FFT_NT : t);
}

// the mean of a density whose partial sums are given, by the CTA's first warp
__device__ __forceinline__ double fft_mean(const double* __restrict__ rho_part, int nparts, double ncell, double* sh) {
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int b = threadIdx.x; b < nparts; b += 32) s += rho_part[b];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) *sh = s / ncell;
    }
    __syncthreads();
    return *sh;
}

// pass 1: `lines` rows per block.  rho is a pitched T field; mean = sum/N.
template <class T, int RB>
__global__ void __launch_bounds__(FFT_NT) fft_rows_fwd_kernel(const T* __restrict__ rho, int pitch, const double* __restrict__ rho_part,
                                    int nparts, double ncell, Cplx<T>* __restrict__ A, int nx, int logn, int lines,
                                    const Cplx<T>* __restrict__ tw, const int* __restrict__ active) {
    if (active && *active == 0) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double s_mean;
    const T mean = (T)fft_mean(rho_part, nparts, ncell, &s_mean);
    const size_t j0 = (size_t)blockIdx.x * lines;
    fft_lines<T, RB, false>(reinterpret_cast<Cplx<T>*>(smem_raw), fft_line_slots(nx), nx, logn, lines, tw,
        [&](int l, int i) { return Cplx<T>{rho[(j0 + l) * pitch + i] - mean, T(0)}; },
        [&](int l, int i, Cplx<T> z) { A[(j0 + l) * nx + i] = z; });
}

// The spectral factor K(k) = -4 pi G / |k|^2 (NS:308-322, continuous |k|^2,
// zero mode removed) between the forward and the inverse transform of a
// column.  The last forward pass and the first inverse one have the same radix
// 2^H, so that a thread's elements q + m n/2^H stay in its registers (one group
// to a thread).  ONLY: they are the whole transforms (n = 2^H), from ld to st.
template <class T, int H, int CW, bool ONLY, class LD, class ST>
__device__ __forceinline__ void fft_turn(Cplx<T>* a, int LS, int n, int logn, double kx, double Ly, double fourpiG,
                                         const Cplx<T>* __restrict__ twf, const Cplx<T>* __restrict__ twi, LD ld, ST st) {
    constexpr int M = 1 << H;
    const int gpl = n >> H, l = threadIdx.x % CW, q = threadIdx.x / CW;
    const bool mine = q < gpl;
    const double two_pi = 2.0 * M_PI, inv_Ly = 1.0 / Ly;
    Cplx<T> y[M];
    if (mine) {
        Cplx<T> x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = ONLY ? ld(l, rev_bits<H>(m)) : a[l * LS + fpad(q + m * gpl)];
        fft_stages<T, H>(x, gpl, q, twf);
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int j = q + m * gpl, nj = (j <= n / 2) ? j : j - n;
            const double ky = quotient(two_pi * (double)nj, Ly, inv_Ly);
            const double k2 = kx * kx + ky * ky;
            const T f = (k2 == 0.0) ? T(0) : (T)(-fourpiG / k2);
            // the inverse's first pass takes element rev(m) n/2^H + q as its m-th
            y[rev_bits<H>(m)] = Cplx<T>{x[m].re * f, x[m].im * f};
        }
        fft_stages<T, H>(y, 1, 0, twi);
    }
    __syncthreads();   // every element of the forward transform is read
    if (mine) {
        const int base = (ONLY ? 0 : bitrev(q, logn - H)) * M;
#pragma unroll
        for (int m = 0; m < M; m++) {
            if (ONLY) st(l, m, y[m]);
            else a[l * LS + fpad(base + m)] = y[m];
        }
    }
    __syncthreads();
}

// line stride of the interleaved columns: half a bank row off, so that the two columns of adjacent
// threads hit distinct banks
__host__ __device__ inline int fft_col_stride(int n) { return (fft_line_slots(n) + 7) / 8 * 8 + 4; }

// pass 2: CW adjacent columns per block: forward FFT along y, spectral
// multiply, inverse FFT along y.
template <class T, int CW, int RB>
__global__ void __launch_bounds__(FFT_NT) fft_cols_solve_kernel(Cplx<T>* __restrict__ A, int nx, int ny, int logn,
                                      const Cplx<T>* __restrict__ twf, const Cplx<T>* __restrict__ twi,
                                      double Lx, double Ly, double G, const int* __restrict__ active) {
    if (active && *active == 0) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Cplx<T>* a = reinterpret_cast<Cplx<T>*>(smem_raw);   // CW padded lines of ny
    const int LS = fft_col_stride(ny), c0 = blockIdx.x * CW, i = c0 + (int)threadIdx.x % CW;
    const double kx = 2.0 * M_PI * (double)((i <= nx / 2) ? i : i - nx) / Lx, fourpiG = 4.0 * M_PI * G;
    const T inv = T(1.0) / (T)ny;   // ny is a power of two: z * inv is z / ny
    auto ld = [&](int l, int j) { return A[(size_t)j * nx + c0 + l]; };
    auto st = [&](int l, int j, Cplx<T> z) { A[(size_t)j * nx + c0 + l] = Cplx<T>{z.re * inv, z.im * inv}; };
    auto none = [](int, int, Cplx<T>) {};
    const int r = (logn - 1) % RB + 1;
    if (r == logn) {
        with_radix<RB>(r, [&](auto R) {
            fft_turn<T, decltype(R)::value, CW, true>(a, LS, ny, logn, kx, Ly, fourpiG, twf, twi, ld, st);
        });
        return;
    }
    with_radix<RB>(r, [&](auto R) { fft_first<T, decltype(R)::value, true, false>(a, LS, ny, logn, CW, twf, ld, none); });
    for (int h0 = 1 << r; (h0 << RB) < ny; h0 <<= RB) fft_next<T, RB, true, false>(a, LS, ny, CW, h0, twf, none);
    fft_turn<T, RB, CW, false>(a, LS, ny, logn, kx, Ly, fourpiG, twf, twi, ld, st);
    int h0 = 1 << RB;
    for (; (h0 << r) < ny; h0 <<= RB) fft_next<T, RB, true, false>(a, LS, ny, CW, h0, twi, none);
    with_radix<RB>(r, [&](auto R) { fft_next<T, decltype(R)::value, true, true>(a, LS, ny, CW, h0, twi, st); });
}

// pass 3: inverse FFT along x, real part -> phi (pitched), `lines` rows per block.
template <class T, int RB>
__global__ void __launch_bounds__(FFT_NT) fft_rows_inv_kernel(const Cplx<T>* __restrict__ A, int nx, int logn, int lines,
                                    const Cplx<T>* __restrict__ tw, T* __restrict__ phi, int pitch,
                                    const int* __restrict__ active) {
    if (active && *active == 0) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const size_t j0 = (size_t)blockIdx.x * lines;
    const T inv = T(1.0) / (T)nx;   // nx is a power of two: x * inv is x / nx
    fft_lines<T, RB, false>(reinterpret_cast<Cplx<T>*>(smem_raw), fft_line_slots(nx), nx, logn, lines, tw,
        [&](int l, int i) { return A[(j0 + l) * nx + i]; },
        [&](int l, int i, Cplx<T> z) { phi[(j0 + l) * pitch + i] = z.re * inv; });
}

// ---------------------------------------------------------------------------
// Red-black SOR, FP64 throughout.
// ---------------------------------------------------------------------------
struct SorArgs {
    int nx, ny;
    AxisMap ax, ay;
    double idx2, idy2, denom, omega, tol;
    int max_iter;
    const double* rhs;      // nx*ny contiguous
    double* phi;            // nx*ny contiguous
    double* part;           // gridDim.x partials
    double* part2;          // gridDim.x partials (residual)
    GridBarrier bar;
    int* iters_out;
    double* res_out;
    const int* active;
    int max_polls = 1 << 26;   // of a wait of sor_cluster_kernel (a second or two), after which it gives up
};

// Lexicographic SOR, the reference's own solve (compute_poisson_gravity_periodic,
// M2:178-237 and EH:288-386) in its own order, for parity runs.  One
// CTA.  A sweep runs as anti-diagonal wavefronts: the cells with i + j = d
// update together, d = 0 .. nx + ny - 2, with a barrier between diagonals.
// Of a cell's neighbours, west and south lie on diagonal d - 1 (already
// updated in this sweep), east and north on d + 1 (not yet), and a periodic
// wrap neighbour on d +- (n - 1): (0, j) reads (nx - 1, j) before this sweep
// updates it and (nx - 1, j) reads (0, j) after, as the row-major loop does;
// a clamped neighbour that is the cell itself is read before its update.  So
// every cell sees exactly the values the reference's loop sees.  The density
// mean and each sweep's mean of phi are summed by one thread in the
// reference's row-major order, and the update is the reference's expression,
// so phi is the reference's to the last bit.  Slow by design (nx + ny - 1
// barriers and an N-term sequential sum per sweep); the red-black kernel is
// the production solve.  tol > 0: stop after the first sweep whose max
// |lap(phi) - rhs|, taken inside the sweep from each cell's update as
// EH:335-368 does, is below tol.
struct SorLexArgs {
    int nx, ny, pitch;
    AxisMap ax, ay;
    double idx2, idy2, denom, omega, fourpiG, tol;
    double floor_rho;       // >= 0: density floored at it first (EH:307-313); < 0: as read (M2)
    int max_iter;
    double* rhs;            // nx*ny contiguous (written)
    double* phi;            // nx*ny contiguous (written)
    int* iters_out;
    double* res_out;
    const int* active;
};

template <class T, int NT>
__global__ void __launch_bounds__(NT) sor_lex_kernel(SorLexArgs a, const T* __restrict__ rho) {
    if (a.active && *a.active == 0) return;
    __shared__ double sh[NT / 32];
    __shared__ double s_val;
    const int nx = a.nx, ny = a.ny, N = nx * ny, tid = threadIdx.x;
    double* __restrict__ phi = a.phi;
    // rhobar and rhs = 4 pi G (rho - rhobar) (M2:187-194; EH:307-321 with the floor)
    auto dens = [&](int i, int j) {
        const double r = (double)rho[(size_t)j * a.pitch + i];
        return (a.floor_rho >= 0.0 && r < a.floor_rho) ? a.floor_rho : r;   // std::max(rho, floor_rho)
    };
    if (tid == 0) {
        double s = 0.0;
        for (int j = 0; j < ny; j++)
            for (int i = 0; i < nx; i++) s += dens(i, j);
        s_val = s / (double)N;
    }
    __syncthreads();
    const double rhobar = s_val;
    for (int j = 0; j < ny; j++)
        for (int i = tid; i < nx; i += NT) {
            const size_t q = (size_t)j * nx + i;
            a.rhs[q] = a.fourpiG * (dens(i, j) - rhobar);
            phi[q] = 0.0;
        }
    __syncthreads();
    int it = 0;
    double res = 0.0;
    for (; it < a.max_iter; ++it) {
        double r = 0.0;   // tol > 0: the residual taken inside the sweep (EH:335-368)
        for (int d = 0; d <= nx + ny - 2; ++d) {
            const int i0 = d - (ny - 1) > 0 ? d - (ny - 1) : 0, i1 = d < nx - 1 ? d : nx - 1;
            for (int i = i0 + tid; i <= i1; i += NT) {
                const int j = d - i;
                const size_t k = (size_t)j * nx + i;
                const double phiE = phi[(size_t)j * nx + a.ax.cell(i + 1)];
                const double phiW = phi[(size_t)j * nx + a.ax.cell(i - 1)];
                const double phiN = phi[(size_t)a.ay.cell(j + 1) * nx + i];
                const double phiS = phi[(size_t)a.ay.cell(j - 1) * nx + i];
                const double phi_new = ((phiE + phiW) * a.idx2 + (phiN + phiS) * a.idy2 - a.rhs[k]) / a.denom;
                const double v = phi[k] + a.omega * (phi_new - phi[k]);
                phi[k] = v;
                if (a.tol > 0.0) {
                    const double lap = (phiE - 2.0 * v + phiW) * a.idx2 + (phiN - 2.0 * v + phiS) * a.idy2;
                    r = fmax(r, fabs(lap - a.rhs[k]));
                }
            }
            __syncthreads();
        }
        // phibar in row-major order (M2:219-222)
        if (tid == 0) {
            double s = 0.0;
            for (int q = 0; q < N; q++) s += phi[q];
            s_val = s / (double)N;
        }
        __syncthreads();
        const double phibar = s_val;
        for (int q = tid; q < N; q += NT) phi[q] -= phibar;
        __syncthreads();
        if (a.tol > 0.0) {
            const double r0 = block_max<NT>(r, sh);   // valid in thread 0
            if (tid == 0) s_val = r0;
            __syncthreads();
            res = s_val;
            __syncthreads();   // s_val is rewritten by the next sweep's mean
            if (res < a.tol) { ++it; break; }
        }
    }
    if (tid == 0) {
        if (a.iters_out) *a.iters_out = it;
        if (a.res_out) *a.res_out = res;
    }
}

// max |lap(phi) - rhs| over the block's cells of the field phi - shift (the
// stored field with a pending mean removal applied on the fly)
template <int NT>
__device__ __forceinline__ double sor_residual_block(const SorArgs& a, double shift, double* sh) {
    double r = 0.0;
    const int N = a.nx * a.ny;
    for (int k = blockIdx.x * NT + threadIdx.x; k < N; k += gridDim.x * NT) {
        const int i = k % a.nx, j = k / a.nx;
        const double c = a.phi[k] - shift;
        const double pE = a.phi[(size_t)j * a.nx + a.ax.cell(i + 1)] - shift;
        const double pW = a.phi[(size_t)j * a.nx + a.ax.cell(i - 1)] - shift;
        const double pN = a.phi[(size_t)a.ay.cell(j + 1) * a.nx + i] - shift;
        const double pS = a.phi[(size_t)a.ay.cell(j - 1) * a.nx + i] - shift;
        const double lap = (pE - 2.0 * c + pW) * a.idx2 + (pN - 2.0 * c + pS) * a.idy2;
        r = fmax(r, fabs(lap - a.rhs[k]));
    }
    return block_max<NT>(r, sh);
}

// One sweep = red update, black update, mean removal, and (tol > 0) the
// residual test.  The mean removal phi -= mean is not a pass of its own: the
// mean of a sweep stays pending (`m`) and every read of a value that the
// sweep has not rewritten subtracts it, which gives the same doubles as
// subtracting first (x - m is the value the reference stores), and x - 0.0 == x
// for the values already rewritten.  The density-independent part of the
// mean (the block partial sums) is formed in the black phase, which also reads
// the red cell of each of its indices, so a sweep needs two grid barriers
// (red, black) plus one for the residual when tol > 0.  A final pass applies
// the last pending mean.
template <int NT>
__global__ void __launch_bounds__(NT) sor_rb_kernel(SorArgs a) {
    if (a.active && *a.active == 0) return;
    __shared__ double sh[NT / 32];
    __shared__ double s_val;
    const unsigned nb = gridDim.x;
    const int N = a.nx * a.ny;
    const int half = (a.nx + 1) / 2;        // cells of one colour per row (upper bound)
    const int M = half * a.ny;
    for (int k = blockIdx.x * NT + threadIdx.x; k < N; k += nb * NT) a.phi[k] = 0.0;
    if (!grid_sync(a.bar, nb)) return;
    // the mean of the block partial sums in block order (the same double in every block)
    auto block_mean = [&]() {
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (unsigned b = 0; b < nb; b++) t += a.part[b];
            s_val = t / (double)N;
        }
        __syncthreads();
        return s_val;
    };
    double m = 0.0;   // mean removal pending on every cell not yet rewritten in this sweep
    int it = 0;
    double res = 0.0;
    for (; it < a.max_iter; ++it) {
        // red: every value read is pending
        for (int k = blockIdx.x * NT + threadIdx.x; k < M; k += nb * NT) {
            const int j = k / half;
            const int i = 2 * (k % half) + (j & 1);
            if (i >= a.nx) continue;
            const size_t q = (size_t)j * a.nx + i;
            const double pE = a.phi[(size_t)j * a.nx + a.ax.cell(i + 1)] - m;
            const double pW = a.phi[(size_t)j * a.nx + a.ax.cell(i - 1)] - m;
            const double pN = a.phi[(size_t)a.ay.cell(j + 1) * a.nx + i] - m;
            const double pS = a.phi[(size_t)a.ay.cell(j - 1) * a.nx + i] - m;
            const double own = a.phi[q] - m;
            const double pn = ((pE + pW) * a.idx2 + (pN + pS) * a.idy2 - a.rhs[q]) / a.denom;
            a.phi[q] = own + a.omega * (pn - own);
        }
        if (!grid_sync(a.bar, nb)) return;
        // black: the red neighbours are rewritten; a clamped neighbour that is
        // the cell itself is still pending.  Sum every cell of the new field.
        double s = 0.0;
        for (int k = blockIdx.x * NT + threadIdx.x; k < M; k += nb * NT) {
            const int j = k / half;
            const int ir = 2 * (k % half) + (j & 1), i = 2 * (k % half) + ((j + 1) & 1);
            if (ir < a.nx) s += a.phi[(size_t)j * a.nx + ir];
            if (i >= a.nx) continue;
            const size_t q = (size_t)j * a.nx + i;
            const int iE = a.ax.cell(i + 1), iW = a.ax.cell(i - 1), jN = a.ay.cell(j + 1), jS = a.ay.cell(j - 1);
            const double pE = a.phi[(size_t)j * a.nx + iE] - (iE == i ? m : 0.0);
            const double pW = a.phi[(size_t)j * a.nx + iW] - (iW == i ? m : 0.0);
            const double pN = a.phi[(size_t)jN * a.nx + i] - (jN == j ? m : 0.0);
            const double pS = a.phi[(size_t)jS * a.nx + i] - (jS == j ? m : 0.0);
            const double own = a.phi[q] - m;
            const double pn = ((pE + pW) * a.idx2 + (pN + pS) * a.idy2 - a.rhs[q]) / a.denom;
            const double v = own + a.omega * (pn - own);
            a.phi[q] = v;
            s += v;
        }
        s = block_sum<NT>(s, sh);
        if (threadIdx.x == 0) a.part[blockIdx.x] = s;
        if (!grid_sync(a.bar, nb)) return;
        m = block_mean();   // this sweep's mean, pending from here on
        if (a.tol > 0.0) {
            const double r = sor_residual_block<NT>(a, m, sh);
            if (threadIdx.x == 0) a.part2[blockIdx.x] = r;
            if (!grid_sync(a.bar, nb)) return;
            if (threadIdx.x == 0) {
                double mx = 0.0;
                for (unsigned b = 0; b < nb; b++) mx = fmax(mx, a.part2[b]);
                s_val = mx;
            }
            __syncthreads();
            res = s_val;
            __syncthreads();   // s_val is rewritten by the next block_mean
            // part and part2 are next written after at least one more grid
            // barrier, when every block has read them
            if (res < a.tol) { ++it; break; }
        }
    }
    // apply the last pending mean
    for (int k = blockIdx.x * NT + threadIdx.x; k < N; k += nb * NT) a.phi[k] -= m;
    if (!(a.tol > 0.0)) {
        if (!grid_sync(a.bar, nb)) return;
        const double r = sor_residual_block<NT>(a, 0.0, sh);
        if (threadIdx.x == 0) a.part2[blockIdx.x] = r;
        if (!grid_sync(a.bar, nb)) return;
        if (threadIdx.x == 0) {
            double mx = 0.0;
            for (unsigned b = 0; b < nb; b++) mx = fmax(mx, a.part2[b]);
            res = mx;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) { *a.iters_out = it; *a.res_out = res; }
}

// The same red-black SOR inside one thread-block cluster, for grids whose two
// colours fit the shared memory of at most 16 CTAs (sor_cluster_plan).  What
// bounds sor_rb_kernel on such grids is its grid barriers: 8.2 us a sweep at
// 256^2 for under 1 us of FP64 work.  Here the potential never leaves the SMs
// and CTAs exchange single values (st.async into the other CTA's shared
// memory, counted by an mbarrier there), so that no phase waits for a fence:
// a cluster barrier of 1024 threads takes 680 cycles with its release fence, an
// exchange by counted stores with a neighbour 380, with all of 16 CTAs 560.
//
// Cells go by pairs k = j half + p, the red and the black cell of columns 2p,
// 2p + 1 of row j: N and S neighbours of either are the other colour's of
// pairs k +- half, E and W those of k itself and of a pair next to it in the
// row.  CTA c owns the pairs [c S, (c + 1) S), S >= half, and keeps both
// colours on the window [c S - half, (c + 1) S + half); whoever updates a pair
// stores it also into the windows of the CTAs that read it, the periodic
// images of the first and last row included, so that every read is local.
// A pair that reads another CTA's values is itself read by that CTA, so a
// CTA's values of a phase can only arrive once every reader of the values
// they replace has read (its own value, which depends on them, is awaited).
// A thread keeps its V pairs and their right-hand sides in registers: a cell
// takes three shared-memory loads instead of six, and the V cells' chains of
// dependent FP64 operations overlap; 512 threads, for the registers (1024
// threads of half as many pairs: 14.1 against 12.8 ms in the 256^2 MHD case).
//
// Measured, per sweep, sor_rb_kernel -> this: 32^2 6.5 -> 1.6 us, 128^2 6.7 ->
// 2.1, 256^2 8.3 -> 3.4, 350^2 9.6 -> 7.2; with the residual test at 50^2
// 10.7 -> 2.9.  V = 8 is the last that gains: ten pairs a thread (400^2) took
// 10.2 us against 10.1.
//
// 1024 consecutive pairs are a block of sor_rb_kernel; S is a multiple of
// 1024, and the field is summed by the same trees and in the same block order:
// every double is that kernel's.
constexpr int SOR_CL_NT = 512;
constexpr int SOR_CL_MAXV = 8;      // pairs per thread
constexpr int SOR_CL_MAXC = 16;     // CTAs of a cluster

__host__ __device__ inline size_t sor_cluster_smem(int S, int half, int nb) {
    return sizeof(double) * (2 * ((size_t)S + 2 * half) + (S / 32) * 33 + (S / 1024) * 33 + 2 * nb);
}

// sum of 32 doubles in the order of a shuffle-down tree (offsets 16, 8, 4, 2, 1)
template <int O> __device__ __forceinline__ double tree32(const double* x, int l) {
    if constexpr (O == 32) return x[l];
    else return tree32<2 * O>(x, l) + tree32<2 * O>(x, l + O);
}
// the same by the four lanes q = 0 .. 3 of a group; every lane gets it
__device__ __forceinline__ double tree32_by4(const double* x, int q) {
    double r = tree32<4>(x, q);
    r += __shfl_down_sync(0xffffffffu, r, 2);
    r += __shfl_down_sync(0xffffffffu, r, 1);
    return __shfl_sync(0xffffffffu, r, 0, 4);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cluster_addr(unsigned local, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// store x at the shared-memory address `local` of CTA `rank` and count its 8 bytes on that CTA's mbarrier
__device__ __forceinline__ void store_counted(unsigned local, unsigned mbar, int rank, double x) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                     cluster_addr(local, rank)),
                 "l"(__double_as_longlong(x)), "r"(cluster_addr(mbar, rank))
                 : "memory");
}

template <int V>
__global__ void __launch_bounds__(SOR_CL_NT, 1) sor_cluster_kernel(SorArgs a) {
    if (a.active && *a.active == 0) return;
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int NT = SOR_CL_NT, S = V * NT;
    static_assert(S % 1024 == 0, "whole blocks");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double s_val, s_res[SOR_CL_MAXC], s_max[NT / 32], s_over[2][SOR_CL_MAXC];
    __shared__ __align__(8) unsigned long long s_bar[6];   // red, black, parts x 2, over x 2
    __shared__ int s_dead, s_any;                          // some thread's wait ran out; some residual is above tol
    const int nc = gridDim.x, c = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nx = a.nx, ny = a.ny, half = (nx + 1) / 2, M = half * ny, W = S + 2 * half;
    const int k0 = c * S, k1 = (k0 + S < M) ? k0 + S : M;
    const int nb = (M + 1023) / 1024, N = nx * ny;
    double* win = reinterpret_cast<double*>(smem_raw);   // red window (slot k - k0 + half), black window (+ W)
    double* scr = win + 2 * W;                           // red + black of each own pair, 33 slots for 32
    double* usum = scr + (S / 32) * 33;                  // sums of 32, 33 slots for the 32 of a block
    double* parts = usum + (S / 1024) * 33;              // every block's sum, of this sweep and the last
    const unsigned bars = smem_addr(s_bar), wins = smem_addr(win);
    enum { RED = 0, BLACK = 8, PARTS = 16, OVER = 32 };
    bool dead = false;
    // Wait for a phase of an mbarrier; bounded: a timeout is recorded, in s_dead too, and ends the thread's further
    // waits.  The CTA must then not arrive again on a phase that is not complete: the next sweep expects nothing and
    // ends where every thread has passed the barrier after the black cells and none can be waiting, so that all of
    // them see the same s_dead.  The other CTAs run out of this one's values in turn.
    auto wait = [&](unsigned bar, unsigned parity) {
        if (dead) return;
        for (int polls = 0;; polls++) {
            unsigned ok = 0;
            asm volatile(
                "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok)
                : "r"(bars + bar), "r"(parity)
                : "memory");
            if (ok) return;
            if (polls >= a.max_polls) { atomicExch(a.bar.err, 1); s_dead = 1; dead = true; return; }
        }
    };
    auto expect = [&](unsigned bar, unsigned bytes) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + bar), "r"(bytes) : "memory");
    };
    // bytes that other CTAs store into a window of this one in a phase (publish, below)
    int halo = (c > 0 ? half : 0) + (c + 1 < nc ? (half < M - k1 ? half : M - k1) : 0);
    if (a.ay.periodic) {
        if (c > 0 && k1 + half > M) halo += k1 + half - M;
        if (c == 0 && nc > 1) halo += half < M - S ? half : M - S;
    }
    const unsigned halo_bytes = 8u * halo, part_bytes = 8u * nb, over_bytes = 8u * nc;
    if (tid == 0) {
        s_dead = 0;
        for (int b = 0; b < 6; b++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8 * b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // What a thread needs of its pairs, formed once: the window slots of the
    // neighbours (16 bits each; .x: the x neighbour beside the pair for the red
    // cell and for the black one, .y: N and S for the red cell, .z for the
    // black one), bits of the pair and where other CTAs hold it (tgt: slot,
    // rank << 16, SEND).  A clamped neighbour is the cell's own slot.
    enum { HAS_R = 1, HAS_B = 2, CLAMPED = 4, ODD = 8, MANY = 16 };
    constexpr unsigned SEND = 0x80000000u;
    uint3 nbr[V];
    unsigned tgt[V];
    unsigned char st[V];
    double vr[V], vb[V], hr[V], hb[V];
    bool edge = false, sends = false;
    // other windows that hold pair k: f(rank, slot in the red window)
    auto holders = [&](int k, auto f) {
        if (c > 0 && k < k0 + half) f(c - 1, k - (k0 - S) + half);
        if (c + 1 < nc && k >= k0 + S - half) f(c + 1, k - (k0 + S) + half);
        if (!a.ay.periodic) return;
        if (k >= M - half) f(0, k - M + half);   // below row 0
        if (k < half)                            // above the last row
            for (int r = nc - 1; r >= 0 && r >= nc - 2; r--) {
                const int end = ((r + 1) * S < M) ? (r + 1) * S : M;
                if (k + M < end + half) f(r, k + M - r * S + half);
            }
    };
    for (int q = tid; q < 2 * W; q += NT) win[q] = 0.0;
    for (int q = tid; q < 2 * nb; q += NT) parts[q] = 0.0;
    for (int q = tid; q < (S / 32) * 33 + (S / 1024) * 33; q += NT) scr[q] = 0.0;
#pragma unroll
    for (int v = 0; v < V; v++) {
        const int own = v * NT + tid, k = k0 + own, me = own + half;
        nbr[v] = make_uint3(0u, 0u, 0u);
        tgt[v] = 0u;
        st[v] = 0;
        vr[v] = vb[v] = hr[v] = hb[v] = 0.0;
        if (k >= k1) continue;
        const int j = k / half, p = k - j * half, odd = j & 1;
        const int ir = 2 * p + odd, ib = 2 * p + 1 - odd;
        const bool perx = a.ax.periodic, pery = a.ay.periodic;
        // A cell's x neighbours: the pair's other cell on one side (east of an even column, west of
        // an odd one), a cell of the pair before or after on the other; a clamped one is the cell itself.
        // slot of the one beside the pair, `oth` the offset of its colour's window
        auto beside = [&](int i, int own_w, int oth) {
            if (i & 1) return i + 1 < nx ? oth + me + 1 : (perx ? oth + me - half + 1 : own_w + me);
            return i > 0 ? oth + me - 1 : (perx ? oth + me + half - 1 : own_w + me);
        };
        int f = odd ? ODD : 0;
        if (ir < nx) f |= HAS_R;
        if (ib < nx) f |= HAS_B;
        // the last pair of an odd nx has one cell, an even column whose east neighbour is clamped
        if ((!pery && (j == 0 || j + 1 == ny)) || (!perx && (ib == 0 || ib == nx - 1 || ir == 0 || ir == nx - 1))) f |= CLAMPED;
        nbr[v].x = (unsigned)beside(ir, 0, W) | ((unsigned)beside(ib, W, 0) << 16);
        const int up = (j + 1 < ny || pery) ? half : 0, down = (j > 0 || pery) ? half : 0;
        nbr[v].y = (unsigned)(me + (up ? W + up : 0)) | ((unsigned)(me + (down ? W - down : 0)) << 16);
        nbr[v].z = (unsigned)(me + (up ? up : W)) | ((unsigned)(me + (down ? -down : W)) << 16);
        int holds = 0;
        holders(k, [&](int rank, int slot) { tgt[v] = SEND | ((unsigned)rank << 16) | (unsigned)slot; holds++; });
        if (holds > 1 || (holds == 1 && (int)((tgt[v] >> 16) & 0xff) == c)) f |= MANY;
        edge |= holds > 0 && nc > 1;
        sends |= holds > 0;
        st[v] = (unsigned char)f;
        if (ir < nx) hr[v] = a.rhs[(size_t)j * nx + ir];
        if (ib < nx) hb[v] = a.rhs[(size_t)j * nx + ib];
    }
    edge = __any_sync(0xffffffffu, edge);   // the warp reads other CTAs' pairs
    // store the value of the thread's pair v also where other CTAs (or the periodic images) read it
    auto publish = [&](int v, int off, unsigned bar, double x) {   // off: 0 the red window, W the black one
        if (!tgt[v]) return;
        if (!(st[v] & MANY)) {
            store_counted(wins + 8 * ((tgt[v] & 0xffffu) + off), bars + bar, (tgt[v] >> 16) & 0xff, x);
            return;
        }
        holders(k0 + v * NT + tid, [&](int rank, int slot) {
            if (rank == c) win[off + slot] = x;
            else store_counted(wins + 8 * (off + slot), bars + bar, rank, x);
        });
    };
    cl.sync();
    const double inv_denom = 1.0 / a.denom, cells = (double)N, inv_cells = 1.0 / cells;
    const bool denom_ok = divisor_inside(a.denom);
    const double omega = a.omega, idx2 = a.idx2, idy2 = a.idy2, tol = a.tol;
    double m = 0.0;   // mean removal pending on every cell not yet rewritten in this sweep
    double res = 0.0;
    int it = 0;
    bool gave_up = false;   // the same in every thread of a CTA
    // the neighbours W, E, N, S of the red (col 0) or black cell of pair v; `other`: the pair's other cell
    auto gather = [&](int v, int col, double other, double& pW, double& pE, double& pN, double& pS) {
        const unsigned y = col ? nbr[v].z : nbr[v].y;
        const double b = win[col ? nbr[v].x >> 16 : nbr[v].x & 0xffffu];
        // red cells of odd rows and black cells of even rows lie in odd columns
        const bool oddcol = ((st[v] & ODD) != 0) != (col != 0);
        pN = win[y & 0xffffu];
        pS = win[y >> 16];
        pW = oddcol ? other : b;
        pE = oddcol ? b : other;
    };
    // whether the quotient a / denom needs the division (an extreme a; a zero does not)
    auto extreme = [&](double q) {
        return !(denom_ok && quotient_inside(q));
    };
    // max |lap(phi - m) - rhs| over the thread's cells
    auto residual = [&]() {
        double r = 0.0;
#pragma unroll
        for (int v = 0; v < V; v++) {
#pragma unroll
            for (int col = 0; col < 2; col++) {
                if (!(st[v] & (col == 0 ? HAS_R : HAS_B))) continue;
                double pW, pE, pN, pS;
                gather(v, col, col == 0 ? vb[v] : vr[v], pW, pE, pN, pS);
                const double x = (col == 0 ? vr[v] : vb[v]) - m;
                pW -= m; pE -= m; pN -= m; pS -= m;
                const double lap = (pE - 2.0 * x + pW) * idx2 + (pN - 2.0 * x + pS) * idy2;
                r = fmax(r, fabs(lap - (col ? hb[v] : hr[v])));
            }
        }
        return r;
    };
    // max over the cluster of the threads' r; every CTA gets it
    auto cluster_max = [&](double r) {
        for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_down_sync(0xffffffffu, r, o));
        if (lane == 0) s_max[warp] = r;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < NT / 32; w++) r = fmax(r, s_max[w]);
            for (int q = 0; q < nc; q++) cl.map_shared_rank(s_res, q)[c] = r;
        }
        cl.sync();
        double x = 0.0;
        for (int q = 0; q < nc; q++) x = fmax(x, s_res[q]);
        return x;
    };
    for (; it < a.max_iter; ++it) {
        const unsigned ph = it & 1, ph2 = (it >> 1) & 1, two = 8 * (it & 1);
        // Red: every value read is pending.  No branch but the rare ones, so that the V cells' chains
        // overlap.  A cell that does not exist (odd nx) takes the value that its neighbour, whose
        // clamped east it stands for, has there.
        {
            double q[V];
            bool rare = false;
#pragma unroll
            for (int v = 0; v < V; v++) {
                double pW, pE, pN, pS;
                gather(v, 0, vb[v], pW, pE, pN, pS);
                q[v] = ((pE - m) + (pW - m)) * idx2 + ((pN - m) + (pS - m)) * idy2 - hr[v];
                rare |= extreme(q[v]);
            }
            if (rare) {
#pragma unroll
                for (int v = 0; v < V; v++) q[v] = q[v] / a.denom;
            } else {
#pragma unroll
                for (int v = 0; v < V; v++) q[v] = quotient_fast(q[v], a.denom, inv_denom);
            }
#pragma unroll
            for (int v = 0; v < V; v++) {
                const double x = vr[v] - m;
                vr[v] = (st[v] & HAS_R) ? x + omega * (q[v] - x) : vb[v] - m;
                if (st[v] & HAS_R) win[v * NT + tid + half] = vr[v];
            }
        }
        if (sends) {
#pragma unroll
            for (int v = 0; v < V; v++) publish(v, 0, RED, vr[v]);
        }
        if (tid == 0 && !s_dead) {   // here rather than first: warp 0 is about to wait
            if (nc > 1) { expect(RED, halo_bytes); expect(BLACK, halo_bytes); }
            expect(PARTS + two, part_bytes);
        }
        if (edge) wait(RED, ph);
        __syncthreads();
        // Black: the red neighbours are rewritten, a clamped one (the cell itself) is
        // pending.  Sum every cell of the new field.
        {
            double q[V], x[V];
            bool rare = false;
#pragma unroll
            for (int v = 0; v < V; v++) {
                x[v] = vb[v] - m;
                if (st[v] & CLAMPED) win[v * NT + tid + half + W] = x[v];   // read back as the clamped neighbour
                double pW, pE, pN, pS;
                gather(v, 1, vr[v], pW, pE, pN, pS);
                q[v] = (pE + pW) * idx2 + (pN + pS) * idy2 - hb[v];
                rare |= extreme(q[v]);
            }
            if (rare) {
#pragma unroll
                for (int v = 0; v < V; v++) q[v] = q[v] / a.denom;
            } else {
#pragma unroll
                for (int v = 0; v < V; v++) q[v] = quotient_fast(q[v], a.denom, inv_denom);
            }
#pragma unroll
            for (int v = 0; v < V; v++) {
                double s = 0.0;
                if (st[v] & HAS_R) s += vr[v];
                const double y = x[v] + omega * (q[v] - x[v]);
                if (st[v] & HAS_B) s += y;
                vb[v] = (st[v] & HAS_B) ? y : vr[v];
                vr[v] = (st[v] & HAS_R) ? vr[v] : y;
                if (st[v] & HAS_B) win[v * NT + tid + half + W] = y;
                scr[(v * (NT / 32) + warp) * 33 + lane] = s;
            }
        }
        if (sends) {
#pragma unroll
            for (int v = 0; v < V; v++) publish(v, W, BLACK, vb[v]);
        }
        __syncthreads();
        // sums of 32 pairs by four lanes each, then the blocks' sums, to every CTA
        const int q4 = tid & 3;
#pragma unroll
        for (int i = 0; i < (4 * S / 32 + NT - 1) / NT; i++) {
            const int u = (i * NT + tid) >> 2;
            if (4 * S / 32 % NT == 0 || u < S / 32) {   // whole warps
                const double s = tree32_by4(scr + 33 * u, q4);
                if (q4 == 0) usum[(u >> 5) * 33 + (u & 31)] = s;
            }
        }
        const int stop = s_dead;   // written before the last barrier or behind the next one
        __syncthreads();
        if (stop) { gave_up = true; break; }
        double* pt = parts + (it & 1) * nb;
        if (warp == 0) {
            const int v = lane >> 2, b = c * (S / 1024) + v;
            const double s = tree32_by4(usum + 33 * (v < S / 1024 ? v : 0), q4);
            if (v < S / 1024 && b < nb)
                for (int q = q4; q < nc; q += 4) store_counted(smem_addr(pt + b), bars + PARTS + two, q, s);
            wait(PARTS + two, ph2);
            if (lane == 0) {   // in block order
                double t = 0.0;
#pragma unroll 8
                for (int q = 0; q < nb; q++) t += pt[q];
                s_val = quotient(t, cells, inv_cells);
            }
        }
        if (edge) wait(BLACK, ph);
        __syncthreads();
        m = s_val;
        if (tol > 0.0) {
            // the sweep's residual is needed only as "below tol or not", except after the last one
            const double r = residual();
            int any = __syncthreads_or(!(r < tol));
            if (nc > 1) {
                if (warp == 0) {
                    if (tid == 0) expect(OVER + two, over_bytes);
                    if (lane < nc) store_counted(smem_addr(&s_over[it & 1][c]), bars + OVER + two, lane, any ? 1.0 : 0.0);
                    wait(OVER + two, ph2);
                    const double o = lane < nc ? s_over[it & 1][lane] : 0.0;
                    any |= __any_sync(0xffffffffu, dead || o != 0.0);
                    if (lane == 0) s_any = any;
                }
                __syncthreads();   // one warp waits and decides, so that every thread goes the same way
                any = s_any;
            }
            if (!any || it + 1 == a.max_iter) res = cluster_max(r);
            if (!any) { ++it; break; }
        }
    }
    if (!(tol > 0.0) || gave_up) res = cluster_max(residual());   // once in every CTA, however it left the sweeps
#pragma unroll
    for (int v = 0; v < V; v++) {
        const int k = k0 + v * NT + tid;
        if (k >= k1) continue;
        const int j = k / half, p = k - j * half, odd = j & 1, ir = 2 * p + odd, ib = 2 * p + 1 - odd;
        if (ir < nx) a.phi[(size_t)j * nx + ir] = vr[v] - m;
        if (ib < nx) a.phi[(size_t)j * nx + ib] = vb[v] - m;
    }
    if (c == 0 && tid == 0) { *a.iters_out = it; *a.res_out = res; }
    cl.sync();   // no CTA leaves while another may still store into its shared memory
    if (s_dead)   // what was under way to it when a wait ran out
        for (int k = 0; k < 100; k++) __nanosleep(1000);
}

// rhs = 4 pi G (rho - mean) (M2:187-194), mean from the density partial sums.
// floor_rho >= 0: the density is floored first (EH:312), and the partial sums
// must then be sums of the floored density.
template <class T>
__global__ void sor_rhs_kernel(const T* __restrict__ rho, int nx, int ny, int pitch, const double* __restrict__ rho_part,
                               int nparts, double fourpiG, double floor_rho, double* __restrict__ rhs,
                               const int* __restrict__ active) {
    if (active && *active == 0) return;
    __shared__ double s_mean;
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int b = 0; b < nparts; b++) s += rho_part[b];
        s_mean = s / ((double)nx * (double)ny);
    }
    __syncthreads();
    const double mean = s_mean;
    const int N = nx * ny;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < N; k += gridDim.x * blockDim.x) {
        const int i = k % nx, j = k / nx;
        double r = (double)rho[(size_t)j * pitch + i];
        if (floor_rho >= 0.0) r = vmax(r, floor_rho);
        rhs[k] = fourpiG * (r - mean);
    }
}

// copy the contiguous FP64 phi into the pitched T field the stage kernel reads
template <class T>
__global__ void phi_to_field_kernel(const double* __restrict__ phi, int nx, int ny, T* __restrict__ out, int pitch,
                                    const int* __restrict__ active) {
    if (active && *active == 0) return;
    const int N = nx * ny;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < N; k += gridDim.x * blockDim.x) {
        const int i = k % nx, j = k / nx;
        out[(size_t)j * pitch + i] = (T)phi[k];
    }
}

// g = -grad(phi) (M2:225-235), written pitched, for the host-facing gravity call
template <class T>
__global__ void gravity_from_phi_kernel(const T* __restrict__ phi, int nx, int ny, int pitch, AxisMap ax, AxisMap ay,
                                        T two_dx, T two_dy, T* __restrict__ gx, T* __restrict__ gy) {
    const int N = nx * ny;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < N; k += gridDim.x * blockDim.x) {
        const int i = k % nx, j = k / nx;
        const size_t q = (size_t)j * pitch + i;
        gx[q] = -(phi[(size_t)j * pitch + ax.cell(i + 1)] - phi[(size_t)j * pitch + ax.cell(i - 1)]) / two_dx;
        gy[q] = -(phi[(size_t)ay.cell(j + 1) * pitch + i] - phi[(size_t)ay.cell(j - 1) * pitch + i]) / two_dy;
    }
}

}  // namespace ccb
