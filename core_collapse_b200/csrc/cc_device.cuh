// Device-side helpers shared by every kernel of libcc_b200: min/max with the
// reference's std::max/std::min semantics, index wrapping, deterministic block
// reductions and a bounded grid barrier for persistent kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ccb {

// std::max(a,b) == (a<b)?b:a, std::min(a,b) == (b<a)?b:a.  Kept exactly so
// that branch-sensitive code (floors, limiter, wave-speed bounds) takes the
// same branches as the reference.
template <class T> __host__ __device__ __forceinline__ T vmax(T a, T b) { return (a < b) ? b : a; }
template <class T> __host__ __device__ __forceinline__ T vmin(T a, T b) { return (b < a) ? b : a; }

// The reference's positive guard 1e-300 (a division or square-root floor); FP32
// cannot hold it and its instantiations use 1e-30, a normal FP32 value far
// below every density floor
template <class T> __host__ __device__ constexpr T tiny_pos() { return sizeof(T) == 4 ? T(1e-30f) : T(1e-300); }

__host__ __device__ __forceinline__ int wrap_idx(int i, int n) { int r = i % n; return (r < 0) ? r + n : r; }
__host__ __device__ __forceinline__ int clamp_idx(int i, int lo, int hi) { return i < lo ? lo : (i > hi ? hi : i); }

// Correctly rounded FP64 quotients without a branch.  A division waits for the
// one before it: measured, a chain of 120 cycles each, and 107 cycles of a
// warp's issue instead of 27 when the numerator is a zero, which the velocity and
// field components that a planar flow does not have are.  The forms below
// overlap, and quotients of one denominator share its reciprocal.
//   y = RN(1/b): two Newton-Raphson steps y <- y + y (1 - b y), each of which
//   squares the relative error, from a starting value within 2^-14: 2^-28, then
//   2^-56 before the rounding of y, so y is within one ulp; then one more step,
//   which rounds it correctly unless b's significand is all ones.
//   a / b from y: q0 = a y is within two ulps, q1 = q0 + (a - b q0) y is a
//   faithful quotient, and from a faithful quotient the same step gives RN(a/b).
// The Newton-Raphson iteration with fused multiply-adds, its last step and the
// quotient's are Markstein's (P. Markstein, Computation of elementary functions
// on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  They hold
// while nothing leaves the normal range: divisor_inside and quotient_inside; what
// they refuse, a caller divides.
__device__ __forceinline__ double recip_start(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
}
__device__ __forceinline__ double newton_step(double b, double y) { return __fma_rn(y, __fma_rn(-b, y, 1.0), y); }
__device__ __forceinline__ double recip_fast(double b) {
    return newton_step(b, newton_step(b, newton_step(b, recip_start(b))));
}
__device__ __forceinline__ double quotient_fast(double a, double b, double y) {
    const double q0 = a * y;
    const double q1 = __fma_rn(-__fma_rn(b, q0, -a), y, q0);
    return __fma_rn(-__fma_rn(b, q1, -a), y, q1);
}
__device__ __forceinline__ bool divisor_inside(double b) {    // 2^-100 <= |b| < 2^101, significand not all ones
    const unsigned hi = (unsigned)__double2hiint(b);
    return (hi & 0x7fffffffu) - 0x39b00000u < 0x0c900000u && ((hi | 0xfff00000u) & (unsigned)__double2loint(b)) != ~0u;
}
__device__ __forceinline__ bool quotient_inside(double a) {   // a zero, or 2^-895 <= |a| < 2^769 (1 + 2^-20)
    const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return hi - 0x08000000u <= 0x68000000u || (hi | (unsigned)__double2loint(a)) == 0u;
}
// a / b with y = RN(1/b) at hand (by a zero the sign of the zero may be the other one for b < 0)
__device__ __forceinline__ double quotient(double a, double b, double y) {
    return divisor_inside(b) && quotient_inside(a) ? quotient_fast(a, b, y) : a / b;
}

// The divisions of a pointwise function in type T.  FP32: one reciprocal per
// shared denominator and products with it.  FP64: the host and PLAIN divide; the
// device forms quotients by the functions above and sets `rare` where one of
// them is outside their range: the caller then evaluates the function again
// with PLAIN.  So every FP64 result is the divisions' own.
template <class T, bool PLAIN> struct Div {
    bool rare = false;
#if defined(__CUDA_ARCH__)
    static constexpr bool FAST64 = sizeof(T) == 8 && !PLAIN;
#else
    static constexpr bool FAST64 = false;
#endif
    // what quot takes beside the denominator b
    __host__ __device__ __forceinline__ T recip(T b) {
#if defined(__CUDA_ARCH__)
        if constexpr (FAST64) {
            rare |= !divisor_inside(b);
            return recip_fast(b);
        }
#endif
        if constexpr (sizeof(T) == 4) return T(1.0) / b;
        else return T(0.0);
    }
    __host__ __device__ __forceinline__ T quot(T a, T b, T y) {
#if defined(__CUDA_ARCH__)
        if constexpr (FAST64) {
            rare |= !quotient_inside(a);
            return quotient_fast(a, b, y);
        }
#endif
        if constexpr (sizeof(T) == 4) return a * y;
        else return a / b;
    }
    // the same with a reciprocal that the host has rounded (constants of the grid)
    __host__ __device__ __forceinline__ T quot_by(T a, T b, T y) {
#if defined(__CUDA_ARCH__)
        if constexpr (FAST64) rare |= !divisor_inside(b);
#endif
        return quot(a, b, y);
    }
    // a / b by a constant of the grid whose reciprocal y the host has rounded; FP32 divides (quot_by: a y, which
    // rounds differently)
    __host__ __device__ __forceinline__ T quot_grid(T a, T b, T y) {
        if constexpr (sizeof(T) == 4) return a / b;
        else return quot_by(a, b, y);
    }
    // a / b, a denominator of its own
    __host__ __device__ __forceinline__ T div(T a, T b) {
        if constexpr (FAST64) return quot(a, b, recip(b));
        else return a / b;
    }
};

// f(d) with the fast divisions, again with the plain ones where they do not apply
template <class T, class F> __host__ __device__ __forceinline__ auto divided(F f) {
    Div<T, false> d;
    auto r = f(d);
    if constexpr (Div<T, false>::FAST64) {
        if (d.rare) {
            Div<T, true> p;
            r = f(p);
        }
    }
    return r;
}

// One grid axis.  Cell indices wrap modulo n (periodic) or clamp to [0,n-1];
// face indices along the axis wrap modulo n+1 or clamp to [0,n]
// (mhd2d_resistive_hlld_ct_gravity.cpp:241-252).
struct AxisMap {
    int n;
    int periodic;
    __host__ __device__ __forceinline__ int cell(int i) const {
        if (i >= 0 && i < n) return i;
        return periodic ? wrap_idx(i, n) : clamp_idx(i, 0, n - 1);
    }
    __host__ __device__ __forceinline__ int face(int i) const {
        if (i >= 0 && i <= n) return i;
        return periodic ? wrap_idx(i, n + 1) : clamp_idx(i, 0, n);
    }
};

// Deterministic sum over a block: fixed shuffle tree inside each warp, then
// warp partials summed in warp order by warp 0.  Result valid in thread 0.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double* sh /* >= NT/32 */) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = (l < NT / 32) ? sh[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    __syncthreads();
    return r;
}

// Max over a block of non-negative values (order-free).  Result in thread 0.
template <int NT>
__device__ __forceinline__ double block_max(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = (l < NT / 32) ? sh[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_down_sync(0xffffffffu, r, o));
    }
    __syncthreads();
    return r;
}

// block_max and block_sum of two values at once, with the same orders (so
// the same bits) and one barrier pair instead of two.  Results in thread 0.
template <int NT>
__device__ __forceinline__ void block_max_sum(double& vmax_, double& vsum, double* sh /* >= 2 NT/32 */) {
    for (int o = 16; o > 0; o >>= 1) {
        vmax_ = fmax(vmax_, __shfl_down_sync(0xffffffffu, vmax_, o));
        vsum += __shfl_down_sync(0xffffffffu, vsum, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sh[w] = vmax_; sh[NT / 32 + w] = vsum; }
    __syncthreads();
    if (w == 0) {
        double m = (l < NT / 32) ? sh[l] : 0.0, r = (l < NT / 32) ? sh[NT / 32 + l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
            r += __shfl_down_sync(0xffffffffu, r, o);
        }
        vmax_ = m;
        vsum = r;
    }
    __syncthreads();
}

// Grid-wide barrier for kernels launched cooperatively (all blocks resident).
// Sense is a generation counter.  The wait is bounded: after max_spins polls the
// block records an error in *err and leaves; callers test the return value and
// stop their loop, so a failed barrier ends the kernel instead of hanging it.
struct GridBarrier {
    unsigned int* count;   // zero-initialised
    unsigned int* gen;     // any start value
    int* err;              // zero-initialised; set to 1 on timeout
};

__device__ __forceinline__ bool grid_sync(const GridBarrier& b, unsigned nblocks) {
    __syncthreads();
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        volatile unsigned int* vgen = b.gen;
        unsigned int g = *vgen;
        __threadfence();
        unsigned int arrived = atomicAdd(b.count, 1u);
        int ok = 1;
        if (arrived == nblocks - 1) {
            atomicExch(b.count, 0u);
            __threadfence();
            atomicAdd(b.gen, 1u);
        } else {
            long long spins = 0;
            while (*vgen == g) {
                if (*(volatile int*)b.err) { ok = 0; break; }
                if (++spins > (1ll << 24)) { atomicExch(b.err, 1); ok = 0; break; }
                __nanosleep(64);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

}  // namespace ccb
