// One RK stage of the 2D FP32 path in registers: a warp owns a strip of 28
// columns (a lane to a column, two halo lanes on either side) over a segment of
// rows and marches up it, one row per step.  x neighbours are shuffles, y
// neighbours are the values a lane carried from the rows below, so the stage
// uses no shared memory and no barrier, and every slope, face and edge of the
// strip is formed once.
//
// Why: the tile kernel (m2_stage_tile) is bound by instruction issue, and of
// its 1800 instructions a cell about half move operands through shared memory
// (primitives, slopes and fluxes written and read back with their index
// arithmetic) or recompute the tile's halo.  Here a cell takes the physics, 35
// shuffles and its global loads; the strip's halo lanes cost 32/28, the rows a
// segment starts with 2 rows of x faces and 4 of primitives.
//
// Same functions as the tile kernel (Stage32, hlld_x2, joule_from), so the same bits.
// That is kept on purpose: some FP32 runs amplify a last bit to 1e-3 of a weak
// field within a hundred steps, so a cheaper HLLD with shared reciprocals (598 /
// 715 us below) would have changed their results.
//
// Bound: issue (73% of the slots at 16 warps an SM; 128 registers allow no more,
// and 20 warps at 96 registers spilled: 722 us) and the latency of a row's two
// HLLD chains.  4096^2 with gravity, first / second stage of a step: tiles 1103
// / 1156 us -> 652 / 771.  On the way: the potential carried instead of read at
// the update (717 -> 611 with the cheaper HLLD: a load there is waited for), the
// state before the update kept in shared memory instead of read again and the
// Joule sub-step from shuffles (864 -> 715, second stage).  1003 x 777: 51 / 54
// us -> 37 / 44.  The rows of a segment and the grids that keep the tiles:
// lane_rows.
#pragma once
#include "mhd2d_kernels.cuh"

namespace ccb {

constexpr int LANE_W = 28;       // columns a warp owns
constexpr int LANE_NT = 128;     // four warps to a CTA, on adjacent strips

__device__ __forceinline__ float lane_up(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }      // from column i - 1
__device__ __forceinline__ float lane_down(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }  // from column i + 1

// components of a row that have slopes: r, u, v, w, P, bz and the transverse in-plane field
struct Row7 { float r, u, v, w, P, bz, bt; };
template <class F> __device__ __forceinline__ Row7 row7(const Row7& a, const Row7& b, F f) {
    return Row7{f(a.r, b.r), f(a.u, b.u), f(a.v, b.v), f(a.w, b.w), f(a.P, b.P), f(a.bz, b.bz), f(a.bt, b.bt)};
}
template <class F> __device__ __forceinline__ Row7 row7(const Row7& a, F f) {
    return Row7{f(a.r), f(a.u), f(a.v), f(a.w), f(a.P), f(a.bz), f(a.bt)};
}

// half the MC slope from its two differences (mc_slope; what a face state adds to the cell's value)
__device__ __forceinline__ float half_mc(float dm, float dp) {
    const float m = fminf(fabsf(0.25f * (dm + dp)), fminf(fabsf(dm), fabsf(dp)));
    return (dm * dp <= 0.0f) ? 0.0f : copysignf(m, dm);
}

// What a lane keeps for the update of a row and needs nowhere else, in its own
// slots of shared memory (no lane reads another's): the state and cell-centred
// B of the last three rows, and of the last row the x-flux differences and
// lower y-face fluxes (rho, mx, my, mz, E, Bz).
struct LaneKeep {
    float4 u[3][2][LANE_NT];
    float4 f[3][LANE_NT];
};

template <bool DEFER, int GMODE, ESum ES>
__device__ __forceinline__ void m2_lane_segment(LaneKeep& keep, const M2Const<float>& c, const Fields<float>& in, const Fields<float>& out,
                                                const float* __restrict__ ga, const float* __restrict__ gb, const float dt,
                                                const int strip, const int j0, const int j1) {
    const int tid = threadIdx.x, lane = tid & 31;
    int slot = 0;   // of keep.u, for row r
    const int P = c.pitch, nx = c.nx, ny = c.ny;
    const int gi = strip * LANE_W - 2 + lane;
    const int ci = c.ax.cell(gi);
    const bool cell = lane >= 2 && lane < 2 + LANE_W && gi < nx;            // owns the cells of column gi
    const bool face = cell || (gi == nx && lane >= 2 && lane <= 2 + LANE_W);   // and its x faces (the last one: face nx)
    const float dtdy = dt / c.dy, dtdx = dt / c.dx;

    // raw state of the next row
    // (DEFER: and what its Joule sub-step reads of the row above it; zN, bN)
    struct Raw { float rho, mx, my, mz, E, Bz, b0, b1, y0, y1, zN, bN, phi; } raw;
    auto load = [&](int row) {
        const size_t q = (size_t)c.ay.cell(row) * P + ci;
        raw.rho = in.rho[q]; raw.mx = in.mx[q]; raw.my = in.my[q]; raw.mz = in.mz[q]; raw.E = in.E[q]; raw.Bz = in.Bz[q];
        raw.b0 = in.bx[q]; raw.b1 = in.bx[q + 1]; raw.y0 = in.by[q]; raw.y1 = in.by[q + P];
        if (GMODE == GRAV_PHI) raw.phi = __ldg(ga + q);
        if (DEFER) {
            // the neighbour rows of the cell that the row stands for (a clamped row repeats it)
            const size_t qn = (size_t)c.ay.cell(c.ay.cell(row) + 1) * P + ci;
            raw.zN = in.Bz[qn]; raw.bN = in.bx[qn];
        }
    };
    float zS = 0.f;   // DEFER: Bz of the row below the one being read
    // the cell's neighbour columns, and whether a lane beside holds them (not at
    // the warp's ends, nor where a clamped halo column repeats the edge cell)
    const int ciE = c.ax.cell(ci + 1), ciW = c.ax.cell(ci - 1);
    const bool readE = lane == 31 || c.ax.cell(gi + 1) != ciE, readW = lane == 0 || c.ax.cell(gi - 1) != ciW;

    // carried from row to row (row r is the one being read; w: row r - 1)
    Prim<float> w{1.f, 0.f, 0.f, 0.f, 1.f, 0.f, 0.f, 0.f};
    Row7 dm{};                    // differences W[r-1] - W[r-2] (bt = Bx: the y direction's)
    Row7 plus{};                  // upper face state of row r - 2
    float F5 = 0.f, Ez = 0.f, bnx = 0.f, byD = 0.f;   // of row r - 2
    float ph1 = 0.f, ph2 = 0.f, ph3 = 0.f;   // potential of rows r - 1, r - 2, r - 3
    float wb0 = 0.f, wb1 = 0.f, wy0 = 0.f;   // x faces and lower y face of row r - 1

    load(j0 - 2);
    for (int r = j0 - 2; r <= j1 + 1; ++r) {
        // ---- primitives of row r (get_prim_cc, M2:278-286) ----
        float rho = raw.rho, E = raw.E, Bz = raw.Bz;
        const float mx = raw.mx, my = raw.my, mz = raw.mz;
        const float Bx = 0.5f * (raw.b0 + raw.b1), By = 0.5f * (raw.y0 + raw.y1);
        if (DEFER && c.resistive) {
            // Joule heating and Bz diffusion of the stored pre-Joule state (joule_cell, M2:631-686)
            const int cj = c.ay.cell(r);
            float zE = lane_down(Bz), zW = lane_up(Bz), yE = lane_down(raw.y0);
            if (readE) { zE = in.Bz[(size_t)cj * P + ciE]; yE = in.by[(size_t)cj * P + ciE]; }
            if (readW) zW = in.Bz[(size_t)cj * P + ciW];
            const int cjS = c.ay.cell(cj - 1);   // the row read before, unless this is a segment's first or a clamped repeat
            if (r == j0 - 2 || c.ay.cell(r - 1) != cjS) zS = in.Bz[(size_t)cjS * P + ci];
            const float zC = Bz;
            float J2, lap;
            joule_from<float, ES>(c, zE, zW, raw.zN, zS, zC, yE - raw.y0, raw.bN - raw.b0, J2, lap);
            joule_add<float, ES>(c, dt, J2, lap, rho, mx, my, mz, E, Bz, Bx, By);
        }
        if (DEFER) zS = raw.Bz;
        const float rb0 = raw.b0, rb1 = raw.b1, ry0 = raw.y0, rphi = GMODE == GRAV_PHI ? raw.phi : 0.f;
        if (r <= j1) load(r + 1);
        keep.u[slot][0][tid] = make_float4(rho, mx, my, mz);
        keep.u[slot][1][tid] = make_float4(E, Bz, Bx, By);
        const Prim<float> W = Stage32<ES>::to_prim(c, rho, mx, my, mz, E, Bx, By, Bz);
        // ---- slopes of row r - 1 along y; its face states ----
        const Row7 dp{W.r - w.r, W.u - w.u, W.v - w.v, W.w - w.w, W.P - w.P, W.bz - w.bz, W.bx - w.bx};
        if (r >= j0) {
            const Row7 sy = row7(dm, dp, half_mc);
            const Row7 c1{w.r, w.u, w.v, w.w, w.P, w.bz, w.bx};
            const Row7 lo = row7(c1, sy, [](float a, float s) { return a - s; });
            const int row = r - 1;                       // x faces of rows j0 - 1 .. j1
            // ---- x faces of row r - 1: lane i holds face gi, between columns gi - 1 and gi ----
            float Fx[7];
            // face gi of the row: the cell's left face, or the last cell's right one (the face arrays do not wrap there)
            float bn = lane_up(wb1);
            if (gi != nx) bn = wb0;
            {
                const Row7 x1{w.r, w.u, w.v, w.w, w.P, w.bz, w.by};
                const Row7 xm = row7(x1, [](float a) { return a - lane_up(a); });
                const Row7 sx = row7(xm, [](float a) { return half_mc(a, lane_down(a)); });
                const Row7 xl = row7(row7(x1, sx, [](float a, float s) { return a + s; }), lane_up);
                const Row7 xr = row7(x1, sx, [](float a, float s) { return a - s; });
                Prim2 S;
                S.r = pk(fmaxf(xl.r, c.floor_rho), fmaxf(xr.r, c.floor_rho));
                S.P = pk(fmaxf(xl.P, c.floor_P), fmaxf(xr.P, c.floor_P));
                S.u = pk(xl.u, xr.u); S.v = pk(xl.v, xr.v); S.w = pk(xl.w, xr.w);
                S.bx = pbc(bn); S.by = pk(xl.bt, xr.bt); S.bz = pk(xl.bz, xr.bz);
                const Flux<float> F = hlld_x2<ES>(c, S, bn);
                Fx[0] = F.f0; Fx[1] = F.f1; Fx[2] = F.f2; Fx[3] = F.f3; Fx[4] = F.f4; Fx[5] = F.f5; Fx[6] = F.f6;
            }
            // ---- y face r - 1, between rows r - 2 and r - 1; edges and faces of that row ----
            float Gy[7] = {}, ez = 0.f, byN = 0.f;
            if (r > j0) {
                const float bnY = row == ny ? in.by[(size_t)ny * P + ci] : wy0;
                Prim2 S;   // in x orientation (hlld_y's swap of (u, v) and (Bx, By))
                S.r = pk(fmaxf(plus.r, c.floor_rho), fmaxf(lo.r, c.floor_rho));
                S.P = pk(fmaxf(plus.P, c.floor_P), fmaxf(lo.P, c.floor_P));
                S.u = pk(plus.v, lo.v); S.v = pk(plus.u, lo.u); S.w = pk(plus.w, lo.w);
                S.bx = pbc(bnY); S.by = pk(plus.bt, lo.bt); S.bz = pk(plus.bz, lo.bz);
                const Flux<float> F = hlld_x2<ES>(c, S, bnY);
                Gy[0] = F.f0; Gy[1] = F.f2; Gy[2] = F.f1; Gy[3] = F.f3; Gy[4] = F.f4; Gy[5] = F.f5; Gy[6] = F.f6;
                // edge EMF at the lower left corner of the row's cells (M2:782-804)
                const float exm = -F5, ex0 = -Fx[5], ey0 = Gy[5], eym = lane_up(ey0);
                const float ideal = 0.25f * (exm + ex0 + eym + ey0);
                float res = 0.f;
                if (c.resistive) {
                    const float dby = bnY - lane_up(bnY), dbx = bn - bnx;
                    res = resistive_emf<float, ES>(c, dby, dbx);
                }
                ez = ideal + res;
                // CT of the row's lower y faces (M2:819-830)
                byN = Stage32<ES>::ct(bnY, dtdx, lane_down(ez) - ez);
                if (cell && (row < j1 || row == ny)) out.by[(size_t)row * P + gi] = byN;
            }
            // ---- finish the cells of row r - 2: update, floors, CT, gravity, store (M2:750-779, 807-832) ----
            if (r >= j0 + 2) {
                const int jr = r - 2;
                const size_t qb = (size_t)jr * P;
                const float bxN = Stage32<ES>::ct(bnx, -dtdy, ez - Ez);
                const float bxR = lane_down(bxN);
                float pE1 = 0.f, pW1 = 0.f;
                if (GMODE == GRAV_PHI) { pE1 = lane_down(ph2); pW1 = lane_up(ph2); }
                if (face) out.bx[qb + gi] = bxN;
                if (cell) {
                    const size_t q = qb + gi;
                    const int old = slot == 2 ? 0 : slot + 1;   // row r - 2
                    const float4 a = keep.u[old][0][tid], b = keep.u[old][1][tid];
                    float u0 = a.x, u1 = a.y, u2 = a.z, u3 = a.w, u4 = b.x, u5 = b.y;
                    const float bxc = b.z, byc = b.w;
                    const float4 f0 = keep.f[0][tid], f1 = keep.f[1][tid], f2 = keep.f[2][tid];
                    using S = Stage32<ES>;
                    u0 = S::update(c, u0, dt, f0.x, Gy[0] - f1.z);
                    u1 = S::update(c, u1, dt, f0.y, Gy[1] - f1.w);
                    u2 = S::update(c, u2, dt, f0.z, Gy[2] - f2.x);
                    u3 = S::update(c, u3, dt, f0.w, Gy[3] - f2.y);
                    u4 = S::update(c, u4, dt, f1.x, Gy[4] - f2.z);
                    u5 = S::update(c, u5, dt, f1.y, Gy[6] - f2.w);
                    S::floors(c, u0, u1, u2, u3, u4, bxc, byc, u5);
                    if (GMODE != GRAV_NONE && c.gravity_on) {
                        float gxq, gyq;
                        if (GMODE == GRAV_ARRAYS) {
                            gxq = ga[q]; gyq = gb[q];
                        } else {
                            gxq = -(pE1 - pW1) * (0.5f * c.inv_dx);
                            gyq = -(ph1 - ph3) * (0.5f * c.inv_dy);
                        }
                        S::kick(c, dt, gxq, gyq, u0, u1, u2, u3, u4, 0.5f * (bxN + bxR), 0.5f * (byD + byN), u5);
                    }
                    out.rho[q] = u0; out.mx[q] = u1; out.my[q] = u2; out.mz[q] = u3; out.E[q] = u4; out.Bz[q] = u5;
                }
            }
            // ---- carry row r - 1 ----
            auto dF = [&](int k) { return lane_down(Fx[k]) - Fx[k]; };
            keep.f[0][tid] = make_float4(dF(0), dF(1), dF(2), dF(3));
            keep.f[1][tid] = make_float4(dF(4), dF(6), Gy[0], Gy[1]);
            keep.f[2][tid] = make_float4(Gy[2], Gy[3], Gy[4], Gy[6]);
            F5 = Fx[5]; Ez = ez; bnx = bn; byD = byN;
            plus = row7(c1, sy, [](float a, float s) { return a + s; });
        }
        dm = dp;
        w = W;
        wb0 = rb0; wb1 = rb1; wy0 = ry0;
        if (GMODE == GRAV_PHI) { ph3 = ph2; ph2 = ph1; ph1 = rphi; }
        slot = slot == 2 ? 0 : slot + 1;
    }
}

template <bool DEFER, int GMODE>
__global__ void __launch_bounds__(LANE_NT, 4)
m2_lane_kernel(const M2Const<float> c, const Fields<float> in, const Fields<float> out, const float* __restrict__ ga,
               const float* __restrict__ gb, const double* __restrict__ dtp, const int* __restrict__ active, const int seg) {
    if (active && *active == 0) return;
    const int strip = blockIdx.x * (LANE_NT / 32) + (threadIdx.x >> 5);
    const int j0 = blockIdx.y * seg, j1 = j0 + seg < c.ny ? j0 + seg : c.ny;
    if (strip * LANE_W >= c.nx) return;   // whole warps
    __shared__ LaneKeep keep;
    m2_lane_segment<DEFER, GMODE, ESUM_GRID>(keep, c, in, out, ga, gb, (float)*dtp, strip, j0, j1);
}

}  // namespace ccb
