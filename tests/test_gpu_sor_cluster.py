"""The red-black SOR inside one thread-block cluster (sor_cluster_kernel in
poisson_kernels.cuh) against the oracle's red-black solve, on the grids where
its decomposition can go wrong: one CTA and sixteen, every number of pairs per
thread, a last CTA with fewer pairs than a row (its rows' images and the
periodic ones then come from two CTAs), rows that end inside a warp, odd and
thin grids, and the sizes just outside, which sor_rb_kernel takes (an odd nx
whose pairs exceed the blocks, a grid beyond the shared memory of the cluster).
The two differ from the oracle only in the order of the density and potential
means (a fixed tree instead of a running sum): 1e-12, the bound of the other
gravity tests.  With a tolerance the sweep counts agree within the rounding of
the residual there (2 sweeps)."""
import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200.mhd2d import Mhd2dSolver, Params, ic_collapse

pytestmark = pytest.mark.gpu

TOL = 1e-12
SWEEPS = 12

SHAPES = [
    (4, 4), (6, 50), (50, 50), (2, 1024),            # one block; a pair to a row
    (66, 62), (64, 64), (64, 66),                    # M = 1024 V exactly, and one row more
    (5, 7), (33, 61), (129, 33),                     # odd: outflow only
    (192, 192), (256, 256), (258, 254),              # nine and sixteen CTAs
    (254, 132), (1022, 34), (2046, 18),              # a last CTA shorter than a row
    (300, 302), (400, 260), (352, 350),              # V = 6, 8, 8
    (402, 400), (63, 131),                           # sor_rb_kernel
]


def _params(shape, px, py, **kw):
    nx, ny = shape
    return Params(Nx=nx, Ny=ny, x0=-1.0, x1=1.0, y0=-1.0, y1=1.3, periodic_x=px, periodic_y=py, gravity_on=True, G=1.0,
                  sor_omega=1.7, poisson="sor", **kw)


def _solve(p):
    U, B = ic_collapse(p, core_amp=6.0, core_width=0.3, noise=0.05, seed=p.Nx + p.Ny, Bx0=0.05)
    want = O.m2_gravity_oracle(p.to_c(), U.rho, mode=1)
    with Mhd2dSolver(p) as s:
        s.upload(U, B)
        g = s.compute_gravity()
        d = s.diagnostics()
    return g, d, want


@pytest.mark.parametrize("px,py", [(True, True), (False, True), (True, False), (False, False)])
@pytest.mark.parametrize("shape", SHAPES)
def test_fixed_sweeps(shape, px, py):
    if (px and shape[0] & 1) or (py and shape[1] & 1):
        pytest.skip("red-black needs an even extent along periodic axes")
    p = _params(shape, px, py, sor_iters=SWEEPS)
    g, d, (gx, gy, it, res) = _solve(p)
    assert d["poisson_iters"] == it == SWEEPS
    assert O.rel_linf(g.gx, gx) <= TOL and O.rel_linf(g.gy, gy) <= TOL
    assert abs(d["poisson_residual"] - res) <= 1e-10 * res


@pytest.mark.parametrize("shape", [(50, 50), (96, 130), (256, 64)])
def test_tolerance(shape):
    p = _params(shape, True, True, sor_iters=20000, sor_tol=1e-3)
    g, d, (gx, gy, it, res) = _solve(p)
    assert abs(d["poisson_iters"] - it) <= 2 and d["poisson_residual"] < 1e-3
    if d["poisson_iters"] == it:
        assert O.rel_linf(g.gx, gx) <= 1e-11 and O.rel_linf(g.gy, gy) <= 1e-11


def test_zero_sweeps_and_uniform_density():
    p = _params((50, 50), True, True, sor_iters=0)
    g, d, _ = _solve(p)
    assert d["poisson_iters"] == 0 and not g.gx.any() and not g.gy.any()
    p = _params((50, 50), True, True, sor_iters=5)
    U, B = ic_collapse(p, core_amp=0.0, core_width=0.3, noise=0.0, seed=1, Bx0=0.05)
    with Mhd2dSolver(p) as s:
        s.upload(U, B)
        g = s.compute_gravity()
    assert np.max(np.abs(g.gx)) <= 1e-12 and np.max(np.abs(g.gy)) <= 1e-12
