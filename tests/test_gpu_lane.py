"""The FP32 stage as a march of warps in registers (m2_lane_kernel,
mhd2d_lane.cuh), the form a handle picks on grids that fill the GPU, against
the tile kernel on the same inputs: the same expressions in the same
contraction, so the same bits in every field.  Grids whose last strip owns 1,
27 and 28 columns, segments that end short, every
boundary (a clamped halo column repeats the edge cell, whose Joule sub-step
needs that cell's own neighbours), with and without resistivity, gravity from
the potential and from arrays."""
import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200.mhd2d import GravField, Mhd2dSolver, Params, ic_collapse, ic_orszag_tang

pytestmark = pytest.mark.gpu


def _run(p, U, B, nsteps, kind=None):
    with Mhd2dSolver(p) as s:
        if kind:
            s.set_stage_kernel(kind)
        s.upload(U, B)
        t = s.advance(nsteps, 0.0)
        return O.state_list(*s.download()), t


def _same(a, b):
    assert [int((x != y).sum()) for x, y in zip(a, b)] == [0] * len(b)


def _swirl(p, U, rng):
    """Velocities and Bz of both signs, so that no limiter or wave sits on a tie."""
    n = p.Nx * p.Ny
    for m in (U.mx, U.my, U.mz):
        m[:] = U.rho * rng.uniform(-0.2, 0.2, n)
    U.Bz[:] = rng.uniform(-0.1, 0.1, n)
    U.E[:] += 0.5 * (U.mx ** 2 + U.my ** 2 + U.mz ** 2) / U.rho + 0.5 * U.Bz ** 2


@pytest.mark.parametrize("px,py", [(True, True), (False, False), (True, False), (False, True)])
@pytest.mark.parametrize("shape,eta", [((896, 700), 1e-3), ((897, 701), 1e-3), ((923, 699), 0.0), ((1003, 777), 1e-3)])
def test_march_matches_tiles(shape, eta, px, py):
    p = Params(Nx=shape[0], Ny=shape[1], x0=-1, x1=1, y0=-1, y1=1, periodic_x=px, periodic_y=py, eta=eta, cfl=0.3,
               gravity_on=False, precision="fp32", t_end=1e30)
    U, B = ic_collapse(p, core_amp=4.0, core_width=0.3, noise=0.1, seed=3, Bx0=0.2)
    _swirl(p, U, np.random.default_rng(shape[0]))
    a, ta = _run(p, U, B, 4)
    b, tb = _run(p, U, B, 4, "tile")
    assert ta == tb and all(np.isfinite(x).all() for x in a)
    _same(a, b)


def test_gravity_from_the_potential():
    p = Params(Nx=1024, Ny=1024, x0=-1, x1=1, y0=-1, y1=1, eta=1e-3, G=1.0, gravity_on=True, poisson="fft", cfl=0.4,
               precision="fp32", t_end=1e30)
    U, B = ic_orszag_tang(p, core_amp=4.0, core_width=0.2)
    a, ta = _run(p, U, B, 4)
    b, tb = _run(p, U, B, 4, "tile")
    assert ta == tb
    _same(a, b)


def test_gravity_arrays():
    p = Params(Nx=1024, Ny=1024, x0=-1, x1=1, y0=-1, y1=1, eta=1e-3, G=1.0, gravity_on=True, poisson="fft", cfl=0.4,
               precision="fp32", t_end=1e30)
    U, B = ic_orszag_tang(p, core_amp=4.0, core_width=0.2)
    rng = np.random.default_rng(0)
    g = GravField(rng.uniform(-1, 1, p.Nx * p.Ny), rng.uniform(-1, 1, p.Nx * p.Ny))
    got = []
    for kind in (None, "tile"):
        with Mhd2dSolver(p) as s:
            if kind:
                s.set_stage_kernel(kind)
            s.upload(U, B)
            s.rk2_step(g, 1e-3)
            got.append(O.state_list(*s.download()))
    _same(*got)
