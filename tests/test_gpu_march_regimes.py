"""The FP32 register march (mhd2d_lane.cuh) against the tile kernels, of a
single grid and of an ensemble, where its expressions take the branches that a
smooth flow never does: cells below the density and pressure floors (after the
update, after the gravity kick and after the Joule sub-step, and cells near
the floors on either side), supersonic faces, faces without a normal field
(the HLL flux), no field at all, and a state at rest.  Both forms have the
same bits, so that neither the size of a grid nor the other instances of an
ensemble, by which the form is chosen, change a result."""
import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200.batch import BatchSolver
from core_collapse_b200.mhd2d import Bfaces, Mhd2dSolver, Params, Ucc

pytestmark = pytest.mark.gpu

REGIMES = ("floors", "supersonic", "no_bn", "no_field", "rest", "mixed")


def _params(regime, nx, ny, **kw):
    floors = regime in ("floors", "mixed")
    return Params(Nx=nx, Ny=ny, x0=-1.0, x1=1.0, y0=-1.0, y1=1.3, eta=1e-3, G=1.0, cfl=0.3, t_end=1e30, precision="fp32",
                  floor_rho=0.8 if floors else 1e-10, floor_P=0.3 if floors else 1e-10, **kw)


def _state(regime, p, seed):
    rng = np.random.default_rng(seed)
    n = p.Nx * p.Ny

    def field(m, a):
        return a * rng.uniform(-1.0, 1.0, m)

    v = {"floors": 0.5, "supersonic": 6.0, "no_bn": 0.5, "no_field": 0.5, "rest": 0.0}.get(regime, 2.0)
    b = {"no_bn": 0.0, "no_field": 0.0}.get(regime, 0.4)
    rho = rng.uniform(0.5, 1.6, n)
    u = [field(n, v) for _ in range(3)]
    bz = field(n, 0.0 if regime in ("no_field", "rest") else 0.3)
    P = rng.uniform(0.05, 0.6, n) if p.floor_P > 0.1 else rng.uniform(0.4, 0.6, n)
    bx, by = field((p.Nx + 1) * p.Ny, b), field(p.Nx * (p.Ny + 1), b)
    if regime == "mixed":   # every second cell of the faces without a field
        bx[::2] = 0.0
        by[1::2] = 0.0
    x, y = bx.reshape(p.Ny, p.Nx + 1), by.reshape(p.Ny + 1, p.Nx)
    cx, cy = 0.5 * (x[:, :-1] + x[:, 1:]).ravel(), 0.5 * (y[:-1] + y[1:]).ravel()
    E = P / (p.gamma - 1.0) + 0.5 * rho * sum(a * a for a in u) + 0.5 * (cx ** 2 + cy ** 2 + bz ** 2)
    return Ucc(rho, rho * u[0], rho * u[1], rho * u[2], E, bz), Bfaces(bx, by)


def _compare(got, want, what):
    differ = [int((~((x == y) | (np.isnan(x) & np.isnan(y)))).sum()) for x, y in zip(got, want)]
    assert differ == [0] * len(want), f"{what}: {differ}"


@pytest.mark.parametrize("px,py", [(True, True), (False, False)])
@pytest.mark.parametrize("regime", REGIMES)
def test_single_grid(regime, px, py):
    p = _params(regime, 700, 513, periodic_x=px, periodic_y=py, gravity_on=False)
    s0 = _state(regime, p, 1)
    out = []
    for kind in ("lane", "tile"):
        with Mhd2dSolver(p) as s:
            s.set_stage_kernel(kind)
            s.upload(*s0)
            s.advance(3, 0.0)
            out.append(O.state_list(*s.download()))
    _compare(*out, regime)


@pytest.mark.parametrize("regime", REGIMES)
def test_single_grid_gravity(regime):
    p = _params(regime, 1024, 512, periodic_x=True, periodic_y=True, gravity_on=True, poisson="fft")
    s0 = _state(regime, p, 2)
    out = []
    for kind in ("lane", "tile"):
        with Mhd2dSolver(p) as s:
            s.set_stage_kernel(kind)
            s.upload(*s0)
            s.advance(3, 0.0)
            out.append(O.state_list(*s.download()))
    _compare(*out, regime)


@pytest.mark.parametrize("gravity", [False, True])
@pytest.mark.parametrize("regime", REGIMES)
def test_ensemble(regime, gravity):
    params = [_params(regime, nx, ny, periodic_x=bool(i & 1), periodic_y=bool(i & 2), gravity_on=gravity, poisson="direct")
              for i in range(4) for nx, ny in ((160, 144), (200, 97), (57, 250), (84, 64))]
    states = [_state(regime, p, 10 + i) for i, p in enumerate(params)]
    out = []
    for shape in (None, 0):
        with BatchSolver(params) as b:
            if shape is None:
                assert b.info()["shape"] == b.info()["n_shapes"] - 1   # the march
            else:
                b.set_shape(shape)
            for i, s in enumerate(states):
                b.upload(i, *s)
            b.advance(3, np.zeros(len(params)))
            out.append([O.state_list(*b.download(i)) for i in range(len(params))])
    for i, (x, y) in enumerate(zip(*out)):
        _compare(x, y, f"{regime}, instance {i}")


@pytest.mark.parametrize("regime", ("floors", "supersonic", "mixed"))
def test_instance_without_gravity_beside_others_with_it(regime):
    """Such an instance runs the stage kernel with gravity, alone it runs the one without."""
    params = [_params(regime, 160, 144, gravity_on=i > 0, poisson="direct") for i in range(12)]
    states = [_state(regime, p, 30 + i) for i, p in enumerate(params)]
    out = []
    for n, shape in ((12, None), (12, 0), (1, None)):
        with BatchSolver(params[:n]) as b:
            if shape is not None:
                b.set_shape(shape)
            for i in range(n):
                b.upload(i, *states[i])
            b.advance(3, np.zeros(n))
            out.append(O.state_list(*b.download(0)))
    _compare(out[0], out[2], regime)
    _compare(out[1], out[2], regime)
