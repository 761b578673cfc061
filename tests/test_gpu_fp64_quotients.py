"""The FP64 kernels' quotients (Div, cc_device.cuh) where their fast form does
not apply and the plain divisions take over: densities beyond 2^101 and below
2^-100, momenta and fields that are zero, subnormal or near the ends of the
range, mixed in one grid with ordinary cells.  Without gravity the FP64 step is
the oracle's, which divides, bit for bit: every wrongly rounded quotient shows."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200.mhd2d import Bfaces, Mhd2dSolver, Params, Ucc
from core_collapse_b200.mhd3d import Mhd3dSolver, Params3, State3

pytestmark = pytest.mark.gpu


def _scales(name, n, rng):
    """(density, velocity, field) factors per cell."""
    if name == "dense":
        return np.full(n, 1e32), np.full(n, 1.0), np.full(n, 1e16)
    if name == "thin":
        return np.full(n, 1e-32), np.full(n, 1.0), np.full(n, 1e-16)
    if name == "mixed":
        d = 10.0 ** rng.choice([0.0, 29.0, 31.5], n)
        return d, np.full(n, 1.0), np.full(n, 1.0)
    if name == "slow":     # momenta and their quotients subnormal
        return np.full(n, 1.0), 10.0 ** rng.choice([-322.0, -310.0, -290.0, 0.0], n), np.full(n, 1.0)
    return np.full(n, 1.0), rng.choice([0.0, -0.0, 1.0], n), rng.choice([0.0, 1.0], n)   # "zeros"


NAMES = ["dense", "thin", "mixed", "slow", "zeros"]


@pytest.mark.parametrize("name", NAMES)
def test_2d_step_bitwise(name):
    rng = np.random.default_rng(NAMES.index(name))
    p = Params(Nx=37, Ny=22, gravity_on=False, eta=1e-3, floor_rho=1e-40, floor_P=1e-40, cfl=0.3, t_end=1e30)
    n = p.Nx * p.Ny
    d, v, b = _scales(name, n, rng)
    rho = d * rng.uniform(0.5, 2.0, n)
    u = [v * rng.uniform(-0.5, 0.5, n) for _ in range(3)]
    bz = b * rng.uniform(-0.3, 0.3, n)
    bx = np.full((p.Nx + 1) * p.Ny, 0.4 * b.max())
    by = np.zeros(p.Nx * (p.Ny + 1))
    E = d * rng.uniform(1.0, 2.0, n) + 0.5 * rho * sum(a * a for a in u) + 0.5 * (bz * bz + (0.4 * b.max()) ** 2)
    U, B = Ucc(rho, rho * u[0], rho * u[1], rho * u[2], E, bz), Bfaces(bx, by)
    S, z = O.state_list(U, B), np.zeros(n)
    cp = p.to_c()
    with Mhd2dSolver(p) as s:
        s.upload(U, B)
        dt = s.compute_dt()
        assert dt == O.oracle().or_mhd2d_compute_dt(C.byref(cp), O.pp(S))
        s.rk2_step(None, dt)
        got = O.state_list(*s.download())
    want = O.m2_rk2_oracle(cp, S, z, z, dt, 1)
    for k, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w, equal_nan=True), f"field {k}: {np.sum(a != w)} differ"


@pytest.mark.parametrize("name", NAMES)
def test_3d_step_bitwise(name):
    rng = np.random.default_rng(10 + NAMES.index(name))
    p = Params3.ideal_gas(Nx=13, Ny=9, Nz=7, eta=1e-3, floor_rho=1e-40, floor_P=1e-40, cfl=0.3, t_end=1e30)
    sizes = p.sizes()
    n = sizes[0]
    d, v, b = _scales(name, n, rng)
    rho = d * rng.uniform(0.5, 2.0, n)
    u = [v * rng.uniform(-0.5, 0.5, n) for _ in range(3)]
    f = [np.full(m, a * b.max()) for m, a in zip(sizes[5:], (0.4, 0.0, -0.2))]
    E = d * rng.uniform(1.0, 2.0, n) + 0.5 * rho * sum(a * a for a in u) + 0.5 * b.max() ** 2 * 0.2
    s0 = State3(rho, rho * u[0], rho * u[1], rho * u[2], E, *f)
    cp = p.to_c()
    with Mhd3dSolver(p) as s:
        s.upload(s0)
        dt = s.compute_dt()
        s.rk2_step(dt)
        got = s.download().arrays()
    want = O.m3_rk2_oracle(cp, [a.copy() for a in s0.arrays()], dt)
    for k, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w, equal_nan=True), f"field {k}: {np.sum(a != w)} differ"
