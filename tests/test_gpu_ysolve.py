"""The y solves of the direct Poisson path (dp_ysolve_kernel: sweeps in groups of 8
rows through a ring of 8 groups, the singular wavenumber by a warp in blocks of 32
rows) against the CPU restatement, bit for bit in FP64: row counts at the ends of a
group, of the ring and of a block, and few rows; x counts at the end of a
warp's 32 wavenumbers; clamped and cyclic."""
import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200.batch import BatchSolver
from core_collapse_b200.mhd2d import Params, ic_collapse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("py", [False, True])
@pytest.mark.parametrize("nx", [33, 34])
def test_y_solve_row_counts(nx, py):
    params, states = [], []
    for ny in (4, 8, 9, 10, 31, 32, 33, 56, 57, 58, 63, 64, 65, 66, 73, 130):
        p = Params(Nx=nx, Ny=ny, x0=-1, x1=1, y0=-1, y1=1, periodic_x=py, periodic_y=py, gravity_on=True, G=1.0, eta=1e-3,
                   cfl=0.3, poisson="direct", t_end=1e30)
        params.append(p)
        states.append(ic_collapse(p, core_amp=6.0, core_width=0.3, noise=0.05, seed=ny, Bx0=0.1))
    with BatchSolver(params) as b:
        for i, s in enumerate(states):
            b.upload(i, *s)
        t = b.advance(2, np.zeros(len(params)))
        got = [b.download(i) for i in range(len(params))]
    for i, p in enumerate(params):
        want, tw = O.m2_main_loop_oracle(p.to_c(), O.state_list(*states[i]), 2, mode=3)
        assert t[i] == tw
        for x, y in zip(got[i][0].arrays() + [got[i][1].Bx_f, got[i][1].By_f], want):
            assert np.array_equal(x, y), f"Ny = {p.Ny}"
