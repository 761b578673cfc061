"""The FP64 spectral solve at every split of its lines: two, three and four
stages a pass (lines to 256, 512 and longer), every remainder of log2 n that
the first pass takes, lines of one pass alone, several rows to a CTA and rows
longer than its threads, against the oracle's radix-2 solve.  The butterflies
and twiddles are the oracle's; the density mean is summed in another order and
the inverse runs columns first: 1e-12, the bound of the other gravity tests."""
import pytest

import oracle_lib as O
from core_collapse_b200.mhd2d import Mhd2dSolver, Params, ic_orszag_tang

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("shape", [(4, 4), (8, 4), (4, 16), (16, 8), (32, 64), (128, 4), (256, 256), (64, 512), (512, 128),
                                   (1024, 32), (16, 1024), (2048, 64), (64, 2048), (8192, 4), (4, 4096)])
def test_fp64_solve(shape):
    nx, ny = shape
    p = Params(Nx=nx, Ny=ny, x0=-1.0, x1=1.0, y0=-1.0, y1=1.5, G=1.0, poisson="fft", gravity_on=True)
    U, B = ic_orszag_tang(p, core_amp=4.0, core_width=0.2)
    gx, gy, _, _ = O.m2_gravity_oracle(p.to_c(), U.rho, mode=2)
    with Mhd2dSolver(p) as s:
        s.upload(U, B)
        g = s.compute_gravity()
    assert O.rel_linf(g.gx, gx) <= TOL and O.rel_linf(g.gy, gy) <= TOL
