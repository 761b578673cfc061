"""The FP32 ensemble's stage as the register march (m2b_lane_kernel), the form
a batch of more than a wave of tiles picks, against the tile kernel on the same
instances: the same bits.  Instances of one strip (28 columns and fewer), of
strips that own one column, of fewer rows than a segment, all boundaries, with
and without gravity and resistivity; a number of (strip, segment) pairs that
does not fill the last CTA; an instance that stops before the others."""
from dataclasses import replace

import numpy as np
import pytest

from core_collapse_b200.batch import BatchSolver
from core_collapse_b200.mhd2d import Params, ic_collapse

pytestmark = pytest.mark.gpu

SHAPES = [(29, 33), (28, 64), (57, 150), (140, 97), (200, 200), (164, 164), (9, 11)]


def _run(params, states, shape):
    with BatchSolver(params) as b:
        if shape is not None:
            b.set_shape(shape)
        for i, s in enumerate(states):
            b.upload(i, *s)
        t = b.advance(5, np.zeros(len(params)))
        return [b.download(i) for i in range(len(params))], t


@pytest.mark.parametrize("gravity", [False, True])
def test_march_matches_tiles(gravity):
    base = Params(x0=-1, x1=1, y0=-1, y1=1, G=1.0, cfl=0.3, poisson="direct", precision="fp32", t_end=1e30)
    params, states = [], []
    for i in range(6 * len(SHAPES)):
        nx, ny = SHAPES[i % len(SHAPES)]
        p = replace(base, Nx=nx, Ny=ny, periodic_x=bool(i & 1), periodic_y=bool(i & 2), eta=0.0 if i % 5 == 0 else 1e-3,
                    gravity_on=gravity and i % 3 != 0, t_end=0.004 if i == 8 else 1e30)
        rng = np.random.default_rng(i)
        U, B = ic_collapse(p, core_amp=4.0, core_width=0.3, noise=0.1, seed=i, Bx0=0.2)
        for m in (U.mx, U.my, U.mz):
            m[:] = U.rho * rng.uniform(-0.2, 0.2, nx * ny)
        U.Bz[:] = rng.uniform(-0.1, 0.1, nx * ny)
        U.E[:] += 0.5 * (U.mx ** 2 + U.my ** 2 + U.mz ** 2) / U.rho + 0.5 * U.Bz ** 2
        params.append(p)
        states.append((U, B))
    a, ta = _run(params, states, None)
    b, tb = _run(params, states, 0)
    assert np.array_equal(ta, tb) and ta[8] == 0.004
    for i in range(len(params)):
        for x, y in zip(a[i][0].arrays() + [a[i][1].Bx_f, a[i][1].By_f], b[i][0].arrays() + [b[i][1].Bx_f, b[i][1].By_f]):
            assert np.isfinite(x).all() and np.array_equal(x, y), f"instance {i}"
