"""Which stage kernel a 2D handle runs (cc_mhd2d_set_stage_kernel,
cc_mhd2d_get_stage_kernel): the choice by the grid, that it can be asked for,
read and returned to, what refuses it, and the register march on grids that
only a caller can give it (thin, wide, smaller than a strip, one segment)
against the tiles: the same bits."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200 import _lib as L
from core_collapse_b200.mhd2d import CcError, Mhd2dSolver, Params, ic_collapse

pytestmark = pytest.mark.gpu


def _params(nx, ny, precision="fp32", **kw):
    return Params(Nx=nx, Ny=ny, x0=-1, x1=1, y0=-1, y1=1, eta=1e-3, cfl=0.3, gravity_on=False, precision=precision, t_end=1e30, **kw)


@pytest.mark.parametrize("p,kind", [
    (_params(1003, 777), "lane"), (_params(896, 700), "lane"), (_params(1024, 512), "lane"), (_params(700, 600), "lane"), (_params(700, 513), "tile"),
    (_params(256, 256), "tile"), (_params(300, 435), "tile"),      # at most 296 tiles
    (_params(1003, 777, compensated=True), "tile"), (_params(1003, 777, "fp64"), "tile")])
def test_choice_by_the_grid(p, kind):
    with Mhd2dSolver(p) as s:
        assert s.stage_kernel()[0] == kind and (s.stage_kernel()[1] > 0) == (kind == "lane")
        auto = s.stage_kernel()
        s.set_stage_kernel("tile")
        assert s.stage_kernel() == ("tile", 0)
        s.set_stage_kernel("auto")
        assert s.stage_kernel() == auto


def test_ask_and_refuse():
    with Mhd2dSolver(_params(64, 48)) as s:
        s.set_stage_kernel("lane")
        assert s.stage_kernel()[0] == "lane" and s.stage_kernel()[1] >= 1
        s.set_stage_kernel("lane", 7)
        assert s.stage_kernel() == ("lane", 7)
        s.set_stage_kernel("march", 24)
        assert s.stage_kernel() == ("march", 24)
        for kind in (-1, 4):
            assert L.lib().cc_mhd2d_set_stage_kernel(s._h, kind, 0) == L.CC_ERR_ARG
        assert s.stage_kernel() == ("march", 24)
        assert L.lib().cc_mhd2d_get_stage_kernel(s._h, None, C.byref(C.c_int())) == L.CC_ERR_ARG
    for p in (_params(64, 48, "fp64"), _params(64, 48, compensated=True)):
        with Mhd2dSolver(p) as s, pytest.raises(CcError) as e:
            s.set_stage_kernel("lane")
        assert e.value.code == L.CC_ERR_UNSUPPORTED


@pytest.mark.parametrize("px,py", [(True, True), (False, False)])
@pytest.mark.parametrize("shape,rows", [((4, 4), 0), ((4, 300), 5), ((29, 33), 64), ((28, 31), 1), ((1500, 5), 0), ((57, 64), 2)])
def test_asked_march_matches_tiles(shape, rows, px, py):
    p = _params(*shape, periodic_x=px, periodic_y=py)
    U, B = ic_collapse(p, core_amp=4.0, core_width=0.3, noise=0.1, seed=3, Bx0=0.2)
    rng = np.random.default_rng(0)
    for m in (U.mx, U.my, U.mz):
        m[:] = U.rho * rng.uniform(-0.2, 0.2, p.Nx * p.Ny)
    U.Bz[:] = rng.uniform(-0.1, 0.1, p.Nx * p.Ny)
    U.E[:] += 0.5 * (U.mx ** 2 + U.my ** 2 + U.mz ** 2) / U.rho + 0.5 * U.Bz ** 2
    out = []
    for kind in ("lane", "tile"):
        with Mhd2dSolver(p) as s:
            s.set_stage_kernel(kind, rows if kind == "lane" else 0)
            assert s.stage_kernel()[0] == kind
            s.upload(U, B)
            s.advance(4, 0.0)
            out.append(O.state_list(*s.download()))
    assert all(np.isfinite(x).all() for x in out[0])
    assert all(np.array_equal(x, y) for x, y in zip(*out))
