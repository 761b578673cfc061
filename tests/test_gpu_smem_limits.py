"""Shared-memory limits of the transforms' kernels: a kernel's limit belongs to
the device and serves every handle, so a handle with short lines (or another
Poisson solver) made after one with long lines must not lower it.  The handle
with the longest lines solves, others are made, and it solves again."""
import ctypes as C

import numpy as np
import pytest

from core_collapse_b200 import _lib as L
from core_collapse_b200.mhd2d import Mhd2dSolver, Params, ic_orszag_tang
from core_collapse_b200.ns2d import Ns2dSolver, ParamsNS

pytestmark = pytest.mark.gpu


def _params(nx, ny, precision, poisson="fft"):
    return Params(Nx=nx, Ny=ny, x0=-1.0, x1=1.0, y0=-1.0, y1=1.0, G=1.0, gravity_on=True, poisson=poisson, precision=precision,
                  sor_iters=4)


def _others():
    """Handles with short lines, of every kind that sets the same kernels' limits."""
    for precision in ("fp64", "fp32"):
        for poisson, n in (("fft", 16), ("sor", 50)):
            yield Mhd2dSolver(_params(n, n, precision, poisson))
        yield Ns2dSolver(ParamsNS(Nx=16, Ny=16, gravity_on=True, precision=precision))


@pytest.mark.parametrize("precision,nx,ny", [("fp64", 8192, 8), ("fp64", 8, 4096), ("fp64", 2048, 2048), ("fp32", 8192, 8),
                                             ("fp32", 8, 4096), ("fp32", 4096, 4096)])
def test_long_lines_after_short_ones(precision, nx, ny):
    p = _params(nx, ny, precision)
    U, B = ic_orszag_tang(p, core_amp=4.0, core_width=0.2)
    with Mhd2dSolver(p) as s:
        s.upload(U, B)
        want = s.compute_gravity()
        for o in _others():
            o.close()
        s.upload(U, B)   # the potential is formed anew
        got = s.compute_gravity()
    assert np.array_equal(got.gx, want.gx) and np.array_equal(got.gy, want.gy) and np.any(want.gx)


def test_noalloc_after_short_lines():
    import torch
    p = _params(64, 4096, "fp64")
    U, B = ic_orszag_tang(p, core_amp=4.0, core_width=0.2)
    rho = torch.from_numpy(U.rho).to("cuda")
    cp = p.to_c()
    out = []
    for k in range(2):
        if k:
            for o in _others():
                o.close()
        g = [torch.zeros_like(rho) for _ in range(2)]
        r = L.lib().cc_mhd2d_gravity_fft_noalloc(C.byref(cp), *(C.c_void_p(t.data_ptr()) for t in (rho, *g)), C.c_void_p(0))
        assert r == L.CC_OK
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in g])
    assert np.any(out[0][0]) and all(np.array_equal(a, b) for a, b in zip(*out))
