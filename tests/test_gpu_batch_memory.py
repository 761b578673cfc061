"""Memory of a batch handle: its buffers for pageable downloads are no larger than
the largest instance's state, and downloads allocate nothing."""
import ctypes as C

import numpy as np
import pytest
import torch

from core_collapse_b200.batch import BatchSolver
from core_collapse_b200.mhd2d import Params, ic_collapse

pytestmark = pytest.mark.gpu


def test_small_handle_stays_small():
    p = Params(Nx=24, Ny=20, x0=-1, x1=1, y0=-1, y1=1, gravity_on=False, precision="fp64")
    state = 8 * 8 * (p.Nx + 1) * (p.Ny + 1)
    pool = 8 * 25 * 32 * (p.Ny + 1)            # three states and a potential, rows of 32
    U, B = ic_collapse(p, noise=0.1, seed=1, Bx0=0.1)
    with BatchSolver([p]) as b:
        held = b.info()["device_bytes"]
        assert held < pool + 2 * state + 65536   # one field, what is packed, and the work-lists and partials
        b.upload(0, U, B)
        pinned = [torch.empty(a.size, dtype=torch.float64, pin_memory=True) for a in U.arrays() + [B.Bx_f, B.By_f]]
        ptrs = (C.POINTER(C.c_double) * 8)(*[C.cast(t.data_ptr(), C.POINTER(C.c_double)) for t in pinned])
        b._check(b._lib.cc_batch_download(b._h, 0, ptrs))
        assert b.info()["device_bytes"] == held
        for _ in range(2):
            V, F = b.download(0)
            assert b.info()["device_bytes"] == held
        for q, g, u in zip(pinned, V.arrays() + [F.Bx_f, F.By_f], U.arrays() + [B.Bx_f, B.By_f]):
            assert np.array_equal(g, u) and np.array_equal(q.numpy(), u)
