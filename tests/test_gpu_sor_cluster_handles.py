"""The cluster SOR (sor_cluster_kernel) of two handles at once.  Grids of the same
number of pairs a thread share one kernel and need different amounts of shared
memory, so its limit must suit both whatever order they launch in: from two host
threads, and from a graph that was captured before the other grid's solve."""
import threading

import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200.mhd2d import Mhd2dSolver, Params, ic_collapse

pytestmark = pytest.mark.gpu

WIDE, NARROW = (1022, 120), (170, 720)   # eight pairs a thread both; rows of 511 and of 85 pairs


def _handle(shape, **kw):
    p = Params(Nx=shape[0], Ny=shape[1], x0=-1.0, x1=1.0, y0=-1.0, y1=1.0, periodic_x=True, periodic_y=True, gravity_on=True,
               G=1.0, sor_omega=1.7, poisson="sor", sor_iters=2, cfl=0.3, t_end=1e30, **kw)
    U, B = ic_collapse(p, core_amp=6.0, core_width=0.3, noise=0.05, seed=1, Bx0=0.05)
    s = Mhd2dSolver(p)
    s.upload(U, B)
    return s, U, B


def test_two_threads():
    """Single steps (no graph), a thousand of each handle: two solves and two launches of the kernel a step."""
    handles = [_handle(x, precision="fp32") for x in (WIDE, NARROW)]
    errors = []

    def work(s, U, B):
        try:
            for _ in range(500):
                s.advance(2)
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=h) for h in handles]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, _, _ in handles:
        s.close()
    assert not errors


def test_graph_captured_before():
    a, U, B = _handle(WIDE)
    b, _, _ = _handle(NARROW)
    a.advance(6, 0.0)
    want = O.state_list(*a.download())
    a.upload(U, B)
    a.advance(3, 0.0)
    b.compute_gravity()
    a.advance(3)
    got = O.state_list(*a.download())
    a.close()
    b.close()
    assert all(np.array_equal(x, y) for x, y in zip(got, want))
