"""The 3D EMF / CT kernel's chunks of planes (m3_edge_kch, 4 to 32 planes by the
number of CTAs) and its quotients against the CPU oracle, bit for bit in FP64:
plane counts on either side of a chunk's end, a last chunk of one plane, chunks of
4, 8 and 16 planes, periodic and clamped."""
import pytest

import cases_mhd3d as C3
import numpy as np
import oracle_lib as O
from core_collapse_b200.mhd3d import Mhd3dSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 6, 3), (8, 6, 4), (33, 9, 8), (31, 8, 17), (62, 28, 63),   # 4 planes
                                   (94, 63, 144), (125, 91, 176)])                                   # 8 and 16
@pytest.mark.parametrize("periodic", [True, False])
def test_chunks_match_the_oracle(shape, periodic, monkeypatch):
    kw = dict(Nx=shape[0], Ny=shape[1], Nz=shape[2], periodic_x=periodic, periodic_y=periodic, periodic_z=periodic,
              eta=7e-4, cfl=0.3)
    monkeypatch.setitem(C3.CASES3, "chunks", (kw, True, False, 11))
    p, s = C3.make_case3("chunks")
    S = [a.copy() for a in s.arrays()]
    want, tw = O.m3_main_loop_oracle(p.to_c(), S, 1)
    with Mhd3dSolver(p) as g:
        g.upload(s)
        t = g.advance(1, 0.0)
        got = g.download().arrays()
    assert t == tw
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
