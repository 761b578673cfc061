"""A batch download into pageable memory (fields packed together into pinned halves
of 4 MB, a larger field in pieces of its own) against one into pinned memory (field
by field): instances whose eight fields fit one half, take two, and whose single
field is larger than a half; and the uploaded values come back in FP64."""
import ctypes as C

import numpy as np
import pytest
import torch

from core_collapse_b200.batch import BatchSolver
from core_collapse_b200.mhd2d import Params, ic_collapse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_pageable_equals_pinned_and_uploaded(precision):
    shapes = [(5, 4), (64, 64), (251, 260), (511, 1021), (1100, 1003), (33, 40)]
    params = [Params(Nx=nx, Ny=ny, x0=-1, x1=1, y0=-1, y1=1, gravity_on=False, precision=precision) for nx, ny in shapes]
    states = []
    for i, p in enumerate(params):
        U, B = ic_collapse(p, noise=0.1, seed=i, Bx0=0.1)
        rng = np.random.default_rng(i)
        for a in U.arrays() + [B.Bx_f, B.By_f]:
            a += rng.uniform(0, 1e-3, a.size)
        states.append((U, B))
    with BatchSolver(params) as b:
        for i, s in enumerate(states):
            b.upload(i, *s)
        for i, (U, B) in enumerate(states):
            given = U.arrays() + [B.Bx_f, B.By_f]
            V, F = b.download(i)
            got = V.arrays() + [F.Bx_f, F.By_f]
            pinned = [torch.empty(a.size, dtype=torch.float64, pin_memory=True) for a in given]
            ptrs = (C.POINTER(C.c_double) * 8)(*[C.cast(t.data_ptr(), C.POINTER(C.c_double)) for t in pinned])
            b._check(b._lib.cc_batch_download(b._h, i, ptrs))
            for g, q, u in zip(got, pinned, given):
                assert np.array_equal(g, q.numpy())
                assert np.array_equal(g, u if precision == "fp64" else u.astype(np.float32).astype(np.float64))
