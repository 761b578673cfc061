"""The FP32 3D kernels divide by the grid spacings: Div::quot_grid and the
resistive EMF (mhd3d_kernels.cuh) have the bits of the written-out divisions in
the FP32 build, on spacings whose FP32 reciprocals are not exact."""
import ctypes as C
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent / "native"))
import build as native_build  # noqa: E402

pytestmark = pytest.mark.gpu

FP32_FLAGS = ["-prec-div=false", "-prec-sqrt=false", "-ftz=true"]   # core_collapse_b200/build.py


def test_fp32_divides():
    n = 1 << 14
    rng = np.random.default_rng(1)
    d1, d2 = (rng.uniform(-1, 1, n).astype(np.float32) for _ in range(2))
    out = np.empty((5, n), np.float32)
    fp = C.POINTER(C.c_float)
    L = C.CDLL(str(native_build.build("grid_quotients", FP32_FLAGS)))
    differ = 0
    for m in range(17, 400, 6):
        h = (2.0 / m, 2.4 / (m + 1))
        r = L.grid_quotients(d1.ctypes.data_as(fp), d2.ctypes.data_as(fp), C.c_long(n), (C.c_double * 2)(*h), C.c_double(1e-3),
                             out.ctypes.data_as(fp))
        assert r == 0, f"cudaError {r}"
        assert np.array_equal(out[0], out[1]) and np.array_equal(out[2], out[3]) and np.isfinite(out).all(), m
        differ += bool((out[4] != out[1]).any())
    assert differ   # a product with the host's reciprocal is told from the division
