"""A wait of the cluster SOR that runs out (sor_cluster_kernel): with a limit of
no polls at all, waits give up at once, in any phase, and in some threads and
CTAs only.  The kernel must end, report it, and leave the device usable: the next
launch with the ordinary limit has the result of the one before."""
import ctypes as C
import sys
import time
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent / "native"))
import build as native_build  # noqa: E402

pytestmark = pytest.mark.gpu


def _solve(nx, ny, sweeps, tol, polls, rhs):
    L = C.CDLL(str(native_build.build("sor_cluster_wait")))
    dp = C.POINTER(C.c_double)
    phi = np.full(nx * ny, np.nan)
    err, iters = C.c_int(-1), C.c_int(-1)
    t = time.perf_counter()
    r = L.sor_cluster_wait(nx, ny, sweeps, C.c_double(tol), polls, rhs.ctypes.data_as(dp), phi.ctypes.data_as(dp),
                           C.byref(err), C.byref(iters))
    assert r == 0, f"cudaError {r}"
    return phi, err.value, iters.value, time.perf_counter() - t


@pytest.mark.parametrize("tol", [0.0, 1e-30])
@pytest.mark.parametrize("nx,ny", [(66, 62), (128, 128), (170, 190)])
def test_wait_runs_out(nx, ny, tol):
    rng = np.random.default_rng(nx)
    rhs = rng.uniform(-1, 1, nx * ny)
    rhs -= rhs.mean()
    want, err, iters, _ = _solve(nx, ny, 50, tol, 1 << 26, rhs)
    assert err == 0 and iters == 50 and np.isfinite(want).all() and want.any()
    failures = 0
    for polls in (0, 0, 0, 3, 10):
        _, err, iters, sec = _solve(nx, ny, 50, tol, polls, rhs)
        assert err in (0, 1) and iters <= 50 and sec < 5.0
        failures += err
    assert failures >= 3   # no poll: some wait always gives up
    got, err, iters, _ = _solve(nx, ny, 50, tol, 1 << 26, rhs)
    assert err == 0 and iters == 50 and np.array_equal(got, want)
