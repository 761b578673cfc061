"""The FP64 reciprocals and quotients of cc_device.cuh (recip_fast,
quotient_fast, quotient, Div) one by one against the host's division: the same
bits over random significands and exponents, quotients next to midpoints of two
doubles, significands of all ones, signed zeros and both sides of every limit
of the range in which the fast forms apply.  What Newton's iteration needs of
its start, 2^-14, is checked too."""
import ctypes as C
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent / "native"))
import build as native_build  # noqa: E402

pytestmark = pytest.mark.gpu

N = 1 << 21
NAMES = ("start", "recip", "fast", "quot", "div", "by")


def _run(a, b):
    L = C.CDLL(str(native_build.build("quotients")))
    dp = C.POINTER(C.c_double)
    out = [np.empty(a.size) for _ in NAMES]
    inside = np.empty(a.size, np.uint8)
    ptr = lambda x: x.ctypes.data_as(dp)  # noqa: E731
    r = L.quotients(ptr(a), ptr(b), C.c_long(a.size), (dp * len(out))(*map(ptr, out)),
                    inside.ctypes.data_as(C.POINTER(C.c_ubyte)))
    assert r == 0, f"cudaError {r}"
    return dict(zip(NAMES, out)), (inside & 1) != 0, (inside & 2) != 0


def _doubles(rng, n, lo, hi):
    """Random sign and significand, exponent uniform in [lo, hi)."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    e = rng.integers(lo + 1023, hi + 1023, n, dtype=np.uint64) << np.uint64(52)
    s = rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
    return (m | e | s).view(np.float64)


def _same(got, want):
    return (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))


def _check(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    with np.errstate(all="ignore"):
        want, y = a / b, 1.0 / b
    o, ob, oa = _run(a, b)
    ones = (b.view(np.uint64) & np.uint64((1 << 52) - 1)) == np.uint64((1 << 52) - 1)
    with np.errstate(invalid="ignore"):
        assert np.array_equal(ob, (np.abs(b) >= 2.0 ** -100) & (np.abs(b) < 2.0 ** 101) & ~ones)
        assert np.array_equal(oa, (a == 0) | ((np.abs(a) >= 2.0 ** -895) & (np.abs(a) < 2.0 ** 769 * (1 + 2.0 ** -20))))
    assert np.max(np.abs(1.0 - b[ob] * o["start"][ob]), initial=0.0) <= 2.0 ** -14
    assert _same(o["recip"], y)[ob].all()
    # a zero's sign by a negative divisor is free
    free = (a == 0) & (b < 0) & ob
    ok = ob & oa & ~free
    assert _same(o["fast"], want)[ok].all()
    for k in ("quot", "div", "by"):
        assert _same(o[k], want)[~free].all(), k
        assert (o[k][free] == 0).all(), k
    return int(ok.sum())


def test_random():
    rng = np.random.default_rng(1)
    assert _check(_doubles(rng, N, -895, 769), _doubles(rng, N, -100, 101)) >= N - 64
    _check(_doubles(rng, N, -1022, 1024), _doubles(rng, N, -1022, 1024))


def test_next_to_midpoints():
    """a = RN(b m), and its neighbours, for midpoints m of adjacent doubles."""
    rng = np.random.default_rng(2)
    b = _doubles(rng, N, -90, 90)
    q = _doubles(rng, N, -90, 90)
    m = (q.astype(np.longdouble) + np.nextafter(q, np.inf).astype(np.longdouble)) / 2
    a = (m * b.astype(np.longdouble)).astype(np.float64)
    for x in (a, np.nextafter(a, np.inf), np.nextafter(a, -np.inf)):
        _check(x, b)


def test_limits():
    """Both sides of every limit, all-ones significands, zeros, infinities, NaN, subnormals."""
    tiny = np.array([0.0, -0.0, 5e-324, 2.0 ** -1022, np.inf, -np.inf, np.nan, 1.0, 2.0, 3.0, 1e300])
    edge_b = np.array([2.0 ** -100, 2.0 ** 101, 2.0 ** -101, 2.0 ** 100])
    edge_a = np.array([2.0 ** -895, 2.0 ** 769, 2.0 ** 769 * (1 + 2.0 ** -20), 2.0 ** -896, 2.0 ** 770])
    around = lambda x: np.concatenate([x, np.nextafter(x, np.inf), np.nextafter(x, -np.inf)])  # noqa: E731
    ones = np.ldexp(2.0 - 2.0 ** -52, np.arange(-102, 104))
    rng = np.random.default_rng(3)
    a = np.concatenate([tiny, around(edge_a), ones[::7], _doubles(rng, 40, -895, 769)])
    b = np.concatenate([tiny, around(edge_b), ones, _doubles(rng, 40, -100, 101)])
    a, b = np.concatenate([a, -a]), np.concatenate([b, -b])
    A, B = np.meshgrid(a, b)
    _check(A.ravel(), B.ravel())


def test_reciprocals_beside_powers_of_two():
    """Divisors just above and below a power of two, whose reciprocals lie next to a binade's end."""
    k = np.arange(1, 2000)
    b = np.concatenate([np.ldexp(1.0 + s * k * 2.0 ** -52, e) for s in (1.0, -0.5) for e in (-99, -1, 0, 1, 99)])
    rng = np.random.default_rng(4)
    _check(_doubles(rng, b.size, -500, 500), b)
