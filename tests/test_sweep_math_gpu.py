"""The FP64 sweeps' reciprocal, roots and erfc/exp pair as they run on the
device, against 64-bit-mantissa and 40-digit host values, over the arguments
they are used on and their edges."""
import ctypes as C
import os
import subprocess

import mpmath
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "device")
RCP, RSQRT, SQRT0, ERFC_EXP = range(4)
ULP = 2.0 ** -53   # half a unit in the last place, relative, at most


@pytest.fixture(scope="module")
def run():
    path = os.path.join(HERE, "libsweep_math.so")
    if not os.path.exists(path):
        subprocess.run(["make", "-C", HERE], check=True)
    fn = C.CDLL(path).sweep_math
    P = C.POINTER(C.c_double)
    fn.argtypes = [C.c_int, C.c_longlong, P, P, P]

    def call(which, x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y, z = np.empty_like(x), np.empty_like(x)
        assert fn(which, len(x), *[a.ctypes.data_as(P) for a in (x, y, z)]) == 0
        return (y, z) if which == ERFC_EXP else y
    return call


def spread(low, high, count=200000):
    """Random mantissas over the binary exponents low .. high, every power of
    two of that range and its neighbours."""
    rng = np.random.default_rng(low + 7 * high)
    e = rng.integers(low, high, count)
    x = np.ldexp(rng.uniform(1.0, 2.0, count), e)
    p = np.ldexp(1.0, np.arange(low, high + 1))
    return np.concatenate([x, p, np.nextafter(p[1:], 0.0), np.nextafter(p[:-1], np.inf)])


def units(got, want):
    """Error in units in the last place of the exact value."""
    exact = want.astype(np.float64)
    return np.max(np.abs((got.astype(np.longdouble) - want) / np.spacing(np.abs(exact))))


def test_rcp(run):
    """1 ulp for 2^-1022 <= |x| <= 2^1021."""
    x = spread(-1022, 1021)
    x = np.concatenate([x, -x])
    assert units(run(RCP, x), 1 / x.astype(np.longdouble)) <= 1.0


def test_rsqrt(run):
    """1 ulp for every normal x > 0."""
    x = np.concatenate([spread(-1022, 1023), [np.finfo(float).max]])
    assert units(run(RSQRT, x), 1 / np.sqrt(x.astype(np.longdouble))) <= 1.0


def test_sqrt0(run):
    """2 ulp (x / sqrt(x) adds a rounding to rsqrt_'s), 0 below the smallest
    normal number."""
    x = np.concatenate([spread(-1022, 1023), [np.finfo(float).max]])
    assert units(run(SQRT0, x), np.sqrt(x.astype(np.longdouble))) <= 2.0
    small = [0.0, -0.0, 5e-324, np.nextafter(np.finfo(float).tiny, 0.0), -1.0]
    assert np.all(run(SQRT0, small) == 0.0)


def test_erfc_exp(run):
    """erfc(x) within 6 and exp(-x^2) within 4 units of 2^-53 relative, for
    |x| <= 26 (the argument reductions and the two Horner schemes lose about
    5 together, tests/test_erfc_host.py)."""
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-6.0, 6.0, 3000), rng.uniform(6.0, 26.0, 1500),
                        rng.uniform(-1e-3, 1e-3, 500), np.linspace(-26.0, 26.0, 53),
                        [1e-300, -1e-20, 1e-9, 0.0]])
    ec, ex = run(ERFC_EXP, x)
    with mpmath.workdps(40):
        worst = [0.0, 0.0]
        for v, a, b in zip(x, ec, ex):
            m = mpmath.mpf(float(v))
            for q, got, want in ((0, a, mpmath.erfc(m)), (1, b, mpmath.exp(-m * m))):
                error = abs((mpmath.mpf(float(got)) - want) / want) / mpmath.mpf(ULP)
                worst[q] = max(worst[q], float(error))
    assert worst[0] <= 6.0 and worst[1] <= 4.0, worst


def test_erfc_exp_beyond(run):
    """Where exp(-x^2) leaves the normal numbers: 0, and 0 or 2."""
    x = np.array([26.7, 27.5, 40.0, 300.0, 1e9, 1e150, 1e300])
    for sign, limit in ((1.0, 0.0), (-1.0, 2.0)):
        ec, ex = run(ERFC_EXP, sign * x)
        assert np.all(ec == limit) and np.all(ex == 0.0)
