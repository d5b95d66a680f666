"""The branch-free square root, reciprocal and quotient of the flux kernels
(vh_math.cuh) are correctly rounded over the ranges their callers check: equal
to the compiler's IEEE results bit for bit."""
import ctypes as C

import numpy as np
import pytest

import vh

pytestmark = pytest.mark.gpu
f = vh.lib.vh_device_round_check
f.restype = C.c_int
f.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]


def both(which, a, b=None):
    out = np.zeros(2 * len(a))
    vh.check(f(which, vh._ptr(a), None if b is None else vh._ptr(b), len(a), vh._ptr(out)), "vh_device_round_check")
    return out[:len(a)].view(np.uint64), out[len(a):].view(np.uint64)


def operands(rng, n, significand, lo, hi):
    m = {"any": rng.integers(0, 1 << 52, n, dtype=np.uint64),
         "small": rng.integers(0, 1 << 16, n, dtype=np.uint64),
         "large": np.uint64((1 << 52) - 1) - rng.integers(0, 1 << 16, n, dtype=np.uint64)}[significand]
    e = rng.integers(1023 + lo, 1023 + hi, n, dtype=np.uint64) << np.uint64(52)
    return (e | m).view(np.float64)


@pytest.mark.parametrize("exponent", [-100, -99, -1, 0, 1, 98, 99])
def test_sqrt_of_every_float_of_a_binade(exponent):
    a = ((np.arange(1 << 23, dtype=np.uint32) | np.uint32((127 + exponent) << 23)).view(np.float32)).astype(np.float64)
    got, want = both(0, a)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("significand", ["any", "small", "large"])
def test_reciprocal_and_quotient(significand):
    rng = np.random.default_rng(7)
    n = 1 << 20
    b = operands(rng, n, significand, -100, 100)
    b = b[(b.view(np.uint64) & np.uint64(0xffffffff)) != np.uint64(0xffffffff)]   # rcp_ok
    got, want = both(1, b)
    assert np.array_equal(got, want)
    for lo, hi in ((-100, 100), (-899, -880), (600, 800)):
        a = operands(rng, len(b), rng.choice(["any", "small", "large"]), lo, hi) * rng.choice([-1.0, 1.0], len(b))
        a[::17] = 0.0
        a[5::17] = -0.0
        got, want = both(2, a, b)
        assert np.array_equal(got, want)
