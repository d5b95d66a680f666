"""The branch-free square root, reciprocal and quotient (vh_math.cuh) over the
ranges their callers reach: every binade of the square root's argument, and
divisors of either sign down to 2^-130 and up to 2^121 (2 p/e and p H of the
table's root solve, at an iterate below zero too).  Equal to the compiler's
IEEE results bit for bit; only the sign of a zero quotient by a negative
divisor is free."""
import ctypes as C

import numpy as np
import pytest

import vh

pytestmark = pytest.mark.gpu
f = vh.lib.vh_device_round_check
f.restype = C.c_int
f.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]


def both(which, a, b=None):
    a = np.ascontiguousarray(a)
    out = np.zeros(2 * len(a))
    vh.check(f(which, vh._ptr(a), None if b is None else vh._ptr(b), len(a), vh._ptr(out)), "vh_device_round_check")
    return out[:len(a)].view(np.uint64), out[len(a):].view(np.uint64)


def test_sqrt_in_every_binade():
    rng = np.random.default_rng(11)
    m = np.concatenate([np.arange(256), (1 << 23) - 1 - np.arange(256), rng.integers(0, 1 << 23, 1 << 14)]).astype(np.uint32)
    e = (np.arange(-100, 100) + 127).astype(np.uint32) << np.uint32(23)
    got, want = both(0, (e[:, None] | m).reshape(-1).view(np.float32).astype(np.float64))
    assert np.array_equal(got, want)


def draw(rng, n, kind, lo, hi):
    m = {"any": rng.integers(0, 1 << 52, n, dtype=np.uint64),
         "small": rng.integers(0, 1 << 10, n, dtype=np.uint64),
         "large": np.uint64((1 << 52) - 1) - rng.integers(0, 1 << 10, n, dtype=np.uint64)}[kind]
    return (rng.integers(1023 + lo, 1023 + hi, n, dtype=np.uint64) << np.uint64(52) | m).view(np.float64)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("kind", ["any", "small", "large"])
def test_reciprocal_and_quotient(kind, sign):
    rng = np.random.default_rng(13)
    b = draw(rng, 1 << 20, kind, -130, 121)
    b = sign * b[(b.view(np.uint64) & np.uint64(0xffffffff)) != np.uint64(0xffffffff)]      # rcp_ok
    got, want = both(1, b)
    assert np.array_equal(got, want)
    for lo, hi in ((-900, -860), (-500, -100), (-100, 100), (600, 800)):
        for ka in ("any", "small", "large"):
            a = draw(rng, len(b), ka, lo, hi) * rng.choice([-1.0, 1.0], len(b))
            got, want = both(2, a, b)
            assert np.array_equal(got, want)
    zero = rng.choice([-0.0, 0.0], len(b))
    got, want = both(2, zero, b)
    if sign > 0:
        assert np.array_equal(got, want)
    else:
        assert not np.any(got << np.uint64(1))
