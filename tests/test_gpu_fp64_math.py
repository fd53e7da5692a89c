"""Sine, cosine and reciprocal square root of the FP64 form against 80-bit values
and CUDA's functions."""
import ctypes as C

import numpy as np
import pytest

from baemm_b200 import _capi

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
rng = np.random.default_rng(5)


def _eval(x):
    """(sin, cos, 1/sqrt|x|) as the FP64 form has them, and CUDA's."""
    x = np.ascontiguousarray(x, np.float64)
    out = np.zeros((6, x.size))
    dp = C.POINTER(C.c_double)
    assert _capi.lib().baemm_selftest_fp64_math(0, x.size, x.ctypes.data_as(dp), out.ctypes.data_as(dp)) == 0
    return out[:3], out[3:]


def _near_multiples(k):
    """Arguments at and beside k pi/2, down to the neighbouring doubles."""
    x = np.float64(k.astype(np.longdouble) * np.longdouble("1.5707963267948966192313216916397514"))
    return np.concatenate([x, np.nextafter(x, 0), np.nextafter(x, np.inf)] + [x + d for d in (1e-12, -1e-9, 1e-4, -0.7853)])


ARGUMENTS = {
    "first octants": rng.uniform(-4.0, 4.0, 200000),
    "all sizes below the switch": rng.uniform(-1e5, 1e5, 200000),
    "small": rng.uniform(-1, 1, 50000) * 10.0 ** rng.uniform(-300, 0, 50000),
    "zero": np.array([0.0, -0.0, 5e-324, -5e-324]),
    "near k pi/2, small k": _near_multiples(np.arange(-2000, 2000)),
    "near k pi/2, large k": _near_multiples(rng.integers(2000, 63661, 20000)),
    "both sides of the switch": np.concatenate([1e5 + rng.uniform(-50, 50, 20000), -1e5 + rng.uniform(-50, 50, 20000)]),
    "beyond": rng.uniform(1e5, 1e9, 50000),
}


@pytest.mark.parametrize("name", ARGUMENTS)
def test_sin_and_cos(name):
    """The reduced argument is within 2^-53 of its own size and 1e-28 (the part of
    pi/2 below its two doubles, 1.5e-33, times k < 63663); a Taylor remainder of
    at most 0.6 units of 2^-53, about 0.3 from the correction terms and one from the
    last rounding follow: below 4 units of the value.  CUDA's functions are within 2
    units in the last place, at most 4 of 2^-53, by themselves."""
    x = ARGUMENTS[name]
    own, cuda = _eval(x)
    lx = x.astype(np.longdouble)
    for f, a, b in ((np.sin(lx), own[0], cuda[0]), (np.cos(lx), own[1], cuda[1])):
        bound = 4 * U * np.abs(f) + 1e-28 + 5e-324
        assert np.all(np.abs(a - f) <= bound), (np.abs(a - f) / (np.abs(f) + 1e-300)).max() / U
        assert np.all(np.abs(a - b) <= 2 * bound)


def test_reciprocal_square_root():
    """A remainder of 5/16 e^3 with e below 2^-18, half a unit of 2^-53 from the
    rounding of e and one from the last: below 2 units over every normal exponent."""
    x = np.concatenate([2.0 ** rng.uniform(-1021, 1023, 400000), rng.uniform(0.5, 4.0, 400000),
                        np.array([2.2250738585072014e-308, 1.7976931348623157e308, 1.0, 4.0])])
    own, cuda = _eval(x)
    ref = 1 / np.sqrt(x.astype(np.longdouble))
    assert np.all(np.abs(own[2] - ref) <= 2 * U * ref), (np.abs(own[2] - ref) / ref).max() / U
    assert np.all(np.abs(own[2] - cuda[2]) <= 4 * U * cuda[2])


def test_invalid_arguments():
    dp = C.POINTER(C.c_double)
    x = np.ones(1)
    p = x.ctypes.data_as(dp)
    lib = _capi.lib()
    assert lib.baemm_selftest_fp64_math(0, 0, p, p) == 1
    assert lib.baemm_selftest_fp64_math(-1, 1, p, p) == 1
    assert lib.baemm_selftest_fp64_math(0, 1, None, p) == 1
