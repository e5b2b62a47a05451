"""The step's quotient, reciprocal, square root estimate and limited slope on
the device (vah_math_values) against IEEE arithmetic.

Bounds: the reciprocal's last Newton-Raphson step leaves e^2 (2^-80) and two
roundings, 2^-52 relative; the quotient's residual correction leaves its
roundings of q and of the result, 2^-52; the square root estimate enters
admission tests with margins of 1e-5 only, and has to be within a fifth of that."""
import ctypes as C

import numpy as np
import pytest

import vahlib as V

D = C.POINTER(C.c_double)
QUOTIENT, RECIPROCAL, SQRT_ESTIMATE, SLOPE, SLOPE_FP32 = range(5)


def values(op, a, b):
    L = V.library()
    L.vah_math_values.argtypes = [C.c_int, C.c_int, D, D, C.c_int, D]
    a, b = (np.ascontiguousarray(x, dtype=np.float64) for x in np.broadcast_arrays(a, b))
    out = np.empty_like(a)
    assert L.vah_math_values(0, op, *(x.ctypes.data_as(D) for x in (a, b)), a.size, out.ctypes.data_as(D)) == 0
    return out


def spread(rng, n, lo, hi):
    return np.exp2(rng.uniform(lo, hi, n)) * rng.choice([-1.0, 1.0], n)


def test_math_values_argument_errors():
    L = V.library()
    L.vah_math_values.argtypes = [C.c_int, C.c_int, D, D, C.c_int, D]
    x = (C.c_double * 1)(1.0)
    for op, n, a in ((-1, 1, x), (5, 1, x), (0, 0, x), (0, 1, None)):
        assert L.vah_math_values(0, op, a, x, n, x) == -1


@pytest.mark.gpu
def test_quotient_is_the_ieee_one_to_an_ulp():
    rng = np.random.default_rng(1)
    n = 400_000
    f = np.concatenate([spread(rng, n, -20, 20), spread(rng, n, -400, 400), spread(rng, n, -1074, 1023)])
    d = np.concatenate([spread(rng, n, -20, 20), spread(rng, n, -400, 400), spread(rng, n, -1074, 1023)])
    # the edges of the band in which the estimate is used
    edge = np.exp2(np.array([-1001.0, -1000, -999, 1000, 1001, 1002])) * np.array([[0.75], [1 - 2.0 ** -53], [1.0], [1.5]])
    f = np.concatenate([f, spread(rng, 24, -2, 2)])
    d = np.concatenate([d, edge.ravel()])
    with np.errstate(all="ignore"):
        want = f / d
    got = values(QUOTIENT, f, d)
    big = np.isinf(want)
    assert np.array_equal(got[big], want[big])
    err = np.abs(got - want)[~big]
    assert np.all(err <= np.maximum(2.0 ** -52 * np.abs(want[~big]), 5e-324))


@pytest.mark.gpu
def test_quotient_of_infinities_zeros_and_nans():
    """As IEEE's: an infinite numerator or an overflowing quotient is infinite, not NaN."""
    x = np.array([0.0, -0.0, 5e-324, 1e-300, 1.0, -3.0, 1e10, 1e300, 1.7e308, np.inf, -np.inf, np.nan])
    f, d = (a.ravel() for a in np.meshgrid(x, x))
    with np.errstate(all="ignore"):
        want = f / d
    got = values(QUOTIENT, f, d)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    sure = ~np.isfinite(want) | (want == 0)
    assert np.array_equal(got[sure], want[sure], equal_nan=True)
    assert np.array_equal(np.signbit(got[~np.isnan(want)]), np.signbit(want[~np.isnan(want)]))


@pytest.mark.gpu
def test_reciprocal_and_square_root_estimate():
    rng = np.random.default_rng(2)
    x = np.concatenate([spread(rng, 300_000, -332, 335), spread(rng, 300_000, -3, 3)])
    assert np.max(np.abs(values(RECIPROCAL, x, x) * x - 1)) <= 2.0 ** -52 + 2.0 ** -53  # the check's own rounding
    x = np.abs(x)
    assert np.max(np.abs(values(SQRT_ESTIMATE, x, x) / np.sqrt(x) - 1)) <= 2e-6
    assert np.array_equal(values(SQRT_ESTIMATE, [0.0], [1.0]), [0.0])


def slope(dl, dr, cc):
    """The limiter by its formula: theta = 1.1, a NaN passed over by the minima
    (fmin) and not below zero."""
    t = dl.dtype.type
    with np.errstate(all="ignore"):
        m = np.fmin(t(1.1) * np.fmin(abs(dl), abs(dr)), abs(cc * t(0.5)))
        neg = dl < 0
        return np.where(neg == (dr < 0), np.where(neg, -m, m), t(0))


@pytest.mark.gpu
@pytest.mark.parametrize("op,t", [(SLOPE, np.float64), (SLOPE_FP32, np.float32)])
def test_limited_slope_equals_the_limiter(op, t):
    """Value for value, beside NaNs and infinities too: the device's own NaN of
    an FP64 difference has its sign bit set, which is not a negative slope."""
    rng = np.random.default_rng(3)
    x = np.array([0.0, -0.0, 1e-30, -1e-30, 1.0, -1.0, 1.1, 3.0, -2.5, 1e30, np.inf, -np.inf, np.nan, -np.nan])
    a, b = (v.ravel() for v in np.meshgrid(x, x))
    a = np.concatenate([a, rng.normal(size=300_000), rng.normal(size=300_000)]).astype(t)
    b = np.concatenate([b, rng.normal(size=300_000), a[-300_000:] * t(-1) + t(1e-3) * rng.normal(size=300_000).astype(t)]).astype(t)
    with np.errstate(all="ignore"):
        want = slope(t(0) - a, b - t(0), b - a)
    got = values(op, a.astype(np.float64), b.astype(np.float64)).astype(t)
    assert np.array_equal(got, want, equal_nan=True)
