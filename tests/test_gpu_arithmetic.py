"""The FP64 square root, its reciprocal and the reciprocal of the N-body kernels and the quotients of the LU against 80-bit
arithmetic (B200).

All three are formed from an approximation by steps of their own.  Bounds, in units in the last place:
  1/sqrt(x)  1.01: half a unit of the last rounding, half a unit of the rounding of x y in the residual, and the
             remainder of a third-order step from a seed of relative error 2^-20 (CUDA's rsqrt: 1);
  1/x        0.51: half a unit of the last rounding and the remainder 2^-60 (CUDA's: 0.5);
  sqrt(x)    0.78: half a unit of the last rounding, half of the half unit of x y (it enters halved) and the
             remainder;
  x/y        the correctly rounded quotient, as the division gives it.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_P = C.POINTER(C.c_double)
RSQRT, RECIPROCAL, QUOTIENT, QUOTIENT_F32, SQRT = range(5)


def _call(kind, x, y=None):
    import uvlm_b200 as U

    x = np.ascontiguousarray(x, np.float64)
    y = x if y is None else np.ascontiguousarray(y, np.float64)
    out = np.empty_like(x)
    U._capi.check(U.lib().uvlm_check_arithmetic(kind, x.ctypes.data_as(_P), y.ctypes.data_as(_P), x.size,
                                                out.ctypes.data_as(_P)))
    return out


def _mantissas(rng, n):
    """In [1, 2): spread, and within a few units of either end."""
    ends = rng.integers(0, 8, n // 8) * 2.0 ** -52
    m = rng.uniform(1, 2, n)
    m[: n // 8], m[n // 8: n // 4] = 1 + ends, 2 - 2.0 ** -52 - ends
    return m


# the squares of distances that the cuts admit begin at 1e-20, the denominators at 1e-30
@pytest.mark.parametrize("kind,low,high,bound", [(RSQRT, -67, 40, 1.01), (RSQRT, -1020, 1023, 1.01),
                                                 (RECIPROCAL, -100, 60, 0.51), (RECIPROCAL, -1020, 1021, 0.51)])
def test_nbody_reciprocals(kind, low, high, bound):
    rng = np.random.default_rng(kind + high)
    n = 1 << 20
    x = _mantissas(rng, n) * 2.0 ** rng.integers(low, high, n)
    x[:2] = 2.0 ** low, (2 - 2.0 ** -52) * 2.0 ** (high - 1)
    ref = 1 / (np.sqrt(x.astype(np.longdouble)) if kind == RSQRT else x.astype(np.longdouble))
    err = np.abs((_call(kind, x) - ref) / np.spacing(ref.astype(np.float64)))
    assert float(err.max()) <= bound


@pytest.mark.parametrize("kind,dtype,low,high", [(QUOTIENT, np.float64, -880, 880), (QUOTIENT_F32, np.float32, -95, 95)])
def test_lu_quotients(kind, dtype, low, high):
    """Multipliers (|x| <= |y|), quotients above 1 as of locally pivoted factors, pivots at the ends of the range (where
    the quotient is a division) and zero pivots (0: the factor is singular)."""
    rng = np.random.default_rng(kind)
    n = 1 << 20
    y = (_mantissas(rng, n) * 2.0 ** rng.integers(low, high, n) * rng.choice([-1, 1], n)).astype(dtype)
    scale = np.where(rng.random(n) < 0.2, rng.uniform(1, 64, n), rng.uniform(-1, 1, n))
    x = (y * scale).astype(dtype)
    info = np.finfo(dtype)
    y[:4], x[:4] = [info.tiny, info.max, -info.tiny, info.max / 2], [info.tiny / 2, info.max / 3, info.tiny, -info.max]
    np.testing.assert_array_equal(_call(kind, x, y).astype(dtype), x / y)
    assert np.all(_call(kind, x[:100], np.zeros(100)) == 0)
    assert np.all(np.isnan(_call(kind, x[:100], np.full(100, np.nan))))


@pytest.mark.parametrize("low,high", [(-67, 40), (-1020, 1023)])
def test_nbody_lengths(low, high):
    rng = np.random.default_rng(high)
    n = 1 << 20
    x = _mantissas(rng, n) * 2.0 ** rng.integers(low, high, n)
    x[:2] = 2.0 ** low, (2 - 2.0 ** -52) * 2.0 ** (high - 1)
    ref = np.sqrt(x.astype(np.longdouble))
    err = np.abs((_call(SQRT, x) - ref) / np.spacing(ref.astype(np.float64)))
    assert float(err.max()) <= 0.78
