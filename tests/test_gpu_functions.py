"""The reciprocals, roots, quotients and compares that the passes use in place
of CUDA's functions, against exact rational arithmetic.  u is half a unit in
the last place of 1: a correctly rounded result is within 1 u of the exact
one, relatively, in any binade."""
import ctypes as C
import math
from fractions import Fraction

import numpy as np
import pytest

from mysph_gb300._lib import dp, load

pytestmark = pytest.mark.gpu

RSQRT, RCP, DIV, RSQRT_F32, DIV_F32, RCP_DF, RSQRT_DF, FROM_U32, NEGATIVE, NAN, CUDA_RSQRT = range(11)
U64, U32 = Fraction(1, 1 << 53), Fraction(1, 1 << 24)


def call(fn, a, b=None):
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = None if b is None else np.ascontiguousarray(b, dtype=np.float64)
    out, low = np.full(len(a), -7.0), np.full(len(a), -7.0)
    ptr = lambda v: None if v is None else v.ctypes.data_as(dp)
    assert load().sph_check_function(fn, len(a), ptr(a), ptr(b), ptr(out), ptr(low)) == 0
    return out, low


def values(lo_exp, hi_exp, n, seed, mantissas=True):
    """n doubles over the binary exponents [lo_exp, hi_exp], among them each
    exponent of the ends and the mantissas next to powers of two."""
    rng = np.random.default_rng(seed)
    e = rng.integers(lo_exp, hi_exp + 1, n)
    e[:40] = np.repeat([lo_exp, lo_exp + 1, hi_exp - 1, hi_exp], 10)
    m = 1.0 + rng.random(n)
    m[::7] = 1.0
    m[1::7] = 2.0 - 2.0 ** -52
    m[2::7] = 1.0 + 2.0 ** -52
    m = np.minimum(m, 2.0 - 2.0 ** -52)
    return np.ldexp(m, e)


def units(got, exact, u):
    """|got - exact| / exact in units u (all Fractions)."""
    return float(abs(got - exact) / abs(exact) / u)


def rsqrt_units(got, x, u):
    """The error of got as 1 / sqrt(x), relative: (got sqrt x - 1) to first
    order is (got^2 x - 1) / 2."""
    return float(abs(got * got * x - 1) / 2 / u)


SPECIAL = np.array([0.0, -0.0, 5e-324, -5e-324, 1e-310, -1e-310, np.inf, -np.inf, np.nan, -np.nan, -1.0, -2.5e-300])


# 1 / sqrt: the last operation rounds (1 u); before it stands the truncation
# of the third-order step, 5/16 e^3 with e below 2e-6 (0.03 u)
def test_rsqrt(gpu):
    x = np.concatenate([values(-1022, 1023, 12000, 1), values(-60, 20, 12000, 2)])
    got, _ = call(RSQRT, x)
    worst = max(rsqrt_units(Fraction(g), Fraction(v), U64) for g, v in zip(got, x))
    assert worst <= 1.04
    cuda, _ = call(CUDA_RSQRT, x)
    off = np.abs(got.view(np.int64) - cuda.view(np.int64))
    assert off.max() <= 2   # CUDA's is within one ulp, this one within a little over half of one
    got, _ = call(RSQRT, SPECIAL)
    want, _ = call(CUDA_RSQRT, SPECIAL)
    want[:2] = 0.0   # coincident particles
    assert np.array_equal(got, want, equal_nan=True)


# 1 / x: likewise, with e^3
def test_rcp(gpu):
    x = np.concatenate([values(-1021, 1020, 12000, 3), values(-60, 60, 12000, 4)])
    x[::3] *= -1.0
    got, _ = call(RCP, x)
    assert max(units(Fraction(g), 1 / Fraction(v), U64) for g, v in zip(got, x)) <= 1.04
    with np.errstate(divide="ignore", over="ignore"):
        ends = np.concatenate([SPECIAL, values(-1022, -1022, 50, 5), values(1021, 1023, 50, 6)])
        ex = np.frexp(ends)[1] - 1
        out = ~np.isfinite(ends) | (ends == 0) | (ex < -1021) | (ex > 1020)   # beyond the estimate: the division itself
        got, want = call(RCP, ends)[0], 1.0 / ends
    assert out.sum() > 80 and np.array_equal(got[out], want[out], equal_nan=True)
    assert max(units(Fraction(g), 1 / Fraction(v), U64) for g, v in zip(got[~out], ends[~out])) <= 1.04


# n / d: the residual of the quotient is exact, so only the last rounding stays
def test_div(gpu):
    n = np.concatenate([values(-383, 384, 12000, 7), values(-60, 40, 12000, 8)])
    d = np.concatenate([values(-383, 384, 12000, 9), values(-60, 40, 12000, 10)])
    n[::5] *= -1.0
    got, _ = call(DIV, n, d)
    assert max(units(Fraction(g), Fraction(p) / Fraction(q), U64) for g, p, q in zip(got, n, d)) <= 1.0 + 1e-9
    # beyond those exponents, and for zeros, infinities and NaN: the division itself
    far = np.concatenate([SPECIAL, values(-1022, -384, 300, 11), values(385, 1023, 300, 12), [1.0, 3.0]])
    rng = np.random.default_rng(13)
    p, q = rng.choice(far, 4000), rng.choice(far, 4000)
    with np.errstate(all="ignore"):
        ok = (np.abs(np.frexp(p)[1]) > 384) | (np.abs(np.frexp(q)[1]) > 385) | ~np.isfinite(p) | ~np.isfinite(q)
        ok |= (p == 0) | (q == 0)
        got, want = call(DIV, p, q)[0], p / q
    assert ok.sum() > 3000 and np.array_equal(got[ok], want[ok], equal_nan=True)


# double-float 1 / a: three roundings of 2^-48 at most
def test_rcp_df(gpu):
    a = values(-100, 100, 12000, 14)
    hi, lo = call(RCP_DF, a)
    f = a.astype(np.float32)
    x = [Fraction(float(p)) + Fraction(float(np.float32(v - float(p)))) for p, v in zip(f, a)]
    assert max(float(abs((Fraction(g) + Fraction(h)) * v - 1)) for g, h, v in zip(hi, lo, x)) <= 2.0 ** -46


def test_integers_and_signs(gpu):
    rng = np.random.default_rng(15)
    k = np.concatenate([[0, 1, 2, 3, (1 << 32) - 1, 1 << 31, (1 << 31) - 1, 1 << 24, (1 << 24) + 1],
                        rng.integers(0, 1 << 32, 4000), 1 << rng.integers(0, 32, 200)]).astype(np.float64)
    assert np.array_equal(call(FROM_U32, k)[0], k)
    x = np.concatenate([SPECIAL, values(-1022, 1023, 2000, 16) * rng.choice([-1.0, 1.0], 2000)])
    assert np.array_equal(call(NEGATIVE, x)[0], (x < 0).astype(np.float64))
    assert np.array_equal(call(NAN, x)[0], np.isnan(x).astype(np.float64))


def test_arguments_are_checked(gpu):
    lib, one = load(), np.ones(1)
    p = one.ctypes.data_as(dp)
    assert lib.sph_check_function(11, 1, p, p, p, p) != 0
    assert lib.sph_check_function(-1, 1, p, p, p, p) != 0
    assert lib.sph_check_function(DIV, 1, p, None, p, p) != 0
    assert lib.sph_check_function(RSQRT_DF, 1, p, None, p, None) != 0
    assert lib.sph_check_function(RCP, -1, p, None, p, None) != 0
