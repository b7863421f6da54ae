"""1 / sqrt of the FP32 and double-float passes over the whole range of FP32
squared distances, subnormal ones among them, against exact arithmetic."""
from fractions import Fraction

import numpy as np
import pytest

from tests.test_gpu_functions import RSQRT_DF, RSQRT_F32, call, rsqrt_units, values

pytestmark = pytest.mark.gpu


# CUDA's bound for rsqrtf: 2 units in the last place, 2^-22 relative
def test_rsqrt_f32(gpu):
    with np.errstate(over="ignore"):
        x = np.concatenate([values(-126, 127, 8000, 21), values(-149, -127, 2000, 22)]).astype(np.float32)
    x = np.abs(x[(x > 0) & np.isfinite(x)]).astype(np.float64)
    got, _ = call(RSQRT_F32, x)
    assert max(rsqrt_units(Fraction(g), Fraction(v), 1) for g, v in zip(got, x)) <= 2.0 ** -22
    assert np.array_equal(call(RSQRT_F32, [0.0, -0.0])[0], [0.0, 0.0])


# double-float: the estimate is within 2^-22, its residual (below 2^-21) is
# formed with at most three roundings of 2^-46, halved, and the correction
# rounds once more, 2^-46: 2.5 x 2^-46, under 2^-44
def test_rsqrt_df(gpu):
    a = values(-125, 126, 12000, 23)
    hi, lo = call(RSQRT_DF, a)
    f = a.astype(np.float32)
    x = [Fraction(float(p)) + Fraction(float(np.float32(v - float(p)))) for p, v in zip(f, a)]
    err = [rsqrt_units(Fraction(g) + Fraction(h), v, 1) if np.isfinite(g) and np.isfinite(h) else np.inf
           for g, h, v in zip(hi, lo, x)]
    assert max(err) <= 2.0 ** -44
