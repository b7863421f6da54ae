"""The quotients of the mixed artificial viscosity: as good as the correctly
rounded division, and the division itself where an operand is out of range."""
from fractions import Fraction

import numpy as np
import pytest

from tests.test_gpu_functions import DIV_F32, U32, call, units, values

pytestmark = pytest.mark.gpu


# the last operation rounds (1 u); before it, the reciprocal estimate (2^-23)
# scales the residual of a quotient that is off by at most 2^-22: 2^-45
def test_div_f32(gpu):
    n = np.concatenate([values(-60, 60, 12000, 31), values(-20, 20, 12000, 32)]).astype(np.float32).astype(np.float64)
    d = np.concatenate([values(-60, 60, 12000, 33), values(-20, 20, 12000, 34)]).astype(np.float32).astype(np.float64)
    n[::2] *= -1.0
    got, _ = call(DIV_F32, n, d)
    assert max(units(Fraction(g), Fraction(p) / Fraction(q), U32) for g, p, q in zip(got, n, d)) <= 1.0 + 2.0 ** -20


def test_div_f32_out_of_range(gpu):
    far = np.concatenate([[0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-40, 3e38, 1.2e-38],
                          values(-149, -64, 200, 35), values(64, 127, 200, 36)])
    with np.errstate(all="ignore"):
        far = far.astype(np.float32)
        rng = np.random.default_rng(37)
        p, q = rng.choice(far, 4000), rng.choice(far, 4000)
        want = p / q
    got, _ = call(DIV_F32, p.astype(np.float64), q.astype(np.float64))
    assert np.array_equal(got, want.astype(np.float64), equal_nan=True)
