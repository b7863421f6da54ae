"""arti_heat as a module call on a context whose flags do not ask for the
artificial heat: the term is the call's, whatever the flags and the lanes per
target, against the oracle; at one lane per target also the bits of a context
with the flag set (with more lanes the flag decides how pass A sums the
divergence, and so its rounding)."""
import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuSolver
from oracle.oracle import Oracle
from tests.conftest import rel_l2
from tests.helpers import perturb, with_heat

pytestmark = pytest.mark.gpu

FLUIDS = {
    "dam2d": lambda: cases.dam_break_2d(dx=0.04),
    "dam3d": lambda: cases.dam_break_3d(dx=0.05),
    "dam2d_large": lambda: cases.dam_break_2d(dx=0.008),   # too many particles for shared pairs
}


@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("name", list(FLUIDS))
def test_heat_without_the_flag(gpu, name, lanes):
    c = with_heat(perturb(FLUIDS[name](), seed=71, v_amp=0.3, x_frac=0.1))
    o = Oracle(c, covering_band=True)
    o.rates()
    want = o.field("AH_DEDT")[: c.n_real]
    assert np.any(want != 0.0)
    off = c.params.copy()
    off.flags &= ~P.F_ARTI_HEAT
    got = []
    for prm in (c.params, off):
        with GpuSolver(c, params=prm) as s:
            s.set_option(P.OPT_LANES, lanes)
            s.nnps()
            got.append(s.arti_heat())
    assert rel_l2(got[1], want) <= 1e-10
    if lanes == 1:
        assert np.array_equal(got[0], got[1])
