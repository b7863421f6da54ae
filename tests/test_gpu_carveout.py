"""SPH_OPT_SMEM_CARVEOUT reaches the kernels that a step's passes A and B run:
small FP64 systems (shared pairs), large ones, lanes per target, XSPH, solids
with and without the artificial stress, and the mixed forms."""
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuSolver

pytestmark = pytest.mark.gpu


def changed(c, on=0, off=0, precision=P.PREC_FP64):
    c.params = c.params.copy()
    c.params.flags = (c.params.flags | on) & ~off
    c.params.precision = precision
    return c


FORMS = {
    "small_2d": (lambda: cases.dam_break_2d(dx=0.05), 1),
    "small_3d": (lambda: cases.dam_break_3d(dx=0.05), 1),
    "small_beam": (lambda: changed(cases.cantilever_2d(dx=2e-3), off=P.F_ARTI_STRESS), 1),
    "large_2d": (lambda: cases.dam_break_2d(dx=0.006), 1),
    "lanes": (lambda: cases.dam_break_2d(dx=0.05), 4),
    "xsph": (lambda: changed(cases.dam_break_2d(dx=0.05), on=P.F_AVER_VELOCITY), 1),
    "gate_stress": (lambda: cases.gate_2d(dx=0.0025), 1),
    "mixed_2d": (lambda: changed(cases.dam_break_2d(dx=0.05), precision=P.PREC_MIXED), 1),
    "mixed_gate": (lambda: changed(cases.gate_2d(dx=0.0025), precision=P.PREC_MIXED), 1),
    "mixed_xsph": (lambda: changed(cases.dam_break_2d(dx=0.05), on=P.F_AVER_VELOCITY, precision=P.PREC_MIXED), 1),
}


@pytest.mark.parametrize("name", list(FORMS))
def test_option_reaches_the_passes(gpu, name):
    make, lanes = FORMS[name]
    with GpuSolver(make()) as s:
        s.set_option(P.OPT_LANES, lanes)
        try:
            s.set_option(P.OPT_SMEM_CARVEOUT, 73)
            assert s.carveout() == (73, 73)
        finally:
            s.set_option(P.OPT_SMEM_CARVEOUT, -1)   # the attribute is the kernels', not the context's
        assert s.carveout() == (-1, -1)
