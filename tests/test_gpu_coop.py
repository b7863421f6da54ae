"""Small FP64 systems share each target's pairs among lanes without a change
of the order of the sums: the bits are those of one lane per target, which the
same system gets in a batch too large for the sharing."""
import dataclasses

import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuBatch, GpuSolver
from tests.helpers import perturb

pytestmark = pytest.mark.gpu


def few(c, n):
    """The first n real particles of the case, and its walls."""
    return c.subset_real(np.arange(c.n_real) < n)


def flagged(c, flags=0, beta=None):
    prm = c.params.copy()
    prm.flags |= flags
    if beta is not None:
        prm.av_beta = prm.av_beta_solid = beta
    return dataclasses.replace(c, params=prm)


def dam2(dx, **kw):
    return perturb(cases.dam_break_2d(dx=dx), seed=11, v_amp=0.5, x_frac=0.2)


def dam3(dx):
    return perturb(cases.dam_break_3d(dx=dx), seed=12, v_amp=0.5, x_frac=0.2)


def beam(dx):
    return perturb(cases.cantilever_2d(dx=dx), seed=13, v_amp=0.5)


# 32, 16, 8, 4 and 2 lanes a target; one and a few particles; solids; beta != 0
@pytest.mark.parametrize("name,small,filler", [
    ("2d_32", lambda: dam2(0.05), lambda: dam2(0.006)),
    ("2d_16", lambda: dam2(0.032), lambda: dam2(0.006)),
    ("2d_8", lambda: dam2(0.0205), lambda: dam2(0.006)),
    ("2d_4", lambda: dam2(0.0151), lambda: dam2(0.006)),
    ("2d_2", lambda: dam2(0.0107), lambda: dam2(0.006)),
    ("2d_one", lambda: few(dam2(0.05), 1), lambda: dam2(0.006)),
    ("2d_few", lambda: few(dam2(0.05), 37), lambda: dam2(0.006)),
    ("2d_beta", lambda: flagged(dam2(0.03), beta=0.3), lambda: flagged(dam2(0.006), beta=0.3)),

    ("3d_32", lambda: dam3(0.05), lambda: dam3(0.0115)),
    ("3d_8", lambda: dam3(0.03), lambda: dam3(0.0115)),
    ("3d_2", lambda: dam3(0.0185), lambda: dam3(0.0115)),
    ("beam", lambda: beam(1.5e-3), lambda: beam(2.5e-4)),
    ("beam_wide", lambda: beam(4e-4), lambda: beam(2.5e-4)),
])
def test_small_system_bits(gpu, name, small, filler):
    a, b = small(), filler()
    steps = 4
    with GpuSolver(a) as s:
        s.advance(steps)
        want = {f: s.field(f) for f in ("X", "V", "RHO", "E", "P", "NNEIGH")}
    with GpuBatch(b.params, 2, a.n_real + b.n_real, a.n_wall + b.n_wall + 1) as g:
        g.add(b)
        k = g.add(a)
        g.advance(steps)
        for f in want:
            assert np.array_equal(g.field(k, f), want[f]), f


def test_lanes_option_keeps_its_own_order(gpu):
    """With SPH_OPT_LANES above 1 the option's order holds, small or not."""
    a = dam2(0.03)
    with GpuSolver(a) as s, GpuBatch(a.params, 2, 200000, 20000) as g:
        s.set_option(P.OPT_LANES, 4)
        g.set_option(P.OPT_LANES, 4)
        g.add(dam2(0.006))
        k = g.add(a)
        s.advance(4)
        g.advance(4)
        assert np.array_equal(s.field("V"), g.field(k, "V"))
