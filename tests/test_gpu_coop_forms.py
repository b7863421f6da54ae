"""Shared pairs of small FP64 systems beyond the plain fluid: other kernels,
several Types, fluid and solid targets in one warp, targets without gravity,
and cells so large that the candidate buffer fills.  The bits are those of one
lane per target, which the same system gets in a large batch."""
import dataclasses

import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuBatch, GpuSolver
from tests.helpers import fsi_block_3d, perturb, two_fluid_dam_break
from tests.test_gpu_coop import beam, dam2, dam3

pytestmark = pytest.mark.gpu


def changed(c, on=0, off=0, **kw):
    prm = c.params.copy()
    prm.flags = (prm.flags | on) & ~off
    for k, v in kw.items():
        setattr(prm, k, v)
    return dataclasses.replace(c, params=prm)


def wide_cells(c, factor):
    return changed(c, cell_size=factor * 2.0 * float(c.h.max()))


def gate(dx, **kw):
    return changed(perturb(cases.gate_2d(dx=dx), seed=14, v_amp=0.05, x_frac=0.1), **kw)


NO_STRESS = dict(off=P.F_ARTI_STRESS)
SKIP = dict(on=P.F_GRAVITY | P.F_GRAVITY_SKIP_SOLIDS, off=P.F_ARTI_STRESS)


def fsi():
    return changed(fsi_block_3d(), dt=1e-6)


def like(c, small):
    """The filler with the small system's model."""
    return changed(c, on=small.params.flags, off=~small.params.flags, skf=small.params.skf,
                   pen_factor=small.params.pen_factor, pen_n1=small.params.pen_n1, pen_n2=small.params.pen_n2)


@pytest.mark.parametrize("name,small,filler", [
    ("2d_gauss", lambda: changed(dam2(0.03), skf=2), lambda: dam2(0.006)),
    ("2d_quintic", lambda: changed(dam2(0.03), skf=3), lambda: dam2(0.006)),
    ("3d_gauss", lambda: changed(dam3(0.04), skf=2), lambda: dam3(0.0115)),
    ("3d_quintic", lambda: changed(dam3(0.04), skf=3), lambda: dam3(0.0115)),
    ("beam_quintic", lambda: changed(beam(1e-3), skf=3), lambda: beam(2.5e-4)),
    ("two_fluids", two_fluid_dam_break, lambda: dam2(0.006)),
    ("gate", lambda: gate(0.0025), lambda: gate(8e-4)),
    ("gate_no_stress", lambda: gate(0.0025, **NO_STRESS), lambda: gate(8e-4, **NO_STRESS)),
    ("gate_skip_gravity", lambda: gate(0.0025, **SKIP), lambda: gate(8e-4, **SKIP)),
    ("block_in_water_3d", fsi, lambda: dam3(0.0115)),
    ("2d_full_buffer", lambda: wide_cells(dam2(0.03), 4.0), lambda: dam2(0.006)),
    ("3d_full_buffer", lambda: wide_cells(dam3(0.04), 4.0), lambda: dam3(0.0115)),
])
def test_small_system_bits(gpu, name, small, filler):
    a = small()
    b = like(filler(), a)
    steps = 4
    fields = ("X", "V", "RHO", "E", "P", "NNEIGH") + (("SHEAR",) if np.any(np.abs(a.type) > 100) else ())
    with GpuSolver(a) as s:
        s.advance(steps)
        want = {f: s.field(f) for f in fields}
    with GpuBatch(a.params, 2, a.n_real + b.n_real, a.n_wall + b.n_wall + 1) as g:
        g.add(b)
        k = g.add(a)
        g.advance(steps)
        for f in want:
            assert np.array_equal(g.field(k, f), want[f]), f
