"""The counted reorder on both sides of the limits of its one-block form
(16,384 particles; 11,264 cell counts, one of them behind the last cell)
against the order of the sorted keys, which a State == -1 particle asks for."""
import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300.solver import GpuSolver
from tests.helpers import perturb
from tests.test_gpu_coop import few
from tests.test_gpu_reorder import with_inactive

pytestmark = pytest.mark.gpu


def in_grid(c, nx, ny, cs):
    """The case in a grid of nx x ny cells of side cs."""
    c.params = c.params.copy()
    c.params.cell_size = cs
    for a, n in enumerate((nx, ny)):
        c.params.domain_lo[a] = -0.9
        c.params.domain_hi[a] = -0.9 + (n - 0.5) * cs
    return c


def dam(dx):
    return perturb(cases.dam_break_2d(dx=dx), seed=15, v_amp=0.5, x_frac=0.2)


@pytest.mark.parametrize("name,make", [
    ("16384_particles", lambda: in_grid(few(dam(0.0109), 16384), 110, 100, 0.06)),
    ("16385_particles", lambda: in_grid(few(dam(0.0109), 16385), 110, 100, 0.06)),
    ("11263_cells", lambda: in_grid(dam(0.1), 1609, 7, 0.7)),
    ("11264_cells", lambda: in_grid(dam(0.1), 1024, 11, 0.7)),
])
def test_counted_equals_sorted_at_the_limits(gpu, name, make):
    c = make()
    assert name not in ("16384_particles", "16385_particles") or c.n_real == int(name[:5])
    with GpuSolver(c) as a, GpuSolver(with_inactive(c)) as b:
        for s in (a, b):
            s.advance(4)
            s.nnps()
        n = c.n_real
        for f in ("X", "V", "RHO", "E", "NNEIGH"):
            assert np.array_equal(a.field(f)[:n], b.field(f)[:n]), f
