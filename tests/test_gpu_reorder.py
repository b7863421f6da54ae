"""The reorder by cell counts against the one by sorted keys: a State == -1
particle (no neighbour of any other) makes the search sort, and leaves the
order and so the bits of all others as they are."""
import dataclasses

import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300.solver import GpuSolver
from tests.helpers import perturb

pytestmark = pytest.mark.gpu


def with_inactive(c):
    """The case with one more real particle, State == -1, in place of the first."""
    at = np.concatenate([np.arange(c.n_real), [0], np.arange(c.n_real, c.n)])
    new = {k: getattr(c, k)[at] for k in ("x", "v", "mass", "rho", "p", "e", "c", "h", "type", "state", "boundary")}
    new["state"] = new["state"].copy()
    new["state"][c.n_real] = -1
    return dataclasses.replace(c, n_real=c.n_real + 1, **new)


# few cells (one block scans them), more than one tile of cells, a wide grid of mostly empty cells
@pytest.mark.parametrize("name,make", [
    ("2d_small", lambda: cases.dam_break_2d(dx=0.1)),
    ("2d", lambda: cases.dam_break_2d(dx=0.01)),
    ("3d", lambda: cases.dam_break_3d(dx=0.03)),
    ("2d_wide", lambda: cases.dam_break_2d(dx=0.02, tank_w=60.0, tank_h=12.0)),
])
def test_counted_equals_sorted(gpu, name, make):
    c = perturb(make(), seed=5, v_amp=0.5, x_frac=0.3)
    with GpuSolver(c) as a, GpuSolver(with_inactive(c)) as b:
        for s in (a, b):
            s.advance(5)
            s.nnps()
        n = c.n_real
        for f in ("X", "V", "RHO", "E", "NNEIGH"):
            assert np.array_equal(a.field(f)[:n], b.field(f)[:n]), f
        ao, al = a.neighbor_lists()
        bo, bl = b.neighbor_lists()
        # the exports list neighbours in the particles' order; walls come one index later
        bl = np.where(bl > n, bl - 1, bl)
        assert np.array_equal(ao, bo[: n + 1]) and np.array_equal(al, bl[: len(al)])


def test_resumed_state_keeps_inactive(gpu):
    c = with_inactive(perturb(cases.dam_break_2d(dx=0.05), seed=6, v_amp=0.5, x_frac=0.3))
    with GpuSolver(c) as a:
        a.advance(3)
        with GpuSolver.from_state(a.save_state()) as b:
            a.advance(4)
            b.advance(4)
            for f in ("X", "V", "RHO", "E"):
                assert np.array_equal(a.field(f), b.field(f)), f
