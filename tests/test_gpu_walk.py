"""The neighbour walk where its candidate buffer fills: cells far larger than
2h, so that a warp's rows hold several buffers of candidates (FP64 pass B then
walks the approaching and the receding pairs in two parts), and systems of a
few particles.  Tolerances are those of the parity tests."""
import numpy as np
import pytest

from tests.helpers import brute_force_sets, csr_sets, perturb
from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuBatch, GpuSolver
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def with_cells(c, factor, precision=P.PREC_FP64):
    prm = c.params.copy()
    prm.cell_size = factor * 2.0 * float(c.h.max())
    prm.precision = precision
    return prm


def make(dim):
    if dim == 2:
        return perturb(cases.dam_break_2d(dx=0.05), seed=3, v_amp=0.3, x_frac=0.1)
    return perturb(cases.dam_break_3d(dx=0.05), seed=3, v_amp=0.3, x_frac=0.1)


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# cells of 2h; of 3 x 2h (a buffer or two); the whole domain in a few cells (many buffers)
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("factor", [1.0, 3.0, 40.0])
@pytest.mark.parametrize("precision,lanes,tol", [(P.PREC_FP64, 1, 1e-10), (P.PREC_FP64, 4, 1e-10),
                                                 (P.PREC_FP64, 32, 1e-10), (P.PREC_DF64, 1, 1e-10),
                                                 (P.PREC_MIXED, 1, 1e-4)])
def test_rates_any_cell_size(gpu, dim, factor, precision, lanes, tol):
    if precision == P.PREC_MIXED and factor > 3.0:
        pytest.skip("FP32 positions are relative to the cell: their accuracy goes with its size")
    c = make(dim)
    o = Oracle(c, covering_band=True)
    o.bggs()
    o.rates()
    with GpuSolver(c, params=with_cells(c, factor, precision)) as s:
        s.set_option(P.OPT_LANES, lanes)
        s.nnps()
        got = s.rates()
        off, lst = s.neighbor_lists()
    sets, ties = brute_force_sets(c)
    assert not ties and csr_sets(off, lst) == sets[: c.n_real]
    for a, f in zip(got, ("DVDT", "DRHODT", "DEDT")):
        assert rel(a, o.field(f)[: c.n_real]) <= tol, f


@pytest.mark.parametrize("factor", [1.0, 6.0])
@pytest.mark.parametrize("lanes", [1, 8])
def test_batch_equals_alone_any_cell_size(gpu, factor, lanes):
    """The pair order is the target's own, whatever its warp holds."""
    a, b = make(3), perturb(cases.dam_break_3d(dx=0.06), seed=9, v_amp=0.3, x_frac=0.1)
    with GpuSolver(b, params=with_cells(b, factor)) as s:
        s.set_option(P.OPT_LANES, lanes)
        s.advance(4)
        want = {f: s.field(f) for f in ("X", "V", "RHO", "E")}
    with GpuBatch(a.params, 2, a.n_real + b.n_real, a.n_wall + b.n_wall) as g:
        g.set_option(P.OPT_LANES, lanes)
        g.add(a, params=with_cells(a, factor))
        k = g.add(b, params=with_cells(b, factor))
        g.advance(4)
        for f in want:
            assert np.array_equal(g.field(k, f), want[f]), f
