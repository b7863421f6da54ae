"""The exact walk in cells a little and much wider than the reach, where tiles
without a neighbour are dropped, the buffer fills in some warps and not in
others, and pass B goes on with the approaching pairs alone: the rates against
the oracle at the parity tests' tolerance, and the bits of a system alone and
in a batch, whose warps hold other targets."""
import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuBatch, GpuSolver
from oracle.oracle import Oracle
from tests.conftest import rel_l2
from tests.helpers import perturb
from tests.test_gpu_walk import with_cells

pytestmark = pytest.mark.gpu


def dam(dim, seed):
    c = cases.dam_break_2d(dx=0.03) if dim == 2 else cases.dam_break_3d(dx=0.04)
    return perturb(c, seed=seed, v_amp=0.3, x_frac=0.1)


@pytest.mark.parametrize("dim,factor", [(2, 2.0), (2, 5.0), (2, 12.0), (3, 1.3), (3, 2.0), (3, 4.0)])
@pytest.mark.parametrize("precision,lanes", [(P.PREC_FP64, 1), (P.PREC_FP64, 8), (P.PREC_DF64, 1)])
def test_rates_and_bits(gpu, dim, factor, precision, lanes):
    a, b = dam(dim, 21), dam(dim, 22)
    a.x = np.ascontiguousarray(a.x + 0.37 * a.meta["dx"])   # other cells than b's
    o = Oracle(b, covering_band=True)
    o.rates()
    with GpuSolver(b, params=with_cells(b, factor, precision)) as s:
        s.set_option(P.OPT_LANES, lanes)
        s.nnps()
        for got, f in zip(s.rates(), ("DVDT", "DRHODT", "DEDT")):
            assert rel_l2(got, o.field(f)[: b.n_real]) <= 1e-10, f
        s.advance(3)
        want = {f: s.field(f) for f in ("X", "V", "RHO", "E")}
    with GpuBatch(with_cells(a, factor, precision), 2, a.n_real + b.n_real, a.n_wall + b.n_wall) as g:
        g.set_option(P.OPT_LANES, lanes)
        g.add(few_of(a), params=with_cells(a, factor, precision))
        k = g.add(b, params=with_cells(b, factor, precision))
        g.advance(3)
        for f in want:
            assert np.array_equal(g.field(k, f), want[f]), f


def few_of(c):
    """All but seven of the case's particles: the other system's targets fall on other lanes."""
    return c.subset_real(np.arange(c.n_real) < c.n_real - 7)
