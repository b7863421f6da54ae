"""The neighbour sets where the FP32 candidate filter has no finite upper
bound: a reach whose square is beyond FP32, and a domain so sparse that every
candidate takes the exact test.  Both against the O(N^2) enumeration, and the
rates against the oracle at the tolerance of the parity tests."""
import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuSolver
from oracle.oracle import Oracle
from tests.conftest import rel_l2
from tests.helpers import brute_force_sets, csr_sets, perturb

pytestmark = pytest.mark.gpu


def scaled(dim, s):
    """A dam break with every length s times as long (s a power of two: no
    rounding, so ties and sets are those of the unscaled system)."""
    c = perturb(cases.dam_break_2d(dx=0.05) if dim == 2 else cases.dam_break_3d(dx=0.06), seed=72, v_amp=0.3,
                x_frac=0.1)
    c.x, c.h, c.mass = c.x * s, c.h * s, c.mass * s ** dim
    c.params = c.params.copy()
    c.params.wall_r0 *= s
    c.params.contact_delta *= s
    c.params.dt *= s
    return c


# reach 0.12 s: beyond 1.8e19 its square is beyond FP32; wide: the domain box
# spans 1.5e6 reaches or more, where the guard band is the whole range
@pytest.mark.parametrize("dim,scale,wide", [
    (2, 2.0 ** 10, True), (2, 2.0 ** 20, True), (3, 2.0 ** 20, True),
    (2, 2.0 ** 66, False), (2, 2.0 ** 70, False), (3, 2.0 ** 70, False),
])
@pytest.mark.parametrize("lanes", [1, 4])
def test_sets_without_an_fp32_bound(gpu, dim, scale, wide, lanes):
    c = scaled(dim, scale)
    if wide:
        for a in range(dim):
            c.params.domain_lo[a], c.params.domain_hi[a] = -1e5 * scale, 1e5 * scale
    sets, ties = brute_force_sets(c)
    assert not ties
    sets = sets[: c.n_real]
    o = Oracle(c, covering_band=True)
    o.rates()
    with GpuSolver(c) as s:
        s.set_option(P.OPT_LANES, lanes)
        s.nnps()
        got = s.rates()
        assert csr_sets(*s.neighbor_lists()) == sets
        assert np.array_equal(s.field("NNEIGH")[: c.n_real], [len(k) for k in sets])
    for a, f in zip(got, ("DVDT", "DRHODT", "DEDT")):
        assert rel_l2(a, o.field(f)[: c.n_real]) <= 1e-10, f
