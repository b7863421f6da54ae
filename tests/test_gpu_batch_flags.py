"""What a system asks of a batch goes with it: after a system with a
State == -1 particle is removed, the steps of the others issue the launches of
a batch that never held it."""
import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuBatch, GpuSolver
from tests.helpers import perturb, two_fluid_dam_break
from tests.test_gpu_reorder import with_inactive

pytestmark = pytest.mark.gpu


def steps_launches(b, n=3):
    l0 = b.launch_count()
    b.advance(n)
    return b.launch_count() - l0


@pytest.mark.parametrize("resumed", [False, True])
def test_removed_system_takes_its_search_with_it(gpu, resumed):
    c = perturb(cases.dam_break_2d(dx=0.05), seed=17, v_amp=0.3, x_frac=0.2)
    counts = []
    for second in (c, with_inactive(c)):
        with GpuBatch(c.params, 3, 3 * c.n_real + 10, 3 * c.n_wall) as b:
            b.set_option(P.OPT_GRAPHS, 0)
            b.add(c)
            k = b.add(second)
            b.advance(2)
            held = steps_launches(b)
            if resumed:
                blob = b.save_state()
                b.close()
                b = GpuBatch.from_state(blob)
                b.set_option(P.OPT_GRAPHS, 0)
            b.remove(k)
            b.advance(1)      # drops the removed particles
            counts.append((held, steps_launches(b)))
            b.close()
    assert counts[1][0] > counts[0][0]
    assert counts[1][1] == counts[0][1]


def test_systems_keep_their_types(gpu):
    """A system of two Types beside one of a single Type: its pairs across the
    interface stay, after the other is removed and in a resumed batch."""
    two = two_fluid_dam_break()
    one = cases.dam_break_2d(dx=0.05)
    prm = one.params.copy()
    prm.flags = two.params.flags
    with GpuSolver(two) as s:
        s.advance(6)
        want = {f: s.field(f) for f in ("X", "V", "RHO")}
    with GpuBatch(two.params, 3, one.n_real + two.n_real, one.n_wall + two.n_wall) as b:
        a = b.add(one, params=prm)
        k = b.add(two)
        b.advance(2)
        with GpuBatch.from_state(b.save_state()) as r:
            r.remove(a)
            r.advance(4)
            for f in want:
                assert np.array_equal(r.field(k, f), want[f]), f
        b.remove(a)
        b.advance(4)
        for f in want:
            assert np.array_equal(b.field(k, f), want[f]), f
