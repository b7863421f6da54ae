"""Version-4 snapshots of a batch: with a removed system's walls still in
their slots (there the wall range is longer than the live walls), and with a
removed system's particles not yet dropped."""
import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuBatch
from tests.test_gpu_state import FIELDS, _flags
from tests.test_gpu_state_v4 import to_v4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pending", [False, True])
def test_version_4_batch_resumes_bitwise(gpu, pending):
    specs = cases.ensemble_specs(count=3, seed=9, n_lo=300, n_hi=2000)
    ms = [_flags(cases.ensemble_member(sp), 0, P.PREC_MIXED) for sp in specs]
    with GpuBatch(ms[0].params, 4, sum(m.n_real for m in ms) + 100, sum(m.n_wall for m in ms) + 100) as b:
        ids = [b.add(m) for m in ms]
        b.advance(5)
        b.remove(ids[0])
        if not pending:
            b.advance(3)
        blob = b.save_state()
        b.advance(6)
        want = {k: {f: b.field(k, f) for f in FIELDS} for k in ids[1:]}
    old = to_v4(blob, ms[0].params.dim)
    assert old != blob
    with GpuBatch.from_state(old) as r:
        assert sorted(r.slots()) == sorted(ids[1:])
        r.advance(6)
        for k in ids[1:]:
            for f in FIELDS:
                assert np.array_equal(r.field(k, f), want[k][f]), (k, f)
