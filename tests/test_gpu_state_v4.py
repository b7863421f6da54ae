"""Snapshots of version 4 (the FP32 mirrors in arrays of their own) load and
continue bit for bit like one of the present version."""
import struct

import numpy as np
import pytest

from mysph_gb300 import cases
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuSolver
from tests.helpers import perturb
from tests.test_gpu_state import CASES, FIELDS, _flags

pytestmark = pytest.mark.gpu


def to_v4(blob, dim):
    """The same state as version 4 wrote it."""
    b = bytearray(blob)
    hb, pb, ib = struct.unpack_from("<III", b, 12)
    assert struct.unpack_from("<I", b, 8)[0] == 5
    struct.pack_into("<I", b, 8, 4)
    _, max_inst, solid, mirrors, _, _ = struct.unpack_from("<6i", b, hb - 120)
    wall_end, n_real, wall_off = (struct.unpack_from("<q", b, hb - o)[0] for o in (80, 56, 40))
    if not mirrors:
        return bytes(b)
    n, d2 = n_real + wall_end - wall_off, dim * dim
    row, old_row = (16, 12) if dim == 3 else (8, 4)
    pre = hb + (ib + pb + 32) * max_inst + n * (236 + 8 * d2 + (24 * d2 + 32 if solid else 0))
    f = np.frombuffer(bytes(b[pre:]), np.float32)
    pv, f = f[:8 * n].reshape(n, 2, 4).copy(), f[8 * n:]
    ef, f = f[:4 * n].reshape(n, 4).copy(), f[4 * n:]
    rows = []
    for _ in range(2 if solid else 1):
        r, f = f[:row * n].reshape(n, row), f[row * n:]
        rows.append(r)
    m_rho, rho = pv[:, 1, 3].copy(), ef[:, 2].copy()
    pv[:, 1, 3], ef[:, 2] = rho, m_rho
    pf = np.zeros((n, 4), np.float32)
    pf[:, 0], pf[:, 2] = rows[0][:, d2 + 1], rows[0][:, d2 + 2]
    parts = [pv[:, 0], pv[:, 1], ef, pf] + [np.pad(r[:, :d2], ((0, 0), (0, old_row - d2))) for r in rows] + [f]
    tail = b"".join(np.ascontiguousarray(p).tobytes() for p in parts)
    out = b[:pre] + tail
    struct.pack_into("<q", out, hb - 8, len(out) - hb)
    return bytes(out)


@pytest.mark.parametrize("name", ["dam2d_fp64", "dam2d_mixed", "gate_mixed", "dam3d_mixed"])
def test_version_4_resumes_bitwise(gpu, name):
    if name == "dam3d_mixed":
        c = _flags(perturb(cases.dam_break_3d(dx=0.05), seed=45, v_amp=0.3, x_frac=0.2), 0, P.PREC_MIXED)
    else:
        c = CASES[name]()
    with GpuSolver(c) as s:
        s.advance(7)
        blob = s.save_state()
        s.advance(5)
        want = {k: s.field(k) for k in FIELDS}
    old = to_v4(blob, c.params.dim)
    assert old != blob
    with GpuSolver.from_state(old) as r:
        r.advance(5)
        for k in FIELDS:
            assert np.array_equal(r.field(k), want[k]), k
