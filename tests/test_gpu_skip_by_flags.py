"""The skip of absent species against the same step without it, cell by cell. A model whose empty cells hold -1e-38 of every
species has every flag set; its advection clips that to zero, so a step must leave both with the same values: a cell that a flag leaves
out is empty here and not there. (A trace can break a tie of the rounding, which moves a value by an ulp or two: eight are
allowed, and 1e-30 for what the 2-dx filter makes of the traces.)
Hydrometeors sit where a reach of the winds and of the fall speed begins or ends: brick corners, domain edges, single cells."""
import numpy as np
import pytest

import _hurricane_case as HC
from outbreaklab_b200 import _native as N, hurricane as H, model as M, workloads as W

pytestmark = pytest.mark.gpu

TRACE = -1e-38


def _pair(kind):
    out = []
    for _ in range(2):
        if kind == "hurricane":
            c, surf, vort = HC.case()
            out.append(H.setup(c, surf, vort, lat=HC.LAT)[0])
        else:
            c = W.StormCase("skip", 75, 43, 16, 1500.0, 9.0, 1, scheme=1 if kind == "thompson" else 0)
            out.append(M.setup_case(c)[0])
    return c, out


@pytest.mark.parametrize("kind,seed", [("hurricane", 1), ("hurricane", 2), ("lin", 3), ("thompson", 4)])
def test_flags_leave_nothing_out(native, kind, seed):
    c, (a, b) = _pair(kind)
    r = np.random.default_rng(seed)
    nz, ny, nx = c.nz, c.ny, c.nx
    q1 = a.get_field(N.FIELD_Q1).reshape(nz, ny, nx, 4).copy()
    q2 = np.zeros((nz, ny, nx, 4), np.float32)
    for k in (0, 1, nz // 2, nz - 1):
        for j in (0, 3, 4, ny - 1):
            for i in (0, 31, 32, nx - 1):
                s = r.integers(7)   # qc, qi, qr, qs, qg, Nr, spare
                (q1 if s < 3 else q2)[k, j, i, s + 1 if s < 3 else s - 3] = 10.0 ** r.uniform(-8, -3)
                if s == 2 and kind == "thompson":
                    q2[k, j, i, 2] = 1e3
    fields = {N.FIELD_Q1: q1, N.FIELD_Q2: q2}
    try:
        for f, q in fields.items():
            a.set_field(f, q)
        for step in range(6):   # the filter runs among them
            for f, q in fields.items():
                b.set_field(f, np.where(q == 0, np.float32(TRACE), q))
            b.set_field(N.FIELD_V, a.get_field(N.FIELD_V))
            for m in (a, b):
                m.step(c.dt, 1)
                m.sync()
            fields = {f: a.get_field(f).reshape(q.shape) for f, q in fields.items()}
            for f, q in fields.items():
                full = b.get_field(f).reshape(q.shape)
                bad = np.abs(q - full) > 8 * np.spacing(np.maximum(q, full)) + np.float32(1e-30)
                assert not bad.any(), (step, f, np.argwhere(bad)[:4], q[bad][:4], full[bad][:4])
            assert np.allclose(a.get_field(N.FIELD_V), b.get_field(N.FIELD_V), rtol=1e-6, atol=1e-6), step
        assert (fields[N.FIELD_Q2][..., :2] > 0).any() and (fields[N.FIELD_Q1][..., 1:] > 0).any()
    finally:
        a.destroy()
        b.destroy()
