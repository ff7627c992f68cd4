"""Hurricane mode's skip of absent species: hydrometeors placed where a reach of the winds and of the fall speed begins or
ends (brick corners, domain edges, single cells), stepped through a filter pass, against the oracle."""
import numpy as np
import pytest

import _hurricane_case as HC
from _parity import check_field
from outbreaklab_b200 import _native as N, hurricane as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2])
def test_sparse_hydrometeors(oracle_lib, native, seed):
    """Five steps (the 2-dx filter runs before the fourth step's successor); the scalars within the five-step envelope
    of the FP64 oracle, and every cell that the oracle leaves empty of a species empty on the GPU too."""
    c, surf, vort = HC.case()
    g, B, _, _, _ = H.setup(c, surf, vort, lat=HC.LAT)
    f, _, _, _ = HC.oracle_setup(c, surf, vort, 4)
    d, _, _, _ = HC.oracle_setup(c, surf, vort, 8)
    r = np.random.default_rng(seed)
    nz, ny, nx = c.nz, c.ny, c.nx
    q1 = g.get_field(N.FIELD_Q1).reshape(nz, ny, nx, 4).copy()
    q2 = np.zeros((nz, ny, nx, 4), np.float32)
    for k in (0, 1, nz // 2, nz - 1):
        for j in (0, 3, 4, ny - 1):
            for i in (0, 31, 32, nx - 1):
                s = r.integers(5)
                (q1[k, j, i, 1:4] if s < 3 else q2[k, j, i, 0:2])[s if s < 3 else s - 3] = 10.0 ** r.uniform(-6, -3)
    for m in (f, d):
        m.set(oracle_lib.FIELD_Q1, q1.reshape(-1))
        m.set(oracle_lib.FIELD_Q2, q2.reshape(-1))
    g.set_field(N.FIELD_Q1, q1)
    g.set_field(N.FIELD_Q2, q2)
    try:
        for m in (g, f, d):
            m.step(c.dt, 5)
        g.sync()
        bad = []
        for fld in (N.FIELD_Q1, N.FIELD_Q2):
            a, o32, o64 = g.get_field(fld), f.get(fld), d.get(fld, f64=True)
            _, b = check_field(fld, a, o32, o64, 4, tol=1e-4, envelope=4.0)
            bad += b
            both = (np.asarray(o32).reshape(-1) == 0) & (np.asarray(o64).reshape(-1) == 0)
            assert not (a[both] > 1e-12).any()
        assert not bad, bad
        assert g.nan_count == 0
    finally:
        g.destroy()
