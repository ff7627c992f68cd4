"""The tensor-core solve at row lengths that are not whole 16 bytes (T2's padded rows), against the oracle."""
import numpy as np
import pytest

from outbreaklab_b200 import model as M, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(97, 61, 40), (130, 75, 16), (35, 90, 80)])
def test_solve_at_odd_widths(oracle_lib, native, shape):
    """T2's padded rows: widths that are not multiples of 4, in every refined precision."""
    nx, ny, nz = shape
    dx, dz = 1000.0, 20000.0 / nz
    rc = (1.15 * np.exp(-(np.arange(nz) + 0.5) * dz / 9000.0)).astype(np.float32)
    rw = (1.15 * np.exp(-np.arange(nz + 1) * dz / 9000.0)).astype(np.float32)
    rhs = W.gaussian_rhs(nx, ny, nz, dx, seed=nx).astype(np.float32)
    ref = oracle_lib.poisson_solve(rhs.astype(np.float64), dx, dz, rc.astype(np.float64), rw.astype(np.float64), 8)
    f32 = oracle_lib.poisson_solve(rhs, dx, dz, rc, rw, 4)
    e32 = np.abs(f32 - ref).max() / np.abs(ref).max()
    for precision in (2, 4, 5):
        P = M.PoissonDirect(nx, ny, nz, dx, dz, precision)
        P.set_density(rc, rw)
        phi = P.solve(rhs)
        P.destroy()
        err = np.abs(phi - ref).max() / np.abs(ref).max()
        assert err <= max(1e-5, 2 * e32), (precision, err, e32)
