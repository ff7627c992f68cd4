"""The fp32 pressure solve (precision 0) at the edges of its transforms' tiles, of its tridiagonal's batches and at
columns past the shared-memory tridiagonal, from pointers that are not 16-byte aligned, against the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

from outbreaklab_b200 import _native as N, model as M, workloads as W

pytestmark = pytest.mark.gpu


# widths around 96 and 128 (the tiles that span a DST matrix), 16 (the stages of the transforms' sums and the
# tridiagonal's batches of levels) and single columns of a tile; 441 levels leave the shared-memory tridiagonal
@pytest.mark.parametrize("shape", [(96, 128, 16), (97, 129, 17), (95, 127, 15), (193, 33, 9), (31, 257, 5), (2, 3, 2), (160, 130, 33),
                                   (12, 10, 440), (11, 13, 441)])
def test_fp32_solve_at_tile_edges(oracle_lib, native, shape):
    import torch
    nx, ny, nz = shape
    dx, dz = 1000.0, 20000.0 / nz
    rc = (1.15 * np.exp(-(np.arange(nz) + 0.5) * dz / 9000.0)).astype(np.float32)
    rw = (1.15 * np.exp(-np.arange(nz + 1) * dz / 9000.0)).astype(np.float32)
    rhs = np.random.default_rng(nx + ny).standard_normal((nz, ny, nx)).astype(np.float32)
    ref = oracle_lib.poisson_solve(rhs.astype(np.float64), dx, dz, rc.astype(np.float64), rw.astype(np.float64), 8)
    f32 = oracle_lib.poisson_solve(rhs, dx, dz, rc, rw, 4)
    e32 = np.abs(f32 - ref).max() / np.abs(ref).max()
    P = M.PoissonDirect(nx, ny, nz, dx, dz, 0)
    try:
        P.set_density(rc, rw)
        phi = P.solve(rhs)
        # the same on device pointers one float past a 16-byte boundary, with a value behind the result left alone
        buf, out = torch.zeros(rhs.size + 1, device="cuda"), torch.full((rhs.size + 2,), 7.0, device="cuda")
        buf[1:] = torch.from_numpy(rhs.reshape(-1)).cuda()
        torch.cuda.synchronize()
        N.check(N.lib().ob_poisson_solve_device(P.h, C.c_void_p(buf.data_ptr() + 4), C.c_void_p(out.data_ptr() + 4), None))
        torch.cuda.synchronize()
    finally:
        P.destroy()
    err = np.abs(phi.reshape(ref.shape) - ref).max() / np.abs(ref).max()
    assert err <= max(1e-5, 2 * e32), (err, e32)
    got = out.cpu().numpy()
    assert got[0] == 7.0 and got[-1] == 7.0
    assert np.array_equal(got[1:-1].view(np.uint32), phi.reshape(-1).view(np.uint32))
