"""ob_poisson_solve_static in a process of its own, where no plan has ever been created: the hosts it serves create none.
Columns on both sides of 96 levels, from which on the tridiagonal needs more shared memory than a launch has by default."""
import os
import subprocess
import sys

import numpy as np
import pytest

from outbreaklab_b200 import workloads as W

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(70, 52, 40), (129, 33, 17), (40, 36, 130), (12, 10, 440), (11, 13, 441)]

CHILD = """
import ctypes as C, sys
import numpy as np, torch
from outbreaklab_b200 import _native as N
f = np.load(sys.argv[1])
out = {}
for k in range(int(f["n"])):
    nx, ny, nz = (int(v) for v in f["shape%d" % k])
    rc, rw, rhs = (torch.from_numpy(f[a + str(k)]).cuda() for a in ("rc", "rw", "rhs"))
    phi = torch.full_like(rhs, float("nan"))
    s = torch.cuda.current_stream()
    torch.cuda.synchronize()
    N.check(N.lib().ob_poisson_solve_static(nx, ny, nz, 1000.0, 20000.0 / nz, C.c_void_p(rc.data_ptr()), C.c_void_p(rw.data_ptr()),
                                            C.c_void_p(rhs.data_ptr()), C.c_void_p(phi.data_ptr()), C.c_void_p(s.cuda_stream)))
    torch.cuda.synchronize()
    out["phi%d" % k] = phi.cpu().numpy()
np.savez(sys.argv[2], **out)
"""


def test_without_any_plan(oracle_lib, native, tmp_path):
    """The bound is the handle-based solve's: 1e-5, or twice the FP32 oracle's own error."""
    f = {"n": len(SHAPES)}
    for k, (nx, ny, nz) in enumerate(SHAPES):
        dz = 20000.0 / nz
        f["shape%d" % k] = (nx, ny, nz)
        f["rc%d" % k] = (1.15 * np.exp(-(np.arange(nz) + 0.5) * dz / 9000.0)).astype(np.float32)
        f["rw%d" % k] = (1.15 * np.exp(-np.arange(nz + 1) * dz / 9000.0)).astype(np.float32)
        f["rhs%d" % k] = W.gaussian_rhs(nx, ny, nz, 1000.0, corr_len=5000.0, seed=k).astype(np.float32)
    np.savez(tmp_path / "in.npz", **f)
    r = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "in.npz"), str(tmp_path / "out.npz")], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = np.load(tmp_path / "out.npz")
    for k, shape in enumerate(SHAPES):
        rhs, rc, rw, dz = f["rhs%d" % k], f["rc%d" % k], f["rw%d" % k], 20000.0 / shape[2]
        ref = oracle_lib.poisson_solve(rhs.astype(np.float64), 1000.0, dz, rc.astype(np.float64), rw.astype(np.float64), 8)
        e32 = np.abs(oracle_lib.poisson_solve(rhs, 1000.0, dz, rc, rw, 4) - ref).max() / np.abs(ref).max()
        err = np.abs(got["phi%d" % k].reshape(ref.shape) - ref).max() / np.abs(ref).max()
        assert err <= max(1e-5, 2 * e32), (shape, err, e32)
