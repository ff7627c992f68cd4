"""The right-hand side's split into bf16 rows: wide and single loads give the same solve."""
import ctypes as C

import pytest
import torch

from outbreaklab_b200 import _native as N, model as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [32, 97, 100, 132, 260])
@pytest.mark.parametrize("precision", [1, 2, 5])
def test_split_does_not_depend_on_the_alignment(native, nx, precision):
    """A field at a 16-byte boundary and the same field 4 bytes past one: equal bits out (a split rounds each value alone)."""
    ny, nz = 37, 16
    P = M.PoissonDirect(nx, ny, nz, 1000.0, 20000.0 / nz, precision)
    n = nx * ny * nz
    g = torch.Generator(device="cuda").manual_seed(nx)
    r = torch.randn(n, device="cuda", generator=g) * 1e-4
    out = []
    for shift in (0, 1, 2):
        buf = torch.zeros(n + 4, device="cuda")
        buf[shift:shift + n] = r
        f = torch.empty_like(r)
        torch.cuda.synchronize()
        N.check(N.lib().ob_poisson_solve_device(P.h, C.c_void_p(buf[shift:].data_ptr()), C.c_void_p(f.data_ptr()), None))
        torch.cuda.synchronize()
        out.append(f)
    P.destroy()
    assert out[0].abs().max() > 0
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
