"""The maps of a domain of many columns, whose levels fewer warps share, against those of a narrow one that holds the same rows,
bit for bit: a column's sums run in the same order however many warps work on it."""
import numpy as np
import pytest

from outbreaklab_b200 import _native as N, model as M, workloads as W

pytestmark = pytest.mark.gpu

ROWS = 41


def _model(nx, ny, nz, scheme):
    return M.setup_case(W.StormCase("maps", nx, ny, nz, 1000.0, 6.0, 1, scheme=scheme, bubbles=[], noise=0.0))[0]


# row blocks of 32 columns: 2560 (eight warps to a column), 2561 and more (two; rows left over in the last block)
@pytest.mark.parametrize("nx,ny,nz,scheme", [(20, 2560, 16, 0), (20, 2561, 16, 1), (61, 1402, 40, 0), (33, 1300, 28, 1), (17, 2603, 16, 0),
                                             (90, 1001, 9, 1), (64, 1501, 100, 0)])
def test_same_columns_same_maps(native, nx, ny, nz, scheme):
    r = np.random.default_rng(nx + ny)
    wide, narrow = _model(nx, ny, nz, scheme), _model(nx, ROWS, nz, scheme)
    try:
        at = ny - ROWS   # the wide one's last rows
        for f, face in ((N.FIELD_V, 1), (N.FIELD_Q1, 0), (N.FIELD_Q2, 0)):
            a = wide.get_field(f).reshape(nz + face, ny + face, nx + face, 4).copy()
            if f == N.FIELD_V:
                a[..., :3] += r.uniform(-20, 20, a[..., :3].shape).astype(np.float32)
                a[..., 3] += r.uniform(-2, 2, a.shape[:3]).astype(np.float32)
            else:
                some = r.random(a.shape[:3]) < 0.03
                some &= (r.random((1,) + a.shape[1:3]) < 0.4) & (np.arange(nz)[:, None, None] % 5 != 1)
                for c in range(1 if f == N.FIELD_Q1 else 0, 4 if f == N.FIELD_Q1 else 3):
                    a[..., c] = np.where(some, 10.0 ** r.uniform(-7, -2, a.shape[:3]), 0.0)
            wide.set_field(f, a)
            narrow.set_field(f, a[:, at:at + ROWS + face])
        got, want = (np.stack([m[k] for k in ("m0", "m1", "m2", "m3")]) for m in (wide.request_maps(), narrow.request_maps()))
        got = got[:, at:]
        inner = slice(1, ROWS)   # the narrow one's first row looks past its edge
        assert np.isfinite(want).all() and (want[0, ..., 0] > 0).any() and (want[1, ..., 1] > 0).any()
        assert np.array_equal(got[:, inner].view(np.uint32), want[:, inner].view(np.uint32))
    finally:
        wide.destroy()
        narrow.destroy()
