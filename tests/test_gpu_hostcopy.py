"""Readbacks into pageable memory through the pinned ring: sizes around its chunks and its threads, from two threads at
once, after the ring was given back, and into pinned memory."""
import threading

import numpy as np
import pytest

from outbreaklab_b200 import _native as N, model as M

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _radar(m, nbytes):
    import ctypes as C
    h = C.c_void_p()
    N.check(N.lib().ob_radar_create(m.h, nbytes, 4, C.byref(h)))
    return h


# the ring takes copies of 16 MiB and more in chunks of 1 MiB, 8 threads with two chunks in flight each
@pytest.mark.parametrize("nbytes", [4, 2 * MIB, 16 * MIB - 4, 16 * MIB, 16 * MIB + 4, 17 * MIB + 12, 24 * MIB - 4, 37 * MIB + 1000])
def test_readback_sizes(native, nbytes):
    import torch
    m = M.RegionalModel().allocate(spec={"dx": 1000, "n": [8, 8, 16]})
    h = _radar(m, nbytes)
    try:
        a = np.random.default_rng(nbytes).integers(0, 256, nbytes, np.uint8)
        N.check(N.lib().ob_radar_write(h, a.ctypes.data, nbytes))
        out = np.full(nbytes + 8, 77, np.uint8)
        N.check(N.lib().ob_radar_read(h, out.ctypes.data + 4, nbytes))
        assert np.array_equal(out[4:-4], a) and (out[:4] == 77).all() and (out[-4:] == 77).all()
        pinned = torch.empty(nbytes, dtype=torch.uint8, pin_memory=True)
        N.check(N.lib().ob_radar_read(h, pinned.data_ptr(), nbytes))
        assert np.array_equal(pinned.numpy(), a)
    finally:
        N.lib().ob_radar_destroy(h)
        m.destroy()


def test_readbacks_from_threads(native):
    n = 20 * MIB
    models = [M.RegionalModel().allocate(spec={"dx": 1000, "n": [8, 8, 16]}) for _ in range(3)]
    radars = [_radar(m, n) for m in models]
    data = [np.random.default_rng(i).integers(0, 256, n, np.uint8) for i in range(3)]
    for h, a in zip(radars, data):
        N.check(N.lib().ob_radar_write(h, a.ctypes.data, n))
    bad = []

    def loop(i):
        for _ in range(10):
            out = np.empty(n, np.uint8)
            rc = N.lib().ob_radar_read(radars[i], out.ctypes.data, n)
            if rc != N.OB_OK or not np.array_equal(out, data[i]):
                bad.append((i, rc))
    th = [threading.Thread(target=loop, args=(i,)) for i in range(3)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for h in radars:
        N.lib().ob_radar_destroy(h)
    for m in models:
        m.destroy()
    assert not bad
