"""The largest grid: a field's values are reached at unsigned 32-bit byte offsets, so a field of more than 4 GiB is refused
before anything else is tried (no device is needed to say so)."""
import ctypes as C

import pytest

from outbreaklab_b200 import _native as N


def _field_bytes(nx, ny, nz):
    return (nx + 32) // 32 * 32 * (ny + 1) * (nz + 1) * 4


@pytest.mark.parametrize("nx,ny,nz", [(8159, 8255, 15),          # just above 4 GiB: 4.31e9 bytes
                                      (4095, 511, 512),          # 2^32 bytes and one plane
                                      (65535, 65535, 40), (2000000000, 2000000000, 512)])
def test_field_past_32_bit_offsets_is_refused(nx, ny, nz):
    assert _field_bytes(nx, ny, nz) > 1 << 32
    h = C.c_void_p()
    g = N.ObGrid(nx, ny, nz, 1000.0)
    assert N.lib().ob_model_create(C.byref(g), C.byref(h)) == N.OB_ERR_INVALID
    assert b"4 GiB" in N.lib().ob_last_error() and not h.value
