"""The fp32 solve's 64 x 64 tiles, which grids of at most 98 wide tiles take, against its wide tiles, bit for bit: every output
of a transform is one chain of fused multiply-adds in ascending order whatever the tile. Without density at the level faces
the levels do not see each other, so a level of a tall column (many tiles: the wide ones) has the bits that it has in a short
one (few: the small ones)."""
import numpy as np
import pytest

from outbreaklab_b200 import model as M

pytestmark = pytest.mark.gpu


def _tiles(n, rows):
    t = 96 if -(-n // 96) * 96 < -(-n // 128) * 128 else 128
    return -(-n // t) * -(-rows // 128)


# widths around 64, 96 and 128, single columns of a tile and sums that end inside a stage of 16
@pytest.mark.parametrize("nx,ny", [(63, 65), (64, 64), (65, 127), (97, 129), (130, 95), (128, 128), (3, 191), (200, 2), (33, 31)])
def test_small_tiles_are_the_wide_ones_bit_for_bit(native, nx, ny):
    few = 98
    short = max(2, min(128 * few // (nx * max(1, -(-ny // 96))), 128 * few // (ny * max(1, -(-nx // 96)))) // 2)
    tall = 2 + 128 * (few + 1) // min(nx, ny)
    short, tall = min(short, 200), min(tall, 4000)
    assert max(_tiles(nx, ny * short), _tiles(ny, nx * short)) <= few < min(_tiles(nx, ny * tall), _tiles(ny, nx * tall))
    rhs = np.random.default_rng(nx + ny).standard_normal((tall, ny, nx)).astype(np.float32)
    phi = []
    for nz in (short, tall):
        P = M.PoissonDirect(nx, ny, nz, 1000.0, 100.0, 0)
        try:
            P.set_density(np.ones(nz, np.float32), np.zeros(nz + 1, np.float32))
            phi.append(P.solve(rhs[:nz])[:short])
        finally:
            P.destroy()
    assert np.isfinite(phi[0]).all() and np.abs(phi[0]).max() > 0
    assert np.array_equal(phi[0].view(np.uint32), phi[1].view(np.uint32))
