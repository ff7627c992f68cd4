"""The radar's scan for gates that can echo, and its PhiDP chain, where they can go wrong.

A tornado far outside the domain touches no gate, but its presence sends every gate through the whole computation: the
volume must not change by a byte. PhiDP of any number of radials and gates must be the oracle's sum of the same KDP."""
import ctypes as C

import numpy as np
import pytest

from outbreaklab_b200 import _native as N, model as M, radar as RD, workloads as W

pytestmark = pytest.mark.gpu

FAR = [{"x": 1e7, "y": 1e7, "R": 150.0, "v": 60.0, "debrisTop": 1500.0, "debrisDbz": 55.0, "debris": 1.0}]


def _sparse(nx, ny, nz, seed, thompson):
    """Single rainy, snowy and hailing cells: the domain's corners, brick corners and scattered ones."""
    r = np.random.default_rng(seed)
    q1, q2 = np.zeros((nz, ny, nx, 4), np.float32), np.zeros((nz, ny, nx, 4), np.float32)
    q1[..., 0] = 1e-3
    ks = [0, 1, 2, 3, 5, 9, nz // 2, nz - 2, nz - 1]
    js, iz = [0, 3, 4, 7, 8, ny - 1], [0, 31, 32, nx // 2, nx - 1]
    cells = [(k, j, i) for k in ks for j in js for i in iz if j < ny and i < nx]
    cells += [(r.integers(nz), r.integers(ny), r.integers(nx)) for _ in range(300)]
    for n, (k, j, i) in enumerate(cells):
        (q1 if n % 3 == 0 else q2)[k, j, i, (3, 0, 1)[n % 3]] = 10.0 ** r.uniform(-8, -2)
        if thompson:
            q2[k, j, i, 2] = 1e4
    return q1.reshape(-1), q2.reshape(-1)


@pytest.mark.parametrize("nx,ny,nz,dx,scheme,site", [(48, 40, 40, 1000.0, 0, (0.4, 0.5)), (97, 33, 16, 2000.0, 1, (-0.3, 1.2)),
                                                     (150, 130, 20, 100.0, 0, (0.5, 0.02)), (64, 200, 40, 1500.0, 1, (1.0, 0.0)),
                                                     (256, 224, 12, 2500.0, 0, (3.0, 2.0))])
def test_scan_leaves_no_echo_out(native, nx, ny, nz, dx, scheme, site):
    case = W.StormCase("scan", nx, ny, nz, dx, 1.0, 1, scheme=scheme, bubbles=[], noise=0.0)
    m, _ = M.setup_case(case)
    q1, q2 = _sparse(nx, ny, nz, nx, scheme == 1)
    m.set_field(N.FIELD_Q1, q1)
    m.set_field(N.FIELD_Q2, q2)
    geo = RD.Geo(35.9, -97.2, nx * dx, ny * dx, 300.0)
    lat, lon = geo.from_model(site[0] * nx * dx, site[1] * ny * dx)
    sim = RD.RadarSim(m, geo, seed=3)
    R = sim.add_radar({"id": "KTST", "lat": lat, "lon": lon, "h": 305.0}, {"vcp": 212, "minDbz": -1000.0})
    R["vol"], R["az0"] = 1, 0.61
    try:
        vols = []
        for tornadoes in ([], FAR):
            sim.set_tornadoes(tornadoes)
            for c in R["cuts"]:
                sim.enc_cut(R, c, 600.0)
            vols.append(sim.read_volume(R))
        near = max(abs(site[0] - 0.5) * nx, abs(site[1] - 0.5) * ny) * dx < 300000.0   # the last site is out of range
        assert (vols[1] > 0).sum() > 50 or not near, "too few echoes to test"
        assert np.array_equal(vols[0], vols[1]), "%d bytes differ" % (vols[0] != vols[1]).sum()
        # every gate was written: no mark of the scan (1, a code that no moment has) is left
        assert not (vols[0] == 1).any()
    finally:
        sim.destroy()
        m.destroy()


@pytest.mark.parametrize("nrad,ngd", [(1, 4), (31, 92), (32, 96), (33, 100), (360, 192), (720, 196)])
def test_phidp_chain(oracle_lib, native, nrad, ngd):
    case = W.case_small(nx=48, ny=40, nz=40, dx=1000.0, dt=6.0)
    m, B = M.setup_case(case)
    q1, q2 = W.hydrometeor_blob(case, B)
    m.set_field(N.FIELD_Q1, q1)
    m.set_field(N.FIELD_Q2, q2)
    geo = RD.Geo(35.9, -97.2, 48000.0, 40000.0, 300.0)
    lat, lon = geo.from_model(500.0, 20000.0)   # in light rain, and the domain reaches 196 Doppler gates from it
    sim = RD.RadarSim(m, geo, seed=3)
    R = sim.add_radar({"id": "KTST", "lat": lat, "lon": lon, "h": 305.0}, {"vcp": 212})
    R["vol"], R["az0"] = 1, 0.61
    try:
        U = sim.cut_uniforms(R, R["cuts"][0], 600.0)
        U.cut[2], U.cut[3] = 360.0 / nrad, nrad
        U.gates[1] = ngd
        N.check(N.lib().ob_radar_cut(R["h"], C.byref(U)))
        kdp = np.empty(nrad * ngd, np.float32)
        N.check(N.lib().ob_radar_kdp(R["h"], N.fptr(kdp), kdp.size))
        vol = sim.read_volume(R)
        at = int(U.offB[0]) * 4
        phi = vol[at:at + nrad * ngd].reshape(nrad, ngd)
        assert (phi == oracle_lib.radar_phi(U.as_array(), kdp.reshape(nrad, ngd))).all()
        assert (phi > 0).any()
    finally:
        sim.destroy()
        m.destroy()
