"""Workloads for timing the framework through its public entry points, from the smallest calls to the largest.

Storm steps are batches of ``RegionalModel.enc_step`` closed by ``request_maps``, which is how the run loop and the
application drive the model (a batch of steps, then the maps a viewer paints); they start from a developed storm state
(updrafts, rain, ice, graupel, anvils) over the Weisman-Klemp sounding. Pressure solves go through
``ob_poisson_solve_device`` on torch tensors, a radar volume through ``RadarSim`` (every cut of VCP 212, then the
volume's bytes), the surrogate's training through ``MicroSurrogate.train``.

``listed`` are fixed cases, ``draw`` gives more of the same ranges, ``prepare`` builds what a program has in hand
before the call, ``run`` is one pass, ``work`` the bytes and operations a pass cannot do without, and ``exact`` the
pressure solve in 64 bits.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from outbreaklab_b200 import _native as N
from outbreaklab_b200 import hurricane as H
from outbreaklab_b200 import model as M
from outbreaklab_b200 import radar as RD
from outbreaklab_b200 import surrogate as S
from outbreaklab_b200 import workloads as W

DEPTH = 20000.0     # every model domain is 20 km deep
STORM_SPACING = 60  # km between storm centres of a developed state


# ---------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------
def _step(nx, ny, nz, dx, scheme, steps, fronts=False, name=None):
    c = {"kind": "step", "nx": nx, "ny": ny, "nz": nz, "dx": dx, "scheme": scheme, "steps": steps, "fronts": fronts}
    return dict(c, name=name) if name else c


def _solve(nx, ny, nz, dx, precision, name=None):
    c = {"kind": "solve", "nx": nx, "ny": ny, "nz": nz, "dx": dx, "precision": precision}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the small single-storm domain: a step is a chain of short kernels, so launches and latency count
        _step(64, 64, 40, 2000.0, "lin", 5, name="step 64x64x40"),
        # an odd-sized domain with moving fronts, as an outbreak run has them
        _step(203, 157, 40, 2000.0, "thompson", 4, fronts=True, name="step 203x157x40 fronts"),
        # the "quick" grid preset with the Thompson-style microphysics
        _step(320, 320, 56, 2000.0, "thompson", 4, name="step 320x320x56"),
        # the benchmark's domain
        _step(640, 640, 40, 1000.0, "lin", 4, name="step 640x640x40"),
        # the "fine" grid preset, the largest outbreak domain
        _step(640, 640, 64, 1000.0, "lin", 4, name="step 640x640x64"),
        # hurricane mode: a vortex over a warm sea
        {"kind": "hurricane", "name": "hurricane 256x224x40", "nx": 256, "ny": 224, "nz": 40, "dx": 2000.0, "steps": 4},
        # the pressure solve alone: the padded grid of the small domain, ...
        _solve(80, 80, 40, 2000.0, 5, name="solve 80x80x40"),
        # ... an odd width refined in bf16x3, ...
        _solve(333, 275, 40, 1500.0, 2, name="solve 333x275x40"),
        # ... the padded grid of the "standard" preset in fp32, ...
        _solve(464, 464, 60, 1500.0, 0, name="solve 464x464x60 fp32"),
        # ... and the benchmark's large solve
        _solve(1024, 1024, 80, 1000.0, 5, name="solve 1024x1024x80"),
        # one WSR-88D volume over a developed storm field
        {"kind": "radar", "name": "radar volume 256x256x40", "nx": 256, "ny": 256, "nz": 40, "dx": 1000.0, "scheme": "lin"},
        # the surrogate's training at the batch the package trains with
        {"kind": "train", "name": "train 16384", "batch": 16384, "steps": 8, "pairs": 400000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "step", "hurricane", "solve", "solve", "solve", "radar", "train"])
    if kind in ("step", "hurricane"):
        most, steps = (640 * 640 * 64 * 4, rng.choice([3, 4, 5])) if kind == "step" else (384 * 384 * 40 * 4, 4)
        nz = rng.choice([16, 28, 40, 40, 56, 60, 64, 80, 100] if kind == "step" else [40, 40, 56])
        side = 640 if kind == "step" else 384
        while True:
            nx, ny = _log_int(rng, 48, side), _log_int(rng, 48, side)
            if nx * ny * nz * steps <= most and max(nx, ny) <= 6 * min(nx, ny):
                break
        if kind == "hurricane":
            return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "dx": rng.choice([1500.0, 2000.0, 3000.0]), "steps": steps}
        return _step(nx, ny, nz, rng.choice([500.0, 1000.0, 1500.0, 2000.0]), rng.choice(["lin", "thompson"]), steps,
                     fronts=rng.random() < 0.3)
    if kind == "solve":
        precision = rng.choice([0, 2, 5, 5])
        nz = rng.choice([16, 40, 80]) if precision else rng.choice([20, 40, 56, 60, 64, 80, 100])
        while True:
            nx, ny = _log_int(rng, 64, 1024), _log_int(rng, 64, 1024)
            if nx * ny * nz * (nx + ny) <= (1024 ** 3 * 160 if precision else 464 ** 3 * 240):
                return _solve(nx, ny, nz, rng.choice([500.0, 1000.0, 1500.0, 2000.0]), precision)
    if kind == "radar":
        nx, ny = _log_int(rng, 96, 288), _log_int(rng, 96, 288)
        return {"kind": "radar", "nx": nx, "ny": ny, "nz": rng.choice([40, 56]), "dx": rng.choice([500.0, 1000.0, 1500.0]),
                "scheme": rng.choice(["lin", "thompson"])}
    return {"kind": "train", "batch": 128 * rng.randint(16, 160), "steps": rng.choice([4, 8]), "pairs": rng.randint(100000, 600000)}


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _storm_state(nx, ny, nz, dx, B, thompson, seed):
    """A developed storm field in the texel layouts of V, Q1, Q2 and AUX: one storm per 60 km square (at least one),
    each with a warm updraft core, cloud water, rain, graupel, ice and a wider anvil of snow, in noisy air."""
    dev, g, r = "cuda", _gen(seed), random.Random(seed)
    dz = DEPTH / nz
    Bz = torch.tensor(np.asarray(B, np.float32).reshape(nz + 1, 8), device=dev)
    V = torch.zeros(nz + 1, ny + 1, nx + 1, 4, device=dev)
    kk = torch.clamp(torch.arange(nz + 1, device=dev), max=nz - 1)
    V[:nz, :ny, :, 0] = Bz[:nz, 6, None, None]
    V[:nz, :, :nx, 1] = Bz[:nz, 7, None, None]
    V[..., 3] = Bz[kk, 0][:, None, None]
    V[:nz, :ny, :nx, 3] += 0.1 * (2 * torch.rand(nz, ny, nx, device=dev, generator=g) - 1)
    Q1 = torch.zeros(nz, ny, nx, 4, device=dev)
    Q1[..., 0] = Bz[:nz, 1, None, None]
    Q2 = torch.zeros(nz, ny, nx, 4, device=dev)
    AUX = torch.zeros(nz, ny, nx, 2, device=dev)
    z = ((torch.arange(nz, device=dev) + 0.5) * dz)[:, None, None]
    zw = (torch.arange(nz + 1, device=dev) * dz)[:, None, None]
    T = (Bz[:nz, 0] * Bz[:nz, 4])[:, None, None]
    Lx, Ly = nx * dx, ny * dx
    n = max(1, round(Lx * Ly / (STORM_SPACING * 1000.0) ** 2))
    rad = min(9000.0, 0.2 * min(Lx, Ly))
    for _ in range(n):
        R = rad * r.uniform(0.6, 1.2)
        xc, yc, amp = Lx * r.uniform(0.15, 0.85), Ly * r.uniform(0.15, 0.85), r.uniform(0.6, 1.0)
        i0, i1 = max(0, int((xc - 2.5 * R) / dx)), min(nx, int((xc + 2.5 * R) / dx) + 1)
        j0, j1 = max(0, int((yc - 2.5 * R) / dx)), min(ny, int((yc + 2.5 * R) / dx) + 1)
        x = ((torch.arange(i0, i1, device=dev) + 0.5) * dx - xc)[None, None, :]
        y = ((torch.arange(j0, j1, device=dev) + 0.5) * dx - yc)[None, :, None]
        r2 = (x * x + y * y) / (R * R)
        core, anvil = torch.clamp(1 - r2, min=0.0) * amp, torch.clamp(1 - r2 / 5.0, min=0.0) * amp
        rough = 0.7 + 0.3 * torch.rand(nz, j1 - j0, i1 - i0, device=dev, generator=g)
        box = (slice(None), slice(j0, j1), slice(i0, i1))
        V[:nz, j0:j1, i0:i1, 3] += 2.5 * core * torch.exp(-((z - 5000) / 3500) ** 2)
        V[1:nz, j0:j1, i0:i1, 2] += (20.0 * core * torch.sin(math.pi * torch.clamp(zw / 13000.0, max=1.0)))[1:nz]
        Q1[box + (0,)] *= 1 + 0.05 * core
        Q1[box + (1,)] += 1.5e-3 * core * rough * ((z > 1000) & (z < 8000))
        Q1[box + (2,)] += 6e-4 * anvil * rough * (T < 262) * (z < 13000)
        Q1[box + (3,)] += 2.5e-3 * core * rough * (z < 6000)
        Q2[box + (0,)] += 9e-4 * anvil * rough * (T < 270) * (z < 12000)
        Q2[box + (1,)] += 3e-3 * core * rough * ((z > 1500) & (z < 9000))
        AUX[box] += (300.0 * core * (z < 13000))[..., None]
    if thompson:
        Q2[..., 2] = Q1[..., 3] * torch.pow(10.0, 5 + 2 * torch.rand(nz, ny, nx, device=dev, generator=g))
    return V, Q1, Q2, AUX


def _model(c, seed, fronts=False):
    thompson = c["scheme"] == "thompson"
    case = W.StormCase("perf", c["nx"], c["ny"], c["nz"], c["dx"], 6.0 * c["dx"] / 1000.0, 1, scheme=1 if thompson else 0)
    bounds, ci = (W.fronts_setup(case, seed=seed) if fronts else (None, None))
    m = M.RegionalModel().allocate(spec={"dx": case.dx, "n": [case.nx, case.ny, case.nz]})
    m.params["noise"] = 0.0
    m.params["scheme"] = c["scheme"]
    B, _ = W.base_state_for(case)
    m.set_base_state(B)
    if bounds:
        m.set_boundaries(bounds)
        m.set_ci(ci)
    m.reset()
    V, Q1, Q2, AUX = _storm_state(case.nx, case.ny, case.nz, case.dx, B, thompson, seed)
    for f, t in ((N.FIELD_V, V), (N.FIELD_Q1, Q1), (N.FIELD_Q2, Q2), (N.FIELD_AUX, AUX)):
        m.set_field(f, t.reshape(-1).cpu().numpy())
    m.sync()
    return m, case


def _density(nz):
    """An exponential atmosphere: density at the level centres and at their bottom faces."""
    dz = DEPTH / nz
    rc = 1.15 * np.exp(-(np.arange(nz) + 0.5) * dz / 9000.0)
    rw = 1.15 * np.exp(-np.arange(nz + 1) * dz / 9000.0)
    return rc.astype(np.float32), rw.astype(np.float32)


def _rhs(c, seed):
    """A Gaussian random field with a 5 km correlation length and no horizontal mean, as a divergence has none."""
    nx, ny, nz, dx = c["nx"], c["ny"], c["nz"], c["dx"]
    w = torch.randn(nz, ny, nx, device="cuda", generator=_gen(seed))
    kx = torch.fft.rfftfreq(nx, d=dx, device="cuda") * 2 * math.pi
    ky = torch.fft.fftfreq(ny, d=dx, device="cuda") * 2 * math.pi
    filt = torch.exp(-0.5 * (ky[:, None] ** 2 + kx[None, :] ** 2) * 5000.0 ** 2)
    f = torch.fft.irfft2(torch.fft.rfft2(w) * filt, s=(ny, nx))
    f -= f.mean(dim=(1, 2), keepdim=True)
    return (f / f.abs().max() * 1e-3).contiguous()


def _pairs(n, seed):
    """(state, tendency) pairs in the ranges the microphysics meets: mixing ratios over several decades, tendencies of
    the size of the processes that move them."""
    g = _gen(seed)
    u = torch.rand(n, 12, device="cuda", generator=g)
    p = torch.zeros(n, N.MLP_PAIR, device="cuda")
    p[:, 0] = 220 + 80 * u[:, 0]                                   # T
    p[:, 1] = 1e5 * torch.exp(-1.6 * (1 - u[:, 0]))                # p
    p[:, 2] = p[:, 1] / (287.0 * p[:, 0])                          # rho
    p[:, 3] = 0.014 * u[:, 0] ** 3 * (0.6 + 0.4 * u[:, 3])         # qv
    for k, (top, cold) in enumerate(((2e-3, 0), (4e-3, 0), (8e-4, 1), (2e-3, 1), (5e-3, 0))):   # qc qr qi qs qg
        q = top * torch.pow(10.0, -4 * u[:, 4 + k])
        p[:, 4 + k] = torch.where(p[:, 0] < 268, q, torch.zeros_like(q)) if cold else q
    p[:, 9] = p[:, 5] * torch.pow(10.0, 5 + 2 * u[:, 9])           # Nr
    p[:, 11] = 30 * (u[:, 10] - 0.3)                               # w
    auto = 1e-2 * torch.clamp(p[:, 4] - 5e-4, min=0.0)
    accr = 8.0 * p[:, 4] * p[:, 5]
    rime = 6.0 * p[:, 4] * p[:, 8]
    melt = 1e-2 * p[:, 8] * torch.clamp((p[:, 0] - 273.15) / 20, min=0.0)
    evap = 2e-3 * p[:, 5] * (1 - u[:, 3])
    noise = 1 + 0.05 * torch.randn(n, device="cuda", generator=g)
    y = torch.stack([2.5e3 * (rime * 0.13 - evap - 0.13 * melt), evap, -auto - accr - rime, torch.zeros_like(auto),
                     auto + accr + melt - evap, torch.zeros_like(auto), rime - melt, 1e6 * (auto - evap)], 1)
    p[:, 12:20] = y * noise[:, None]
    return p.cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        m, c = _model(case, seed, case["fronts"])
        return {"run": _run_step, "m": m, "dt": c.dt, "steps": case["steps"]}
    if kind == "hurricane":
        c, surf, vort = H.tropical_case(case["nx"], case["ny"], case["nz"], case["dx"], land_cols=case["nx"] // 16)
        m, B, _, _, _ = H.setup(c, surf, vort, noise=0.25)
        _, Q1, Q2, _ = _storm_state(c.nx, c.ny, c.nz, c.dx, B, False, seed)   # rain bands in the moist vortex
        Q1[..., 0] = torch.maximum(Q1[..., 0], torch.tensor(m.get_field(N.FIELD_Q1).reshape(c.nz, c.ny, c.nx, 4)[..., 0], device="cuda"))
        m.set_field(N.FIELD_Q1, Q1.reshape(-1).cpu().numpy())
        m.set_field(N.FIELD_Q2, Q2.reshape(-1).cpu().numpy())
        m.sync()
        return {"run": _run_step, "m": m, "dt": c.dt, "steps": case["steps"]}
    if kind == "solve":
        P = M.PoissonDirect(case["nx"], case["ny"], case["nz"], case["dx"], DEPTH / case["nz"], case["precision"])
        P.set_density(*_density(case["nz"]))
        rhs = _rhs(case, seed)
        return {"run": _run_solve, "P": P, "rhs": rhs, "phi": torch.empty_like(rhs)}
    if kind == "radar":
        m, c = _model(case, seed)
        geo = RD.Geo(35.9, -97.2, c.nx * c.dx, c.ny * c.dx, 350.0)
        lat, lon = geo.from_model(0.35 * c.nx * c.dx, 0.4 * c.ny * c.dx)   # the domain's extent sets the gate counts
        sim = RD.RadarSim(m, geo, seed=seed)
        R = sim.add_radar({"id": "KPRF", "lat": lat, "lon": lon, "h": 355.0}, {"vcp": 212})
        R["vol"], R["az0"] = 0, random.Random(seed).random()
        return {"run": _run_radar, "m": m, "sim": sim, "R": R}
    net = S.MicroSurrogate(seed=1 + seed % 1000)
    pairs = _pairs(case["pairs"], seed)
    net.reserve(len(pairs))
    net.write_pairs(pairs)
    net.fit_norm(6.0)
    return {"run": _run_train, "net": net, "batch": case["batch"], "steps": case["steps"], "seed": 7 + seed % 1000}


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def _run_step(s):
    s["m"].enc_step(s["dt"], s["steps"])
    return s["m"].request_maps()


def _run_solve(s):
    N.check(N.lib().ob_poisson_solve_device(s["P"].h, C.c_void_p(s["rhs"].data_ptr()), C.c_void_p(s["phi"].data_ptr()),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return s["phi"]


def _run_radar(s):
    sim, R = s["sim"], s["R"]
    for c in R["cuts"]:
        sim.enc_cut(R, c, 600.0 + c["t0"])
    return sim.collect({"R": R, "vol": 0, "volStart": 600.0, "az0": R["az0"]}, "perf", 0)["bytes"]


def _run_train(s):
    loss = s["net"].train(s["batch"], s["steps"], 1e-3, s["seed"])
    return {"loss": loss, "params": s["net"].params()}


def run(state):
    return state["run"](state)


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------
def _solve_work(nx, ny, nz):
    n = nx * ny * nz   # right-hand side in, phi out; fast transforms both ways and a tridiagonal sweep
    return 8.0 * n, n * (5.0 * math.log2(nx) + 5.0 * math.log2(ny) + 8.0)


def work(case):
    kind = case["kind"]
    if kind == "solve":
        b, f = _solve_work(case["nx"], case["ny"], case["nz"])
        return {"bytes": b, "flops": f}
    if kind == "train":
        params = N.MLP_NPARAM
        return {"bytes": case["steps"] * (4.0 * 20 * case["batch"] + 24.0 * params), "flops": case["steps"] * 6.0 * params * case["batch"]}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells, texels = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    if kind == "radar":
        geo = RD.radar_layout(nx * case["dx"], ny * case["dx"], 0.5 * nx * case["dx"], 0.5 * ny * case["dx"], RD.VCPS[212])
        gates = sum(c["nrad"] for c in geo[2]) * geo[0]
        return {"bytes": 16.0 * texels + 20.0 * cells + geo[3], "flops": 600.0 * gates}
    pad = M.grid_pad(case["dx"])
    px, py = nx + 2 * pad, ny + 2 * pad
    solve = _solve_work(px, py, nz)
    # a step reads and writes u, v, w, theta and the eight scalars once and stores phi; the maps go to the host
    step = 32.0 * texels + 64.0 * cells + 4.0 * px * py * nz
    return {"bytes": case["steps"] * step + 64.0 * nx * ny, "flops": case["steps"] * (solve[1] + 800.0 * cells)}


# ---------------------------------------------------------------------------------------------------------------
# the pressure solve in 64 bits: rho_c lap_h(phi) + d/dz(rho_w dphi/dz) = rhs, phi = 0 beyond the lateral faces,
# Neumann in z, with the operator's coefficients as the plan stores them (fp32: the near-singular lowest mode magnifies
# their rounding, so another rounding of them is another problem)
# ---------------------------------------------------------------------------------------------------------------
def _dst(n):
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    q = torch.sin(math.pi * (i[:, None] + 1) * (i[None, :] + 0.5) / n) * math.sqrt(2.0 / n)
    q[n - 1] *= math.sqrt(0.5)
    return q   # row l: the l-th sine mode


def exact(case, seed):
    if case["kind"] != "solve":
        return None
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    rc, rw = _density(nz)
    a = 1.0 / (DEPTH / nz) ** 2
    lo = np.array([float(rw[k]) * a if k > 0 else 0.0 for k in range(nz)])
    up = np.array([float(rw[k + 1]) * a if k < nz - 1 else 0.0 for k in range(nz)])
    lo32, up32, di32 = lo.astype(np.float32).astype(np.float64), up.astype(np.float32).astype(np.float64), (-(lo + up)).astype(np.float32).astype(np.float64)

    def eig(n):
        lam = -4.0 / dx ** 2 * np.sin(math.pi * (np.arange(n) + 1) / (2 * n)) ** 2
        return torch.tensor(lam.astype(np.float32).astype(np.float64), device="cuda")
    shift = eig(nx)[None, :] + eig(ny)[:, None]
    qx, qy = _dst(nx), _dst(ny)
    h = [qy @ (r.double() @ qx.T) for r in _rhs(case, seed)]
    cp, d = [], []
    for k in range(nz):
        den = di32[k] + shift * float(rc[k]) - (lo32[k] * cp[-1] if k else 0.0)
        d.append((h[k] - (lo32[k] * d[-1] if k else 0.0)) / den)
        cp.append(up32[k] / den)
        h[k] = None
    for k in range(nz - 2, -1, -1):
        d[k] = d[k] - cp[k] * d[k + 1]
    return torch.stack([qy.T @ (x @ qx) for x in d])
