"""The radar's scan against the gates that it leaves out: no gate that may_echo drops comes out of gate() with anything in it, by
the domain's edges, its lid and inside. The sources are compiled into a program of the test's own, because the library has no
way round the scan."""
import subprocess

import numpy as np
import pytest

from outbreaklab_b200 import build, radar as RD

import _radar_case as RC

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "ob_radar.cu"
using namespace ob;

// [0] the gates that gate() fills, [1] those of them that may_echo drops, [2] gates that may_echo passes, [3] the first dropped
__global__ void k_gates(RadarU R, ScanU S, Grid g, Fields F, unsigned* n) {
  const int gi = blockIdx.x * blockDim.x + threadIdx.x, ri = blockIdx.y;
  if (gi >= int(R.gates.x)) return;
  const bool may = may_echo(R, S, g, F, ri, gi);
  const GateOut G = gate(R, g, F, 0, nullptr, ri, gi);
  const bool filled = G.c[0] != 0u || G.kdp != -1.f || G.m[0] == G.m[0];
  if (filled) atomicAdd(n, 1u);
  if (filled && !may) { atomicAdd(n + 1, 1u); atomicMin(n + 3, unsigned(ri) << 16 | unsigned(gi)); }
  if (may) atomicAdd(n + 2, 1u);
}
static void* dev(const void* host, size_t bytes) {
  void* d = nullptr;
  if (cudaMalloc(&d, bytes) != cudaSuccess) { std::printf("cudaMalloc\n"); std::exit(2); }
  if (host) cudaMemcpy(d, host, bytes, cudaMemcpyHostToDevice);
  else cudaMemset(d, 0, bytes);
  return d;
}
int main(int argc, char** argv) {
  unsigned* n = static_cast<unsigned*>(dev(nullptr, 16));
  unsigned h[4] = {0u, 0u, 0u, ~0u};
  cudaMemcpy(n, h, 16, cudaMemcpyHostToDevice);
  if (argc != 2) return 2;
  {
    FILE* f = std::fopen(argv[1], "rb");   // RadarU, 8 floats of base state per level and one more level
    RadarU R;
    if (!f || std::fread(&R, sizeof(R), 1, f) != 1) return 2;
    Grid g{};
    g.nx = int(R.mdl.x); g.ny = int(R.mdl.y); g.nz = int(R.mdl.z);
    g.px = (g.nx + 32) / 32 * 32; g.py = g.ny + 1; g.plane = g.px * g.py;
    std::vector<float> B(size_t(g.nz + 1) * 8);
    if (std::fread(B.data(), 4, B.size(), f) != B.size()) return 2;
    const size_t cells = size_t(g.plane) * (g.nz + 1);
    std::vector<float> rain(cells, 0.f), theta(cells, 300.f), wet(cells, 0.f);
    // rain in every cell of the outermost columns and levels, of a plane through the middle, and in scattered cells
    for (int k = 0; k < g.nz; k++)
      for (int j = 0; j < g.ny; j++)
        for (int i = 0; i < g.nx; i++)
          if (i == 0 || i == g.nx - 1 || j == 0 || j == g.ny - 1 || k == 0 || k >= g.nz - 2 || i == g.nx / 2 ||
              (unsigned(i * 73856093) ^ unsigned(j * 19349663) ^ unsigned(k * 83492791)) % 97u == 0u)
            rain[g.at(i, j, k)] = 1e-3f;
    Fields F{};
    F.nbx = (g.nx + 31) / 32; F.nby = (g.ny + 3) / 4;
    std::vector<unsigned> act(size_t(F.nbx) * F.nby * g.nz, 0u);
    for (int k = 0; k < g.nz; k++)
      for (int j = 0; j < g.ny; j++)
        for (int i = 0; i < g.nx; i++)
          if (rain[g.at(i, j, k)] != 0.f) act[i / 32 + size_t(F.nbx) * (j / 4 + size_t(F.nby) * k)] |= 1u << 3;
    float* zero = static_cast<float*>(dev(nullptr, cells * 4));
    for (int q = 0; q < 8; q++) F.Q[0][q] = F.Q[1][q] = zero;
    F.Q[0][3] = static_cast<float*>(dev(rain.data(), cells * 4));
    for (int c = 0; c < 4; c++) F.V[0][c] = F.V[1][c] = zero;
    F.V[0][3] = static_cast<float*>(dev(theta.data(), cells * 4));
    F.aux[0] = F.aux[1] = zero;
    F.B = static_cast<float*>(dev(B.data(), B.size() * 4));
    F.actQ0 = static_cast<unsigned*>(dev(act.data(), act.size() * 4));
    k_gates<<<dim3((int(R.gates.x) + 127) / 128, int(R.cut.w)), 128>>>(R, scan_uniforms(R), g, F, n);
  }
  const cudaError_t e = cudaDeviceSynchronize();
  cudaMemcpy(h, n, 16, cudaMemcpyDeviceToHost);
  std::printf("%s %u %u %u %u\n", cudaGetErrorName(e), h[0], h[1], h[2], h[3]);
  return e == cudaSuccess ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("bounds")
    (d / "bounds.cu").write_text(PROGRAM)
    exe = str(d / "bounds")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-I", build.CSRC, str(d / "bounds.cu"), "-o", exe], check=True)
    return exe


def _run(program, *args):
    r = subprocess.run([program, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    name, *n = r.stdout.split()
    assert name == "cudaSuccess"
    return [int(v) for v in n]


# the domain's size and spacing, where the site stands in it (parts of its extent), the latitude of its centre, and cuts from
# the lowest to the one that meets the lid nearest by
@pytest.mark.parametrize("nx,ny,nz,dx,site,lat", [(48, 40, 40, 1000.0, (0.4, 0.5), 35.9), (97, 33, 16, 2000.0, (-0.3, 1.2), 35.9),
                                                  (150, 130, 20, 100.0, (0.5, 0.02), 35.9), (64, 200, 40, 1500.0, (1.0, 0.0), -20.0),
                                                  (256, 224, 12, 2500.0, (0.5, 0.5), 60.0), (400, 300, 40, 250.0, (0.1, 0.9), 0.0),
                                                  (150, 130, 20, 100.0, (0.5, 0.5), 89.9), (120, 160, 20, 250.0, (0.2, 0.3), -89.7),
                                                  (300, 300, 16, 1000.0, (0.2, 0.3), 84.0)])
def test_no_gate_with_an_echo_is_dropped(program, tmp_path, nx, ny, nz, dx, site, lat):
    geo = RD.Geo(lat, -97.2, nx * dx, ny * dx, 350.0)
    la, lo = geo.from_model(site[0] * nx * dx, site[1] * ny * dx)

    class Case:
        pass
    c = Case()
    c.nx, c.ny, c.nz, c.dx = nx, ny, nz, dx
    dz = 20000.0 / nz
    z = (np.arange(nz + 1) + 0.5) * dz
    B = np.zeros((nz + 1, 8), np.float32)
    B[:, 0], B[:, 2], B[:, 3] = 300.0, 1.15 * np.exp(-z / 9000.0), 1.15 * np.exp(-z / 9000.0)
    B[:, 4], B[:, 5] = np.exp(-z / 30000.0), 1e5 * np.exp(-z / 8000.0)
    plan, ngr, _, _ = RC.cut_plan(c, geo, {"id": "KTST", "lat": la, "lon": lo, "h": 355.0}, B.reshape(-1), cut_indices=(0, 4, 8, 12, 16),
                                  az0=0.61, min_dbz=-1000.0)
    total = 0
    for k, (cut, U) in enumerate(plan):
        f = tmp_path / ("cut%d" % k)
        f.write_bytes(U.as_array().tobytes() + B.tobytes())
        filled, dropped, may, first = _run(program, str(f))
        total += filled
        assert dropped == 0, "cut %d: %d of %d, the first at radial %d, gate %d" % (k, dropped, filled, first >> 16, first & 0xffff)
        assert may < cut["nrad"] * ngr or abs(lat) > 80   # the scan drops some, but near a pole
    assert total > 50, "too few echoes to test"
