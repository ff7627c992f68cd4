"""The bound that lets a cloudless cell skip the saturation adjustment, in the device's own arithmetic: no vapour that
far_below_saturation passes over exceeds the saturation value that the adjustment would compare it with, and where it does not
exceed it the adjustment's first iteration changes nothing. The function is compiled into a program of the test's own."""
import subprocess

import pytest

from outbreaklab_b200 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "ob_common.cuh"
#include "ob_micro.cuh"
using namespace ob;
// [0] cells passed over, [1] those of them above the saturation value, [2] cells that are not
__global__ void k_vapour(unsigned* n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;   // 2^20 temperatures
  const float w = float(t & 0xfffff) / 1048576.f;
  // a third each over 100 to 400 K, around 0 degrees C and around -40
  const float T = t % 3 == 0 ? 100.f + 300.f * w : (t % 3 == 1 ? 273.15f : 233.15f) + 0.1f * (w - 0.5f);
  const float p0s[6] = {100.f, 101.f, 611.2f, 5.0e3f, 3.0e4f, 1.05e5f};
  unsigned passed = 0, above = 0, rest = 0;
  for (int i = 0; i < 6; i++) {
    const float q = qvsat1(T, p0s[i], fIce(T));
    for (int e = -64; e <= 16; e++) {   // 0.97 to 1.0075 of the lower of the two saturation values, and of the mix
      for (int k = 0; k < 2; k++) {
        const float base = k ? q : fminf(q, 0.622f * fminf(esl(T), esi(T)) / p0s[i]);
        const float qv = base * (1.f + float(e) * (0.03f / 64.f));
        const bool far = far_below_saturation(T, p0s[i], qv);
        passed += far;
        above += far && !(qv <= q);
        rest += !far;
      }
    }
  }
  atomicAdd(n, passed);
  atomicAdd(n + 1, above);
  atomicAdd(n + 2, rest);
}
int main() {
  unsigned *n = nullptr, h[3] = {};
  if (cudaMalloc(&n, 12) != cudaSuccess || cudaMemset(n, 0, 12) != cudaSuccess) return 2;
  k_vapour<<<4096, 256>>>(n);
  const cudaError_t e = cudaMemcpy(h, n, 12, cudaMemcpyDeviceToHost);
  std::printf("%s %u %u %u\n", cudaGetErrorName(e), h[0], h[1], h[2]);
  return e == cudaSuccess ? 0 : 2;
}
"""


def test_vapour_passed_over_is_below_saturation(tmp_path):
    (tmp_path / "bound.cu").write_text(PROGRAM)
    exe = str(tmp_path / "bound")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-I", build.CSRC, str(tmp_path / "bound.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    passed, above, rest = (int(v) for v in r.stdout.split()[1:])
    assert passed > 1e7 and rest > 1e7, (passed, rest)
    assert above == 0, "%d of %d" % (above, passed)
