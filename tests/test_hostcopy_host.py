"""The readback ring's host code (ob_hostcopy.cu) against a stand-in for the CUDA runtime with two devices: what a machine
with one GPU cannot show. The stand-in refuses what the runtime refuses: an event recorded on another device's stream."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "outbreaklab_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidResourceHandle = 400 };
enum cudaMemcpyKind { cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1, cudaMemoryTypeDevice = 2 };
struct cudaPointerAttributes { cudaMemoryType type; int device; };
struct FakeStream { int device; };
struct FakeEvent { int device; };
using cudaStream_t = FakeStream*;
using cudaEvent_t = FakeEvent*;
constexpr unsigned cudaHostAllocDefault = 0, cudaEventDisableTiming = 2;
extern thread_local int fake_device;
extern const uint8_t* fake_mem[2];   // one array of device memory on each device
extern size_t fake_bytes;
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int* d) { *d = fake_device; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) { fake_device = d; return cudaSuccess; }
template <class T> cudaError_t cudaHostAlloc(T** p, size_t n, unsigned) { *p = static_cast<T*>(std::malloc(n)); return cudaSuccess; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = static_cast<FakeEvent*>(std::malloc(sizeof(FakeEvent))); (*e)->device = fake_device; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return e->device == s->device ? cudaSuccess : cudaErrorInvalidResourceHandle; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  *a = {cudaMemoryTypeUnregistered, -2};
  for (int d = 0; d < 2; d++)
    if (p >= fake_mem[d] && p < fake_mem[d] + fake_bytes) *a = {cudaMemoryTypeDevice, d};
  return cudaSuccess;
}
"""

HEAD = r"""
#include <algorithm>
#include <cstdio>
#include <new>
#include <vector>
#include "ob_hostcopy.cuh"
thread_local int fake_device = 0;
const uint8_t* fake_mem[2];
size_t fake_bytes;
static std::vector<uint8_t> mem[2];
static FakeStream stream[2] = {{0}, {1}};
static void fill(size_t n) {
  fake_bytes = n;
  for (int d = 0; d < 2; d++) {
    mem[d].resize(n);
    for (size_t i = 0; i < n; i++) mem[d][i] = uint8_t(i * 2654435761u >> 24) + uint8_t(d);
    fake_mem[d] = mem[d].data();
  }
}
// a readback of device d's memory while cur is the current device
static bool read_back(int d, int cur, size_t n) {
  std::vector<uint8_t> out(n, 7);
  fake_device = cur;
  const cudaError_t e = ob::copy_to_host(out.data(), fake_mem[d], n, &stream[d]);
  return e == cudaSuccess && std::memcmp(out.data(), mem[d].data(), n) == 0 && fake_device == cur;
}
"""


def _run(tmp_path, main):
    cxx = shutil.which("g++") or pytest.skip("no g++")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(HEAD + main)
    exe = str(tmp_path / "run")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", str(tmp_path), "-I", CSRC, "-x", "c++", os.path.join(CSRC, "ob_hostcopy.cu"),
                    str(tmp_path / "main.cpp"), "-o", exe], check=True)
    return subprocess.run([exe], capture_output=True, text=True, timeout=120)


def test_memory_of_another_device_than_the_current_one(tmp_path):
    """As cudaMemcpyAsync allows it: a thread that never chose a device reads back a model of the second one."""
    r = _run(tmp_path, r"""
int main() {
  const size_t n = (size_t(37) << 20) + 1000;
  fill(n);
  ob::host_copy_retain();
  bool ok = true;
  for (int rep = 0; rep < 2; rep++)   // the second time round the ring exists already
    for (int d = 0; d < 2; d++)
      for (int cur = 0; cur < 2; cur++)
        if (!read_back(d, cur, n)) { std::printf("device %d read back under device %d failed\n", d, cur); ok = false; }
  ob::host_copy_release();
  return ok ? 0 : 1;
}
""")
    assert r.returncode == 0, r.stdout + r.stderr


def test_no_memory_for_the_threads(tmp_path):
    """Any failure to start the draining threads leaves their chunks to the caller's thread; nothing escapes a C entry."""
    r = _run(tmp_path, r"""
static thread_local int fail_in = -1;   // allocations of this thread until one fails (-1: none does)
void* operator new(size_t n) {
  if (fail_in == 0) throw std::bad_alloc();
  if (fail_in > 0) fail_in--;
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
int main() {
  const size_t n = (size_t(21) << 20) + 12;
  fill(n);
  std::vector<uint8_t> out(n);
  ob::host_copy_retain();
  for (int k = 0; k < 9; k++) {
    std::fill(out.begin(), out.end(), uint8_t(7));
    fail_in = k;
    const cudaError_t e = ob::copy_to_host(out.data(), fake_mem[0], n, &stream[0]);
    fail_in = -1;
    if (e != cudaSuccess || out != mem[0]) { std::printf("allocation %d\n", k); return 1; }
  }
  ob::host_copy_release();
  return 0;
}
""")
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
