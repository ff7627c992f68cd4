// ob_hostcopy.cu — device-to-host copies into ordinary (pageable) memory of the caller.
//
// The driver moves such a copy through a small pinned buffer of its own, and one thread empties it into the caller's
// pages, which take a fault each in a fresh array: 36 MB took 8.1 ms where the link needs 0.7 ms. A large copy (pinned
// memory of the caller takes the driver's copy as it is) goes here through a ring of pinned slots that several host
// threads drain: each thread owns two slots and queues the copy of its next chunk into one while it empties the other
// into the caller's memory. 36 MB into a fresh array: 2.0-2.5 ms; 26 MB of maps with the pages at hand: 1.6 -> 1.1 ms. With 4
// threads 2.5-2.9 ms, with chunks of half the size or 12 threads no less.
//
// The ring is one per process (16 MiB), made at the first large copy and given back when the last model goes
// (host_copy_release). A copy that finds it taken by another thread, made for another device, or not to be had, and one from
// another device than the current one, goes the driver's way.
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>

#include "ob_hostcopy.cuh"

namespace ob {

namespace {
constexpr size_t kChunk = size_t(1) << 20;
constexpr int kThreads = 8, kSlots = 2 * kThreads;
// below it the driver's copy is as good: 6.6 MB of maps after a batch of steps took 0.4 ms longer by the ring
constexpr size_t kMinBytes = 16 * kChunk;

struct Ring {
  std::mutex use;          // held by the copy that uses the slots
  std::mutex owners_lock;
  int owners = 0;
  uint8_t* mem = nullptr;
  cudaEvent_t ev[kSlots] = {};
  int device = -1;

  bool make() {
    if (mem) return true;
    if (cudaHostAlloc(&mem, kSlots * kChunk, cudaHostAllocDefault) != cudaSuccess) { mem = nullptr; cudaGetLastError(); return false; }
    for (cudaEvent_t& e : ev)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); drop(); return false; }
    cudaGetDevice(&device);
    return true;
  }
  void drop() {
    for (cudaEvent_t& e : ev)
      if (e) { cudaEventDestroy(e); e = nullptr; }
    if (mem) cudaFreeHost(mem);
    mem = nullptr;
    device = -1;
  }
};
Ring& ring() {
  static Ring r;   // no destructor: handles may outlive static destruction
  return r;
}
}  // namespace

void host_copy_retain() {
  Ring& R = ring();
  std::lock_guard<std::mutex> g(R.owners_lock);
  R.owners++;
}
void host_copy_release() {
  Ring& R = ring();
  std::lock_guard<std::mutex> g(R.owners_lock);
  if (--R.owners > 0) return;
  std::lock_guard<std::mutex> u(R.use);
  R.drop();
}

cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  Ring& R = ring();
  int dev = -1;
  std::unique_lock<std::mutex> use(R.use, std::defer_lock);
  cudaPointerAttributes at{}, from{};
  const bool ordinary = bytes >= kMinBytes && cudaPointerGetAttributes(&at, dst) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
  // the ring's events belong to the device that is current when it is made, and are recorded on s
  const bool here = ordinary && cudaGetDevice(&dev) == cudaSuccess && cudaPointerGetAttributes(&from, src) == cudaSuccess && from.device == dev;
  if (!here || !use.try_lock() || !R.make() || R.device != dev) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
  }
  // the work queued before is waited for here, by one thread and not by all of them
  const cudaError_t before = cudaStreamSynchronize(s);
  if (before != cudaSuccess) return before;
  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  const int nt = int(chunks < size_t(kThreads) ? chunks : size_t(kThreads));
  std::atomic<int> err{int(cudaSuccess)};
  // chunks t, t + nt, ... through slots 2 t and 2 t + 1
  auto work = [&](int t) {
    auto fail = [&](cudaError_t e) {
      int none = int(cudaSuccess);
      if (e != cudaSuccess) err.compare_exchange_strong(none, int(e));
      return e != cudaSuccess;
    };
    if (fail(cudaSetDevice(dev))) return;
    auto size = [&](size_t c) { return c + 1 < chunks ? kChunk : bytes - c * kChunk; };
    auto queue = [&](size_t c, int half) {
      const int sl = 2 * t + half;
      return fail(cudaMemcpyAsync(R.mem + sl * kChunk, static_cast<const uint8_t*>(src) + c * kChunk, size(c), cudaMemcpyDeviceToHost, s)) ||
             fail(cudaEventRecord(R.ev[sl], s));
    };
    if (queue(size_t(t), 0)) return;
    int half = 0;
    for (size_t c = size_t(t); c < chunks; c += size_t(nt), half ^= 1) {
      if (c + size_t(nt) < chunks && queue(c + size_t(nt), half ^ 1)) break;
      const int sl = 2 * t + half;
      if (fail(cudaEventSynchronize(R.ev[sl]))) break;
      std::memcpy(static_cast<uint8_t*>(dst) + c * kChunk, R.mem + sl * kChunk, size(c));
    }
  };
  std::thread th[kThreads];
  int started = 1;
  try {
    for (; started < nt; started++) th[started] = std::thread(work, started);
  } catch (...) {   // no more threads to be had, or no memory for them: this one takes over their chunks below
  }
  for (int t = started; t < nt; t++) work(t);
  work(0);
  for (int t = 1; t < started; t++) th[t].join();
  // every queued copy has landed before the slots (and, on an error, the caller's memory) are given up
  const cudaError_t e = cudaStreamSynchronize(s);
  return err.load() != int(cudaSuccess) ? cudaError_t(err.load()) : e;
}

}  // namespace ob
