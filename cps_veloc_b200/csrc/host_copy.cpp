// Pageable host <-> device copies through pinned staging chunks filled by
// several threads.
//
// The CPS-side callers hand over ordinary (pageable) vectors.  The driver's
// own path for those is one thread copying through its staging buffer:
// 10-17 GB/s measured, and 5 GB/s into freshly allocated pages, on a host
// whose PCIe link moves 55 GB/s from pinned memory.  Here a few threads copy
// each chunk between the vector and a ring of pinned chunks while the DMA of
// the neighbouring chunks runs; into fresh pages they also share the page
// faults.  Measured, whole calls
// before / with: RHMC force, DWF 16^4 Ls=8, 4 poles (275 MB) 24.1 / 7.2 ms;
// MatPcDagMatPc, DWF 8^4 Ls=8 (6 MB) 0.46 / 0.28 ms; 12 batched solves on
// 8^3x16 (226 MB) 48.3 / 38.2 ms
//
// The ring (RING chunks of at most CHUNK bytes, 16 MiB) and the threads
// belong to one device; they are made by the first copy that needs them,
// shared by every lattice of the device and given back by cpsgpu_finalize.
// They do not go with the last lattice: pinning the ring takes 6-9 ms, and a
// program that makes a lattice per configuration would pay it each time
// (an 8^4 lattice made, its links uploaded and closed: 6.7 ms, 18-22 with the
// ring made and freed each time, 6.3 with the driver's path).  One transfer uses them at a time: a second thread's transfer that
// finds them busy takes the driver's path, and so do all for a while after a
// copy thread lost its core in the middle of a copy (CopyPool::crowded).
#include "host_copy.h"

#include <sched.h>

#include <algorithm>
#include <cstdio>
#include <map>
#include <memory>
#include <mutex>
#include <thread>

#include "copy_pool.h"
#include "cpsgpu_impl.h"

namespace cpsgpu {

namespace {

constexpr size_t CHUNK = size_t(2) << 20;
// 8 x 4 MiB copies no faster; the force with 8 x 1 MiB 8.8 ms, with 5 x 2 MiB
// 8.0, with 8 x 2 MiB 7.3
constexpr int RING = 8;
// below this the driver's path is as fast (one chunk, no overlap)
constexpr size_t SMALLEST = size_t(256) << 10;

// the cores this process may run on: its affinity mask and its CPU quota
// (cgroup v2), either of which a container may set
int usable_cores() {
  int n = (int)std::thread::hardware_concurrency();
  cpu_set_t set;
  CPU_ZERO(&set);
  if (sched_getaffinity(0, sizeof(set), &set) == 0) n = CPU_COUNT(&set);
  if (FILE *f = std::fopen("/sys/fs/cgroup/cpu.max", "r")) {
    long quota = 0, period = 0;  // "max 100000" without a limit
    if (std::fscanf(f, "%ld %ld", &quota, &period) == 2 && quota > 0 && period > 0)
      n = std::min(n, (int)std::max(1L, quota / period));
    std::fclose(f);
  }
  return n;
}

struct Stager {
  std::mutex busy;
  char *ring = nullptr;
  cudaEvent_t ev[RING] = {};
  std::unique_ptr<CopyPool<>> pool;
  ~Stager() {
    if (ring)
      for (auto e : ev) cudaEventSynchronize(e);
    for (auto e : ev)
      if (e) cudaEventDestroy(e);
    if (ring) cudaFreeHost(ring);
  }
  // the buffers and threads; false when the host has none to give
  bool ready() {
    if (ring) return true;
    const int cores = usable_cores();
    if (!pool) pool.reset(new CopyPool<>(cores >= 16 ? 7 : cores >= 4 ? cores / 2 - 1 : 0));
    if (pool->workers() == 0) return false;
    for (auto &e : ev)
      if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
    void *p = nullptr;
    if (cudaHostAlloc(&p, CHUNK * RING, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    ring = static_cast<char *>(p);
    return true;
  }
};

std::mutex g_mu;
// by device; never destroyed, as the CUDA runtime may be gone when statics are
std::map<int, std::shared_ptr<Stager>> &g_stagers = *new std::map<int, std::shared_ptr<Stager>>;

std::shared_ptr<Stager> stager_of(int device) {
  std::lock_guard<std::mutex> lk(g_mu);
  std::shared_ptr<Stager> &s = g_stagers[device];
  if (!s) s = std::make_shared<Stager>();
  return s;
}

bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// the stager, locked, when this copy goes through it
std::shared_ptr<Stager> take(const void *host, size_t bytes, std::unique_lock<std::mutex> &lk) {
  if (bytes < SMALLEST || !pageable(host)) return nullptr;
  int dev = 0;
  CPSGPU_CUDA(cudaGetDevice(&dev));
  std::shared_ptr<Stager> s = stager_of(dev);
  lk = std::unique_lock<std::mutex>(s->busy, std::try_to_lock);
  if (!lk.owns_lock() || !s->ready() || s->pool->crowded()) {
    if (lk.owns_lock()) lk.unlock();
    return nullptr;
  }
  return s;
}

// at least four chunks in a transfer, so that its copies and DMAs overlap
size_t chunk_of(size_t bytes) {
  const size_t c = (bytes / 4 + 65535) & ~size_t(65535);
  return c < CHUNK ? c : CHUNK;
}

}  // namespace

void host_copy_finalize() {
  std::map<int, std::shared_ptr<Stager>> gone;  // a transfer on another thread keeps its own until it ends
  std::lock_guard<std::mutex> lk(g_mu);
  gone.swap(g_stagers);
}

void copy_to_device(cudaStream_t stream, void *dst, const void *src, size_t bytes) {
  std::shared_ptr<Stager> s;  // outlives its lock
  std::unique_lock<std::mutex> lk;
  s = take(src, bytes, lk);
  if (!s) {
    CPSGPU_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream));
    return;
  }
  const size_t chunk = chunk_of(bytes);
  int slot = 0;
  for (size_t at = 0; at < bytes; at += chunk, slot = (slot + 1) % RING) {
    const size_t n = bytes - at < chunk ? bytes - at : chunk;
    char *buf = s->ring + CHUNK * slot;
    CPSGPU_CUDA(cudaEventSynchronize(s->ev[slot]));  // its last DMA, this transfer's or an earlier one's
    s->pool->copy(buf, static_cast<const char *>(src) + at, n);
    CPSGPU_CUDA(cudaMemcpyAsync(static_cast<char *>(dst) + at, buf, n, cudaMemcpyHostToDevice, stream));
    CPSGPU_CUDA(cudaEventRecord(s->ev[slot], stream));
  }
}

void copy_to_host(cudaStream_t stream, void *dst, const void *src, size_t bytes) {
  std::shared_ptr<Stager> s;  // outlives its lock
  std::unique_lock<std::mutex> lk;
  s = take(dst, bytes, lk);
  if (!s) {
    CPSGPU_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream));
    return;
  }
  const size_t chunk = chunk_of(bytes);
  const size_t count = (bytes + chunk - 1) / chunk;
  auto issue = [&](size_t k) {
    const int slot = (int)(k % RING);
    const size_t at = k * chunk, n = bytes - at < chunk ? bytes - at : chunk;
    // an earlier transfer's copy out of this slot may still run on another stream
    CPSGPU_CUDA(cudaEventSynchronize(s->ev[slot]));
    CPSGPU_CUDA(cudaMemcpyAsync(s->ring + CHUNK * slot, static_cast<const char *>(src) + at, n, cudaMemcpyDeviceToHost, stream));
    CPSGPU_CUDA(cudaEventRecord(s->ev[slot], stream));
  };
  for (size_t k = 0; k < count && k < RING; k++) issue(k);
  for (size_t k = 0; k < count; k++) {
    const int slot = (int)(k % RING);
    const size_t at = k * chunk, n = bytes - at < chunk ? bytes - at : chunk;
    CPSGPU_CUDA(cudaEventSynchronize(s->ev[slot]));
    s->pool->copy(static_cast<char *>(dst) + at, s->ring + CHUNK * slot, n);
    if (k + RING < count) issue(k + RING);
  }
}

}  // namespace cpsgpu
