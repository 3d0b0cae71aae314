"""The threads behind the pageable host copies (copy_pool.h), compiled alone: no GPU."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "cps_veloc_b200" / "csrc"

SOURCE = r"""
#include "copy_pool.h"
#include <system_error>

// a thread of which only the first `allowed` can be started
struct Limited : std::thread {
  static inline int allowed = 0;
  template <class F> explicit Limited(F &&f) : std::thread(start(std::forward<F>(f))) {}
  Limited(Limited &&) = default;
  template <class F> static std::thread start(F &&f) {
    if (allowed-- <= 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    return std::thread(std::forward<F>(f));
  }
};

extern "C" void limited_copy(int allowed, int workers, void *dst, const void *src, size_t n, int reps) {
  Limited::allowed = allowed;
  cpsgpu::CopyPool<Limited> pool(workers);
  for (int k = 0; k < reps; k++) pool.copy(dst, src, n);
}

// milliseconds of a copy in chunks by one thread, then by the pool, while `spinners` threads keep a core each, as a
// caller's own threads do for a while after a parallel loop
extern "C" void crowded_copy(int spinners, int workers, char *dst, const char *src, size_t n, size_t chunk, double *one,
                             double *pooled) {
  using clk = std::chrono::steady_clock;
  std::atomic<bool> stop{false};
  std::vector<std::thread> th;
  cpsgpu::CopyPool<> pool(workers);
  for (int k = 0; k < spinners; k++)
    th.emplace_back([&] {
      while (!stop.load(std::memory_order_relaxed)) {
      }
    });
  auto ms = [&](auto &&copy) {
    const clk::time_point t0 = clk::now();
    for (size_t at = 0; at < n; at += chunk) copy(dst + at, src + at, n - at < chunk ? n - at : chunk);
    return std::chrono::duration<double, std::milli>(clk::now() - t0).count();
  };
  *one = ms([](char *d, const char *s, size_t m) { std::memcpy(d, s, m); });
  *pooled = ms([&](char *d, const char *s, size_t m) { pool.copy(d, s, m); });
  stop = true;
  for (auto &t : th) t.join();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pool")
    (d / "pool.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "pool.cpp"), "-o", str(d / "pool.so"),
                    "-lpthread"], check=True)
    so = C.CDLL(str(d / "pool.so"))
    so.crowded_copy.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_size_t, C.c_size_t, C.POINTER(C.c_double),
                                C.POINTER(C.c_double)]
    so.limited_copy.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    return so


@pytest.mark.parametrize("allowed", [0, 1, 3, 7])
def test_threads_that_cannot_be_started(lib, allowed):
    """a process at its thread limit copies with the workers it could start"""
    src = np.random.default_rng(1).integers(0, 256, (3 << 20) + 17, dtype=np.uint8)
    dst = np.zeros_like(src)
    lib.limited_copy(allowed, 7, dst.ctypes.data, src.ctypes.data, src.nbytes, 20)
    np.testing.assert_array_equal(dst, src)


@pytest.mark.parametrize("n", [1, 4096, 32768, 65536, 65537, (1 << 20) + 1, (2 << 20) - 5, 7 << 20])
@pytest.mark.parametrize("workers", [0, 1, 3, 7])
def test_every_byte_once(lib, workers, n):
    """sizes about the blocks' edges; repeated, so that workers come late, early and from sleep"""
    src = np.random.default_rng(2).integers(0, 256, n, dtype=np.uint8)
    dst = np.zeros(n + 64, dtype=np.uint8)
    lib.limited_copy(workers, workers, dst.ctypes.data, src.ctypes.data, n, 200)
    np.testing.assert_array_equal(dst[:n], src)
    assert not dst[n:].any()


def test_busy_cores(lib):
    """With every core taken by the caller's own threads the pool is no slower than one thread by more than the
    scheduling slices (some ms) of a stall or two; a wait for every worker took one per chunk, 100-250 ms here.  The
    best of a few tries: the host is shared."""
    n, chunk = 64 << 20, 2 << 20
    src = np.random.default_rng(3).integers(0, 256, n, dtype=np.uint8)
    dst = np.zeros_like(src)
    over = []
    for _ in range(6):
        one, pooled = C.c_double(), C.c_double()
        lib.crowded_copy(len(os.sched_getaffinity(0)), 7, dst.ctypes.data, src.ctypes.data, n, chunk, C.byref(one), C.byref(pooled))
        np.testing.assert_array_equal(dst, src)
        dst[:] = 0
        over.append(pooled.value - 2 * one.value)
    assert min(over) < 20.0, over
