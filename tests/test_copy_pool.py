"""The threads behind the pageable host copies (copy_pool.h), compiled alone: no GPU."""
import ctypes as C
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
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pool")
    (d / "pool.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "pool.cpp"), "-o", str(d / "pool.so"),
                    "-lpthread"], check=True)
    so = C.CDLL(str(d / "pool.so"))
    so.limited_copy.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    return so


@pytest.mark.parametrize("allowed", [0, 1, 3, 7])
def test_threads_that_cannot_be_started(lib, allowed):
    """a process at its thread limit copies with the workers it could start"""
    src = np.random.default_rng(1).integers(0, 256, (3 << 20) + 17, dtype=np.uint8)
    dst = np.zeros_like(src)
    lib.limited_copy(allowed, 7, dst.ctypes.data, src.ctypes.data, src.nbytes, 20)
    np.testing.assert_array_equal(dst, src)
