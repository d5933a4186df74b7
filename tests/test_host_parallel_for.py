"""parallel_for (csrc/internal.h), which the plans are built with: an exception
of a worker reaches the caller (it ended the process), and work goes on where no
thread can be started."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dolfin_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cerrno>
#include <cstring>
#include <new>
#include <pthread.h>
#include "internal.h"

#ifdef NO_THREADS
extern "C" int pthread_create(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*) { return EAGAIN; }
#endif

int main() {
  const int64_t n = 1000;
  std::atomic<int64_t> sum{0};
  db2::parallel_for(n, [&](int64_t b, int64_t e) { for (int64_t i = b; i < e; ++i) sum += i; }, 1);
  if (sum != n * (n - 1) / 2) return 1;
  std::atomic<int64_t> done{0};
  try {
    db2::parallel_for(n, [&](int64_t b, int64_t e) {
      done += e - b;
      if (b <= n / 2 && n / 2 < e) throw std::bad_alloc();
    }, 1);
  } catch (const std::bad_alloc&) {
    return done == n ? 0 : 3;
  }
  return 2;
}
"""


@pytest.mark.parametrize("flags", [[], ["-DNO_THREADS"]], ids=["threads", "no threads"])
def test_worker_exception_reaches_the_caller(tmp_path, flags):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-rdynamic", "-I", CSRC, *flags, str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
