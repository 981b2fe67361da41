"""The host loops over several threads (host_parallel.h), compiled and run on the CPU: every element is
visited once, also where a thread cannot be started or there is no memory to start one."""
import subprocess

import pytest

from totem_b200 import build

# operator new fails from the ``left``-th call on (a thread's start is one); -1 never
PROGRAM = r"""
#include <cstdio>
#include <new>
#include "host_parallel.h"
static long left = -1;
void* operator new(std::size_t n) {
  if (left == 0) throw std::bad_alloc();
  if (left > 0) --left;
  void* p = std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
static int seen[100003];
int main(int argc, char** argv) {
  for (std::size_t n : {0, 1, 7, 8, 4096, 100003}) {
    for (std::size_t i = 0; i < n; ++i) seen[i] = 0;
    left = std::atol(argv[1]);
    totem::host_parallel(n, 3, [&](std::size_t lo, std::size_t hi) {
      for (std::size_t i = lo; i < hi; ++i) ++seen[i];
    });
    left = -1;
    for (std::size_t i = 0; i < n; ++i)
      if (seen[i] != 1) return std::printf("%zu of %zu: %d\n", i, n, seen[i]), 1;
  }
  return std::puts("ok"), 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_parallel")
    (d / "m.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", build.CSRC, str(d / "m.cpp"), "-o", str(d / "m")], check=True)
    return str(d / "m")


@pytest.mark.parametrize("allocations", [-1, 0, 1, 2, 3, 6, 7])
def test_every_element_once_whatever_threads_start(program, allocations):
    r = subprocess.run([program, str(allocations)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
