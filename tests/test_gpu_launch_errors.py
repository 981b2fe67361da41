"""A launch that fails reports its error once: the next kernel's own check does not find it again.  The
launch asks for more threads than a block may have, which the runtime refuses on the host."""
import subprocess

import pytest

from totem_b200 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "common.cuh"
__global__ void k_nothing(int) {}
int main() {
  for (bool overlap : {false, true}) {
    const cudaError_t e = totem::launch_kernel(k_nothing, 1, 4096, 0, nullptr, overlap, 0);
    const cudaError_t left = cudaGetLastError();
    std::printf("%d %d\n", e != cudaSuccess, left == cudaSuccess);
  }
}
"""


def test_failed_launch_leaves_no_error_behind(tmp_path):
    (tmp_path / "m.cu").write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-I", build.CSRC, "-I", build.INCLUDE,
                    str(tmp_path / "m.cu"), "-o", str(tmp_path / "m")], check=True)
    out = subprocess.run([str(tmp_path / "m")], capture_output=True, text=True, check=True, timeout=120).stdout
    assert out == "1 1\n1 1\n", out
