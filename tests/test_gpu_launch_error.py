"""A refused kernel launch is reported once: launch() returns the error and the
runtime's last error is clear again, so that the caller's next error check does
not see it. The launch here asks for more threads than a block may have, which
the runtime refuses on the host."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include "mans_internal.h"
__global__ void nothing(int) {}
int main() {
  const cudaError_t e = mans::launch(nothing, 1, 4096, 0, nullptr, 0);
  const cudaError_t left = cudaPeekAtLastError();
  std::printf("%s, left: %s\n", cudaGetErrorName(e), cudaGetErrorName(left));
  return e != cudaSuccess && left == cudaSuccess ? 0 : 1;
}
"""


def test_refused_launch_leaves_no_error(tmp_path):
    src, exe = tmp_path / "launch.cu", tmp_path / "launch"
    src.write_text(SOURCE)
    from mans_b200.build import ARCH
    nvcc = os.environ.get("NVCC", "nvcc")
    subprocess.run([nvcc, *ARCH, "-std=c++17", "-I", os.path.join(ROOT, "mans_b200", "csrc"), "-o",
                    str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
