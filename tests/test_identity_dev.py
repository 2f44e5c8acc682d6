"""identity_dev (common.cuh), compiled for the host: the deviation that decides
whether an environment block is replaced by the exact identity must not pass
over a value of which one part is not a number."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SRC = """
#include "common.cuh"
#include <cstdio>
int main() {
  const double n = NAN, i = INFINITY;
  const double v[][3] = {{1, 0, 1},   {1.5, 0, 1}, {1, -0.25, 1}, {0, 0, 0}, {n, 0, 1}, {1, n, 1},
                         {n, n, 0}, {0, n, 0},   {i, 0, 0},     {0, -i, 0}, {i, n, 0}};
  for (const auto& q : v) printf("%g\\n", identity_dev(make_double2(q[0], q[1]), q[2]));
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_parts_that_are_not_numbers_count_as_infinite(tmp_path):
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run([NVCC, "-arch=sm_100", "-I", os.path.join(ROOT, "yaqs_julia_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0.5", "0.25", "0"] + ["inf"] * 7
