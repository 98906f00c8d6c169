"""quarter_rest, the integer part of the fused kernels' phases, compiled for the host with the
undefined-behaviour sanitizer: edges of the quadrants and random phases."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "frequencydriftratetransforms.jl_b200", "csrc")

PROGRAM = r"""
#include <stdio.h>
#include "fdr_internal.cuh"
static int check(unsigned u) {
  unsigned q = 99;
  const int r = fdr::quarter_rest((int)u, &q);
  const long long turn = 1LL << 32, whole = (long long)q * (turn / 4) + r;
  const bool ok = q < 4 && r >= -(1 << 29) && r < (1 << 29) && (whole - (long long)u) % turn == 0;
  if (!ok) printf("phase %08x: q %u rest %d\n", u, q, r);
  return ok ? 0 : 1;
}
int main() {
  int bad = 0;
  for (unsigned e = 0; e < 8; ++e)
    for (unsigned d = 0; d < 5; ++d) bad += check((e << 29) + d - 2u);
  unsigned u = 1;
  for (int i = 0; i < 1000000; ++i) bad += check(u = u * 1664525u + 1013904223u);
  return bad ? 1 : 0;
}
"""


def test_quarter_rest_without_overflow(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "quarter.cu", tmp_path / "quarter"
    src.write_text(PROGRAM)
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
             "-Xcompiler", "-fsanitize=undefined", "-Xcompiler", "-fno-sanitize-recover=all"]
    r = subprocess.run([nvcc, *flags, "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
