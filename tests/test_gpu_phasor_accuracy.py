"""The phasors of fftfdr!: cos and sin of Float32 half-turns by the packed polynomials against float64,
in rms and at most no further off than sincospif, over the ranges of small and large arguments."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "frequencydriftratetransforms.jl_b200", "csrc")

PROGRAM = r"""
#include <stdio.h>
#include "fdr_internal.cuh"
using namespace fdr;
__device__ double sums[2];
__device__ unsigned long long most[2];
// random half-turns h in (-range, range): sincospif (0) and the packed polynomials (1)
__global__ void errors(unsigned n, float range) {
  double s[2] = {0, 0}, m[2] = {0, 0};
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    unsigned long long z = (i + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    const float h = (float)(long long)(z ^ (z >> 31)) * (1.f / 9223372036854775808.f) * range;
    double ds, dc;
    sincospi((double)h, &ds, &dc);
    const float2 p = cispif(h);
    const float2 h2 = pk_set(h + h), q = pk_add(h2, pk_set(12582912.f));
    const float2 rest = csub(h2, pk_add(q, pk_set(-12582912.f)));
    float2 c, sn;
    cis_quarter_pk<true>(rest, __float_as_uint(q.x), __float_as_uint(q.y), c, sn);
    const double e[2][2] = {{p.x - dc, p.y - ds}, {c.x - dc, sn.y - ds}};
    for (int k = 0; k < 2; ++k)
      for (int j = 0; j < 2; ++j) {
        s[k] += e[k][j] * e[k][j];
        m[k] = fmax(m[k], fabs(e[k][j]));
      }
  }
  for (int k = 0; k < 2; ++k) {
    atomicAdd(&sums[k], s[k]);
    atomicMax(&most[k], (unsigned long long)__double_as_longlong(m[k]));
  }
}
int main() {
  const float ranges[] = {1.f, 5.f, 80.f, 4000.f, 500000.f};
  int bad = 0;
  for (float r : ranges) {
    double s[2] = {0, 0}, m[2] = {0, 0};
    cudaMemcpyToSymbol(sums, s, sizeof(s));
    cudaMemcpyToSymbol(most, m, sizeof(m));
    errors<<<1184, 256>>>(1u << 24, r);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpyFromSymbol(s, sums, sizeof(s));
    cudaMemcpyFromSymbol(m, most, sizeof(m));
    printf("range %g: rms %.4e and %.4e, most %.3e and %.3e\n", r, sqrt(s[0] / (1u << 25)), sqrt(s[1] / (1u << 25)), m[0], m[1]);
    bad += !(s[1] <= s[0]) || !(m[1] <= m[0]);
  }
  return bad ? 1 : 0;
}
"""


def test_phasors_no_further_off_than_sincospif(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "phasor.cu", tmp_path / "phasor"
    src.write_text(PROGRAM)
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
