"""The four-step twiddles of the pass kernels, products of a coarse and a fine factor from tables in
shared memory, against float64 for lengths across the rule that sets the tables' sizes.

Tolerance, in units of the errors of correctly rounded values (2^-25 at most): the fine factor's
difference from 1 is below 2 pi / 16 = 0.39, so its rounding and those of the two products with it are
below 2^-26 each.  At most 1 + 3 / 2 = 2.5; the rms of the three, uniform and below half that size on
average, adds a tenth to the square of the final rounding's: sqrt(1.12) = 1.06."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "frequencydriftratetransforms.jl_b200", "csrc")

PROGRAM = r"""
#include <stdio.h>
#include "fft_stages.cuh"
using namespace fdr;
__device__ double sums[2];
__device__ unsigned long long most;
// every l of 4 transforms from b0 on: squared errors of the product and of rounded values
template <int SIGN>
__global__ void errors(TwiddleTables t, int L, long long b0, long long N) {
  extern __shared__ float4 sm4[];
  fill_twiddles<SIGN>(t, sm4, 4, L, b0, 2.0 / (double)N);
  __syncthreads();
  const float2* const sm = reinterpret_cast<const float2*>(sm4);
  double s[2] = {0, 0}, m = 0;
  for (int e = threadIdx.x; e < 4 * L; e += blockDim.x) {
    const int i = e & 3, l = e >> 2;
    const float2 w = twiddle_at(sm4 + t.hi + i * t.nh, sm + t.lo + (i << t.lg) + i, t.lg, l);
    double sn, cs;
    sincospi(2.0 * (double)(l * (b0 + i)) / (double)N, &sn, &cs);
    sn *= SIGN;
    const double ex = w.x - cs, ey = w.y - sn, rx = (float)cs - cs, ry = (float)sn - sn;
    s[0] += ex * ex + ey * ey;
    s[1] += rx * rx + ry * ry;
    m = fmax(m, fmax(fabs(ex), fabs(ey)));
  }
  atomicAdd(&sums[0], s[0]);
  atomicAdd(&sums[1], s[1]);
  atomicMax(&most, (unsigned long long)__double_as_longlong(m));
}
int main() {
  const int L1[] = {2, 25, 31, 32, 52, 63, 64, 91, 100, 127, 128, 160, 255, 256, 400, 511, 512, 1000, 1024, 4096, 8192};
  int bad = 0;
  for (int L : L1) {
    const long long L2 = L + 37, N = L * L2;
    StageDesc d;
    memset(&d, 0, sizeof(d));
    d.L = L;
    d.bpc = 4;
    d.SS = 3;
    const TwiddleTables t = twiddle_tables(d);
    const size_t bytes = 4 * 3 * sizeof(float2) + tw_bytes(L, 4);
    double s[2] = {0, 0}, m = 0;
    cudaMemcpyToSymbol(sums, s, sizeof(s));
    cudaMemcpyToSymbol(most, &m, sizeof(m));
    for (long long b0 = 0; b0 + 4 <= L2; b0 += (L2 + 39) / 40) {
      if (b0 % 2) errors<+1><<<1, 256, bytes>>>(t, L, b0, N);
      else errors<-1><<<1, 256, bytes>>>(t, L, b0, N);
    }
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    cudaMemcpyFromSymbol(s, sums, sizeof(s));
    cudaMemcpyFromSymbol(&m, most, sizeof(m));
    const double ratio = s[1] > 0 ? sqrt(s[0] / s[1]) : 1.0, top = m * 33554432.0;
    printf("%d: rms %.4f, most %.3f\n", L, ratio, top);
    bad += !(ratio <= 1.06) || !(top <= 2.5);
  }
  return bad ? 1 : 0;
}
"""


def test_twiddles_against_float64(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "twiddles.cu", tmp_path / "twiddles"
    src.write_text(PROGRAM)
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
