"""rfft and irfft of the generic engine against float64 on columns of normal numbers, for lengths of each
radix in one pass and two.

Tolerance: a level of radix 2 adds a rounded sum, 0.42 * 2^-24 rms relative (a uniform error of half a unit
in the last place over all mantissas), and about every third level a product with a rounded twiddle,
0.6 * 2^-24; together 0.55 * 2^-24 a level.  With 0.65 for the spread over radices, and three
levels' worth for packing and unpacking: 0.65 * 2^-24 * sqrt(log2(N) + 3) relative L2."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [256, 1000, 1024, 4096, 6000, 8000, 9000, 12000, 14400, 2 ** 14, 20000, 2 ** 16,
                               100000, 200000, 2 ** 18, 2 ** 20])
def test_rms_error(fdr, N):
    tol = 0.65 * 2.0 ** -24 * np.sqrt(np.log2(N) + 3)
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn((max(2, min(400, (1 << 22) // N)), N), device="cuda", generator=g)
    ws = fdr.fftfdr_workspace(x.t())
    F = ws.dest_rfft.clone().t().to(torch.complex128)
    ref = torch.fft.rfft(x.double(), dim=1)
    assert float((F - ref).norm() / ref.norm()) <= tol
    back = fdr.fdshift(ws, 0.0).t().double()  # no shift: irfft of F
    exact = torch.fft.irfft(F, n=N, dim=1)
    assert float((back - exact).norm() / exact.norm()) <= tol
