"""The real transforms of the Fourier-shift workspace (rfft of every time step, irfft back)
over lengths that take each radix of the pass kernels, one or two passes, partial CTAs, odd
column counts, and a prime above 13 (the generic passes).

Tolerance: a radix pass rounds each value a few times at 2^-24 relative to the column's norm;
with at most ten passes and independent roundings the relative L2 error stays below
10 * 2^-24 = 6e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 10 * 2.0 ** -24


@pytest.mark.parametrize("Nf,Nt", [
    (2, 1), (3, 3), (16, 2), (30, 5), (49, 3), (121, 2), (169, 4), (1001, 3), (4096, 7), (5040, 1),
    (8192, 2), (9 * 1001, 3), (10000, 5), (2 ** 14, 3), (13 * 1024, 2), (200000, 3), (3 ** 10, 2),
    (2 ** 20, 3), (17 * 600, 3)])
def test_rfft_and_back(fdr, Nf, Nt):
    rng = np.random.default_rng(Nf + Nt)
    spec = rng.exponential(1.0, (Nf, Nt)).astype(np.float32)
    ws = fdr.fftfdr_workspace(spec)
    F = ws.dest_rfft.cpu().numpy()
    ref = np.fft.rfft(spec.astype(np.float64), axis=0)
    assert np.linalg.norm(F - ref) <= TOL * np.linalg.norm(ref)
    back = fdr.fdshift(ws, 0.0).cpu().numpy()  # no shift: irfft(rfft(spec))
    assert np.linalg.norm(back - spec) <= 2 * TOL * np.linalg.norm(spec)
