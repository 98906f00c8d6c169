"""The two-pass real transforms of the generic engine with so many columns that a CTA takes as many
transforms as its shared memory holds: first passes of 52 points (the one length whose padded
buffer and twiddle tables for 128 transforms exceed it), 91, 96 and 128 points.

Tolerance: as in test_gpu_fft_stages.py, ten roundings at 2^-24 of the column's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 10 * 2.0 ** -24


@pytest.mark.parametrize("Nf", [8788, 8918, 9216, 2 ** 14])
@pytest.mark.parametrize("Nt", [294, 297])
def test_rfft_and_back(fdr, Nf, Nt):
    rng = np.random.default_rng(Nf + Nt)
    spec = rng.exponential(1.0, (Nf, Nt)).astype(np.float32)
    ws = fdr.fftfdr_workspace(spec)
    F = ws.dest_rfft.cpu().numpy()
    ref = np.fft.rfft(spec.astype(np.float64), axis=0)
    assert np.linalg.norm(F - ref) <= TOL * np.linalg.norm(ref)
    back = fdr.fdshift(ws, 0.0).cpu().numpy()
    assert np.linalg.norm(back - spec) <= 2 * TOL * np.linalg.norm(spec)
