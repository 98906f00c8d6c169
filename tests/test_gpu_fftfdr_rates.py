"""fftfdr! where the phasor kernel's forms change: rates of 2^19 / Nt and more (their quarter turns
come from cispif), NaN rates, both in one call with small ones, channel counts beyond the exact
Float32 products 2k * t (Nf >= 2^24), and few bins.

Tolerance: relative L-infinity 2e-5 against the FP32 mirror, as in test_gpu_fftfdr.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-5


@pytest.mark.parametrize("Nf", [4096, 3000])
@pytest.mark.parametrize("rates", [[1e6, 2.0, float("nan"), 1.0], [1.0, float("nan"), 3.0, 4e5, 0.5],
                                   [32767.9, -32768.1], [-1e7, 0.25, 0.5]])
def test_large_and_nan_rates(fdr, oracle, Nf, rates):
    """Every column whose two-for-one partner is finite; a NaN rate gives NaN."""
    Nt = 16
    spec, _ = oracle.synth_spectrogram(Nf, Nt, 2, 20, 20, 4, seed=Nf)
    out = fdr.fftfdr(fdr.fftfdr_workspace(spec), rates).cpu().numpy()
    mws = oracle.fftfdr_workspace(spec)
    for j, r in enumerate(rates):
        pair = [x for x in rates[j & ~1:(j & ~1) + 2]]
        if np.isnan(r):
            assert np.isnan(out[:, j]).all()
        elif not np.isnan(pair).any():
            assert oracle.rel_linf(out[:, j], oracle.fftfdr(mws, [r])[:, 0]) < TOL


@pytest.mark.parametrize("Nf", [4096, 3000, 200000])
def test_columns_do_not_depend_on_other_rates(fdr, oracle, Nf):
    """The same pairs of rates beside large or NaN ones: bit for bit the same columns."""
    spec, _ = oracle.synth_spectrogram(Nf, 16, 2, 20, 20, 4, seed=Nf)
    ws = fdr.fftfdr_workspace(spec)
    alone = fdr.fftfdr(ws, [1.25, -0.5, 3.0, 2.0]).cpu().numpy()
    for more in ([1e6, 5.0], [float("nan"), 1e8], [0.1] * 30):
        both = fdr.fftfdr(ws, [1.25, -0.5, 3.0, 2.0] + more).cpu().numpy()
        assert np.array_equal(alone, both[:, :4])


@pytest.mark.parametrize("Nf", [2 ** 24, 4000 * 5000])
def test_products_beyond_float32(fdr, oracle, Nf):
    rng = np.random.default_rng(Nf)
    spec = rng.exponential(1.0, (Nf, 3)).astype(np.float32)
    rates = [1.5, -0.7, 3e5]
    out = fdr.fftfdr(fdr.fftfdr_workspace(spec), rates).cpu().numpy()
    mws = oracle.fftfdr_workspace(spec)
    for j, r in enumerate(rates):
        assert oracle.rel_linf(out[:, j], oracle.fftfdr(mws, [r])[:, 0]) < TOL
