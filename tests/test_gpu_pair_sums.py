"""zdtfdr! where the sums by rate pairs about the grid's centre have their edges: step counts at
and beside the middle step's parity and the kernels' limits (1, 2, 15 to 17, 31 to 33, 63, 64),
rate counts that leave half or unused super pairs (1 to 9, 33), every four-step split, one-sided
and descending grids; rate subsets bit for bit against the whole grid in every czt kernel.

Tolerance: relative L-infinity 1e-5 against the FP64 sums, the bound of the other ZDT tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _run(fdr, oracle, Nf, Nt, Nr, r0, dr, cols=None):
    spec, _ = oracle.synth_spectrogram(Nf, Nt, 2, 10.0, 30.0, 2.0, seed=Nf % 1000 + 7 * Nt + Nr)
    ws = fdr.ZDTWorkspace(spec, r0, dr, Nr)
    assert ws.fused
    out = fdr.zdtfdr(ws)
    cols = list(range(Nr)) if cols is None else cols
    got = out[:, cols].cpu().numpy()
    rates = [float(np.float32(r0)) + j * float(np.float32(dr)) for j in cols]
    assert oracle.rel_linf(got, oracle.fdr_truth(spec, rates)) < TOL
    return spec, ws, out


@pytest.mark.parametrize("Nt", [1, 2, 3, 4, 7, 8, 12, 15, 16, 17, 24, 31, 32, 33, 48, 63, 64])
def test_step_counts(fdr, oracle, Nt):
    _run(fdr, oracle, 1 << 12, Nt, 21, -1.25, 0.125)


@pytest.mark.parametrize("Nr", [1, 2, 3, 4, 5, 6, 7, 8, 9, 33])
@pytest.mark.parametrize("Nt", [16, 21, 40])
def test_rate_counts(fdr, oracle, Nr, Nt):
    _run(fdr, oracle, 1 << 14, Nt, Nr, 0.7, -0.1)


@pytest.mark.parametrize("Nf,Nt,Nr", [
    (1 << 12, 16, 24), (1 << 13, 9, 40), (1 << 15, 16, 33), (1 << 16, 16, 33), (1 << 18, 16, 27),
    (1 << 13, 20, 24), (1 << 14, 64, 17), (1 << 17, 32, 26), (1 << 17, 64, 41), (1 << 18, 19, 33),
    (1 << 20, 64, 49), (1 << 20, 33, 24), (1 << 21, 16, 17), (1 << 21, 40, 16)])
def test_rate_subsets_equal_whole_grid(fdr, oracle, Nf, Nt, Nr):
    spec, ws, out = _run(fdr, oracle, Nf, Nt, Nr, -1.5, 1 / 16, cols=[0, Nr // 2, Nr - 1])
    blocks = list(range(Nr // 8))[::-1]
    sub = fdr.fortran_empty(Nf, 8 * len(blocks))
    fdr.zdtfdr_blocks_(sub, ws, spec, blocks, w="hamming")
    whole = fdr.zdtfdr(ws, spec, w="hamming")
    for i, b in enumerate(blocks):
        assert (sub[:, 8 * i:8 * i + 8] == whole[:, 8 * b:8 * b + 8]).all()
