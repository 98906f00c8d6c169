"""Rate subsets in every form that their rounds of rate pairs take: blocks of which the mirror about
the grid's centre is wanted too (in part, or an odd number of super pairs of them), blocks on one
side, across the centre, in any order and given twice; rate counts with an even and an odd number
of super pairs; each czt kernel, rectangular and Hamming windows.  Bit for bit the whole grid's
columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nf,Nt", [(1 << 13, 16), (1 << 16, 7), (1 << 18, 16), (1 << 13, 24), (1 << 15, 24), (1 << 14, 64),
                                   (1 << 17, 32), (1 << 17, 64), (1 << 20, 40), (1 << 21, 16)])
@pytest.mark.parametrize("Nr", [56, 57, 63, 64, 65])
def test_any_blocks_equal_the_whole_grid(fdr, oracle, Nf, Nt, Nr):
    spec, _ = oracle.synth_spectrogram(Nf, Nt, 2, 10.0, 30.0, 2.0, seed=Nr + Nt)
    ws = fdr.ZDTWorkspace(spec, -1.5, 1 / 16, Nr)
    rng = np.random.default_rng(Nr * Nt)
    nb = Nr // 8
    subsets = [[0], [nb - 1], [nb // 2], [nb // 2 - 1, nb // 2], [nb - 1, 0], [3, 3], [2, 5, 2], list(range(nb)),
               rng.permutation(nb)[:3].tolist(), rng.permutation(nb)[:5].tolist(), rng.integers(0, nb, nb).tolist()]
    if Nf >= 1 << 20:
        subsets = subsets[3:7] + subsets[9:]
    for w in ("rect", "hamming"):
        whole = fdr.zdtfdr(ws, spec, w=w)
        for blocks in subsets:
            sub = fdr.fortran_empty(Nf, 8 * len(blocks))
            fdr.zdtfdr_blocks_(sub, ws, None, blocks, w=w)
            for i, b in enumerate(blocks):
                assert (sub[:, 8 * i:8 * i + 8] == whole[:, 8 * b:8 * b + 8]).all(), (w, blocks, i)
