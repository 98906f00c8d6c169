"""Error of zdtfdr! against the FP64 sums in every czt kernel, within what its rounding steps account for.

Bound on the relative L2 error, eps = 2^-24: each of the 2 log2(Nf) halving levels of the two transforms and
each of the Nt terms of a sum adds an independent error of at most eps rms, sqrt(2 log2(Nf) + Nt) eps together.
The rounding of a rate's start phase (at most eps / 2 per component) enters with the step's distance u from
the middle, Nt / (2 sqrt(3)) rms, for the noise alone: at bin 0, which holds all but 1 / (Nt + 1) of the
squared norm of a sum of exponential(1) steps, every phase is exactly 1."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nf,Nt,Nr", [
    (1 << 12, 16, 17), (1 << 16, 16, 33), (1 << 20, 16, 24), (1 << 21, 16, 12),  # F in registers
    (1 << 13, 24, 33), (1 << 14, 64, 33),                                        # sums, then transforms
    (1 << 15, 32, 33), (1 << 18, 32, 33), (1 << 17, 64, 33),                     # side by side
    (1 << 20, 64, 12), (1 << 20, 33, 12)])                                       # clusters
def test_error_against_float64(fdr, oracle, Nf, Nt, Nr):
    spec = np.asfortranarray(np.random.default_rng(Nf + Nt).exponential(size=(Nf, Nt)).astype(np.float32))
    r0, dr = -2.0, 1 / 8
    ws = fdr.ZDTWorkspace(spec, r0, dr, Nr)
    assert ws.fused
    want = oracle.fdr_truth(spec, [r0 + j * dr for j in range(Nr)])
    err = oracle.rel_l2(fdr.zdtfdr(ws).cpu().numpy(), want)
    eps = 2.0 ** -24
    bound = eps * (math.sqrt(2 * math.log2(Nf) + Nt) + Nt / (2 * math.sqrt(3)) / math.sqrt(Nt + 1))
    assert err < bound, (err, bound)
