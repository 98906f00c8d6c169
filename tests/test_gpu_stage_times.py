"""Stage times of a staged zdtfdr!: a time of its own for each stage, the FDR of an untimed call.

The two FDRs differ by the order of the convolution's stages only: relative L-infinity 1e-5, the
bound of the other ZDT tests."""
import pytest

pytestmark = pytest.mark.gpu


def test_every_stage_has_its_own_time(fdr, oracle):
    Nf, Nt, Nr = 100000, 21, 81
    spec, _ = oracle.synth_spectrogram(Nf, Nt, 2, 10.0, 30.0, 2.0, seed=3)
    ws = fdr.ZDTWorkspace(spec, -4.0, 0.1, Nr)
    assert not ws.fused
    plain = fdr.zdtfdr(ws, spec).cpu().numpy()
    ws.set_timing(True)
    fdr.zdtfdr(ws, spec)
    ws.stage_times()
    timed = fdr.zdtfdr(ws, spec).cpu().numpy()
    times = ws.stage_times()
    assert [n for n, _ in times] == ["input", "preprocess", "convolve", "postprocess", "output"]
    t = dict(times)
    # convolve! reads and writes all of Y twice and reads V, postprocess! all of Ys once,
    # preprocess! writes Y once
    assert t["convolve"] > t["preprocess"] and t["postprocess"] > 0.1 * t["preprocess"]
    assert oracle.rel_linf(timed, plain) < 1e-5
