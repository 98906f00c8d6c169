"""Gradients of the proposal network where the selected bins crowd or meet the ends of the bin
axis: few bins (every window's bin and its neighbours overlap), tile edges, all windows on one
bin, and one sample.

Tolerance: a float32 sum of n products is off by about sqrt(n) 2^-24 relative; the longest chain
has six sums of up to 64 * 5 products, so 6 * sqrt(320) * 2^-24 = 6.4e-6 relative L2 against FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 6 * np.sqrt(320) * 2.0 ** -24


@pytest.mark.parametrize("B,cin,X", [(1, 16, 1), (2, 3, 2), (3, 16, 5), (2, 33, 17), (1, 16, 128),
                                     (4, 16, 255), (2, 16, 256), (3, 33, 257), (2, 64, 600)])
def test_gradients_at_crowded_bins(fdr, oracle, B, cin, X):
    rng = np.random.default_rng(100 * B + cin + X)
    net = fdr.proposal.ProposalNet(nbins=X, cin=cin, max_batch=B, seed=X)
    x = rng.normal(0, 1, (B, cin, X)).astype(np.float32)
    lab = (rng.random((B, 16)) < 0.5).astype(np.float32)
    g, loss = net.gradients(torch.from_numpy(x).cuda(), torch.from_numpy(lab).cuda())
    L, ref = oracle.propose_loss_and_grad(net.get_state()["params"], x, lab, cin, half_weights=True)
    assert abs(loss - L) <= TOL * abs(L)
    assert np.linalg.norm(g.cpu().numpy() - ref) <= TOL * np.linalg.norm(ref)


def test_one_bin_for_all_windows(fdr, oracle):
    """A spike at the last bin of a tile is every window's maximum."""
    B, cin, X = 2, 16, 300
    rng = np.random.default_rng(5)
    net = fdr.proposal.ProposalNet(nbins=X, cin=cin, max_batch=B, seed=9)
    st = net.get_state()
    off = sum(ci * co * k + co for ci, co, k in oracle.propose_layers(cin)[:3])
    st["params"][off:off + 512] = np.abs(st["params"][off:off + 512])  # positive 1x1 layer
    net.set_state(st)
    x = (0.01 * rng.normal(0, 1, (B, cin, X))).astype(np.float32)
    x[:, :, 255] += 10.0
    lab = (rng.random((B, 16)) < 0.5).astype(np.float32)
    g, _ = net.gradients(torch.from_numpy(x).cuda(), torch.from_numpy(lab).cuda())
    _, ref = oracle.propose_loss_and_grad(net.get_state()["params"], x, lab, cin, half_weights=True)
    assert np.linalg.norm(g.cpu().numpy() - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("X,at", [(300, 0), (300, 1), (300, 150), (300, 255), (300, 257), (300, 299), (256, 255)])
def test_nan_outside_the_selected_bins(fdr, X, at):
    """A NaN input makes every sum over the bins that it enters NaN (zero gradients included, up to
    the end of the last tile of 256 bins), and no other: the hidden layers' ReLU takes it to 0."""
    cin, ci = 16, 5
    rng = np.random.default_rng(X + at)
    net = fdr.proposal.ProposalNet(nbins=X, cin=cin, max_batch=2, seed=3)
    x = rng.normal(0, 1, (2, cin, X)).astype(np.float32)
    x[1, ci, at] = np.nan
    lab = (rng.random((2, 16)) < 0.5).astype(np.float32)
    g, _ = net.gradients(torch.from_numpy(x).cuda(), torch.from_numpy(lab).cuda())
    bad = np.isnan(g.cpu().numpy())
    want = np.zeros((32, cin, 5), bool)
    for k in range(5):
        want[:, ci, k] = 0 <= at + 2 - k < -(-X // 256) * 256
    assert (bad[:want.size] == want.ravel()).all() and not bad[want.size:].any()
