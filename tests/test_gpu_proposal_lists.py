"""The lists of bins that the proposal network's backward pass builds for its three hidden layers
(144, 80 and 16 bins when the selected bins lie apart): the same gradients on every pass, bit for
bit, and those of the oracle.

Tolerance: as in test_gpu_proposal_backward.py, 6 * sqrt(320) * 2^-24 = 6.4e-6 relative L2."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 6 * np.sqrt(320) * 2.0 ** -24


@pytest.mark.parametrize("B,X", [(8, 2048), (1, 700)])
def test_gradients_repeat_bit_for_bit(fdr, oracle, B, X):
    cin = 4
    rng = np.random.default_rng(B + X)
    net = fdr.proposal.ProposalNet(nbins=X, cin=cin, max_batch=B, seed=X)
    x = rng.normal(0, 1, (B, cin, X)).astype(np.float32)
    lab = (rng.random((B, 16)) < 0.5).astype(np.float32)
    xd, ld = torch.from_numpy(x).cuda(), torch.from_numpy(lab).cuda()
    first = net.gradients(xd, ld)[0].clone()
    for _ in range(200):
        assert torch.equal(net.gradients(xd, ld)[0], first)
    _, ref = oracle.propose_loss_and_grad(net.get_state()["params"], x, lab, cin, half_weights=True)
    assert np.linalg.norm(first.cpu().numpy() - ref) <= TOL * np.linalg.norm(ref)
