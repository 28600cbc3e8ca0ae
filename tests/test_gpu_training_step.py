"""One training step of the far-field network: what a call leaves to its caller."""
import torch
import pytest

from fluxvortex_gb300 import learned as L

pytestmark = pytest.mark.gpu


def _batch(rows, seed):
    g = torch.Generator().manual_seed(seed)
    X = (0.5 * torch.randn(rows, L.IN, generator=g)).to(torch.bfloat16)
    X[:, L.NFEAT:] = 0.0
    return X.cuda(), (0.3 * torch.randn(rows, L.OUT, generator=g)).cuda()


def test_a_loss_outlives_batches_of_other_sizes(cuda):
    """As a loop that keeps the full batches' last loss over a ragged one, and back."""
    net = L.FarFieldMLP(seed=1)
    kept = []
    for k, rows in enumerate((256, 130, 256, 256, 7)):
        loss, _ = net.gradients(*_batch(rows, k))
        if k == 3:             # (of as many rows as the one before, which it overwrites)
            kept.pop()
        kept.append((loss, float(loss), net.gw, float(net.gw.abs().sum())))
    assert all(float(loss) == value and value > 0.0 for loss, value, _, _ in kept)
    assert all(gw is net.gw for _, _, gw, _ in kept)
    again, _ = L.FarFieldMLP(seed=1).gradients(*_batch(7, 4))
    assert float(again) == pytest.approx(kept[-1][1], rel=1e-6)
