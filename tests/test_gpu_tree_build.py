"""Cells and moments of the treecode's build at the edges of its blocks (1,024
particles), on a sweep and on the sweep that reuses its structure."""

import numpy as np
import pytest
import torch

from fluxvortex_gb300 import _capi
from fluxvortex_gb300.tree import TreeSweeper
from oracle import treecode as OT
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 9, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("leaf", [1, 24])
def test_build_matches_the_oracle_algorithm(cuda, n, leaf):
    """A dense cloud, a long thin one and repeated positions; 2e-5 is what FP32
    arithmetic leaves of the same algorithm in FP64."""
    rng = np.random.default_rng(n)
    pos = rng.standard_normal((n, 3)) * 0.1
    pos[::3] = rng.uniform([0.0, -0.1, -0.1], [8.0, 0.1, 0.1], size=pos[::3].shape)
    pos[::7] = pos[0]
    gam, sig = rng.standard_normal((n, 3)), np.full(n, 0.05)
    tr = OT.build(pos, theta=0.5, leaf_target=leaf)
    OT.moments(tr, pos, gam)
    u, _ = OT.evaluate(tr, pos, gam, sig, kernel="winckelmans")
    lists = OT.lists(tr)
    ts = TreeSweeper(theta=0.5, leaf_target=leaf)
    dev = [torch.as_tensor(v, dtype=torch.float64, device=cuda) for v in (pos, gam, sig)]
    out = torch.empty((n, 3), dtype=torch.float64, device=cuda)
    for again in range(2):
        if again:
            _capi.check(_capi.load().fvx_tree_hint_same_positions(ts.handle))
        st = ts.sweep(_capi.PAIR_VELOCITY, "winckelmans", *dev, n, out, None, check=True).copy()
        torch.cuda.synchronize()
        assert st[0] == tr["L"] and st[1] == len(tr["levels"][-1]["start"])
        assert st[2] == sum(len(a) for a, _ in lists) and st[3] == sum(len(b) for _, b in lists)
        got = out.cpu().numpy()
        assert rel_err(got, u) < 2e-5 if n > 2 else np.abs(got - u).max() < 2e-5 * (1 + np.abs(u).max())
    assert _capi.status_read_and_clear() == 0
