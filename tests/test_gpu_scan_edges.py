"""The sort's scans around the sizes where their launches change (256 digit counts
per 1,024 particles; 8,192 elements a tile, 65,536 a CTA)."""

import numpy as np
import pytest
import torch

from fluxvortex_gb300 import _capi
from fluxvortex_gb300.tree import TreeSweeper
from oracle import treecode as OT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 1025, 32768, 32769, 262144, 262145])
def test_every_particle_is_sorted_into_its_cell(cuda, n):
    """The oracle's leaves, and a result for every particle: a scan that is off
    breaks runs of equal keys and writes some particles twice, others never."""
    rng = np.random.default_rng(n)
    pos, gam = rng.uniform(0.0, 1.0, (n, 3)), rng.standard_normal((n, 3))
    tr = OT.build(pos, theta=0.5, leaf_target=64)
    ts = TreeSweeper(theta=0.5, leaf_target=64)
    dev = [torch.as_tensor(v, dtype=torch.float64, device=cuda)
           for v in (pos, gam, np.full(n, 0.01))]
    out = torch.full((n, 3), float("nan"), dtype=torch.float64, device=cuda)
    st = ts.sweep(_capi.PAIR_VELOCITY, "winckelmans", *dev, n, out, None, check=True)
    torch.cuda.synchronize()
    assert st[0] == tr["L"] and st[1] == len(tr["levels"][-1]["start"])
    assert bool(torch.isfinite(out).all())
    assert _capi.status_read_and_clear() == 0
