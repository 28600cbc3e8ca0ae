"""The FP64 sums of the judge's classes, on both forms of their core."""

import numpy as np
import pytest
import torch

from fluxvortex_gb300 import _capi
from fluxvortex_gb300 import kernel as K
from fluxvortex_gb300.tree import TreeSweeper

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["velocity", "stretch"])
@pytest.mark.parametrize("core,scale", [(0.05, 1.0), (1e-7, 1.0), (40.0, 1000.0)])
def test_far_cloud_is_summed_in_fp64(cuda, mode, core, scale):
    """A cloud of no strength sees another one ten lengths away only through
    cells, and tol ~ 0 sends every class to FP64: what it gets is the direct sum, to
    the rounding of 700 FP64 terms (700 x 2^-53 of their magnitudes' sum, some ten
    roundings each).  Cores and offsets within the three-float range, a core below
    it, offsets beyond it."""
    rng = np.random.default_rng(5)
    n = 700
    pos = rng.uniform(0.0, 1.0, (2 * n, 3))
    pos[n:, 0] += 10.0
    pos *= scale
    gam = rng.standard_normal((2 * n, 3))
    tgt_gam = gam.copy()
    gam[:n] = 0.0
    sig = np.full(2 * n, core)
    P, G, S, T = [torch.as_tensor(v, dtype=torch.float64, device=cuda)
                  for v in (pos, gam, sig, tgt_gam)]
    ts = TreeSweeper(theta=0.5, leaf_target=16)
    ts.set_far_field("m2l")
    ts.set_validation(samples=65536, tol=1e-30)
    out = torch.empty((2 * n, 3), dtype=torch.float64, device=cuda)
    m = _capi.PAIR_VELOCITY if mode == "velocity" else _capi.PAIR_STRETCH
    stats = ts.sweep(m, "winckelmans", P, G, S, 2 * n, out, None,
                     tgt_gamma=T if mode == "stretch" else None, check=True)
    torch.cuda.synchronize()
    assert int(stats[4]) > 0 and ts.last_validation()["fallback"] > 0
    if mode == "velocity":
        ref = K.velocity_from_particles(P[:n].contiguous(), P, G, S, "winckelmans", "f64")
    else:
        ref = K.stretching_from_particles(P[:n].contiguous(), T[:n].contiguous(), P, G, S,
                                          "winckelmans", "f64")
    d = np.linalg.norm(pos[:n, None] - pos[None, n:], axis=2)
    size = np.linalg.norm(gam[n:], axis=1) / (4 * np.pi)
    size = ((size / d ** 2).sum(1) if mode == "velocity" else
            (size * 4 / d ** 3).sum(1) * np.linalg.norm(tgt_gam[:n], axis=1))
    err = (out[:n] - torch.as_tensor(ref, device=cuda)).abs().max(1).values.cpu().numpy()
    assert np.all(err <= 710 * 2.0 ** -53 * size)
    assert _capi.status_read_and_clear() == 0
