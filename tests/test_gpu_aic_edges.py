"""The influence coefficients (fvx_uvlm_aic) where the FP64 fast path of the line
vortices hands over to its general path: non-finite collocation points."""
import numpy as np
import pytest
import torch

from fluxvortex_gb300 import _capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu
RC0, NU = 0.03, 1.5e-5


def _rings(m, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-2, 2, (m, 3))
    q = [np.array(v, float) for v in ((1, .5, 0), (0, .5, .1), (0, -.5, 0), (1, -.5, .2))]
    return [o + v + 0.05 * rng.standard_normal((m, 3)) for v in q]


def _aic(colloc, normal, corners, rc0=RC0):
    n = len(colloc)
    dev = [torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
           for a in (colloc, normal, *corners)]
    out = torch.empty((n, n), dtype=torch.float64, device="cuda")
    _capi.check(_capi.load().fvx_uvlm_aic(1, n, *[a.data_ptr() for a in dev], rc0, NU,
                                          out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy()


def _aic_oracle(colloc, normal, corners, rc0=RC0):
    m = len(corners[0])
    v = O.expanded_velocities_from_ring_vortices(
        colloc, *corners, np.ones(m), np.full(m, rc0), np.zeros(4, np.int64), np.zeros(m), NU)
    return (v * normal[:, None]).sum(2)


# a NaN's sign is the host's: inf - inf has it set on x86, clear on Arm
@pytest.mark.parametrize("value", [np.nan, np.copysign(np.nan, -1.0), np.inf, -np.inf])
@pytest.mark.parametrize("component", [0, 1, 2])
def test_a_bad_collocation_point_is_not_a_zero_row(cuda, value, component):
    m = 8
    corners = _rings(m, 1)
    rng = np.random.default_rng(2)
    colloc = rng.uniform(-2, 2, (m, 3))
    normal = np.tile([0.6, 0.48, 0.64], (m, 1))
    colloc[3, component] = value
    got, want = _aic(colloc, normal, corners), _aic_oracle(colloc, normal, corners)
    assert np.isnan(want[3]).all() and np.isnan(got[3]).all()
    keep = np.arange(m) != 3
    assert np.abs(got - want)[keep].max() <= 1e-12 * np.abs(want[keep]).max()
