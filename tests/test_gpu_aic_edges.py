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


# on the corners, on and around the legs' lines and just inside and outside of the
# skip tolerances (1e-10 of a leg); without a core the points next to them are
# ill conditioned in r3 = d_a x d_b: its products round by eps / 2 |d_a||d_b|
# and |r3| is 1e-10 |d_a||d_b| at least, so kernel and oracle, each with 4 eps /
# 1e-10 = 1e-5, agree to 2e-5
@pytest.mark.parametrize("core,tol", [(RC0, 1e-12), (0.0, 2e-5)])
def test_points_on_and_near_the_skip_tolerances(cuda, core, tol):
    m = 40
    c = _rings(m, 3)
    c[1][5] = c[0][5]                  # zero-length legs
    c[3][9] = c[2][9]
    leg = c[1] - c[0]
    length = np.linalg.norm(leg, axis=1, keepdims=True)
    side = np.cross(leg, [0.3, 0.2, 1.0])
    side /= np.maximum(np.linalg.norm(side, axis=1, keepdims=True), 1e-300)
    pts = [*c, c[0] + 0.37 * leg, c[0] - 2.0 * leg]
    for k in (0.1, 0.9, 1.1, 1.9, 2.1, 10.0, 1e4):
        pts += [c[0] + k * 1e-10 * length * side, c[0] + k * 1e-10 * leg,
                c[0] + 0.5 * leg + k * 0.5e-10 * length * side]
    normal = np.random.default_rng(4).standard_normal((m, 3))
    got = np.concatenate([_aic(p, normal, c, core) for p in pts])
    want = np.concatenate([_aic_oracle(p, normal, c, core) for p in pts])
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


# the fast path's range is lengths of 2^-120 to 2^120 (8e-37 to 1e36); legs below
# 2.22e-16 are skipped whatever the rest
@pytest.mark.parametrize("scale", [1e-16, 3e-14, 1e-3, 1e5, 1e30, 3e35, 1e37, 1e40])
@pytest.mark.parametrize("m", [1, 33])
def test_scales_at_the_ends_of_the_range(cuda, scale, m):
    c = [q * scale for q in _rings(m, 5)]
    rng = np.random.default_rng(6)
    colloc, normal = rng.uniform(-2, 2, (m, 3)) * scale, rng.standard_normal((m, 3))
    got, want = (f(colloc, normal, c, RC0 * scale) for f in (_aic, _aic_oracle))
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
