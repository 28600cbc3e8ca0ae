"""Line vortices at the ends of the three-float range (coordinates below 2^13, legs
of 2^-20 to 2^15): vortices and points on either side of it in one call, in one
warp and in one CTA, take different paths.  Against the FP64 oracle at the
path's parity bar of 1e-12 (max |d| / max |ref|), with equal skip counts."""
import numpy as np
import pytest
import torch

from fluxvortex_gb300 import _capi
from fluxvortex_gb300 import aerodynamics as A
from oracle import oracle as O
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-12
FUNCTIONS = ("collapsed_velocities_from_ring_vortices",
             "collapsed_velocities_from_ring_vortices_chordwise_segments",
             "collapsed_velocities_from_horseshoe_vortices",
             "expanded_velocities_from_ring_vortices",
             "expanded_velocities_from_horseshoe_vortices")


def _wake(m, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-2, 2, (m, 3))
    q = [np.array(v, float) for v in ((1, .5, 0), (0, .5, .1), (0, -.5, 0), (1, -.5, .2))]
    return [(o + v + 0.05 * rng.standard_normal((m, 3))) * scale for v in q]


def _check(name, pts, c, core, seed=5):
    m = len(c[0])
    rng = np.random.default_rng(seed)
    s, rc, ages = rng.standard_normal(m), np.full(m, core), rng.uniform(0, 1, m)
    tail = (1.5e-5,) if "horseshoe" in name else (ages, 1.5e-5)
    cg, co = np.zeros(4, np.int64), np.zeros(4, np.int64)
    g = getattr(A, name)(pts, *c, s, rc, cg, *tail)
    o = getattr(O, name)(pts, *c, s, rc, co, *tail)
    assert rel_err(g, o) < TOL
    assert list(cg) == list(co)


# one vortex or point out of range, every other, all; sizes at the edges of the
# expanded CTAs' 64 vortices and of the collapsed ones' 128 points (not so few
# that only pairs thousands of legs apart are left: the oracle loses them)
@pytest.mark.parametrize("name", FUNCTIONS)
@pytest.mark.parametrize("n,m", [(40, 33), (129, 65), (200, 130)])
@pytest.mark.parametrize("out", ["vortex", "vortices", "point", "points", "all"])
def test_both_sides_of_the_range_in_one_call(cuda, name, n, m, out):
    rng = np.random.default_rng(n * 1000 + m)
    c = _wake(m, 3)
    pts = rng.uniform(-2, 2, (n, 3))
    pts[: min(n, m)] = c[1][: min(n, m)]          # points on corners on either side
    far = np.array([0.0, 2.0 ** 13, 0.0])
    if out == "vortex":
        c = [np.where(np.arange(m)[:, None] == m // 2, q + far, q) for q in c]
    elif out == "vortices":
        c[1] = np.where(np.arange(m)[:, None] % 2 == 0, c[0], c[1])     # legs of length zero
    elif out == "point":
        pts[n // 2] += far
    elif out == "points":
        pts[::2] += far
    else:
        pts, c = pts * 1e4, [q * 1e4 for q in c]
    _check(name, pts, c, 0.03 * (1e4 if out == "all" else 1.0))


@pytest.mark.parametrize("name", FUNCTIONS)
def test_skip_tolerances_out_of_the_range(cuda, name):
    """Points around 1e-10 of a leg from its ends and its line, legs of 1e4 and
    beyond: the tolerance's root is taken only for such points."""
    m = 33
    c = _wake(m, 7, 1e4)
    leg = c[1] - c[0]
    side = np.cross(leg, [0.3, 0.2, 1.0])
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    length = np.linalg.norm(leg, axis=1, keepdims=True)
    pts = [c[0], c[1], c[2], c[3], c[0] + 0.37 * leg, c[0] - 2.0 * leg]
    for k in (0.9, 1.1, 10.0, 1e4, 1e9):
        pts += [c[0] + k * 1e-10 * length * side, c[1] + k * 1e-10 * leg]
    for j in (0, 17, 32):
        _check(name, np.concatenate([p[j:j + 1] for p in pts]), [q[j:j + 1] for q in c], 300.0)
    _check(name, np.concatenate(pts), c, 300.0)


# odd counts over several blocks of 128 points: runs that start at odd vortices, where
# no bulk copy is aligned; runs of less than a tile, around it and of several;
# arrays of their own alignment and 8 bytes off it
@pytest.mark.parametrize("name", FUNCTIONS[:3])
@pytest.mark.parametrize("n,m", [(129, 1), (129, 3), (300, 101), (1000, 333), (2500, 1025),
                                 (2500, 1153), (9001, 577)])
@pytest.mark.parametrize("offset", [0, 1])
def test_runs_from_odd_vortices(cuda, name, n, m, offset):
    rng = np.random.default_rng(m)
    c = _wake(m, 9)
    pts = rng.uniform(-2, 2, (n, 3))
    s, rc, ages = rng.standard_normal(m), np.full(m, 0.03), rng.uniform(0, 1, m)

    def device(a):
        flat = torch.empty(a.size + offset, dtype=torch.float64, device=cuda)[offset:]
        return flat.copy_(torch.as_tensor(a.reshape(-1))).reshape(a.shape)

    tail = (1.5e-5,) if "horseshoe" in name else (ages, 1.5e-5)
    co = np.zeros(4, np.int64)
    want = getattr(O, name)(pts, *c, s, rc, co, *tail)
    cg = torch.zeros(4, dtype=torch.int64, device=cuda)
    tail = (1.5e-5,) if "horseshoe" in name else (device(ages), 1.5e-5)
    got = getattr(A, name)(*[device(a) for a in (pts, *c, s, rc)], cg, *tail)
    assert rel_err(got.cpu().numpy(), want) < TOL
    assert cg.tolist() == list(co)
    assert _capi.status_read_and_clear() == 0
