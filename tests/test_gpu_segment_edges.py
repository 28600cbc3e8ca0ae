"""Line-vortex sweeps where their fast path can go wrong: points on corners, on
and next to a leg's line and just inside and outside the skip tolerances,
degenerate legs, cores of zero, values at the ends of the fast path's range and
non-finite ones, and sizes at the edges of the CTAs' runs.  Against the FP64
oracle at the path's parity bar of 1e-12 (max |d| / max |ref|), with equal skip
counts.  Without a core the points next to the tolerances are ill conditioned
in r3 = d_a x d_b alone: its products round by eps / 2 |d_a||d_b| and |r3| is
1e-10 |d_a||d_b| at least, so the oracle and the kernel, each with 4 eps / 1e-10
= 1e-5, agree to 2e-5."""
import numpy as np
import pytest

from fluxvortex_gb300 import aerodynamics as A
from oracle import oracle as O
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-12
COLLAPSED = ("collapsed_velocities_from_ring_vortices",
             "collapsed_velocities_from_ring_vortices_chordwise_segments",
             "collapsed_velocities_from_horseshoe_vortices")
EXPANDED = ("expanded_velocities_from_ring_vortices",
            "expanded_velocities_from_horseshoe_vortices")


def _rings(m, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-2, 2, (m, 3))
    q = [np.array(v, float) for v in ((1, .5, 0), (0, .5, .1), (0, -.5, 0), (1, -.5, .2))]
    c = [(o + v + 0.05 * rng.standard_normal((m, 3))) * scale for v in q]
    return c, rng.standard_normal(m), np.full(m, 0.03 * scale), rng.uniform(0, 1, m)


def _both(name, pts, c, s, rc, ages, nu=1.5e-5):
    cg, co = np.zeros(4, np.int64), np.zeros(4, np.int64)
    tail = (nu,) if "horseshoe" in name else (ages, nu)
    return (getattr(A, name)(pts, *c, s, rc, cg, *tail), cg,
            getattr(O, name)(pts, *c, s, rc, co, *tail), co)


@pytest.mark.parametrize("name", COLLAPSED + EXPANDED)
@pytest.mark.parametrize("core", [0.03, 0.0])
def test_points_on_and_near_the_skip_tolerances(cuda, name, core):
    m = 40
    c, s, rc, ages = _rings(m, 3)
    rc[:] = core
    ages[:] = 0.0 if core == 0.0 else ages
    c[1][5] = c[0][5]                  # zero-length legs
    c[3][9] = c[2][9]
    a, b = c[0], c[1]
    leg = b - a
    length = np.linalg.norm(leg, axis=1, keepdims=True)
    side = np.cross(leg, [0.3, 0.2, 1.0])
    side /= np.maximum(np.linalg.norm(side, axis=1, keepdims=True), 1e-300)
    pts = [a, b, c[2], c[3], a + 0.37 * leg, a - 2.0 * leg]
    for k in (0.1, 0.9, 1.1, 1.9, 2.1, 10.0, 1e4):       # around 1e-10 of the leg
        pts += [a + k * 1e-10 * length * side, a + k * 1e-10 * leg,
                a + 0.5 * leg + k * 0.5e-10 * length * side]
    # one ring at a time: every point against the ring it was made for and its
    # neighbour, so that a single wrong decision shows in a count
    pts = np.stack(pts, axis=1)
    for r in (0, 5, 9, 20, 39):
        k = slice(max(r - 1, 0), r + 1)
        g, cg, o, co = _both(name, pts[r], [x[k] for x in c], s[k], rc[k], ages[k])
        assert np.array_equal(cg, co), (r, cg, co)
        assert np.isfinite(g).all() and rel_err(g, o) < (TOL if core else 2e-5)


@pytest.mark.parametrize("name", COLLAPSED + EXPANDED)
@pytest.mark.parametrize("scale", [1e-12, 1e-6, 1e20, 1e35, 1e36, 1e37, 1e60])
def test_scales_across_the_fast_range(cuda, name, scale):
    c, s, rc, ages = _rings(70, 4, scale)
    ages[:] = 0.0                                          # the core law has a length scale
    pts = np.random.default_rng(5).uniform(-3, 3, (33, 3)) * scale
    pts[0] = c[2][3]
    g, cg, o, co = _both(name, pts, c, s, rc, ages)
    assert np.array_equal(cg, co)
    assert rel_err(g, o) < TOL


@pytest.mark.parametrize("name", COLLAPSED)
def test_non_finite_inputs_stay_where_they_are(cuda, name):
    c, s, rc, ages = _rings(9, 6)
    pts = np.random.default_rng(7).uniform(-3, 3, (130, 3))
    pts[3, 1], pts[64, 0] = np.nan, np.inf
    g = _both(name, pts, c, s, rc, ages)[0]
    bad = ~np.isfinite(g).all(axis=1)
    assert bad[3] and bad[64] and bad.sum() == 2
    s[4] = np.nan
    assert np.isnan(_both(name, pts, c, s, rc, ages)[0]).all()


@pytest.mark.parametrize("n,m", [(1, 1), (1, 5000), (127, 3), (128, 2), (129, 1), (129, 65),
                                 (257, 333), (1000, 64), (4000, 1001), (19457, 77), (38913, 5),
                                 (39000, 130)])
@pytest.mark.parametrize("name", COLLAPSED)
def test_runs_of_any_size(cuda, name, n, m):
    c, s, rc, ages = _rings(m, n)
    pts = np.random.default_rng(m).uniform(-3, 3, (n, 3))
    g, cg, o, co = _both(name, pts, c, s, rc, ages)
    assert np.array_equal(cg, co)
    assert rel_err(g, o) < TOL
