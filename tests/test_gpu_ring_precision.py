"""Line vortices and influence coefficients against extended precision (np.longdouble:
113 bits on Arm, 64 on x86).

Bound of a leg's velocity k S num / den r3, k = Gamma / 8 pi, S = 1/A + 1/B, num =
2 (A B - a.b), den = |r3|^2 + r0^2 rc^2, r3 = a x b, u = 2^-53.  The offsets a, b
round by u in each component, so r3 by 4 u A B in each (two products of two
rounded factors, their rounding and the sum's) and 7 u A B in length; den by 14 u
A B |r3| and its own terms' 6 u; S, the quotient and the products by 14 u.  num:
  FP64, both ends a leg length away, r0^2 - (A - B)^2: the lengths by 3 u, so 4 u
    r0^2 + 8 u r0 (A + B); nearer, 2 (A B - a.b): 24 u A B;
  three floats, lengths to 2^-58: 4 u num + 2^-58 (r0^2 + r0 (A + B)), down to 2^-10 of
    a leg; nearer, as FP64.
A sum of n terms adds n u times their magnitudes.  Roots and reciprocals that are
off by more than a few ulps exceed it, and so does A B - a.b at any distance
(the wake's points are up to 60 legs away)."""
import numpy as np
import pytest
import torch

from fluxvortex_gb300 import _capi
from fluxvortex_gb300 import aerodynamics as A

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
LEGS = {"ring": ((0, 1), (1, 2), (2, 3), (3, 0)), "chordwise": ((0, 1), (2, 3)),
        "horseshoe": ((0, 1), (1, 2), (2, 3))}


def _wake(n, seed):
    rng = np.random.default_rng(seed)
    cols = 10
    rows = -(-n // cols)
    x = 1.0 + 0.15 * np.arange(rows + 1)[:, None] + 0.02 * rng.standard_normal((rows + 1, cols + 1))
    y = np.linspace(-5, 5, cols + 1)[None] + 0.02 * rng.standard_normal((rows + 1, cols + 1))
    v = np.stack([x, y, 0.2 * np.sin(0.8 * x + 0.3 * y)], -1)
    return [np.ascontiguousarray(q.reshape(-1, 3)[:n])
            for q in (v[1:, 1:], v[:-1, 1:], v[:-1, :-1], v[1:, :-1])]


def _reference(legs, pts, c, s, rc, x3):
    """(n, m, 3) velocities in extended precision, their bounds (n, m) and magnitudes."""
    L = np.longdouble
    d = [q.astype(L)[None] - pts.astype(L)[:, None] for q in c]
    n2 = [(q * q).sum(2) for q in d]
    length = [np.sqrt(q) for q in n2]
    v = np.zeros(d[0].shape, L)
    bound = np.zeros(d[0].shape[:2])
    size = np.zeros(d[0].shape[:2])
    k = np.abs(s.astype(L)) / (8 * L(np.pi))
    for a, b in LEGS[legs]:
        r0sq = ((c[b].astype(L) - c[a].astype(L)) ** 2).sum(1)[None]
        r3 = np.cross(d[a], d[b])
        r3sq = (r3 * r3).sum(2)
        AB, dot = length[a] * length[b], (d[a] * d[b]).sum(2)
        num = 2 * np.where(dot > 0, r3sq / (AB + np.abs(dot)), AB - dot)
        den = r3sq + r0sq * (rc.astype(L) ** 2)[None]
        S = 1 / length[a] + 1 / length[b]
        w = S * num / den
        v += (s.astype(L) / (8 * L(np.pi)))[None, :, None] * w[..., None] * r3
        f = lambda q: np.asarray(q, float)  # noqa: E731
        r0, r3n, AB, num, den, kS = (f(q) for q in (np.sqrt(r0sq), np.sqrt(r3sq), AB, num, den,
                                                    k[None] * S))
        sum_, near = f(length[a] + length[b]), np.minimum(f(length[a]), f(length[b])) / r0
        by_dot = 24 * U * AB
        if x3:
            dnum = 4 * U * num + 2.0 ** -58 * (r0 * r0 + r0 * sum_)
            dnum = np.where(near < 2.0 ** -10 * 1.01, np.maximum(dnum, by_dot), dnum)
        else:
            dnum = 4 * U * r0 * r0 + 8 * U * r0 * sum_
            dnum = np.where(near < 1.01, np.maximum(dnum, by_dot), dnum)
        bound += kS / den * (dnum * r3n + num * 7 * U * AB
                             + num * r3n * (14 * U * AB * r3n / den + 20 * U))
        size += kS / den * num * r3n
    return v, bound, size


def _case(m, n, seed):
    rng = np.random.default_rng(seed)
    c = _wake(m, seed)
    pts = np.concatenate([rng.uniform([0, -5, -0.3], [3, 5, 0.3], (n - n // 2, 3)),
                          rng.uniform([1, -5, -0.3], [4, 5, 0.3], (n // 2, 3))])
    pts[::4, 2] *= 1e-3            # in the sheet, between its rings
    return c, pts, 0.3 * rng.standard_normal(m) + 0.5, np.full(m, 0.03)


@pytest.mark.parametrize("legs", sorted(LEGS))
def test_sweeps(cuda, legs):
    m, n = 120, 200
    c, pts, s, rc = _case(m, n, 11)
    v, bound, size = _reference(legs, pts, c, s, rc, True)
    name = {"ring": "ring_vortices", "chordwise": "ring_vortices_chordwise_segments",
            "horseshoe": "horseshoe_vortices"}[legs]
    tail = (15e-6,) if legs == "horseshoe" else (np.zeros(m), 15e-6)
    got = getattr(A, "collapsed_velocities_from_" + name)(pts, *c, s, rc, np.zeros(4, np.int64),
                                                          *tail)
    err = np.abs(got - v.sum(1)).max(1).astype(float)
    assert (err <= bound.sum(1) + 4 * m * U * size.sum(1)).all()
    if legs == "chordwise":
        return
    got = getattr(A, "expanded_velocities_from_" + name)(pts, *c, s, rc, np.zeros(4, np.int64),
                                                         *tail)
    err = np.abs(got - v).max(2).astype(float)
    assert (err <= bound + 16 * U * size).all()


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -31 * 1.3, 2.0 ** 33 * 1.7])
def test_influence_coefficients(cuda, scale):
    m = 120
    c, pts, _, rc = _case(m, m, 12)
    c, pts, rc = [q * scale for q in c], pts * scale, rc * scale
    normal = np.random.default_rng(13).standard_normal((m, 3))
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    v, bound, size = _reference("ring", pts, c, np.ones(m), rc, False)
    dev = [torch.as_tensor(q, dtype=torch.float64, device=cuda) for q in (pts, normal, *c)]
    out = torch.empty((m, m), dtype=torch.float64, device=cuda)
    _capi.check(_capi.load().fvx_uvlm_aic(1, m, *[q.data_ptr() for q in dev], float(rc[0]), 15e-6,
                                          out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    want = (v * normal[:, None].astype(np.longdouble)).sum(2)
    err = np.abs(out.cpu().numpy() - want).astype(float)
    # |error . n| <= |error|: the bound is of each component, so sqrt(3) of it
    assert (err <= np.sqrt(3.0) * (bound + 16 * U * size)).all()
