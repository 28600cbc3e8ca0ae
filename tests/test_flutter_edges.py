"""The flutter kernel at the edges of its splits: panel counts on both sides of
a warp and of the cluster's row shares, threads below three per point, particle
stores smaller than one step's edges; and the mixed-precision offset (three floats
per coordinate) against the rounded FP64 difference it stands for."""
import numpy as np
import pytest

from fluxvortex_gb300.flutter import FlutterSweep, goland


@pytest.mark.gpu
@pytest.mark.parametrize("nc,ns,threads,envs,store", [
    (2, 8, 32, 1, 48), (2, 8, 512, 90, 20), (4, 16, 128, 2, 33), (4, 16, 512, 80, 1),
    (2, 16, 64, 80, 31), (3, 16, 96, 2, 2048), (8, 4, 64, 3, 7)])
def test_shapes_match_oracle(cuda, nc, ns, threads, envs, store):
    from oracle.flutter import FlutterOracle
    cfg = goland(num_chords=5.0, n_keep=2, nc=nc, ns=ns, max_particles=store)
    V = np.linspace(110.0, 150.0, envs)
    sw = FlutterSweep(cfg, V, precision="f64", threads=threads)
    sw.run()
    hw, ht = sw.histories()
    for e in {0, envs - 1}:
        w, th = FlutterOracle(cfg, V[e]).run()
        # the bar of the histories' parity test
        assert np.abs(hw[e] - w).max() <= 1e-9 * np.abs(w).max(), e
        assert np.abs(ht[e] - th).max() <= 1e-9 * np.abs(th).max(), e
    from fluxvortex_gb300 import _capi
    assert _capi.status_read_and_clear() == 0


def _split(x):
    h = x.astype(np.float32)
    y = x - h.astype(np.float64)
    lo = y.astype(np.float32)
    return h, lo, (y - lo.astype(np.float64)).astype(np.float32)


@pytest.mark.parametrize("kind", ["apart", "near", "ties", "floats", "equal"])
def test_difference_in_parts_is_the_rounded_fp64_difference(kind):
    """The kernel's diff_f32 restated in NumPy: wherever it does not send the
    pair to the FP64 way, its float is that of the FP64 difference."""
    rng = np.random.default_rng(17)
    n = 400000
    f32, f64 = np.float32, np.float64
    x = rng.uniform(-20, 20, n)
    y = rng.uniform(-20, 20, n)
    if kind == "near":
        y = x + rng.standard_normal(n) * 2.0 ** -rng.integers(0, 50, n)
    elif kind == "ties":
        f = (x - y).astype(f32)
        mid = 0.5 * (f.astype(f64) + np.nextafter(f, f32(np.inf)))
        y = np.nextafter(x - mid, np.where(rng.random(n) < 0.5, np.inf, -np.inf))
    elif kind == "floats":
        x = x.astype(f32).astype(f64)
        y = x * (1.0 + 2.0 ** -rng.integers(8, 52, n).astype(f64))
    elif kind == "equal":
        y = x.copy()
    (xh, xl, xr), (yh, yl, yr) = _split(x), _split(y)
    h = xh - yh
    bb = h - xh
    e = (xh - (h - bb)) - (yh + bb)
    a, b = xl - yl, xr - yr
    low = e + (a + b)
    t = (np.abs(e) + (np.abs(a) + np.abs(b))) * f32(2.0 ** -22)
    w = (np.abs(h).astype(f64) * 2.0 ** -52 + t.astype(f64)).astype(f32)   # fma: one rounding
    r0, r1 = h + (low - w), h + (low + w)
    ref = (x - y).astype(f32)
    same = r0 == r1
    assert np.array_equal(r0[same], ref[same])
    if kind in ("apart", "equal"):
        assert same.mean() > 0.9999
