"""FP64 particle sweeps at the edges of their tiles, slices and splits, and where
a tile leaves the three-float arithmetic's range (coordinates beyond 2^13, cores
below 2^-22 or beyond 2^13, non-finite values): against the FP64 oracle at the
path's bar of 1e-12 (max |d| / max |ref|)."""
import numpy as np
import pytest

from fluxvortex_gb300 import _capi
from fluxvortex_gb300 import kernel as K
from tests.conftest import rel_err
from tests.test_gpu_particles import MODES, TOL64, _field, _oracle_mode

pytestmark = pytest.mark.gpu


def _check(mode, kernel, t, tg, p, g, s):
    a, b = K.particle_pairs(getattr(_capi, "PAIR_" + mode.upper()), t, tg, p, g, s, kernel, "f64")
    oa, ob = _oracle_mode(mode, t, tg, p, g, s, kernel)
    assert rel_err(a, oa) < TOL64
    if ob is not None:
        assert rel_err(b, ob) < TOL64


@pytest.mark.parametrize("kernel", ["winckelmans", "gaussianerf"])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("M,N", [(1, 2), (1, 4001), (127, 63), (128, 64), (129, 65), (130, 129),
                                 (385, 31), (2049, 130), (20000, 66)])
def test_sizes(cuda, kernel, mode, M, N):
    rng = np.random.default_rng(M + 7 * N)
    p, g, s = _field(rng, N)
    t = rng.uniform([0, -1, -0.2], [2, 1, 0.2], size=(M, 3))
    t[: min(M, N) // 2] = p[: min(M, N) // 2]
    _check(mode, kernel, t, rng.normal(0, 1e-3, size=(M, 3)), p, g, s)


@pytest.mark.parametrize("kernel", ["winckelmans", "gaussianerf"])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("case", ["far source", "far target", "tiny core", "large core", "scaled up",
                                  "scaled down"])
def test_range_of_the_scalar_core(cuda, kernel, mode, case):
    rng = np.random.default_rng(5)
    p, g, s = _field(rng, 300)
    t = np.vstack([p[:50], rng.uniform([0, -1, -0.2], [2, 1, 0.2], size=(100, 3))])
    if case == "far source":
        p[130] = [1e4, 0.0, 3.0]          # one tile of the five
    elif case == "far target":
        t[60] = [0.0, -9000.0, 1.0]
    elif case == "tiny core":
        s[200] = 1e-7
        p[200] = [0.5, 0.5, 0.5]          # not a target: its own core would be all there is
    elif case == "large core":
        s[10] = 1e4
    elif case == "scaled up":
        t, p, s = t * 3000.0, p * 3000.0, s * 3000.0
    else:
        t, p, s = t * 1e-4, p * 1e-4, s * 1e-4
    _check(mode, kernel, t, rng.normal(0, 1e-3, size=(150, 3)), p, g, s)


@pytest.mark.parametrize("kernel", ["winckelmans", "gaussianerf"])
def test_non_finite_and_lone_particles(cuda, kernel):
    rng = np.random.default_rng(8)
    p, g, s = _field(rng, 100)
    t = rng.uniform([0, -1, -0.2], [2, 1, 0.2], size=(5, 3))
    t[2, 1] = np.nan
    u = K.velocity_from_particles(t, p, g, s, kernel)
    assert np.array_equal(np.isnan(u).any(axis=1), [False, False, True, False, False])
    p[70, 0] = np.inf
    assert not np.isfinite(K.velocity_from_particles(t, p, g, s, kernel)).all(axis=1).any()
    # a particle does not move itself
    assert not K.velocity_from_particles(p[:1], p[:1], g[:1], s[:1], kernel).any()


@pytest.mark.parametrize("kernel", ["winckelmans", "gaussianerf"])
def test_scratch_of_the_coarser_split_is_still_enough(cuda, kernel):
    """A caller whose scratch holds six splits' sums (304 KB here) and not this
    kernel's gets the same sums from fewer CTAs; one with less is refused."""
    import torch
    lib = _capi.load()
    rng = np.random.default_rng(9)
    p, g, s = (torch.as_tensor(a, device=cuda) for a in _field(rng, 1501))
    n, out = 1501, torch.empty((1501, 3), dtype=torch.float64, device=cuda)
    kid = _capi.KERNELS[kernel]
    coarse = 6 * n * 24                       # ceil(1501 / 256) splits of three values
    assert lib.fvx_particle_pairs_scratch_bytes(0, 0, n, n) > coarse
    sc = torch.empty(coarse, dtype=torch.uint8, device=cuda)
    st = torch.cuda.current_stream().cuda_stream

    def call(nbytes):
        return lib.fvx_particle_pairs(0, kid, 0, p.data_ptr(), None, n, p.data_ptr(), g.data_ptr(),
                                      s.data_ptr(), n, out.data_ptr(), None, sc.data_ptr(), nbytes,
                                      st)

    assert call(coarse) == _capi.FVX_OK
    ref = K.velocity_from_particles(p, p, g, s, kernel)
    assert rel_err(out.cpu().numpy(), ref.cpu().numpy()) < TOL64
    assert call(coarse - 1) == _capi.FVX_ERR_SCRATCH
