"""The paired FP32 sweeps at the edges of their tiles (256 targets, 128 sources)
and for cores whose squares FP32 holds only as subnormal numbers."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = [0, 1, 2, 3, 4]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("nt,ns", [(1, 1), (255, 127), (257, 129), (513, 255), (300, 1000)])
@pytest.mark.parametrize("tiny", [False, True])
def test_paired_sweep_against_fp64(cuda, mode, nt, ns, tiny):
    """Coordinates are multiples of 2^-10 (targets half a step off), so that the
    separations are exact in FP32.  A pair's value takes fewer than 64 roundings
    and a tile's sum 128 more: 192 x 2^-24 of the sum of the magnitudes."""
    import torch
    from fluxvortex_gb300 import _capi
    lib = _capi.load()
    rng = np.random.default_rng(mode + 10 * ns)
    pos = rng.integers(-2048, 2048, (ns, 3)) / 1024.0
    tgt = (rng.integers(-2048, 2048, (nt, 3)) + 0.5) / 1024.0
    alpha, tg = rng.standard_normal((ns, 3)), rng.standard_normal((nt, 3))
    sigma = np.full(ns, 0.125)
    if tiny:
        sigma[::5] = 1e-20
    nc = [3, 3, 6, 9, 3][mode]
    dev = [torch.as_tensor(v, device="cuda").contiguous() for v in (tgt, tg, pos, alpha, sigma)]
    p = [v.data_ptr() for v in dev]
    got = []
    for precision in (0, 1):
        a = torch.zeros(nt * (3 if mode == 2 else nc), dtype=torch.float64, device="cuda")
        b = torch.zeros(nt * 3, dtype=torch.float64, device="cuda")
        nb = int(lib.fvx_particle_pairs_scratch_bytes(mode, precision, nt, ns))
        scratch = torch.empty(max(nb, 1), dtype=torch.uint8, device="cuda")
        _capi.check(lib.fvx_particle_pairs(mode, 1, precision, p[0], p[1], nt, p[2], p[3], p[4],
                                           ns, a.data_ptr(), b.data_ptr(), scratch.data_ptr(), nb,
                                           None))
        torch.cuda.synchronize()
        rows = [a.cpu().numpy().reshape(nt, -1)]
        if mode == 2:
            rows.append(b.cpu().numpy().reshape(nt, 3))
        got.append(rows)
    d = tgt[:, None] - pos[None]
    r2, s2 = (d * d).sum(-1), (sigma ** 2)[None]
    f = (r2 + 2.5 * s2) * (r2 + s2) ** -2.5 / (4 * np.pi)
    fp = (3 * r2 + 10.5 * s2) * (r2 + s2) ** -3.5 / (4 * np.pi)
    na = np.linalg.norm(alpha, axis=1)[None]
    vel = (f * np.sqrt(r2) * na).sum(1)
    grad = ((fp * r2 + 2 * f) * na).sum(1)
    size = {0: [vel], 1: [grad * np.linalg.norm(tg, axis=1)],
            2: [vel, grad * np.linalg.norm(tg, axis=1)], 3: [grad], 4: [grad]}[mode]
    assert _capi.status_read_and_clear() == 0
    for want, have, s in zip(got[0], got[1], size):
        assert np.all(np.abs(have - want) <= 192 * 2.0 ** -24 * s[:, None])
