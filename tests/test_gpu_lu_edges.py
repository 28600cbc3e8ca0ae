"""The cluster forms of the LU solve against the single-CTA form, bit for bit:
a system bordered by an identity to more than 192 unknowns takes the single-CTA
form, whose operations on the original unknowns are the same."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 2, 8, 9, 31, 32, 33, 64, 65, 96, 161, 191, 192])
@pytest.mark.parametrize("scale", [0, 30, 140])
def test_cluster_lu_is_the_single_cta_form(cuda, P, scale):
    """``scale``: rows over 10^+-scale, so that quotients leave the range of the
    reciprocal form on both sides."""
    import torch
    from fluxvortex_gb300 import _capi
    lib = _capi.load()
    rng = np.random.default_rng(1000 * scale + P)
    A = rng.standard_normal((2, P, P)) * 10.0 ** rng.uniform(-scale, scale, (2, P, 1))
    b = rng.standard_normal((2, P))
    n = 256
    big = np.tile(np.eye(n), (2, 1, 1))
    big[:, :P, :P] = A
    rhs = np.zeros((2, n))
    rhs[:, :P] = b
    dev = [torch.as_tensor(v, device="cuda").contiguous() for v in (A, b, A, b, big, rhs)]
    work = torch.empty(2 * lib.fvx_lu_workspace_bytes(P) // 8, dtype=torch.float64, device="cuda")
    p = [t.data_ptr() for t in dev]
    _capi.check(lib.fvx_lu_solve_batched(2, P, p[0], p[1], None))
    _capi.check(lib.fvx_lu_factor_batched(2, P, p[2], work.data_ptr(), None))
    _capi.check(lib.fvx_lu_solve_factored_batched(2, P, work.data_ptr(), p[3], None))
    _capi.check(lib.fvx_lu_solve_batched(2, n, p[4], p[5], None))
    torch.cuda.synchronize()
    assert _capi.status_read_and_clear() == 0
    assert torch.equal(dev[1], dev[5][:, :P])
    assert torch.equal(dev[3], dev[5][:, :P])
