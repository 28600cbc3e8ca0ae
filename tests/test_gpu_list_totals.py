"""Lists longer than their 32-bit offsets are refused: the totals of the counts are
64-bit sums, not the last prefix sum's wrapped value."""
import numpy as np
import pytest
import torch

from fluxvortex_gb300 import _capi
from fluxvortex_gb300.tree import TreeSweeper

pytestmark = pytest.mark.gpu


# one tile of a CTA, several, the last size and the first beyond one CTA, many
@pytest.mark.parametrize("n", [1, 33, 8192, 8193, 65536, 65537, 1 << 20])
# the greatest counts: 2^31 - 1; totals just below and above 2^32; small ones
@pytest.mark.parametrize("kind", ["greatest", "at 2^32", "small"])
def test_totals_are_64_bit_sums(cuda, n, kind):
    rng = np.random.default_rng(n)
    counts = rng.integers(0, 600, n)
    if kind == "greatest":
        counts[:] = (1 << 31) - 1
    elif kind == "at 2^32":
        counts[:] = min((1 << 32) // n, (1 << 31) - 1)
        counts[-1] += 5 if n > 2 else 0
    d = torch.as_tensor(counts.astype(np.int32), device=cuda)
    tmp = torch.empty(512, dtype=torch.int64, device=cuda)
    lib, st = _capi.load(), torch.cuda.current_stream().cuda_stream
    for inclusive in (0, 1):
        out = torch.full((n + 1,), -7, dtype=torch.int32, device=cuda)
        total = torch.full((1,), -1, dtype=torch.int64, device=cuda)
        _capi.check(lib.fvx_probe_scan(d.data_ptr(), n, inclusive, out.data_ptr(),
                                       total.data_ptr(), tmp.data_ptr(), st))
        want = np.cumsum(counts.astype(np.int64))
        assert int(total) == int(want[-1])
        pre = want if inclusive else want - counts
        assert np.array_equal(out[:n].cpu().numpy().view(np.uint32),
                              (pre & 0xFFFFFFFF).astype(np.uint32))
        assert int(out[n]) == -7


def test_an_empty_list_has_a_total_of_zero(cuda):
    d = torch.zeros(4, dtype=torch.int32, device=cuda)
    total = torch.full((1,), -1, dtype=torch.int64, device=cuda)
    tmp = torch.empty(512, dtype=torch.int64, device=cuda)
    _capi.check(_capi.load().fvx_probe_scan(d.data_ptr(), 0, 0, d.data_ptr(), total.data_ptr(),
                                            tmp.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))
    assert int(total) == 0


def test_a_list_that_wraps_to_a_small_number_is_refused(cuda):
    """Leaves of single particles that nothing opens: the near list has leaves^2
    entries, 2^32 and some 5 x 10^8 here; nothing is filled."""
    n, m = 41 ** 3, 41
    g = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) / m
    dev = [torch.as_tensor(v, dtype=torch.float64, device=cuda)
           for v in (g, np.full((n, 3), 1e-3), np.full(n, 0.02))]
    ts = TreeSweeper(theta=1e-3, leaf_target=1)
    out = torch.empty((n, 3), dtype=torch.float64, device=cuda)
    with pytest.raises(_capi.FvxError, match="too long"):
        ts.sweep(_capi.PAIR_VELOCITY, "winckelmans", *dev, n, out)
    torch.cuda.synchronize()
    ts.theta = 0.5             # the handle is usable afterwards
    ts.sweep(_capi.PAIR_VELOCITY, "winckelmans", *dev, n, out)
    assert bool(torch.isfinite(out).all())
    assert _capi.status_read_and_clear() == 0
