"""One training step of the far-field network: what a call leaves to its caller, and
the step in one kernel against the same by the separate entry points."""
import torch
import pytest

from fluxvortex_gb300 import _capi
from fluxvortex_gb300 import learned as L

pytestmark = pytest.mark.gpu


def _batch(rows, seed):
    g = torch.Generator().manual_seed(seed)
    X = (0.5 * torch.randn(rows, L.IN, generator=g)).to(torch.bfloat16)
    X[:, L.NFEAT:] = 0.0
    return X.cuda(), (0.3 * torch.randn(rows, L.OUT, generator=g)).cuda()


def test_a_loss_outlives_batches_of_other_sizes(cuda):
    """As a loop that keeps the full batches' last loss over a ragged one, and back."""
    net = L.FarFieldMLP(seed=1)
    kept = []
    for k, rows in enumerate((256, 130, 256, 256, 7)):
        loss, _ = net.gradients(*_batch(rows, k))
        if k == 3:             # (of as many rows as the one before, which it overwrites)
            kept.pop()
        kept.append((loss, float(loss), net.gw, float(net.gw.abs().sum())))
    assert all(float(loss) == value and value > 0.0 for loss, value, _, _ in kept)
    assert all(gw is net.gw for _, _, gw, _ in kept)
    again, _ = L.FarFieldMLP(seed=1).gradients(*_batch(7, 4))
    assert float(again) == pytest.approx(kept[-1][1], rel=1e-6)


def _step_by_step(net, X, T, weights):
    """The batch by the separate C entry points: forward with stores, loss gradient,
    and per layer GEMMs, SiLU backward and column sums."""
    lib, st = net.lib, torch.cuda.current_stream().cuda_stream
    rows, dev = X.shape[0], X.device
    Y, Z, H = net.forward(X, store=True)
    dY = torch.empty(rows, L.OUT, dtype=torch.bfloat16, device=dev)
    dY32, dH = torch.empty(rows, L.OUT, device=dev), torch.empty(rows, L.HID, device=dev)
    dZ = torch.empty(rows, L.HID, dtype=torch.bfloat16, device=dev)
    loss, gw, gb = torch.zeros(1, device=dev), torch.zeros_like(net.w32), torch.zeros_like(net.b)

    def gemm(a, lda, ta, b, ldb, tb, c, ldc, m, n, k, split, add):
        _capi.check(lib.fvx_mlp_gemm(a.data_ptr(), lda, ta, b.data_ptr(), ldb, tb, c.data_ptr(),
                                     ldc, m, n, k, split, add, st))

    _capi.check(lib.fvx_mlp_loss_grad(rows, Y.data_ptr(), T.data_ptr(),
                                      None if weights is None else weights.data_ptr(),
                                      dY.data_ptr(), dY32.data_ptr(), loss.data_ptr(), st))
    split = max(1, rows // 128)
    gemm(dY, L.OUT, 1, H[2], L.HID, 1, gw[L.W_OFFSETS[3]:], L.HID, L.OUT, L.HID, rows, split, 1)
    _capi.check(lib.fvx_mlp_colsum(rows, L.OUT, dY32.data_ptr(), gb[L.B_OFFSETS[3]:].data_ptr(),
                                   st))
    gemm(dY, L.OUT, 0, net.wb[L.W_OFFSETS[3]:], L.HID, 1, dH, L.HID, rows, L.HID, L.OUT, 1, 0)
    for l in (2, 1, 0):
        n_in, inp = (L.HID, H[l - 1]) if l else (L.IN, X)
        _capi.check(lib.fvx_mlp_silu_back(rows, L.HID, dH.data_ptr(), Z[l].data_ptr(),
                                          dZ.data_ptr(), gb[L.B_OFFSETS[l]:].data_ptr(), st))
        gemm(dZ, L.HID, 1, inp, n_in, 1, gw[L.W_OFFSETS[l]:], n_in, L.HID, n_in, rows, split, 1)
        if l:
            gemm(dZ, L.HID, 0, net.wb[L.W_OFFSETS[l]:], n_in, 1, dH, L.HID, rows, L.HID, L.HID,
                 1, 0)
    return loss, Y, gw, gb


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 500, 1300])
@pytest.mark.parametrize("weighted", [False, True])
def test_one_kernel_and_the_separate_entries_agree(cuda, rows, weighted):
    """Same operations and roundings per row, so Y is the same; sums in another order.
    The loss: up to 30 x 1,300 FP32 terms, 1e-5.  Gradients: FP32 sums in another
    order (2^-24 of the terms, which cancel to a sixth of their root-mean-square
    sum at worst) may round a few of the BF16 dZ the other way, 2^-8 of it; one in
    2^12 of them is 2^-14 of a gradient's norm.  1e-3 leaves a factor of 16."""
    net = L.FarFieldMLP(seed=3)
    X, T = _batch(rows, rows)
    w = None
    if weighted:
        w = torch.rand(rows, generator=torch.Generator().manual_seed(9)).cuda() * 3.0
    loss, Y = net.gradients(X, T, w)
    loss_s, Y_s, gw_s, gb_s = _step_by_step(net, X, T, w)
    assert torch.equal(Y, Y_s)
    assert abs(float(loss) - float(loss_s)) <= 1e-5 * float(loss_s)
    for l in range(4):
        for g, s, at in ((net.gw, gw_s, L.W_OFFSETS), (net.gb, gb_s, L.B_OFFSETS)):
            end = at[l + 1] if l < 3 else g.numel()
            a, b = g[at[l]:end].double(), s[at[l]:end].double()
            assert float((a - b).norm()) <= 1e-3 * float(b.norm())
