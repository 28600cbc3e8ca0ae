"""The training GEMM's staging at the edges of its wide accesses: odd leading
dimensions, operands and results that start off a 16-byte boundary, and
remainders of the 8-element, 16-column and 128-row steps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K,split", [(1, 1, 1, 1), (129, 31, 7, 1), (127, 129, 300, 2),
                                         (130, 96, 136, 1)])
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (0, 1), (2, 2), (8, 8)])
def test_gemm_strides_and_offsets(cuda, tA, tB, M, N, K, split, pad, off):
    from fluxvortex_gb300 import _capi
    lib = _capi.load()
    g = torch.Generator().manual_seed(M + 3 * N + 7 * K + pad)

    def operand(r, c):
        ld = c + pad
        buf = torch.randn(off + r * ld, generator=g).to(torch.bfloat16)
        return buf.cuda(), buf[off:].reshape(r, ld)[:, :c].double(), ld

    a, ah, lda = operand(*((K, M) if tA else (M, K)))
    b, bh, ldb = operand(*((K, N) if tB else (N, K)))
    ldc = N + pad
    C = torch.zeros(off + M * ldc, dtype=torch.float32, device="cuda")
    _capi.check(lib.fvx_mlp_gemm(a.data_ptr() + 2 * off, lda, tA, b.data_ptr() + 2 * off, ldb, tB,
                                 C.data_ptr() + 4 * off, ldc, M, N, K, split, 1,
                                 torch.cuda.current_stream().cuda_stream))
    ref = (ah.T if tA else ah) @ (bh if tB else bh.T)
    got = C[off:].cpu().reshape(M, ldc)
    # exact BF16 products, FP32 sums of K terms: K 2^-24 of sum |a||b| at most
    bound = K * 2.0 ** -23 * ((ah.T if tA else ah).abs() @ (bh if tB else bh.T).abs()).max()
    assert (got[:, :N].double() - ref).abs().max() <= bound
    assert not got[:, N:].any() and not C[:off].any()      # nothing outside the result
    assert _capi.status_read_and_clear() == 0


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 1000, 152 * 128 + 5])
@pytest.mark.parametrize("weighted", [False, True])
def test_gradient_kernel_rows_and_weights(cuda, rows, weighted):
    """The one-kernel gradient pass at partial tiles, more tiles than SMs and with
    row weights: outputs bit for bit the training forward's, gradients against the
    oracle with the same BF16 rounding points, at the gradient check's bounds."""
    import numpy as np
    from fluxvortex_gb300 import _capi
    from fluxvortex_gb300 import learned as L
    from oracle import learned as OL
    rng = np.random.default_rng(rows)
    w, _ = L.init_weights(5)
    m = L.FarFieldMLP(w, (rng.standard_normal(L.NB) * 0.1).astype(np.float32))
    X = np.zeros((rows, L.IN), np.float32)
    X[:, :L.NFEAT] = rng.standard_normal((rows, L.NFEAT))
    Xd = torch.tensor(X).to(torch.bfloat16).cuda()
    T = rng.standard_normal((rows, L.OUT)).astype(np.float32)
    wr = rng.uniform(0.5, 2.0, rows).astype(np.float32) if weighted else np.ones(rows, np.float32)
    loss, Y = m.gradients(Xd, torch.tensor(T).cuda(), torch.tensor(wr).cuda() if weighted else None)
    Yf, _, _ = m.forward(Xd, store=True)
    assert torch.equal(Y, Yf)
    e = (Y.cpu().double() - torch.tensor(T).double())[:, :L.NOUT]
    ref = (torch.tensor(wr).double()[:, None] * e * e).sum().item()
    # FP32 squares and row sums (31 roundings), FP64 above, one addition per CTA
    assert abs(loss.item() - ref) <= (31 + 152) * 2.0 ** -24 * ref
    # the oracle's backward with the row weights in dY
    ws, bs = m.weights_numpy()
    gw, gb = m.gw.cpu().numpy(), m.gb.cpu().numpy()
    Wl, Bl = OL.unpack(ws, bs)
    Yo, (Zs, Hs) = OL.forward(ws, bs, Xd.float().cpu().numpy())
    E = np.zeros_like(Yo)
    E[:, :L.NOUT] = Yo[:, :L.NOUT] - T[:, :L.NOUT]
    dY = 2.0 * wr[:, None] * E / (rows * L.NOUT)
    g = OL.bf16(dY)
    refs_w, refs_b, dH = {3: g.T @ Hs[3]}, {3: dY.sum(0)}, g @ OL.bf16(Wl[3])
    for l in (2, 1, 0):
        dZ = dH * OL._silu_grad(Zs[l])
        gz = OL.bf16(dZ)
        refs_w[l], refs_b[l], dH = gz.T @ Hs[l], dZ.sum(0), gz @ OL.bf16(Wl[l])
    for l, ((r, c), o) in enumerate(zip(L.LAYERS, L.W_OFFSETS)):
        a, b = gw[o:o + r * c], refs_w[l].reshape(-1)
        assert np.abs(a - b).max() < 2e-2 * np.abs(b).max(), l
        a, b = gb[L.B_OFFSETS[l]:L.B_OFFSETS[l] + r], refs_b[l]
        assert np.abs(a - b).max() < 2e-2 * np.abs(b).max(), l
    assert _capi.status_read_and_clear() == 0
