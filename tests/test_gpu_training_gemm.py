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
