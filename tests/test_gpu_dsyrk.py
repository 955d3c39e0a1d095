"""FP64 exchange update K = sum_Q W_Q W_Q^T (``dfb_dsyrk``) against an FP64 product.

Both sum the same products in another order: the error of a sum of k terms grows at most like k ulp of the
sum of magnitudes; 1e-14 of the largest element is about 45 ulp, and the products here have random signs."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("naux,nao,nocc", [
    (1, 1, 1), (3, 5, 1),          # one partial tile, k below a chunk
    (7, 64, 16), (33, 65, 17),     # one tile exactly, one element more; k not a multiple of the chunk
    (40, 127, 5), (5, 128, 40), (64, 200, 41),
    (700, 70, 40),                 # several k spans
])
def test_exchange_update(naux, nao, nocc):
    from asuka_b200.linalg import exchange_update

    g = torch.Generator(device="cuda")
    g.manual_seed(naux)
    W = torch.randn((naux, nao, nocc), generator=g, dtype=torch.float64, device="cuda")
    K0 = torch.randn((nao, nao), generator=g, dtype=torch.float64, device="cuda")
    K0 = K0 + K0.T
    K = exchange_update(W, K0.clone())
    ref = K0 + torch.einsum("qmi,qni->mn", W, W)
    assert float((K - ref).abs().max()) <= 1e-14 * float(ref.abs().max()) * max(1.0, (naux * nocc) ** 0.5 / 16)
    Wt = W.transpose(1, 2).contiguous().transpose(1, 2)  # strided input
    assert float((exchange_update(Wt, K0.clone()) - K).abs().max()) <= 1e-13 * float(ref.abs().max())


def test_exchange_update_rejects_bad_sizes():
    from asuka_b200 import _lib

    L = _lib.lib()
    assert L.dfb_dsyrk(4, 2, 3, 0, 12, 3, 0, 4, None) == -1   # no pointers
    assert L.dfb_dsyrk(4, 2, 3, 0, 12, 3, 0, 3, None) == -1   # ldc < n
    assert L.dfb_dsyrk(0, 2, 3, 0, 12, 3, 0, 0, None) == 0    # nothing to do


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 255, 256, 257, 300, 520])
@pytest.mark.parametrize("nb", [32, 96, 256])
def test_diag_block_inverses(n, nb):
    """Block inverses by forward substitution (``dfb_tri_inv``), row- and column-major factors: the residual of
    a substitution is within n ulp of the magnitudes of L times its inverse."""
    from asuka_b200.linalg import diag_block_inverses

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    A = torch.randn((n, n + 8), generator=g, dtype=torch.float64, device="cuda")
    L = torch.linalg.cholesky(A @ A.T + n * torch.eye(n, dtype=torch.float64, device="cuda"))
    for F in (L.contiguous(), L.T.contiguous().T):
        for i, inv in enumerate(diag_block_inverses(F, nb)):
            r0 = i * nb
            blk = L[r0:r0 + nb, r0:r0 + nb]
            eye = torch.eye(blk.shape[0], dtype=L.dtype, device="cuda")
            bound = nb * 2.3e-16 * float((blk.abs() @ inv.abs()).max())
            assert float((blk @ inv - eye).abs().max()) <= bound
            assert float(torch.triu(inv, 1).abs().max()) == 0.0 if inv.shape[0] > 1 else True
