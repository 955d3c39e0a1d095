"""``linalg.exchange_update`` and the J/K contractions built on it, over the inputs that torch's own products
take: the FP64 kernel reads raw pointers, so every other type, layout or context has to reach torch.

Both forms sum the same products in another order; the tolerances are 1e-13 (FP64) and 1e-5 (FP32) of the
largest element, about sqrt(terms) ulp with a factor of ten to spare."""

import pytest

torch = pytest.importorskip("torch")

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]
NAUX, NAO, NOCC = 33, 20, 5


def _inputs(device, dtype=torch.float64):
    g = torch.Generator().manual_seed(5)
    B = torch.randn((NAUX, NAO, NAO), generator=g, dtype=torch.float64)
    B = (B + B.transpose(1, 2)).to(device, dtype)
    return B, torch.randn((NAO, NOCC), generator=g, dtype=torch.float64).to(device, dtype)


def _k(B, Cw):
    U = torch.matmul(B, Cw)
    return torch.einsum("qmi,qni->mn", U, U)


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_factor_types(device, dtype):
    """FP32 factors: their products summed into the FP64 K by type promotion."""
    from asuka_b200.jk import df_JK_from_BQ, df_K_from_BQ_Cw

    B, Cw = _inputs(device, dtype)
    ref = _k(B.double(), Cw.double())
    tol = 1e-13 if dtype == torch.float64 else 1e-5
    for q in (7, 256):
        K = df_K_from_BQ_Cw(B, Cw, q_block=q)
        assert K.dtype == torch.float64
        assert float((K - ref).abs().max()) <= tol * float(ref.abs().max())
    _J, K = df_JK_from_BQ(B, Cw, Cw @ Cw.T)
    assert float((K - ref).abs().max()) <= tol * float(ref.abs().max())


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("layout", ["rows", "columns", "padded", "fp32 W", "neg"])
def test_layouts_of_the_accumulator(device, layout):
    """Row-major (also with padded rows) and column-major accumulators, FP32 W into an FP64 accumulator, and a
    lazily negated one: the sum goes to the elements the caller sees, and nothing beside them changes."""
    from asuka_b200.linalg import exchange_update

    B, Cw = _inputs(device)
    W = torch.matmul(B, Cw)
    buf = torch.zeros((NAO, NAO + 3), dtype=torch.float64, device=device)
    out = {"columns": torch.zeros((NAO, NAO), dtype=torch.float64, device=device).T,
           "padded": buf[:, :NAO], "neg": torch._neg_view(buf[:, :NAO])}.get(
               layout, torch.zeros((NAO, NAO), dtype=torch.float64, device=device))
    if layout == "fp32 W":
        W = W.float()
    ref = torch.einsum("qmi,qni->mn", W.double(), W.double())
    assert exchange_update(W, out) is out
    assert float((out - ref).abs().max()) <= (1e-13 if W.dtype == torch.float64 else 1e-5) * float(ref.abs().max())
    assert float(buf[:, NAO:].abs().max()) == 0.0


def test_the_kernel_takes_fp64_of_one_gpu_only():
    """The rule on the CPU, with stand-ins that carry the attributes it reads."""
    from types import SimpleNamespace as NS

    from asuka_b200.linalg import _kernel_update

    def t(shape, dtype=torch.float64, device="cuda:0", stride=None, neg=False):
        n = shape[-1]
        stride = stride or ((n, 1) if len(shape) == 2 else (shape[1] * n, n, 1))
        d = torch.device(device)
        return NS(shape=shape, dtype=dtype, device=d, is_cuda=d.type == "cuda", stride=lambda i: stride[i],
                  is_neg=lambda: neg)

    W, out = t((4, 6, 2)), t((6, 6))
    assert _kernel_update(W, out)
    assert _kernel_update(W, t((6, 6), stride=(9, 1)))
    for bad in (t((4, 6, 2), dtype=torch.float32), t((4, 6, 2), device="cpu"), t((4, 6, 2), device="cuda:1"),
                t((4, 6, 2), neg=True)):
        assert not _kernel_update(bad, out)
    for bad in (t((6, 6), dtype=torch.float32), t((6, 6), stride=(1, 6)), t((6, 6), stride=(0, 1)), t((5, 6)),
                t((6, 6), neg=True)):
        assert not _kernel_update(W, bad)
