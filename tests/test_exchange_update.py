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


@pytest.mark.parametrize("device", DEVICES)
def test_k_is_differentiable(device):
    """K carries its graph, as J does: d/dCw and d/dBQ of <T, K> against the closed forms 2 sum_Q B_Q Ts B_Q Cw
    and 2 Ts B_Q Cw Cw^T (Ts = (T + T^T) / 2, B_Q taken as independent elements: right factor Cw Cw^T)."""
    from asuka_b200.jk import df_JK_from_BQ, df_K_from_BQ_Cw

    B, Cw = _inputs(device)
    T = torch.arange(NAO * NAO, dtype=torch.float64, device=device).reshape(NAO, NAO).cos()
    Ts = 0.5 * (T + T.T)
    C = Cw.clone().requires_grad_(True)
    (gC,) = torch.autograd.grad((df_K_from_BQ_Cw(B, C) * T).sum(), C)
    ref = 2.0 * torch.einsum("qmn,mk,qkl,li->ni", B, Ts, B, Cw)
    assert float((gC - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
    Bg = B.clone().requires_grad_(True)
    (gB,) = torch.autograd.grad((df_K_from_BQ_Cw(Bg, Cw) * T).sum(), Bg)
    ref = 2.0 * torch.einsum("mk,qkl,li,ni->qmn", Ts, B, Cw, Cw)
    assert float((gB - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
    J, K = df_JK_from_BQ(B, C, C @ C.T)
    assert J.requires_grad and K.requires_grad
    with torch.no_grad():
        assert not df_K_from_BQ_Cw(B, C).requires_grad


@pytest.mark.parametrize("device", DEVICES)
def test_forward_mode_and_hooks(device):
    """The tangent of K along a direction of Cw, by dual numbers and by ``torch.func.jvp``, and saved-tensor
    hooks on the way."""
    import torch.autograd.forward_ad as fwd

    from asuka_b200.jk import df_K_from_BQ_Cw

    B, Cw = _inputs(device)
    V = Cw.sin()
    U, dU = torch.matmul(B, Cw), torch.matmul(B, V)
    ref = torch.einsum("qmi,qni->mn", U, dU)
    ref = ref + ref.T
    with fwd.dual_level():
        K = df_K_from_BQ_Cw(B, fwd.make_dual(Cw, V))
        dK = fwd.unpack_dual(K).tangent
    assert float((dK - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
    _K, dK = torch.func.jvp(lambda c: df_K_from_BQ_Cw(B, c), (Cw,), (V,))
    assert float((dK - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
    packed = []
    C = Cw.clone().requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t, lambda t: t):
        df_K_from_BQ_Cw(B, C)
    assert packed


@pytest.mark.gpu
def test_written_accumulator_is_noted():
    """An accumulator that autograd saved before the kernel wrote to it is refused in backward, as for torch's
    in-place sums; a default device does not take the kernel away."""
    from asuka_b200 import _lib
    from asuka_b200.linalg import exchange_update

    B, Cw = _inputs("cuda")
    W = torch.matmul(B, Cw)
    out = torch.zeros((NAO, NAO), dtype=torch.float64, device="cuda")
    x = torch.ones((NAO, NAO), dtype=torch.float64, device="cuda", requires_grad=True)
    y = (x * out).sum()
    L = _lib.lib()
    with torch.device("cuda"):
        n = L.dfb_launch_count()
        exchange_update(W, out)
        assert L.dfb_launch_count() > n
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()


@pytest.mark.parametrize("device", DEVICES)
def test_block_inverses_are_differentiable(device):
    """d/dL of <T, inverse of a diagonal block> = -(inv^T T inv^T) on the block."""
    from asuka_b200.linalg import diag_block_inverses

    n = 40
    A = torch.randn((n, n + 4), generator=torch.Generator().manual_seed(2), dtype=torch.float64)
    L = torch.linalg.cholesky(A @ A.T).to(device).requires_grad_(True)
    T = torch.arange(32.0 * 32, dtype=torch.float64, device=device).reshape(32, 32).cos()
    inv = diag_block_inverses(L, 32)[0]
    (g,) = torch.autograd.grad((inv * T).sum(), L)
    ref = -(inv.detach().T @ T @ inv.detach().T).tril()
    assert float((g[:32, :32].tril() - ref).abs().max()) <= 1e-10 * float(ref.abs().max())


def test_launches_enter_the_tensors_device(monkeypatch):
    """The launch helper with recorded torch.cuda calls: the tensors' device is made current around the call
    when it is not, and the stream is that device's."""
    from contextlib import contextmanager

    from asuka_b200 import linalg

    state = {"current": 0}

    @contextmanager
    def device(d):
        was, state["current"] = state["current"], d.index
        yield
        state["current"] = was

    monkeypatch.setattr(torch.cuda, "current_device", lambda: state["current"])
    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(linalg._lib, "current_stream", lambda index: 100 + index)
    for idx in (0, 1):
        assert linalg._launch(torch.device("cuda", idx), lambda x, st: (x, st, state["current"]), 7) == (7, 100 + idx, idx)
        assert state["current"] == 0


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_tensors_of_another_device():
    from asuka_b200.jk import df_K_from_BQ_Cw
    from asuka_b200.linalg import diag_block_inverses

    B, Cw = _inputs("cuda:1")
    with torch.cuda.device(0):
        K = df_K_from_BQ_Cw(B, Cw)
        (inv,) = diag_block_inverses(torch.eye(32, dtype=torch.float64, device="cuda:1"), 32)
    assert float((K - _k(B, Cw)).abs().max()) <= 1e-13 * float(K.abs().max())
    assert float((inv - torch.eye(32, dtype=torch.float64, device="cuda:1")).abs().max()) == 0.0


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("precision", ["fp64", pytest.param("mixed", marks=pytest.mark.gpu)])
def test_blocks_within_the_memory_there_is(monkeypatch, device, precision):
    """Larger blocks than q_block only up to a quarter of B, never for factors whose blocks are copied, and none
    where they cannot be allocated: a build that q_block rows fit runs through."""
    from asuka_b200 import jk

    if precision == "mixed" and device == "cpu":
        pytest.skip("tensor-core products take CUDA tensors")
    B, Cw = _inputs(device)
    ref = _k(B, Cw)
    tol = 1e-13 if precision == "fp64" else 1e-5
    owner = torch if precision == "fp64" else jk._tc
    product, rows = owner.matmul, []

    def limited(limit):
        def matmul(A, *a, **k):
            if A.shape[0] > limit * NAO:
                raise torch.OutOfMemoryError("no room")
            rows.append(A.shape[0] // NAO)
            return product(A, *a, **k)
        return matmul

    for factors, limit, most in ((B, NAUX, NAUX), (B, 7, 7), (B.permute(1, 2, 0).contiguous().permute(2, 0, 1), NAUX, 7)):
        rows.clear()
        with monkeypatch.context() as m:
            m.setattr(owner, "matmul", limited(limit))
            K = jk.df_K_from_BQ_Cw(factors, Cw, q_block=7, precision=precision)
        assert max(rows) == most and sum(rows) == NAUX
        assert float((K - ref).abs().max()) <= tol * float(ref.abs().max())
    with monkeypatch.context() as m:
        m.setattr(owner, "matmul", limited(6))
        with pytest.raises(torch.OutOfMemoryError):
            jk.df_K_from_BQ_Cw(B, Cw, q_block=7, precision=precision)
    wide = torch.ones((NAO, 2 * NAO), dtype=torch.float64, device=device)  # U of all rows: twice B
    assert jk._half_rows(B, wide.shape[1], 1) * NAO * wide.shape[1] <= B.numel() // 4
    with pytest.raises(ValueError):
        jk.df_K_from_BQ_Cw(B, Cw, q_block=0, precision=precision)


@pytest.mark.gpu
@pytest.mark.parametrize("naux,nao,nocc", [(3, 5, 1), (40, 64, 13), (900, 65, 7), (700, 70, 40), (333, 300, 11), (60, 1100, 3)])
def test_exchange_sum_repeats_and_stays_close(naux, nao, nocc):
    """Equal calls give equal bits and a symmetric sum, beside each other on two streams too.  Error: chains of
    at most 512 terms, then the sums of a span and of the spans; 512 + K/512 roundings of random sign stay below
    4 sqrt(512 + K/512) ulp of the magnitudes summed."""
    from asuka_b200.linalg import exchange_update

    g = torch.Generator(device="cuda")
    g.manual_seed(nao)
    W = torch.randn((naux, nao, nocc), generator=g, dtype=torch.float64, device="cuda")

    def run():
        return exchange_update(W, torch.zeros((nao, nao), dtype=torch.float64, device="cuda"))

    K = run()
    assert torch.equal(K, K.T)
    for _ in range(3):
        assert torch.equal(run(), K)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        K1 = run()
    K2 = run()
    torch.cuda.synchronize()
    assert torch.equal(K1, K) and torch.equal(K2, K)
    rows = slice(0, min(nao, 96))
    A = (W.permute(1, 0, 2).reshape(nao, -1).cpu())[rows]
    ref = torch.zeros((A.shape[0], A.shape[0]), dtype=torch.float64)
    comp = torch.zeros_like(ref)
    for k0 in range(0, A.shape[1], 8):  # compensated sums of short products
        p = A[:, k0:k0 + 8]
        hi = p.float().double()
        lo = p - hi
        for t in (hi @ hi.T, hi @ lo.T, lo @ hi.T, lo @ lo.T):
            y = t - comp
            s = ref + y
            comp = (s - ref) - y
            ref = s
    k = naux * nocc
    mag = A.abs() @ A.abs().T
    assert bool(((K.cpu()[rows, rows] - ref).abs() <= 4 * (512 + k / 512) ** 0.5 * 1.2e-16 * mag).all())


@pytest.mark.gpu
def test_exchange_workspace_is_checked():
    from asuka_b200 import _lib

    L = _lib.lib()
    need = L.dfb_dsyrk_scratch(70, 700, 40)
    assert need > 0 and L.dfb_dsyrk_scratch(5, 3, 1) == 0 and L.dfb_dsyrk_scratch(0, 3, 1) == 0
    W = torch.ones((700, 70, 40), dtype=torch.float64, device="cuda")
    C = torch.zeros((70, 70), dtype=torch.float64, device="cuda")
    ws = torch.empty(need, dtype=torch.float64, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    args = (70, 700, 40, W.data_ptr(), 2800, 40, C.data_ptr(), 70)
    assert L.dfb_dsyrk_ws(*args, ws.data_ptr(), need - 1, st) == -1
    assert L.dfb_dsyrk_ws(*args, ws.data_ptr(), need, st) == 0
    assert L.dfb_dsyrk(*args, st) == 0  # without a workspace: atomics
    torch.cuda.synchronize()
    assert float((C - 2 * 28000.0).abs().max()) == 0.0
