"""Triangular solves with the metric's Cholesky factor as blocked GEMMs.

The DF step solves with the lower factor L of the aux metric twice per step:
W = L^-1 Y (Y = X Cw, naux x nao*nocc) and Z = L^-T M (M = Cw^T W,
naux x nocc^2).  A single library TRSM call with a few-thousand-row triangle and
tens of thousands of right-hand sides runs far below the FP64 GEMM rate, so the
solve is done by block substitution instead: the diagonal blocks of L are
inverted once (one kernel), and every step of
the substitution is then two FP64 GEMMs -- the update with the rows already
solved, and the product with the inverted diagonal block.  The work is the same
naux^2 * ncol multiply-adds as the TRSM.
"""

from __future__ import annotations

import functools

import torch
import torch.autograd.forward_ad as _fwd
from torch.utils._device import DeviceContext

from . import _lib

NB = 256  # rows per diagonal block
_PLAIN = (torch.Tensor, torch.nn.Parameter)


def diag_block_inverses(L: torch.Tensor, nb: int = NB) -> list[torch.Tensor]:
    """Inverses of the nb x nb diagonal blocks of the lower-triangular L: one kernel (``dfb_tri_inv``) on the
    GPU for row-major FP64 factors and blocks of a multiple of 32 up to 256 rows, a triangular solve against
    the identity per block otherwise."""
    n = L.shape[0]
    starts = range(0, n, nb)
    if not (L.is_cuda and L.dtype == torch.float64 and nb % 32 == 0 and 32 <= nb <= 256) or _observed(L):
        out = []
        for r0 in starts:
            r1 = min(n, r0 + nb)
            eye = torch.eye(r1 - r0, dtype=L.dtype, device=L.device)
            out.append(torch.linalg.solve_triangular(L[r0:r1, r0:r1], eye, upper=False))
        return out
    Lr = L if L.stride(1) == 1 and L.stride(0) >= n else L.contiguous()  # cuSOLVER returns its factor column-major
    inv = torch.empty((len(starts), nb, nb), dtype=L.dtype, device=L.device)
    rc = _launch(L.device, _lib.lib().dfb_tri_inv, n, nb, _lib.ptr(Lr), max(Lr.stride(0), n), _lib.ptr(inv))
    _lib.check(rc, "dfb_tri_inv")
    return [inv[i, : min(n, r0 + nb) - r0, : min(n, r0 + nb) - r0] for i, r0 in enumerate(starts)]


def solve_lower(L: torch.Tensor, Y: torch.Tensor, inv: list[torch.Tensor] | None = None, nb: int = NB,
                out: torch.Tensor | None = None) -> torch.Tensor:
    """W = L^-1 Y by forward block substitution; ``out`` may be Y itself (in place)."""
    n = L.shape[0]
    if inv is None:
        inv = diag_block_inverses(L, nb)
    W = out if out is not None else torch.empty_like(Y)
    for i, r0 in enumerate(range(0, n, nb)):
        r1 = min(n, r0 + nb)
        rhs = Y[r0:r1].clone() if r0 == 0 else torch.addmm(Y[r0:r1], L[r0:r1, :r0], W[:r0], alpha=-1.0)
        torch.mm(inv[i], rhs, out=W[r0:r1])
    return W


def solve_lower_T(L: torch.Tensor, M: torch.Tensor, inv: list[torch.Tensor] | None = None, nb: int = NB,
                  out: torch.Tensor | None = None) -> torch.Tensor:
    """Z = L^-T M by backward block substitution; ``out`` may be M itself (in place)."""
    n = L.shape[0]
    if inv is None:
        inv = diag_block_inverses(L, nb)
    Z = out if out is not None else torch.empty_like(M)
    starts = list(range(0, n, nb))
    for i in range(len(starts) - 1, -1, -1):
        r0 = starts[i]
        r1 = min(n, r0 + nb)
        rhs = M[r0:r1].clone() if r1 == n else torch.addmm(M[r0:r1], L[r1:, r0:r1].T, Z[r1:], alpha=-1.0)
        torch.mm(inv[i].T, rhs, out=Z[r0:r1])
    return Z


def solve_lower_right_T(L: torch.Tensor, X: torch.Tensor, inv: list[torch.Tensor] | None = None, nb: int = NB,
                        out: torch.Tensor | None = None) -> torch.Tensor:
    """B = X L^-T (X is (m, n), the solve runs over its columns); ``out`` may be X itself."""
    n = L.shape[0]
    if inv is None:
        inv = diag_block_inverses(L, nb)
    B = out if out is not None else torch.empty_like(X)
    for i, r0 in enumerate(range(0, n, nb)):
        r1 = min(n, r0 + nb)
        rhs = X[:, r0:r1] if r0 == 0 else torch.addmm(X[:, r0:r1], B[:, :r0], L[r0:r1, :r0].T, alpha=-1.0)
        B[:, r0:r1] = rhs @ inv[i].T
    return B


def _launch(device: torch.device, fn, *args) -> int:
    """fn(*args, the device's current stream) with that device current: a kernel is launched on the current
    device, and its stream has to belong to it."""
    stream = _lib.current_stream(device.index)
    if device.index in (None, torch.cuda.current_device()):
        return fn(*args, stream)
    with torch.cuda.device(device):
        return fn(*args, stream)


def _observed(*tensors: torch.Tensor) -> bool:
    """True when something follows the operations on these tensors that a kernel on raw pointers would pass by:
    autograd, forward-mode or function transforms, a tensor subclass, a mode or a tracer."""
    grad = torch.is_grad_enabled()
    for t in tensors:
        if type(t) not in _PLAIN or (grad and t.requires_grad):
            return True
    c = torch._C
    if (c._functorch.maybe_current_level() is not None or c._len_torch_dispatch_stack() or torch.compiler.is_compiling()
            or c._get_tracing_state() is not None):
        return True
    if c._len_torch_function_stack():  # a default device is a mode too, which only creates tensors
        if any(not isinstance(m, DeviceContext) for m in torch.overrides._get_current_function_mode_stack()):
            return True
    return _fwd._current_level >= 0 and any(_fwd.unpack_dual(t).tangent is not None for t in tensors)


def _kernel_update(W: torch.Tensor, out: torch.Tensor) -> bool:
    """True when the exchange kernel can take W (naux, nao, nocc) and out: FP64 on one GPU, out a row-major
    (nao, nao) matrix.  Its pointers carry neither a type nor a device, so everything else stays with torch."""
    n, f64 = W.shape[1], torch.float64
    if not (W.is_cuda and W.dtype is f64 and out.dtype is f64 and out.device == W.device and out.shape == (n, n)):
        return False
    return (out.stride(1) == 1 and out.stride(0) >= n or n <= 1) and not (W.is_neg() or out.is_neg())


@functools.lru_cache(maxsize=256)
def _syrk_scratch(nao: int, naux: int, nocc: int, device: int) -> int:
    with torch.cuda.device(device):
        return int(_lib.lib().dfb_dsyrk_scratch(nao, naux, nocc))


def exchange_update(W: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out += sum_Q W_Q W_Q^T for W (naux, nao, nocc), without a transposed copy of W in FP64 on the GPU.

    There the library's symmetric kernel runs (``dfb_dsyrk``: half the multiply-adds of a full product, k
    split over the chip and its spans added in a fixed order: equal calls give equal bits).  Other types and
    layouts, and tensors that autograd or a transform follows, take the product of a transposed copy, with
    torch's type promotion."""
    naux, nao, nocc = W.shape
    if not _kernel_update(W, out) or _observed(W, out):
        W2 = W.permute(1, 0, 2).reshape(nao, naux * nocc)
        out += W2 @ W2.T
        return out
    W = W.contiguous()
    device = W.device
    need = _syrk_scratch(nao, naux, nocc, device.index)
    ws = torch.empty(need, dtype=torch.float64, device=device) if need else None  # freed in stream order
    rc = _launch(device, _lib.lib().dfb_dsyrk_ws, nao, naux, nocc, W.data_ptr(), nao * nocc, nocc, out.data_ptr(),
                 max(out.stride(0), nao), _lib.ptr(ws), need)
    _lib.check(rc, "dfb_dsyrk")
    if not out.is_inference():
        torch.autograd.graph.increment_version(out)  # written behind autograd's back
    return out
