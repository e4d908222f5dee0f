"""bf16 GEMM on tcgen05 tensor cores (TMEM accumulators, TMA-fed) and the
autograd ``linear`` built on it.

The native kernel computes ``D[b,m,n] (+)= sum_k A[b,m,k] * B[b,n,k] (+ bias[n])``
with each operand either K-major or MN-major, so forward (``x @ w.T``),
data-gradient (``dy @ w``) and weight-gradient (``dy.T @ x``) run without
transposition copies.  It stands where the reference calls
``torch.nn.functional.linear`` / ``torch.einsum`` (cuBLAS):
``src/distdl/nn/linear_ag.py:486``, ``src/distdl/nn/linear_rs.py:361``,
``src/distdl/nn/linear_ag_zero.py:35-61``.
"""
from __future__ import annotations

import ctypes
import functools

import torch

from .. import _native
from ._util import main_grad_now, ptr, stream_ptr, use_native

_v, _i, _ll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
_native.declare("dd_gemm_bf16_rows", [_v, _i, _ll, _ll, _v, _i, _ll, _ll, _v, _ll, _ll, _i, _i, _i, _i, _i, _v, _i, _v])
_native.declare("dd_gemm_split", [_i, _i, _i])
_native.declare("dd_gemm_bf16_split", [_v, _i, _ll, _v, _i, _ll, _v, _ll, _v, _i, _i, _i, _i, _i, _v, _v])
_native.declare("dd_colsum_parts", [_ll, _i])
_native.declare("dd_colsum", [_v, _ll, _i, _v, _v, _i, _v])

F_OUT_F32 = 1
F_ACCUMULATE = 2
F_BIAS = 4
F_BIAS_F32 = 8


def _major(t: torch.Tensor):
    """Classifies a 2-D/3-D operand view [.., rows, k]: returns (mn_major, ld, batch_stride)."""
    if t.stride(-1) == 1:
        return 0, t.stride(-2), (t.stride(0) if t.dim() == 3 else 0)
    if t.stride(-2) == 1:
        return 1, t.stride(-1), (t.stride(0) if t.dim() == 3 else 0)
    raise ValueError("GEMM operand needs unit stride in one of its last two dimensions")


# Short cuts past the rule of dd_gemm_split, which answers 1 beyond them on a GPU of 148 SMs: outputs of more elements
# have tiles for half the SMs, contractions of less than 4096 gain less than the second launch costs.
_SPLIT_MAX_MN = 37 * 256 * 256


@functools.lru_cache(maxsize=1024)
def _split(M, N, K):
    return _native.lib().dd_gemm_split(M, N, K)


def gemm(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor = None, *, bias: torch.Tensor = None,
         accumulate: bool = False, out_dtype: torch.dtype = None, max_ctas: int = 0, rows: torch.Tensor = None,
         bound_k: bool = False) -> torch.Tensor:
    """``out[.., m, n] (+)= a[.., m, k] @ b[.., n, k].T (+ bias)`` on bf16 operands.

    ``a`` and ``b`` are *views*: pass ``w`` for ``x @ w.T``, ``w.t()`` for
    ``dy @ w``, and ``dy.t(), x.t()`` for ``dy.T @ x``; any combination of
    row-/column-contiguous views with 16-byte-aligned leading dimensions is
    accepted.  ``out`` may be bf16 or fp32 and may be a strided row-major view.

    ``rows`` (int32 ``[batch]`` on the device, for 3-D operands without a bias) promises that ``a[b]`` is zero after
    its first ``rows[b]`` rows, or, with ``bound_k``, that the terms of the contraction after the first ``rows[b]``
    are zero: the result is the same, the work on those zeros is left out.

    ``max_ctas`` below the number of SMs leaves the others to work of other streams; the next product does not start on
    them before this one has ended.
    """
    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16, "bf16 operands required"
    assert a.dim() == b.dim() and a.dim() in (2, 3)
    M, K = a.shape[-2], a.shape[-1]
    N = b.shape[-2]
    assert b.shape[-1] == K, f"contraction mismatch {a.shape} x {b.shape}"
    batch = a.shape[0] if a.dim() == 3 else 1
    if out is None:
        shape = (batch, M, N) if a.dim() == 3 else (M, N)
        out = torch.empty(shape, dtype=out_dtype or torch.bfloat16, device=a.device)
        assert not accumulate
    assert out.stride(-1) == 1
    if M == 0 or N == 0:
        return out
    if K == 0:
        if not accumulate:
            out.zero_()
        return out
    a_mn, lda, sa = _major(a)
    b_mn, ldb, sb = _major(b)
    flags = 0
    if out.dtype == torch.float32:
        flags |= F_OUT_F32
    else:
        assert out.dtype == torch.bfloat16
    if accumulate:
        flags |= F_ACCUMULATE
    if bias is not None:
        flags |= F_BIAS
        if bias.dtype == torch.float32:
            flags |= F_BIAS_F32
        assert bias.is_contiguous() and bias.numel() == N
    ldd = out.stride(-2)
    sd = out.stride(0) if out.dim() == 3 else 0
    if rows is not None:
        assert bias is None and rows.dtype == torch.int32 and rows.numel() == batch and rows.is_contiguous()
        _native.call("dd_gemm_bf16_rows", a.data_ptr(), a_mn, lda, sa, b.data_ptr(), b_mn, ldb, sb, out.data_ptr(), ldd,
                     sd, M, N, K, batch, flags, rows.data_ptr(), int(bound_k), stream_ptr())
        return out
    if K >= 4096 and batch == 1 and max_ctas == 0 and M * N <= _SPLIT_MAX_MN:
        split = _split(M, N, K)
        if split > 1:
            ws = torch.empty(split * M * ((N + 3) & ~3), dtype=torch.float32, device=a.device)
            _native.call("dd_gemm_bf16_split", a.data_ptr(), a_mn, lda, b.data_ptr(), b_mn, ldb, out.data_ptr(), ldd,
                         ptr(bias), M, N, K, flags, split, ws.data_ptr(), stream_ptr())
            return out
    _native.call("dd_gemm_bf16", a.data_ptr(), a_mn, lda, sa, b.data_ptr(), b_mn, ldb, sb, out.data_ptr(), ldd, sd,
                 ptr(bias), M, N, K, batch, flags, max_ctas, stream_ptr())
    return out


def grad_target(w: torch.Tensor):
    """What a weight-gradient GEMM needs to know about the weight ``w`` ([out, in], possibly a
    transposed view), as a small tuple that a backward pass can keep without keeping ``w``
    itself alive: ``(main_grad, transposed_storage, main_grad_owner)``."""
    return (getattr(w, "main_grad", None), not w.is_contiguous() and w.t().is_contiguous(),
            getattr(w, "main_grad_owner", None))


def weight_grad(dy2: torch.Tensor, x2: torch.Tensor, w: torch.Tensor = None, target=None, ctx=None):
    """Gradient of ``y = x @ w.T`` with respect to ``w`` ([out, in]) from
    ``dy2 [tokens, out]`` and ``x2 [tokens, in]``; give either ``w`` or ``target =
    grad_target(w)``, and the ``ctx`` of the running backward pass if ``w`` is its input 1.

    * ``w.main_grad`` (an fp32 tensor in the layout of ``w``, possibly a
      transposed view): the GEMM epilogue accumulates into it and ``None`` is
      returned, so no bf16 gradient is ever written; with ``w.main_grad_owner``, the
      leaf behind ``w``, only where :func:`main_grad_now` allows it.
    * ``w`` a transposed view of a contiguous ``[in, out]`` tensor: the gradient
      is produced in that storage order (``x^T dy``) and returned as the matching
      view, so autograd's transpose back is free instead of a strided copy.
    """
    mg, transposed, owner = target if target is not None else grad_target(w)
    mg = main_grad_now(mg, owner, ctx, 1)
    if mg is not None:
        if mg.is_contiguous():
            gemm(dy2.t(), x2.t(), out=mg, accumulate=True)
        else:
            gemm(x2.t(), dy2.t(), out=mg.t(), accumulate=True)
        return None
    if transposed:
        return gemm(x2.t(), dy2.t()).t()
    return gemm(dy2.t(), x2.t())


def column_sum(x2: torch.Tensor, acc: torch.Tensor = None) -> torch.Tensor:
    """``x2.sum(0)`` of a contiguous bf16 matrix in fp32; with ``acc`` (flat fp32) added to it in place."""
    rows, n = x2.shape
    if rows == 0 or n % 8 or x2.data_ptr() % 16 or x2.dtype != torch.bfloat16 \
            or not (acc is None or (acc.dtype == torch.float32 and acc.is_contiguous())):
        s = x2.sum(0, dtype=torch.float32)
        return s if acc is None else acc.add_(s)
    out = acc if acc is not None else torch.empty(n, dtype=torch.float32, device=x2.device)
    parts = torch.empty(_native.lib().dd_colsum_parts(rows, n), n, dtype=torch.float32, device=x2.device)
    _native.call("dd_colsum", x2.data_ptr(), rows, n, parts.data_ptr(), out.data_ptr(), int(acc is not None), stream_ptr())
    return out


class _LinearFn(torch.autograd.Function):
    """y = x @ w.T + b with all three GEMMs on the native kernel.

    When the weight carries a ``main_grad`` fp32 buffer (set by the optimizer
    for gradient accumulation) the weight gradient is accumulated straight into
    it from the GEMM epilogue and ``None`` is returned for ``w.grad``.
    """

    @staticmethod
    def forward(ctx, x, w, b):
        x2 = x.reshape(-1, x.shape[-1])
        # the result is allocated in its final shape (never a view), so that
        # in-place ops such as the rotary embedding may follow
        y = torch.empty(*x.shape[:-1], w.shape[0], dtype=x.dtype, device=x.device)
        gemm(x2, w, out=y.view(-1, w.shape[0]), bias=b)
        ctx.save_for_backward(x2, w)
        ctx.has_bias = b is not None
        # (not the weight itself: a gathered ZeRO weight must not be held from forward to backward)
        ctx.wgrad = grad_target(w)
        ctx.b_main_grad = (getattr(b, "main_grad", None), getattr(b, "main_grad_owner", None))
        ctx.xshape = x.shape
        return y

    @staticmethod
    def backward(ctx, dy):
        x2, w = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = gemm(dy2, w.t()).view(ctx.xshape)
        if ctx.needs_input_grad[1]:
            dw = weight_grad(dy2, x2, target=ctx.wgrad, ctx=ctx)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            mg = main_grad_now(*ctx.b_main_grad, ctx, 2)
            s = column_sum(dy2, mg)
            if mg is None:
                db = s.to(dy.dtype)
        return dx, dw, db


def linear(x: torch.Tensor, w: torch.Tensor, b: torch.Tensor = None) -> torch.Tensor:
    """Drop-in for ``torch.nn.functional.linear`` (bf16 CUDA operands run the tcgen05 kernel)."""
    if use_native(x, w) and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and w.dim() == 2 \
            and w.shape[1] % 8 == 0 and (w.shape[0] % 8 == 0):
        return _LinearFn.apply(x, w, b)
    return torch.nn.functional.linear(x, w, b)


def matmul(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """``a @ b`` for 2-D / 3-D bf16 CUDA tensors through the native kernel (no autograd)."""
    return gemm(a, b.transpose(-1, -2))
