"""Flash attention (causal or full, grouped-query) on tcgen05 tensor cores.

New relative to the reference, which has no attention code; required by the
decoder model shapes.  Forward and backward never materialise the
[seq, seq] score matrix: scores live in TMEM, probabilities pass through
shared memory as bf16, and only the output and the per-row log-sum-exp reach
HBM.  Tensors use the layout ``[tokens, heads, head_dim]`` so that the packed
output of a fused QKV projection is consumed in place (strided views).
"""
from __future__ import annotations

import ctypes
import functools
import math

import torch

from .. import _native
from ._util import env, stream_ptr, use_native
from .pad import _plain

_native.declare("dd_attn_fwd", [_native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p, _native.c_ll,
                                _native.c_ll, _native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p,
                                _native.c_void_p, _native.c_int, _native.c_int, _native.c_int, _native.c_int,
                                _native.c_int, _native.c_int, _native.c_float, _native.c_void_p])
_native.declare("dd_attn_fwd2", [_native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p, _native.c_ll,
                                 _native.c_ll, _native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p,
                                 _native.c_void_p, _native.c_int, _native.c_int, _native.c_int, _native.c_int,
                                 _native.c_int, _native.c_int, _native.c_float, _native.c_void_p])
_BWD_ARGS = [_native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p, _native.c_ll,
             _native.c_ll, _native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p,
             _native.c_void_p, _native.c_void_p, _native.c_void_p, _native.c_void_p,
             _native.c_ll, _native.c_ll, _native.c_void_p, _native.c_ll, _native.c_ll,
             _native.c_void_p, _native.c_ll, _native.c_ll, _native.c_int, _native.c_int,
             _native.c_int, _native.c_int, _native.c_int, _native.c_int, _native.c_float,
             _native.c_void_p]
_native.declare("dd_attn_bwd2", _BWD_ARGS)
_native.declare("dd_attn_bwd", [_native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p, _native.c_ll,
                                _native.c_ll, _native.c_void_p, _native.c_ll, _native.c_ll, _native.c_void_p,
                                _native.c_void_p, _native.c_void_p, _native.c_void_p, _native.c_void_p,
                                _native.c_ll, _native.c_ll, _native.c_void_p, _native.c_ll, _native.c_ll,
                                _native.c_void_p, _native.c_ll, _native.c_ll, _native.c_int, _native.c_int,
                                _native.c_int, _native.c_int, _native.c_int, _native.c_int, _native.c_float,
                                _native.c_void_p])
_native.declare("dd_attn_bwd3", _BWD_ARGS[:13] + [_native.c_ll] + _BWD_ARGS[13:])
_native.declare("dd_attn_fwd_two_tiles", [_native.c_int] * 4)
_native.declare("dd_attn_ragged", [_native.c_int] * 5)
_native.declare("dd_attn_bwd_one_pass", [_native.c_int] * 6 + [_native.c_void_p])


@functools.lru_cache(maxsize=1024)
def _one_pass_words(device, batch, seq, Hq, Hkv, D, causal):
    words = ctypes.c_longlong()
    one = _native.lib().dd_attn_bwd_one_pass(batch, seq, Hq, Hkv, D, int(causal), ctypes.byref(words))
    return words.value if one else 0


@functools.lru_cache(maxsize=1024)
def _two_tiles(device, batch, seq, Hq, causal):
    return bool(_native.lib().dd_attn_fwd_two_tiles(batch, seq, Hq, int(causal)))


@functools.lru_cache(maxsize=1024)
def _ragged_faster(device, batch, seq, Hq, Hkv, causal):
    return bool(_native.lib().dd_attn_ragged(batch, seq, Hq, Hkv, int(causal)))


def _one_pass(batch, seq, Hq, Hkv, D, causal):
    """Words of scratch for a backward pass in one kernel, 0 where two kernels are the faster way on this device."""
    return _one_pass_words(torch._C._cuda_getDevice(), batch, seq, Hq, Hkv, D, bool(causal))


def _strides(t):
    # [tokens, heads, D] view with unit stride in D
    assert t.stride(2) == 1
    return t.stride(0), t.stride(1)


def attention_forward(q, k, v, batch, seq, causal=True, scale=None):
    """Returns (out [tokens, Hq, D], lse [batch, Hq, seq])."""
    tokens, Hq, D = q.shape
    Hkv = k.shape[1]
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    out = torch.empty(tokens, Hq, D, dtype=q.dtype, device=q.device)
    lse = torch.empty(batch, Hq, seq, dtype=torch.float32, device=q.device)
    # the two-tile kernel (scores and probabilities in tensor memory, two query tiles alternating on the tensor cores)
    two_tile = D in (64, 128) and (seq % 128 != 0 or (
        env("DISTDL_ATTN_FWD2", "1") != "0" and _two_tiles(torch._C._cuda_getDevice(), batch, seq, Hq, bool(causal))))
    _native.call("dd_attn_fwd2" if two_tile else "dd_attn_fwd", q.data_ptr(), *_strides(q), k.data_ptr(), *_strides(k),
                 v.data_ptr(), *_strides(v), out.data_ptr(), lse.data_ptr(), batch, seq, Hq, Hkv, D, int(causal),
                 float(scale), stream_ptr())
    return out, lse


def attention_backward(dout, q, k, v, out, lse, batch, seq, causal=True, scale=None, dq=None, dk=None, dv=None):
    """Gradients of :func:`attention_forward`; writes into ``dq/dk/dv`` views when given."""
    tokens, Hq, D = q.shape
    Hkv = k.shape[1]
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if dq is None:
        dq = torch.empty(tokens, Hq, D, dtype=q.dtype, device=q.device)
    if dk is None:
        dk = torch.empty(tokens, Hkv, D, dtype=q.dtype, device=q.device)
    if dv is None:
        dv = torch.empty(tokens, Hkv, D, dtype=q.dtype, device=q.device)
    dout, out = dout.contiguous(), out.contiguous()
    if seq % 128 and dout.data_ptr() % 16:
        dout = dout.clone()
    in_tmem = env("DISTDL_ATTN_BWD2", "1") != "0" or seq % 128 != 0
    words = _one_pass(batch, seq, Hq, Hkv, D, causal) if in_tmem and D in (64, 128) else 0
    scratch = None
    if words:
        try:
            scratch = torch.empty(words, dtype=torch.float32, device=q.device)
        except torch.OutOfMemoryError:
            if seq % 128:
                raise                       # (no other kernel takes such a length)
    if scratch is not None:
        # one kernel for all three gradients; without room for its sums, the two that need none
        _native.call("dd_attn_bwd3", q.data_ptr(), *_strides(q), k.data_ptr(), *_strides(k), v.data_ptr(), *_strides(v),
                     out.data_ptr(), dout.data_ptr(), lse.data_ptr(), scratch.data_ptr(), words, dq.data_ptr(),
                     *_strides(dq), dk.data_ptr(), *_strides(dk), dv.data_ptr(), *_strides(dv), batch, seq, Hq, Hkv, D,
                     int(causal), float(scale), stream_ptr())
        return dq, dk, dv
    # the kernels that keep P / dS in tensor memory (scratch: delta and the base-2 lse)
    in_tmem = D in (64, 128) and env("DISTDL_ATTN_BWD2", "1") != "0"
    delta = torch.empty(2 if in_tmem else 1, batch, Hq, seq, dtype=torch.float32, device=q.device)
    _native.call("dd_attn_bwd2" if in_tmem else "dd_attn_bwd", q.data_ptr(), *_strides(q), k.data_ptr(), *_strides(k),
                 v.data_ptr(), *_strides(v), out.data_ptr(), dout.data_ptr(), lse.data_ptr(), delta.data_ptr(),
                 dq.data_ptr(), *_strides(dq), dk.data_ptr(), *_strides(dk), dv.data_ptr(), *_strides(dv), batch, seq,
                 Hq, Hkv, D, int(causal), float(scale), stream_ptr())
    return dq, dk, dv


class _AttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, batch, seq, causal, scale):
        out, lse = attention_forward(q, k, v, batch, seq, causal, scale)
        ctx.save_for_backward(q, k, v, out, lse)
        ctx.cfg = (batch, seq, causal, scale)
        return out

    @staticmethod
    def backward(ctx, dout):
        q, k, v, out, lse = ctx.saved_tensors
        batch, seq, causal, scale = ctx.cfg
        dq, dk, dv = attention_backward(dout, q, k, v, out, lse, batch, seq, causal, scale)
        return dq, dk, dv, None, None, None, None


def _reference(q, k, v, batch, seq, causal, scale):
    tokens, Hq, D = q.shape
    Hkv = k.shape[1]
    qh = q.reshape(batch, seq, Hq, D).transpose(1, 2)
    kh = k.reshape(batch, seq, Hkv, D).transpose(1, 2)
    vh = v.reshape(batch, seq, Hkv, D).transpose(1, 2)
    # grouped-query heads are handled by the library kernel itself on CUDA (no expanded copy of K / V)
    if Hkv != Hq and not q.is_cuda:
        kh = kh.repeat_interleave(Hq // Hkv, dim=1)
        vh = vh.repeat_interleave(Hq // Hkv, dim=1)
    o = torch.nn.functional.scaled_dot_product_attention(qh, kh, vh, is_causal=causal, scale=scale,
                                                         enable_gqa=Hkv != Hq and q.is_cuda)
    return o.transpose(1, 2).reshape(tokens, Hq, D)


def attention(q, k, v, batch: int, seq: int, causal: bool = True, scale: float = None):
    """Scaled-dot-product attention over ``[tokens = batch*seq, heads, head_dim]``
    tensors (strided views allowed); ``k``/``v`` may have fewer heads (GQA)."""
    D = q.shape[-1]
    native = (use_native(q) and q.dtype == torch.bfloat16 and D in (64, 128) and seq % 128 == 0
              and env("DISTDL_ATTN_IMPL", "native") == "native")
    if native:
        return _AttnFn.apply(q, k, v, batch, seq, causal, scale)
    return _reference(q, k, v, batch, seq, causal, scale)


def _operators(dout, qkv, Hq, Hkv, batch, seq, causal, scale):
    """The packed gradient by the library's operators: for a backward pass that is itself differentiated, or runs under
    a function transform (batched gradients), a dispatch mode or a tracer."""
    with torch.enable_grad():
        out = _reference(qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:], batch, seq, causal, scale)
        return torch.autograd.grad(out, qkv, dout, create_graph=True)[0]


def _ragged_ok(qkv, Hq, Hkv, batch, seq, scale=None, causal=True):
    """Sequences that are not whole tiles of 128, in training at head dim 128: the kernels take over from the library's
    operators, whose packed gradient is put together by copies, where they are the faster way (``dd_attn_ragged``), where
    nobody looks for the operators themselves and where the tensor maps can address the projection.  The kernels mask with
    -inf before they multiply by the scale: one of 0 or below is the library's.  Without a gradient (2 x 1531 tokens, 32 / 8
    heads: 54 against 68 us) and at head dim 64 the library's kernels are the faster ones."""
    return (qkv.dim() == 3 and qkv.shape[2] == 128 and qkv.requires_grad and torch.is_grad_enabled() and batch > 0
            and seq > 0 and Hkv > 0 and Hq > 0 and Hq % Hkv == 0 and qkv.shape[0] == batch * seq
            and qkv.shape[1] == Hq + 2 * Hkv and (scale is None or (isinstance(scale, (int, float)) and 0 < scale < math.inf))
            and qkv.data_ptr() % 16 == 0 and _plain(qkv)
            and not (torch.is_autocast_enabled() and torch.get_autocast_dtype("cuda") != torch.bfloat16)
            and _ragged_faster(torch._C._cuda_getDevice(), batch, seq, Hq, Hkv, bool(causal)))


class _PackedAttnFn(torch.autograd.Function):
    """Attention on a packed ``[tokens, Hq + 2*Hkv, D]`` projection output; the
    backward kernels write dq / dk / dv straight into one packed gradient."""

    @staticmethod
    def forward(ctx, qkv, Hq, Hkv, batch, seq, causal, scale):
        q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]
        out, lse = attention_forward(q, k, v, batch, seq, causal, scale)
        ctx.save_for_backward(qkv, out, lse)
        ctx.cfg = (Hq, Hkv, batch, seq, causal, scale)
        return out

    @staticmethod
    def backward(ctx, dout):
        qkv, out, lse = ctx.saved_tensors
        Hq, Hkv, batch, seq, causal, scale = ctx.cfg
        q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]
        if seq % 128 and (torch.is_grad_enabled() or not _plain(dout)):
            return _operators(dout, qkv, Hq, Hkv, batch, seq, causal, scale), None, None, None, None, None, None
        dqkv = torch.empty_like(qkv)
        attention_backward(dout, q, k, v, out, lse, batch, seq, causal, scale, dq=dqkv[:, :Hq],
                           dk=dqkv[:, Hq:Hq + Hkv], dv=dqkv[:, Hq + Hkv:])
        return dqkv, None, None, None, None, None, None


def attention_packed(qkv, Hq: int, Hkv: int, batch: int, seq: int, causal: bool = True, scale: float = None):
    """Attention over a packed projection ``[tokens, Hq + 2*Hkv, head_dim]`` (heads
    ordered q..., k..., v...).  Returns ``[tokens, Hq, head_dim]``."""
    D = qkv.shape[-1]
    native = (use_native(qkv) and qkv.dtype == torch.bfloat16 and D in (64, 128) and qkv.is_contiguous()
              and env("DISTDL_ATTN_IMPL", "native") == "native"
              and (seq % 128 == 0 or _ragged_ok(qkv, Hq, Hkv, batch, seq, scale, causal)))
    if native:
        return _PackedAttnFn.apply(qkv, Hq, Hkv, batch, seq, causal, scale)
    return _reference(qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:], batch, seq, causal, scale)
