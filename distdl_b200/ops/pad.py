"""Constant padding of the spatial dimensions of ``[batch, channel, *space]`` tensors and its adjoint, the crop,
on this library's kernel (``csrc/pad.cu``).  Stands where the reference calls ``torch.nn.functional.pad``
(``src/distdl/nn/conv_feature.py``, ``src/distdl/nn/pooling.py``)."""
from __future__ import annotations

import ctypes

import torch

from .. import _native
from ._util import stream_ptr, use_native

_i3 = ctypes.c_int * 3
_v, _ll, _i = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
_native.declare("dd_shift_channels", [_v, _v, _i, _i, _i, _i3, _i3, _i3, _v])
_native.declare("dd_shift_copy", [_v, _v, _i, _ll, _i3, _i3, _i3, ctypes.c_uint, _v])
# the bits of 0 and -inf
_FILL = {torch.bfloat16: (0, 0xFF80), torch.float16: (0, 0xFC00), torch.float32: (0, 0xFF800000)}


def _three(v, fill):
    v = [int(a) for a in v]
    return _i3(*([fill] * (3 - len(v)) + v))


def _plain(x) -> bool:
    """A tensor and a moment at which a kernel may stand for the library's operators: no subclass, no dispatch
    mode, tracer, compiler, function transform or forward-mode differentiation, which know the operators only."""
    return (type(x) in (torch.Tensor, torch.nn.Parameter) and torch._C._len_torch_dispatch_stack() == 0
            and not torch._C._are_functorch_transforms_active() and not torch._C._functorch.is_functorch_wrapped_tensor(x)
            and not torch._C._functorch.is_legacy_batchedtensor(x) and torch.autograd.forward_ad._current_level < 0
            and not torch.jit.is_tracing() and not torch.compiler.is_compiling())


def _operators(dy, lo, space):
    """The shifted copy by the library's operators, contiguous: for a backward pass under a function transform (batched
    gradients), a dispatch mode or a tracer."""
    pads = []
    for n, a, m in reversed(list(zip(dy.shape[-len(space):], lo, space))):
        pads += [a, m - n - a]
    return torch.nn.functional.pad(dy, pads).contiguous()


class _ShiftCopyFn(torch.autograd.Function):
    """``y[o] = x[o - lo]`` in a tensor of spatial shape ``space``, ``fill`` outside ``x``; its adjoint is the
    shift back, filled with zeros."""

    @staticmethod
    def forward(ctx, x, lo, space, lowest):
        ctx.lo, ctx.space = lo, tuple(x.shape[2:])
        x = x.contiguous()
        y = torch.empty(tuple(x.shape[:2]) + space, dtype=x.dtype, device=x.device)
        _native.call("dd_shift_copy", x.data_ptr(), y.data_ptr(), x.element_size(), x.shape[0] * x.shape[1],
                     _three(x.shape[2:], 1), _three(space, 1), _three(lo, 0), _FILL[x.dtype][int(lowest)], stream_ptr())
        return y

    @staticmethod
    def backward(ctx, dy):
        lo = tuple(-a for a in ctx.lo)
        dx = _ShiftCopyFn.apply(dy, lo, ctx.space, False) if _plain(dy) else _operators(dy, lo, ctx.space)
        return dx, None, None, None


_LAST = {2: torch.channels_last, 3: torch.channels_last_3d}


def _shift_channels(x, to_last, lo, space):
    nd = len(space)
    y = torch.empty(tuple(x.shape[:2]) + space, dtype=x.dtype, device=x.device,
                    memory_format=_LAST[nd] if to_last else torch.contiguous_format)
    _native.call("dd_shift_channels", x.data_ptr(), y.data_ptr(), int(to_last), x.shape[0], x.shape[1],
                 _three(x.shape[2:], 1), _three(space, 1), _three(lo, 0), stream_ptr())
    return y


class _ToChannelsLastFn(torch.autograd.Function):
    """``y[o] = x[o - lo]``, zero outside ``x``, in channels-last memory; the adjoint of
    :class:`_FromChannelsLastFn` with the opposite shift."""

    @staticmethod
    def forward(ctx, x, lo, space):
        ctx.lo, ctx.space = lo, tuple(x.shape[2:])
        return _shift_channels(x.contiguous(), True, lo, space)

    @staticmethod
    def backward(ctx, dy):
        lo = tuple(-a for a in ctx.lo)
        return (_FromChannelsLastFn.apply if _plain(dy) else _operators)(dy, lo, ctx.space), None, None


class _FromChannelsLastFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, lo, space):
        ctx.lo, ctx.space = lo, tuple(x.shape[2:])
        return _shift_channels(x.contiguous(memory_format=_LAST[len(space)]), False, lo, space)

    @staticmethod
    def backward(ctx, dy):
        lo = tuple(-a for a in ctx.lo)
        return (_ToChannelsLastFn.apply if _plain(dy) else _operators)(dy, lo, ctx.space), None, None


def channels_last_usable(x: torch.Tensor, pad_tuple, weight: torch.Tensor) -> bool:
    """Whether a convolution of ``x`` should run in channels-last memory: its tensor-core kernels work in that layout
    and convert every operand on the way in and every result on the way out otherwise.  bf16 and fp16 only, where the
    errors against fp32 of output and gradients are alike in both layouts (200 shapes).  fp32 stays channels-first:
    channels-last always runs in tf32 (errors of 2.9e-4), channels-first for some shapes, directions and channel counts
    only (of 240 convolutions with windows of 3 x 3 x 3, 61 had a gradient exact to 1e-7)."""
    nd = x.dim() - 2
    if nd not in _LAST or not use_native(x) or not x.is_contiguous() or x.numel() == 0 or x.shape[0] > 65535:
        return False
    return (x.dtype in (torch.bfloat16, torch.float16) and x.shape[1] % 8 == 0 and weight.shape[0] % 8 == 0
            and len(pad_tuple) >= 2 * nd and min(pad_tuple) >= 0 and not any(pad_tuple[2 * nd:]) and _plain(x))


def pad_channels_last(x: torch.Tensor, pad_tuple) -> torch.Tensor:
    """``x`` padded with zeros, in channels-last memory (see :func:`channels_last_usable`)."""
    nd = x.dim() - 2
    lo = tuple(int(a) for a in pad_tuple[:2 * nd:2][::-1])
    hi = tuple(int(a) for a in pad_tuple[1:2 * nd:2][::-1])
    return _ToChannelsLastFn.apply(x, lo, tuple(int(n) + a + b for n, a, b in zip(x.shape[2:], lo, hi)))


def channels_first(y: torch.Tensor) -> torch.Tensor:
    """``y.contiguous()`` of a channels-last tensor."""
    return _FromChannelsLastFn.apply(y, (0,) * (y.dim() - 2), tuple(int(n) for n in y.shape[2:]))


def pad(x: torch.Tensor, pad_tuple, value: float = 0.0) -> torch.Tensor:
    """``torch.nn.functional.pad(x, pad_tuple, value=value)``."""
    nd = x.dim() - 2
    spatial, rest = pad_tuple[:2 * nd], pad_tuple[2 * nd:]
    if (1 <= nd <= 3 and len(spatial) == 2 * nd and use_native(x) and x.dtype in _FILL
            and value in (0.0, float("-inf")) and x.numel() > 0 and x.is_contiguous() and any(spatial)
            and min(spatial) >= 0 and not any(rest) and _plain(x)):
        lo = tuple(int(a) for a in spatial[::2][::-1])
        hi = tuple(int(a) for a in spatial[1::2][::-1])
        return _ShiftCopyFn.apply(x, lo, tuple(int(n) + a + b for n, a, b in zip(x.shape[2:], lo, hi)), value != 0.0)
    return torch.nn.functional.pad(x, pad_tuple, mode="constant", value=value)
