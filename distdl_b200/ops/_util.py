"""Small helpers shared by the op wrappers."""
from __future__ import annotations

import os

import torch

from .. import _native


def stream_ptr(t: torch.Tensor = None) -> int:
    """Raw handle of the current CUDA stream (kernels launch on torch's stream).  Asked for at every
    launch: 0.3 us this way, 5 us through a ``torch.cuda.Stream`` object."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


# the process environment as os.environ keeps it (bytes on POSIX): a look-up per launch that sees every
# change made through os.environ, without the encoding and the exception of os.environ.get
_environ = getattr(os.environ, "_data", None)


def env(name: str, default: str) -> str:
    """``os.environ.get(name, default)`` at a third of its cost."""
    if _environ is None:
        return os.environ.get(name, default)
    v = _environ.get(name.encode())
    return default if v is None else os.fsdecode(v)


def ptr(t):
    return 0 if t is None else t.data_ptr()


def _leaf_node(owner, ctx, k):
    """The node that accumulates into the leaf ``owner``: the end of the views that lead from input ``k`` of the running
    node ``ctx`` to it, a microsecond away; asked of the leaf itself, for four, where that is not the way."""
    if ctx is not None:
        node = ctx.next_functions[k][0]
        further = node.next_functions
        while len(further) == 1:
            node = further[0][0]
            further = node.next_functions
        if getattr(node, "variable", None) is owner:
            return node
    return torch.autograd.graph.get_gradient_edge(owner).node


def main_grad_now(acc, owner, ctx=None, k=0):
    """``acc``, the fp32 accumulator that stands for the gradient of the leaf ``owner``, if the backward pass that is
    running would hand that gradient to nobody but the optimizer's own hook; None where it has to go through autograd:
    the leaf has hooks of the user's, or the pass does not accumulate into it (``torch.autograd.grad``, ``inputs=`` of
    ``backward``) or builds a graph.  Asked in the backward pass (of ``ctx``, whose input ``k`` the leaf became), so that
    hooks of any moment count.  ``owner`` None: a gathered weight, whose gradient is never autograd's."""
    if acc is None or owner is None:
        return acc
    after = owner._post_accumulate_grad_hooks
    if torch.is_grad_enabled() or owner._backward_hooks \
            or (after and not all(getattr(h, "into_main_grad", False) for h in after.values())):
        return None
    try:
        runs = torch._C._will_engine_execute_node(_leaf_node(owner, ctx, k))
    except RuntimeError:            # the pass captures the gradient of this leaf
        return None
    return acc if runs else None


def use_native(*tensors) -> bool:
    """True when the operands live on a CUDA device: the hand-written kernels run.

    CPU tensors take the plain PyTorch path, which exists for the gloo
    plumbing and adjoint tests only.  On a CUDA device a missing native
    library is an error, never a silent fallback.
    """
    if env("DISTDL_FORCE_TORCH", "0") == "1":
        return False            # baseline arm: library kernels (cuBLAS / cuDNN / ATen) everywhere
    for t in tensors:
        if t is not None and t.is_cuda:
            if not _native.available():
                raise ImportError("distdl_b200 native library missing on a CUDA machine; "
                                  "run `python -m distdl_b200._build`")
            return True
    return False
