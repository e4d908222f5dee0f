"""Base class of every distributed layer.

The call runs the layer's set-up lazily, on the first call and again
whenever the structure of the input (shape, dtype, requires_grad) changes
(``src/distdl/nn/module.py:34-56``, ``:101-112``); set
``DISTDL_CHECK_INPUT_CHANGED=0`` to skip the re-check.  The backend that is
active when the layer is built is captured on the instance.
"""
import torch
from torch.nn.modules import module as _torch_module

from .. import backends, config


def hooked(module):
    """True where a call of ``module`` is more than its ``forward``: it, or every module, has hooks."""
    return bool(module._forward_pre_hooks or module._forward_hooks or module._backward_pre_hooks
                or module._backward_hooks or _torch_module._has_any_global_hook())


class Module(torch.nn.Module):
    def __init__(self):
        super().__init__()
        self._distdl_backend = backends.backend
        self._distdl_is_setup = False

    # Set in every forward pass: plain attributes, never parameters, buffers or sub-modules (also where a gather
    # that is the identity hands the Parameter itself on), so that they skip torch.nn.Module's registration.
    _distdl_plain = frozenset(("weight_buffer", "bias_buffer", "buffers_gathered", "gamma_buffer", "beta_buffer",
                               "_distdl_is_setup", "_input_tensor_structure"))

    def __setattr__(self, name, value):
        if name in Module._distdl_plain:
            object.__setattr__(self, name, value)
        else:
            super().__setattr__(name, value)

    def __call__(self, *input, **kwargs):
        # a registered pre-hook only beside others, so that a module without hooks takes torch.nn.Module's short way
        if self._forward_pre_hooks or _torch_module._global_forward_pre_hooks:
            self._register_set_up()
        elif self._distdl_module_requires_reset(input):
            Module._distdl_forward_pre_hook(self, input)
        return super().__call__(*input, **kwargs)

    def register_forward_pre_hook(self, hook, *, prepend=False, with_kwargs=False):
        self._register_set_up()
        return super().register_forward_pre_hook(hook, prepend=prepend, with_kwargs=with_kwargs)

    def _register_set_up(self):
        """Set-up sees the input that global pre-hooks and those registered with ``prepend`` leave, and runs before the
        module's other pre-hooks."""
        if all(h is not Module._distdl_forward_pre_hook for h in self._forward_pre_hooks.values()):
            super().register_forward_pre_hook(Module._distdl_forward_pre_hook)

    @staticmethod
    def _distdl_forward_pre_hook(self, input):
        if self._distdl_module_requires_reset(input):
            if self._distdl_is_setup:
                self._distdl_module_teardown(input)
            self._distdl_module_setup(input)

    def _distdl_module_setup(self, input):
        """Layer-specific set-up from the structure of ``input``."""

    def _distdl_module_teardown(self, input):
        """Releases whatever set-up allocated."""

    def _distdl_input_changed(self, input):
        """Layer-specific definition of "the input changed"."""
        return False

    def _distdl_module_requires_reset(self, input):
        if not self._distdl_is_setup:
            return True
        return bool(config.check_input_changed) and bool(self._distdl_input_changed(input))


def reset_setup(module: torch.nn.Module):
    """Makes every distributed layer below ``module`` run its set-up again at its next call.

    Set-up is collective, but a layer re-runs it only when THIS worker sees its input structure change.
    When shapes change in a way some workers cannot see (a new sequence length that leaves one worker's
    shard as long as before; a worker that feeds zero-volume tensors), call this on all workers before
    the next forward pass, so that all of them take part."""
    for m in module.modules():
        if isinstance(m, Module) and m._distdl_is_setup:
            m._distdl_module_teardown(None)
            m._distdl_is_setup = False
