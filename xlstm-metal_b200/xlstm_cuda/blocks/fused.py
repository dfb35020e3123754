"""When a fused launch may stand in for calls of modules.

The fused kernels have no backward and read the weights of the modules they replace.  They are taken where nobody can tell the
difference: no gradient is recorded, and each of those modules is the class the kernel restates, with nothing attached to its call.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch
import torch.nn as nn
from torch._C import _len_torch_dispatch_stack, _len_torch_function_stack
from torch._C._functorch import peek_interpreter_stack
from torch.autograd import forward_ad as _forward_ad
from torch.nn.modules import module as _module
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext


_PLAIN = frozenset((nn.Parameter, torch.Tensor, type(None)))


def _no_mode() -> bool:
    """No dispatch mode, and no function mode but the default device's."""
    return (_len_torch_dispatch_stack() == 0 and
            (_len_torch_function_stack() == 0 or all(type(m) is DeviceContext for m in _get_current_function_mode_stack())))


def plain_tensor(x: torch.Tensor, *weights: Optional[torch.Tensor]) -> bool:
    """Whether ``x`` and the weights are ordinary tensors whose memory a kernel may be handed: not subclasses, not wrapped by a
    function transform (vmap, grad, jvp; an ensemble's stacked weights are wrapped where ``x`` is not) or a forward-mode level,
    not being traced or compiled, no mode listens to the operators (make_fx, a counter), and not under autocast (which would pick
    another type for the module)."""
    if type(x) is not torch.Tensor or peek_interpreter_stack() is not None or _forward_ad._current_level >= 0 or not _no_mode():
        return False   # (the interpreter stack: every function transform that is running, whatever it has wrapped)
    for w in weights:
        if type(w) not in _PLAIN:
            return False
    return not (torch.jit.is_tracing() or torch.compiler.is_compiling() or torch.is_autocast_enabled(x.device.type))


def may_fuse(owner: nn.Module, x: torch.Tensor, *replaced: Tuple[nn.Module, type]) -> bool:
    """``replaced``: the modules whose calls the fused launch leaves out, with the class each is expected to be."""
    if torch.is_grad_enabled() and (x.requires_grad or any(p.requires_grad for p in owner.parameters())):
        return False
    if _module._global_forward_hooks or _module._global_forward_pre_hooks:
        return False
    return all(type(m) is cls and not m._forward_hooks and not m._forward_pre_hooks and "forward" not in m.__dict__
               for m, cls in replaced)


__all__ = ["may_fuse", "plain_tensor"]
