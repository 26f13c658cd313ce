import torch
from torch.nn.modules.module import (_global_backward_hooks, _global_backward_pre_hooks, _global_forward_hooks,
                                     _global_forward_pre_hooks)

from .._lib import fast


def forward_is(layer: torch.nn.Module, cls, forward) -> bool:
    """Whether layer.forward is `forward`, the one `cls` was defined with: not a subclass's, and replaced neither on the
    instance (as offloading wrappers attach) nor on the class."""
    return type(layer) is cls and cls.forward is forward and "forward" not in layer.__dict__


def calls_plainly(layer: torch.nn.Module, cls, forward) -> bool:
    """Whether layer(x) runs `forward` and nothing else: no hook of its own and none of all modules, either.  (Asked three
    times per block and step: straight from the instance's dictionary it takes a third of a microsecond.)"""
    d = layer.__dict__
    return not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"]
                or _global_forward_hooks or _global_forward_pre_hooks or _global_backward_hooks or _global_backward_pre_hooks
                or "forward" in d or "_compiled_call_impl" in d and d["_compiled_call_impl"] is not None) \
        and type(layer) is cls and cls.forward is forward


class LinearBase(torch.nn.Module):
    """Common base of the quantized linear layers (ref: runtime/nn_models/modules/linear/linear_base.py)."""

    def forward(self, x):
        raise NotImplementedError


def tensor_key(*tensors):
    """Identity + in-place-version key of tensors, used to invalidate caches derived from buffers."""
    return fast.tensor_key(*tensors)
