"""RMSNorm with the reference's interface (runtime/nn_models/modules/nonlinear/norm.py:4-16), one kernel."""
import torch
from torch import nn

from .. import glue
from ..linear.linear_base import calls_plainly


class RMSNorm(nn.Module):
    def __init__(self, weight, eps=1e-6):
        super().__init__()
        self.weight = weight
        self.variance_epsilon = eps

    def forward(self, hidden_states):
        y, _, _, _ = glue.rmsnorm(hidden_states, self.weight.to(hidden_states.dtype), self.variance_epsilon)
        return y

    def add(self, hidden_states, residual):
        """(h, forward(h)) with h = hidden_states + residual: one kernel where it has that form."""
        if hidden_states.dtype == residual.dtype and hidden_states.shape == residual.shape and hidden_states.is_cuda \
                and hidden_states.device == residual.device and calls_plainly(self, RMSNorm, _FORWARD) \
                and not (torch.is_grad_enabled() and (hidden_states.requires_grad or residual.requires_grad)):
            y, h, _, _ = glue.rmsnorm(hidden_states, self.weight.to(hidden_states.dtype), self.variance_epsilon,
                                      residual=residual)
            return h, y
        h = hidden_states + residual
        return h, self(h)


_FORWARD = RMSNorm.forward
