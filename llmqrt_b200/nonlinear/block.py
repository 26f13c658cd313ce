"""Pre-norm decoder block and layer stack with the reference's interfaces
(runtime/nn_models/modules/nonlinear/block.py:8-78, model.py:11-62)."""
from __future__ import annotations

from typing import List

import torch
import torch.nn as nn

from .._lib import fast
from ..fused_utils import FusedGateUpMLP
from ..linear import WQLinear_GEMM
from ..linear import linear_base
from .attn import QuantAttentionFused
from .cache import WindowedCache
from .norm import RMSNorm


class LlamaLikeBlock(nn.Module):
    def __init__(self, hidden_size, n_heads, n_kv_heads, qkv_layer, q_proj, k_proj, v_proj, o_proj, mlp, norm_1,
                 norm_2, dev, max_seq_len, rope_theta=10000, partial_rotary_factor=1.0, use_alibi=False,
                 head_dim=None):
        super().__init__()
        self.n_heads, self.n_kv_heads = n_heads, n_kv_heads
        self.head_dim = head_dim if head_dim else hidden_size // n_heads
        self.hidden_size = hidden_size
        self.norm_1 = norm_1.to(dev)
        self.attn = QuantAttentionFused(hidden_size, n_heads, n_kv_heads, qkv_layer, o_proj, dev=dev, q_proj=q_proj,
                                        k_proj=k_proj, v_proj=v_proj, max_seq_len=max_seq_len, use_alibi=use_alibi,
                                        rope_theta=rope_theta, partial_rotary_factor=partial_rotary_factor,
                                        head_dim=head_dim).to(dev)
        self.norm_2 = norm_2.to(dev)
        self.mlp = mlp.to(dev)
        self.device = dev

    def forward(self, hidden_states):
        out = fast.awq_block_step(self, hidden_states)       # a few 4-bit tokens: the whole step, one native call
        if out is not None:
            return out
        attn_output, _, _ = self.attn.forward(hidden_states=self.norm_1(hidden_states))
        hidden_states = hidden_states.to(attn_output.device)
        if type(self.norm_2) is RMSNorm:
            h, y = self.norm_2.add(hidden_states, attn_output)
        else:
            h = hidden_states + attn_output
            y = self.norm_2(h)
        return self.mlp.add_to(h, y) if type(self.mlp) is FusedGateUpMLP else h + self.mlp.forward(y)


class LlamaLikeModel(nn.Module):
    def __init__(self, vocab_size, blocks, embedding, norm):
        super().__init__()
        self.vocab_size = vocab_size
        self.embedding = embedding
        self.blocks: List[LlamaLikeBlock] = nn.ModuleList(blocks)
        self.norm = norm
        self.last_forward_num_tokens = 0

    @property
    def embed_tokens(self):
        return self.embedding

    @property
    def layers(self):
        return self.blocks

    @torch.inference_mode()
    def forward(self, input_ids: torch.Tensor, *args, **kwargs):
        # keep only the new tokens once the context has been processed (ref fused_utils.py:28-40)
        n_in = input_ids.shape[-1]
        n_new = n_in
        if n_in != 1:
            n_new = n_in - self.last_forward_num_tokens
            if n_new == 1:
                input_ids = input_ids[:, -1:]
        self.last_forward_num_tokens += n_new
        seqlen = input_ids.shape[1]
        for block in self.blocks:            # reset / roll the caches (ref fused_utils.py:12-25)
            a = block.attn
            exceeded = a.start_pos + seqlen > a.max_seq_len
            if seqlen > 1 and (exceeded or a.start_pos > 0):
                a.start_pos = a.cache.roll_kv_n_steps(a.start_pos, n=a.start_pos)
            elif seqlen == 1 and exceeded:
                a.start_pos = a.cache.roll_kv_n_steps(a.start_pos, n=100)
        h = self.embedding(input_ids)
        for layer in self.blocks:
            h = layer(h.to(layer.device))
        return self.norm(h)


# What has to be as it was defined for the native step to stand for the modules' own code, on the classes and on each object.
fast.set_block_classes(
    RMSNorm, QuantAttentionFused, FusedGateUpMLP, WQLinear_GEMM, WindowedCache,
    tuple((cls, name, getattr(cls, name)) for cls, names in
          ((RMSNorm, ("__call__", "forward", "add")), (QuantAttentionFused, ("forward",)),
           (FusedGateUpMLP, ("forward", "add_to", "_hidden")),
           (WQLinear_GEMM, ("__call__", "forward", "packed", "takes_tail", "silu_halves", "add_to")), (WindowedCache, ("to",)))
          for name in names),
    (linear_base._global_forward_hooks, linear_base._global_forward_pre_hooks, linear_base._global_backward_hooks,
     linear_base._global_backward_pre_hooks))
