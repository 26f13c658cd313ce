"""Attention entry points with the call signatures the reference uses from the flash-attn package.

`flash_attn_func` and `flash_attn_with_kvcache` accept the keyword subset of the reference's two
call sites (runtime/nn_models/modules/nonlinear/attn.py:290-298 and :305-315) and run this
package's own sm_100a kernels; arguments of the flash-attn API that the reference never sets are
accepted only at their neutral values.
"""
from __future__ import annotations

import math

import torch

from . import _lib as L


def _check_common(q, softmax_scale, dropout_p=0.0, window_size=(-1, -1), alibi_slopes=None):
    if dropout_p != 0.0:
        raise NotImplementedError("llmqrt_b200 attention: dropout is not supported (inference only)")
    if alibi_slopes is not None:
        raise NotImplementedError("llmqrt_b200 attention: ALiBi is not supported")
    if tuple(window_size) != (-1, -1):
        raise NotImplementedError("llmqrt_b200 attention: sliding windows are not supported")
    d = q.shape[-1]
    if softmax_scale is not None and not math.isclose(softmax_scale, d ** -0.5, rel_tol=1e-6):
        raise NotImplementedError("llmqrt_b200 attention: only the default softmax scale d**-0.5 is supported")
    if q.dtype not in (torch.float16, torch.bfloat16):
        raise TypeError("llmqrt_b200 attention: q/k/v must be fp16 or bf16")


def flash_attn_func(q, k, v, dropout_p=0.0, softmax_scale=None, causal=False, window_size=(-1, -1), softcap=0.0,
                    alibi_slopes=None, deterministic=False, return_attn_probs=False):
    """O = softmax(mask(Q K^T / sqrt(d))) V.  q [B,S,Hq,d]; k, v [B,S,Hkv,d]; returns [B,S,Hq,d]."""
    _check_common(q, softmax_scale, dropout_p, window_size, alibi_slopes)
    if return_attn_probs:
        raise NotImplementedError("llmqrt_b200 attention: attention probabilities are never materialised")
    return L.fast.attn_prefill(q, k, v, causal, softcap)


def kv_append(k_cache, v_cache, k, v, cache_seqlens=None, start_pos: int = 0):
    """cache[b, pos_b + s] = k/v[b, s] with pos_b = cache_seqlens[b] (device int32) or `start_pos`."""
    L.fast.kv_append(k_cache, v_cache, k, v, cache_seqlens, start_pos)


def attn_decode(q, k_cache, v_cache, seqlens, max_seqlen: int, softcap: float = 0.0, quantize: bool = False,
                k_new=None, v_new=None, cos=None, sin=None):
    """q [B, Hq, d] attends to rows [0, seqlens[b]) of the caches [Bc, Smax, Hkv, d]; returns [B, Hq, d].

    q may be a slice of a fused projection output (any batch stride, heads and d contiguous).
    quantize=True returns (out, out_q int8 [B, Hq*d], scale fp32 [B]): the per-token int8
    quantization of out, computed by the kernel that merges the KV splits.
    k_new / v_new [B, Hkv, d] (slices of a fused row allowed): the newest token's key and value are
    written into cache row seqlens[b] - 1 by the attention kernel itself; cos / sin (fp32
    [rows, d/2], see glue.rope_tables): q and the new key are rotated at that row's angle first.
    """
    res = L.fast.attn_decode(q, k_cache, v_cache, seqlens, max_seqlen, softcap, quantize, k_new, v_new, cos, sin)
    return res if quantize else res[0]


def flash_attn_with_kvcache(q, k_cache, v_cache, k=None, v=None, rotary_cos=None, rotary_sin=None,
                            cache_seqlens=None, cache_batch_idx=None, block_table=None, softmax_scale=None,
                            causal=False, window_size=(-1, -1), softcap=0.0, rotary_interleaved=True,
                            alibi_slopes=None, num_splits=0, max_seqlen_k=None):
    """Decode step over the KV cache.

    If k / v are given they are first written in place into the caches at row cache_seqlens[b];
    attention then covers rows [0, cache_seqlens[b] + k.shape[1]).  q is [B, 1, Hq, d] (one new token per
    sequence); the causal flag is immaterial for a single query.  `max_seqlen_k` (an addition to the
    flash-attn signature) bounds the longest sequence after the append so that the split-KV grid can be
    sized without reading cache_seqlens back; it defaults to the cache capacity.
    rotary_cos / rotary_sin ([rows, d/2], with k and v of one token and rotary_interleaved=False): q and
    the new key are rotated at angle row cache_seqlens[b] inside the attention kernel (half-split
    pairing, the convention of the reference's RoPE module); the interleaved pairing is not offered.
    """
    _check_common(q, softmax_scale, 0.0, window_size, alibi_slopes)
    if cache_batch_idx is not None or block_table is not None:
        raise NotImplementedError("llmqrt_b200 attention: batch indirection and paged caches are not supported")
    rotary = rotary_cos is not None or rotary_sin is not None
    if rotary and (rotary_interleaved or k is None or k.shape[1] != 1 or rotary_cos is None or rotary_sin is None):
        raise NotImplementedError("llmqrt_b200 attention: in-kernel rotary needs rotary_interleaved=False, both "
                                  "tables, and k / v of exactly one new token")
    B, Sq, Hq, d = q.shape
    if Sq != 1:
        raise NotImplementedError("flash_attn_with_kvcache: one query token per sequence (use flash_attn_func for prefill)")
    dev = L.require_cuda(q, k_cache, v_cache, k, v)
    if cache_seqlens is None:
        raise RuntimeError("flash_attn_with_kvcache: cache_seqlens is required")
    if k is not None and v is None:
        raise RuntimeError("flash_attn_with_kvcache: k and v must be given together")
    cap = k_cache.shape[1]                                 # (the native call also goes by the shorter of the two caches)
    bound = min(cap, max_seqlen_k) if max_seqlen_k is not None else cap
    if rotary:
        Hkv = k_cache.shape[2]
        if isinstance(cache_seqlens, int):
            cache_seqlens = torch.full((B,), cache_seqlens, dtype=torch.int32, device=dev)
        out = attn_decode(q.reshape(B, Hq, d), k_cache, v_cache, cache_seqlens + 1, bound, softcap,
                          k_new=k.to(k_cache.dtype).reshape(B, Hkv, d).contiguous(),
                          v_new=v.to(v_cache.dtype).reshape(B, Hkv, d).contiguous(),
                          cos=rotary_cos.float().contiguous(), sin=rotary_sin.float().contiguous())
        return out.reshape(B, 1, Hq, d)
    lens, add = (None, cache_seqlens) if isinstance(cache_seqlens, int) else (cache_seqlens, 0)
    if k is not None and k.shape[1] != 1:                  # several tokens: written by a kernel of their own
        kv_append(k_cache, v_cache, k.to(k_cache.dtype), v.to(v_cache.dtype), cache_seqlens=lens, start_pos=add)
        return L.fast.attn_decode_step(q, k_cache, v_cache, None, None, lens, add + k.shape[1], bound, softcap,
                                       None, None, False)
    return L.fast.attn_decode_step(q, k_cache, v_cache, k, v if k is not None else None, lens,
                                   add + (1 if k is not None else 0), bound, softcap, None, None, False)


def decode_rotary_step(q, k, v, k_cache, v_cache, cos, sin, pos: int, twice: bool = False, softcap: float = 0.0):
    """One kernel for a decode step whose sequences all stand at row `pos`: q and k [B, 1, H, d] are rotated at angle
    row `pos` (neither tensor changes), k and v are written to cache row pos -- with `twice` to row pos + 1 as well --
    and q attends to everything up to the last row written."""
    _check_common(q, None)
    n = pos + (2 if twice else 1)
    return L.fast.attn_decode_step(q, k_cache, v_cache, k, v, None, n, n, softcap, cos, sin, twice)
