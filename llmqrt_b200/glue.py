"""Fused block-glue ops of the decode step: RMSNorm, rotary embedding + KV-cache write, SiLU*up."""
from __future__ import annotations

import torch

from . import _lib as L


def rmsnorm(x, weight, eps: float, residual=None, quantize: bool = False, want_y: bool = True, comm=None):
    """y = weight * T(x32 * rsqrt(mean(x32^2) + eps)) over the last dimension.

    residual: if given, h = x + residual (rounded to T) is normalised instead and also returned.
    quantize: also return the per-token int8 quantization (q, scale_f32[M]) of y.
    comm: a tp.PeerAllreduce; `residual` then holds this rank's tensor-parallel PARTIAL sums and is
          all-reduced over the group first -- inside the same kernel when it fits the communicator,
          else by NCCL (`residual` is then summed in place).  `residual` may also be the token returned
          by `comm.linear_push`: the GEMM has then sent the partial sums itself and this kernel only gathers.
    Returns (y or None, h or None, q or None, scale or None).
    """
    if residual is None or (comm is None and isinstance(residual, torch.Tensor)):
        return L.fast.rmsnorm(x, weight, eps, residual, quantize, want_y)
    from .tp import PushedPartial
    pushed = isinstance(residual, PushedPartial)          # the partial sums are already on their way to the peers
    dev = L.require_cuda(x, weight, None if pushed else residual)
    H = x.shape[-1]
    x2 = x.reshape(-1, H).contiguous()
    M = x2.shape[0]
    if pushed:
        if comm is None or (residual.M, residual.H) != (M, H):
            raise RuntimeError("rmsnorm: pushed partial sums need their communicator and the same [M, H]")
        h = torch.empty_like(x2)
        y = torch.empty_like(x2) if want_y else None
        q = torch.empty((M, H), dtype=torch.int8, device=dev) if quantize else None
        s = torch.empty(M, dtype=torch.float32, device=dev) if quantize else None
        with torch.cuda.device(dev):
            L.call("llmqrt_comm_allreduce_rmsnorm", comm.handle, None, L.ptr(x2), L.ptr(h), L.ptr(weight),
                   float(eps), L.ptr(y), L.ptr(q), L.ptr(s), L.dtype_code(x.dtype), M, H, L.stream(dev))
        return (y.reshape(x.shape) if y is not None else None, h.reshape(x.shape), q, s)
    r2 = residual.reshape(-1, H).contiguous()
    if r2.data_ptr() % 16:
        r2 = r2.clone()                                  # rank-local misalignment must not change the path
    if not (comm.eligible(r2) and comm.fits_rows(M, H)):
        torch.distributed.all_reduce(r2, group=comm.group)
        return L.fast.rmsnorm(x, weight, eps, r2, quantize, want_y)
    h = torch.empty_like(x2)
    y = torch.empty_like(x2) if want_y else None
    q = torch.empty((M, H), dtype=torch.int8, device=dev) if quantize else None
    s = torch.empty(M, dtype=torch.float32, device=dev) if quantize else None
    with torch.cuda.device(dev):
        L.call("llmqrt_comm_allreduce_rmsnorm", comm.handle, L.ptr(r2), L.ptr(x2), L.ptr(h), L.ptr(weight),
               float(eps), L.ptr(y), L.ptr(q), L.ptr(s), L.dtype_code(x.dtype), M, H, L.stream(dev))
    shape = x.shape
    return (y.reshape(shape) if y is not None else None, h.reshape(shape), q, s)


def rope_tables(head_dim: int, max_seq_len: int, theta: float, device) -> tuple[torch.Tensor, torch.Tensor]:
    """cos / sin of pos * theta**(-2i/d), fp32 [max_seq_len, d/2], built on the CPU exactly like the
    reference's freqs_cis table (runtime/nn_models/modules/nonlinear/attn.py:37-43) and then moved."""
    freqs = 1.0 / (theta ** (torch.arange(0, head_dim, 2)[: head_dim // 2].float() / head_dim))
    ang = torch.outer(torch.arange(max_seq_len), freqs).float()
    return torch.cos(ang).to(device).contiguous(), torch.sin(ang).to(device).contiguous()


def rope_kv_write(q, k, v, cos, sin, pos0: int = 0, pos_dev=None, k_cache=None, v_cache=None):
    """Rotates q [B,S,Hq,d] and k [B,S,Hkv,d] IN PLACE at positions pos + s and, when caches are given,
    writes the rotated k and v into rows pos + s of the caches [Bc, Smax, Hkv, d]."""
    L.fast.rope_kv_write(q, k, v, cos, sin, pos0, pos_dev, k_cache, v_cache)


def silu_mul(gate_up, quantize: bool = False, want_y: bool = True):
    """h = silu(gate) * up for gate_up [..., 2I] (gate first).  Returns (h or None, q or None, scale or None)."""
    return L.fast.silu_mul(gate_up, quantize, want_y)


def argmax_rows(x, base: int = 0):
    """(values [M] in x's dtype, base + indices [M] int64) of the row maxima of x [M, N] (fp16 / bf16, unit inner
    stride); ties go to the lowest index, a NaN counts as the greatest value."""
    dev = L.require_cuda(x)
    M, N = x.shape
    if x.stride(1) != 1:
        x = x.contiguous()
    val, idx = torch.empty(M, dtype=x.dtype, device=dev), torch.empty(M, dtype=torch.int64, device=dev)
    with torch.cuda.device(dev):
        L.call("llmqrt_argmax_rows", L.ptr(x), x.stride(0) if M > 1 else N, L.dtype_code(x.dtype), M, N, int(base), L.ptr(val),
               L.ptr(idx), L.stream(dev))
    return val, idx
