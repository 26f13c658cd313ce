"""Edges of the decode-sized kernels: splits merged by a cluster, the row appended by the attention kernel, and the
4-bit GEMM of at most eight tokens."""
import pytest
import torch

from tests.util import rel_fro

pytestmark = pytest.mark.gpu


def _attend(q, k, v):
    """q [Hq, d], k / v [L, Hkv, d] in 64 bits on the GPU."""
    Hq, d = q.shape
    rep = Hq // k.shape[1]
    kk, vv = (t.double().repeat_interleave(rep, 1) for t in (k, v))
    p = (torch.einsum("hd,lhd->hl", q.double(), kk) * d ** -0.5).softmax(-1)
    return torch.einsum("hl,lhd->hd", p, vv)


# (before the append) lengths, cache rows, bound on the rows attended to; 1 to 8 splits, the first size beyond the
# cluster's, more blocks than fit at once, sequences without keys and one whose new row lies beyond the bound
@pytest.mark.parametrize("lens,cap,bound", [
    ([5], 64, None), ([64], 65, None), ([127, 0], 128, None), ([199, 3, 60], 200, None), ([480], 512, 500),
    ([511, 512], 520, None), ([4000], 4096, None), ([4090], 4100, None), ([700] * 3 + [1], 2048, 701),
    ([300] * 30, 512, None), ([90, 300, 20], 400, 100)])
@pytest.mark.parametrize("Hq,Hkv,d", [(12, 2, 128), (14, 2, 64), (4, 4, 128)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("append", [True, False])
def test_decode_step(lens, cap, bound, Hq, Hkv, d, dt, append):
    from llmqrt_b200.attention import flash_attn_with_kvcache
    g = torch.Generator(device="cuda").manual_seed(len(lens) + cap)
    B = len(lens)
    kc, vc = (torch.randn(B, cap, Hkv, d, generator=g, device="cuda").to(dt) for _ in range(2))
    row = torch.randn(B, 1, Hq + 2 * Hkv, d, generator=g, device="cuda").to(dt)       # slices of a fused projection
    q, k, v = row[:, :, :Hq], row[:, :, Hq:Hq + Hkv], row[:, :, Hq + Hkv:]
    want_k, want_v = kc.clone(), vc.clone()
    top = min(cap, bound) if bound else cap
    seqlens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    if append:
        for b, n in enumerate(lens):
            want_k[b, n], want_v[b, n] = k[b, 0], v[b, 0]
    want = torch.zeros(B, 1, Hq, d, dtype=torch.float64, device="cuda")
    for b, n in enumerate(lens):
        n = min(n + append, top)
        if n:
            want[b, 0] = _attend(q[b, 0], want_k[b, :n], want_v[b, :n])
    out = flash_attn_with_kvcache(q, kc, vc, k if append else None, v if append else None, cache_seqlens=seqlens,
                                  max_seqlen_k=bound)
    assert torch.equal(kc, want_k) and torch.equal(vc, want_v)
    # one rounding of P and one of the result: 2^-11 (fp16) or 2^-8 (bf16) each
    assert rel_fro(out, want) < (1e-3 if dt == torch.float16 else 8e-3)
    if len(set(lens)) == 1:                                  # the same lengths as one number
        out2 = flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens[0] + append, max_seqlen_k=bound)
        assert rel_fro(out2, out.double()) < (1e-3 if dt == torch.float16 else 8e-3)
