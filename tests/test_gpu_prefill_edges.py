"""Prompt attention at the edges of its 128-key and 128-row tiles, with maxima that keep moving."""
import pytest
import torch

from tests.util import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 63, 64, 65, 127, 128, 129, 192, 193, 255, 256, 257, 320, 385, 641])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dt,d,growth", [(torch.float16, 128, 0), (torch.bfloat16, 64, 0), (torch.float16, 64, 40), (torch.float16, 128, 40),
                                         (torch.bfloat16, 128, -40)])
def test_prefill_halves(S, causal, dt, d, growth):
    """growth: the score rises (falls) by that many powers of e over every 64 keys, so a row's reference maximum moves
    in every tile and the accumulator is rescaled while a product may be on its way (or never again)."""
    from llmqrt_b200.attention import flash_attn_func
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(2, S, h, d, generator=g, device="cuda") for h in (4, 2, 2))
    if growth:
        q[..., 0] = 8.0
        k[..., 0] = growth * d ** 0.5 / 8 * torch.arange(S, device="cuda")[None, :, None] / 64
    q, k, v = (t.to(dt) for t in (q, k, v))
    out = flash_attn_func(q, k, v, causal=causal)
    s = torch.einsum("bshd,bthd->bhst", q.double(), k.double().repeat_interleave(2, 2)) * d ** -0.5
    if causal:
        s.masked_fill_(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.einsum("bhst,bthd->bshd", s.softmax(-1), v.double().repeat_interleave(2, 2))
    # P and the result are rounded to 16 bits: 2^-11 (fp16) or 2^-8 (bf16) each at most
    assert rel_fro(out, want) < (1e-3 if dt == torch.float16 else 8e-3)


def test_prefill_row_sum_order():
    """The eight partial sums of a row's P are added as neighbours, then as neighbouring pairs.  Two keys of weight 1
    share the first one; two of weight 0.8 * 2^-23, each below half a unit of the sum and together above it, lie in the
    third and the fourth.  The result is made a tie of fp16 but for them: added as a pair they tip it, as 64 bits do."""
    from llmqrt_b200.attention import flash_attn_func
    S, d = 128, 64
    q, k, v = (torch.zeros(1, S, 1, d, device="cuda") for _ in range(3))
    q[..., 0] = 16.0
    k[..., 0] = -1000.0                                      # e^-2000: weight 0
    k[:, [0, 8], :, 0] = 0.0
    k[:, [2, 3], :, 0] = -8.0859375                          # 2^(-8.0859 * 16 / 8 * log2(e)) = 0.795 * 2^-23
    v[:, 0], v[:, 8] = 1 + 2 ** -10, 1 + 2 ** -9
    out = flash_attn_func(*(t.half() for t in (q, k, v)), causal=False)
    p = (q[0, :, 0].double() @ k[0, :, 0].double().t() * d ** -0.5).softmax(-1)
    assert torch.equal(out[0, :, 0], (p @ v[0, :, 0].double()).half())


@pytest.mark.parametrize("S,key", [(257, 128), (300, 250), (513, 383), (640, 511)])
@pytest.mark.parametrize("d,dt", [(64, torch.bfloat16), (128, torch.float16)])
def test_prefill_one_row_leaps(S, key, d, dt):
    """The first half of a tile's P is computed with the reference as it stands.  Here the score of ONE key outgrows it by
    far more than 2^8, for one row of a warp only, in either half of a tile after the first: the half is done again, the
    row's earlier sum and output are scaled down, and the warp's other rows keep their reference.  A row that meets a NaN
    is NaN and no other."""
    from llmqrt_b200.attention import flash_attn_func
    g = torch.Generator(device="cuda").manual_seed(S + key)
    q, k, v = (torch.randn(1, S, 2, d, generator=g, device="cuda") for _ in range(3))
    leap, nan = S - 40, S - 3
    q[..., 0], k[..., 0] = 0.0, 0.0
    q[:, leap, :, 0], k[:, key, :, 0] = 40.0, 40.0
    q[:, nan, 0, 1] = float("nan")
    q, k, v = (t.to(dt) for t in (q, k, v))
    out = flash_attn_func(q, k, v, causal=True)
    s = torch.einsum("bshd,bthd->bhst", q.double(), k.double()) * d ** -0.5
    s.masked_fill_(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.einsum("bhst,bthd->bshd", s.softmax(-1), v.double())
    assert out[0, nan, 0].isnan().all() and int(out.isnan().sum()) == d
    keep = [i for i in range(S) if i != nan]
    # as above: P and the result rounded to 16 bits
    assert rel_fro(out[:, keep], want[:, keep]) < (1e-3 if dt == torch.float16 else 8e-3)
    assert rel_fro(out[:, leap], want[:, leap]) < (1e-3 if dt == torch.float16 else 8e-3)


@pytest.mark.parametrize("S", [1, 17, 31, 32, 33, 40, 41])
@pytest.mark.parametrize("d,dt", [(64, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("softcap", [0.0, 5.0])
def test_prefill_short_sequences(S, d, dt, softcap):
    """The form for short sequences and the general one, up to both sides of the line between them: a causal prompt's rows have
    the bits of the same rows of a longer one (keys that a row does not see count as zeros)."""
    from llmqrt_b200.attention import flash_attn_func
    g = torch.Generator(device="cuda").manual_seed(S + d)
    q, k, v = (torch.randn(3, 100, h, d, generator=g, device="cuda").to(dt) for h in (4, 2, 2))
    whole = flash_attn_func(q, k, v, causal=True, softcap=softcap)
    out = flash_attn_func(*(t[:, :S].contiguous() for t in (q, k, v)), causal=True, softcap=softcap)
    assert torch.equal(out, whole[:, :S])
    kk, vv = (t[:, :S].double().repeat_interleave(2, 2) for t in (k, v))
    s = torch.einsum("bshd,bthd->bhst", q[:, :S].double(), kk) * d ** -0.5
    if softcap:
        s = softcap * (s / softcap).tanh()
    want = torch.einsum("bhst,bthd->bshd", s.softmax(-1), vv)
    out = flash_attn_func(*(t[:, :S].contiguous() for t in (q, k, v)), causal=False, softcap=softcap)
    assert rel_fro(out, want) < (1e-3 if dt == torch.float16 else 8e-3)      # P and the result rounded to 16 bits
