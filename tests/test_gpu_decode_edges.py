"""Edges of the decode-sized kernels: splits merged by a cluster, the row appended by the attention kernel, and the
4-bit GEMM of a few tokens with and without the next step on its sums."""
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


def test_decode_step_without_keys():
    """A length of zero, as a number or as a tensor, gives zeros."""
    from llmqrt_b200.attention import flash_attn_with_kvcache
    q, kc = torch.randn(2, 1, 4, 64, device="cuda").half(), torch.randn(2, 40, 2, 64, device="cuda").half()
    for lens in (0, torch.zeros(2, dtype=torch.int32, device="cuda")):
        assert not flash_attn_with_kvcache(q, kc, kc.clone(), cache_seqlens=lens).any()


@pytest.mark.parametrize("pos,cap", [(0, 2), (0, 1), (63, 65), (64, 65), (63, 64), (127, 200), (511, 1000), (700, 708), (4094, 4200)])
@pytest.mark.parametrize("B,Hq,Hkv,d", [(1, 12, 2, 128), (3, 14, 2, 64)])
@pytest.mark.parametrize("twice", [True, False])
def test_decode_rotary_step(pos, cap, B, Hq, Hkv, d, twice):
    """Rotation, one or two cache rows (in one split or in two) and attention, against the kernels it replaces."""
    from llmqrt_b200 import glue
    from llmqrt_b200.attention import decode_rotary_step, flash_attn_with_kvcache
    if pos + 1 + twice > cap:
        pytest.skip("the second row does not fit")
    g = torch.Generator(device="cuda").manual_seed(pos + cap)
    kc, vc = (torch.randn(B, cap, Hkv, d, generator=g, device="cuda").half() for _ in range(2))
    row = torch.randn(B, 1, Hq + 2 * Hkv, d, generator=g, device="cuda").half()
    q, k, v = row[:, :, :Hq], row[:, :, Hq:Hq + Hkv], row[:, :, Hq + Hkv:]
    cos, sin = glue.rope_tables(d, cap, 1e6, "cuda")
    q1, k1, kc1, vc1 = q.clone(), k.clone(), kc.clone(), vc.clone()
    glue.rope_kv_write(q1, k1, v.clone(), cos, sin, pos0=pos, k_cache=kc1, v_cache=vc1)
    if twice:
        kc1[:, pos + 1], vc1[:, pos + 1] = k1[:, 0], v[:, 0]
    want = flash_attn_with_kvcache(q1, kc1, vc1, cache_seqlens=pos + 1 + twice, max_seqlen_k=pos + 1 + twice)
    before = row.clone()
    out = decode_rotary_step(q, k, v, kc, vc, cos, sin, pos, twice)
    assert torch.equal(row, before) and torch.equal(vc, vc1)
    assert rel_fro(kc, kc1.double()) < 1e-4 and rel_fro(out, want.double()) < 1e-3      # (one rounding of the rotated values)


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("K,N,G", [(32, 16, 32), (1536, 17920, 128), (2080, 48, 32), (8960, 1536, 128)])
def test_awq_tail(M, K, N, G):
    """The residual and silu(gate) * up on the GEMM's sums round as the separate kernels do."""
    from llmqrt_b200 import glue
    from llmqrt_b200.linear import WQLinear_GEMM
    g = torch.Generator(device="cuda").manual_seed(M + N)
    layer = WQLinear_GEMM(4, G, K, N, M % 2 == 1, "cuda")
    layer.qweight.random_(-2 ** 31, 2 ** 31 - 1, generator=g)
    layer.qzeros.random_(-2 ** 31, 2 ** 31 - 1, generator=g)
    layer.scales.uniform_(0.0001, 0.002, generator=g)
    if layer.bias is not None:
        layer.bias.normal_(0, 0.1, generator=g)
    x, res = torch.randn(1, M, K, generator=g, device="cuda").half(), torch.randn(1, M, N, generator=g, device="cuda").half()
    assert layer.takes_tail(x, 16)
    y = layer(x)
    assert torch.equal(layer.add_to(res, x), res + y)
    assert torch.equal(layer.silu_halves(x), glue.silu_mul(y)[0])
    assert not layer.takes_tail(torch.zeros(17, K, dtype=torch.float16, device="cuda"))


@pytest.mark.parametrize("M", [9, 12, 13, 16])
@pytest.mark.parametrize("K,N,G", [(3584, 37888, 128), (18944, 3584, 128), (1536, 17920, 64)])
def test_awq_tail_of_large_layers(M, K, N, G):
    """The sizes at which a plain call might prefer another kernel than its tail has."""
    test_awq_tail(M, K, N, G)


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("K,N,G", [(32, 8, 32), (96, 24, 32), (128, 16, 128), (1536, 2056, 128), (2080, 40, 32),
                                   (8960, 1536, 128), (4096, 17920, 64)])
def test_awq_few_tokens(M, K, N, G):
    """Ragged K (a chunk of 128 cut short), N off the 16-row block, every block width, with and without bias."""
    from llmqrt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int32)
    qz = torch.randint(-2 ** 31, 2 ** 31 - 1, (K // G, N // 8), generator=g, device="cuda", dtype=torch.int32)
    sc = torch.rand(K // G, N, generator=g, device="cuda").mul_(0.02).half()
    x = torch.randn(M, K, generator=g, device="cuda").half()
    bias = torch.randn(N, generator=g, device="cuda").half() if N % 16 else None
    want = x.double() @ ops.awq_dequantize(qw, sc, qz).double()
    if bias is not None:
        want += bias.double()
    y = ops.awq_gemm(x, ops.AwqPacked(qw, sc, qz), bias)
    assert rel_fro(y, want) < 5e-4                           # the fp16 rounding of the result (2^-11 at most per value)


@pytest.mark.parametrize("K,N,G", [(32, 8, 32), (40, 24, 8), (1536, 72, 128), (8960, 264, 64)])
def test_awq_expansion_bits(K, N, G):
    """Word counts off the block's 1024, and a K that no 16-byte load divides."""
    from llmqrt_b200 import ops
    from oracle import awq as oa
    qw, qz, sc = oa.random_layer(K, N, G, seed=K)
    packed = ops.AwqPacked(qw.cuda(), sc.cuda(), qz.cuda())
    assert torch.equal(ops.awq_dequantize_t(packed).cpu(), oa.dequantize(qw, qz, sc, G).t())


@pytest.mark.parametrize("lens,cap", [([1], 4096), ([63], 4096), ([64], 2048), ([65], 4096), ([500], 4096), ([511], 4096),
                                      ([512], 4096), ([513, 2, 4000], 4096), ([1025, 64], 2048), ([3000], 3072)])
@pytest.mark.parametrize("Hq,Hkv,d", [(12, 2, 128), (14, 2, 64)])
@pytest.mark.parametrize("append", [True, False])
def test_short_sequences_in_a_large_cache(lens, cap, Hq, Hkv, d, append):
    """A cluster's blocks share out the sequence's own length, whatever the cache could hold."""
    test_decode_step(lens, cap, None, Hq, Hkv, d, torch.float16, append)


@pytest.mark.parametrize("pos,cap", [(0, 2), (0, 1), (63, 65), (64, 66), (127, 200), (700, 2048), (4094, 4200)])
@pytest.mark.parametrize("B,Hq,Hkv,d,dt", [(1, 12, 2, 128, torch.float16), (3, 14, 2, 64, torch.bfloat16)])
@pytest.mark.parametrize("twice", [True, False])
def test_decode_rotary_step_against_64_bits(pos, cap, B, Hq, Hkv, d, dt, twice):
    from llmqrt_b200 import glue
    from llmqrt_b200.attention import decode_rotary_step
    if pos + 1 + twice > cap:
        pytest.skip("the second row does not fit")
    g = torch.Generator(device="cuda").manual_seed(pos + cap)
    kc, vc = (torch.randn(B, cap, Hkv, d, generator=g, device="cuda").to(dt) for _ in range(2))
    row = torch.randn(B, 1, Hq + 2 * Hkv, d, generator=g, device="cuda").to(dt)
    q, k, v = row[:, :, :Hq], row[:, :, Hq:Hq + Hkv], row[:, :, Hq + Hkv:]
    cos, sin = glue.rope_tables(d, cap, 1e6, "cuda")
    ang = pos * 1e6 ** (-torch.arange(0, d, 2, dtype=torch.float64, device="cuda") / d)

    def rotate(x):
        a, b = x[:, 0].double().chunk(2, -1)
        return torch.cat([a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()], -1)

    want_k, want_v = kc.double(), vc.double()
    for r in range(pos, pos + 1 + twice):
        want_k[:, r], want_v[:, r] = rotate(k), v[:, 0].double()
    n, rq = pos + 1 + twice, rotate(q)
    want = torch.stack([_attend(rq[b], want_k[b, :n], want_v[b, :n]) for b in range(B)])
    out = decode_rotary_step(q, k, v, kc, vc, cos, sin, pos, twice)
    eps = 2 ** -11 if dt == torch.float16 else 2 ** -8
    assert torch.equal(vc.double(), want_v)
    # the angle in fp32 (position times 2^-24, twice) and one rounding of the rotated key
    assert rel_fro(kc, want_k) < eps + 4 * pos * 2 ** -24
    # q, k, P and the result rounded once each; scores of d products of unit variance pass on sqrt(2) of q's and k's
    assert rel_fro(out[:, 0], want) < 4 * eps + 8 * pos * 2 ** -24


@pytest.mark.parametrize("B", [16, 17, 18, 33, 35])
@pytest.mark.parametrize("Hq,Hkv,d", [(12, 2, 128), (14, 2, 64), (8, 1, 128)])
def test_as_many_clusters_as_fit_and_more(B, Hq, Hkv, d):
    """The largest batches that clusters merge, and the first ones left to the merge kernel."""
    test_decode_step([300 + 10 * b % 200 for b in range(B)], 512, None, Hq, Hkv, d, torch.float16, True)
