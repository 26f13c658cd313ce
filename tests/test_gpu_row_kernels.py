"""The vectorised row kernels at the edges of their ranges, against the general path or the CPU oracle."""
import pytest
import torch


pytestmark = pytest.mark.gpu


def _g(seed=0):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("B,S,Hq,Hkv,d,dt", [
    (1, 1, 14, 2, 64, torch.float16), (2, 3, 28, 4, 128, torch.bfloat16), (3, 65, 33, 3, 128, torch.float16),
    (1, 7, 1, 1, 16, torch.bfloat16), (2, 5, 64, 8, 256, torch.float16), (1, 2, 0, 4, 128, torch.float16)])
def test_rope_vectorised_equals_general(B, S, Hq, Hkv, d, dt):
    """Rows off a 16-byte boundary take the one-element form; both round the same sums, so the bits agree."""
    from llmqrt_b200 import glue
    g, H, pos0, cap = _g(1), Hq + 2 * Hkv, 9, 9 + S + 2
    x = torch.randn(B, S, H * d, generator=g, device="cuda").to(dt)
    cos, sin = glue.rope_tables(d, cap, 1e4, "cuda")
    got = []
    for pad in (0, 4):                                       # token stride H * d + 4: 8-byte aligned rows only
        buf = torch.zeros(B, S, H * d + pad, dtype=dt, device="cuda")
        buf[..., :H * d] = x
        rows = buf[..., :H * d].unflatten(-1, (H, d))
        q, k, v = rows[:, :, :Hq], rows[:, :, Hq:Hq + Hkv], rows[:, :, Hq + Hkv:]
        kc, vc = (torch.zeros(B, cap, Hkv, d, dtype=dt, device="cuda") for _ in range(2))
        if Hq == 0:
            q = rows[:, :, :0]
        glue.rope_kv_write(q, k, v, cos, sin, pos0=pos0, k_cache=kc, v_cache=vc)
        got.append((buf[..., :H * d].clone(), kc, vc))
    for a, b in zip(*got):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert torch.equal(got[0][2][:, pos0:pos0 + S].flatten(2), x[..., (Hq + Hkv) * d:])
    assert not got[0][1][:, :pos0].any() and not got[0][1][:, pos0 + S:].any()


@pytest.mark.parametrize("I", [8, 24, 4096, 4104, 8960, 12296, 18944, 24584, 32768, 32776])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_silu_one_block_per_row(I, dt):
    """300 rows: one block each, one to eight units per thread (the last size is beyond that form)."""
    from llmqrt_b200 import glue
    from oracle import quant as oq
    gu = torch.randn(300, 2 * I, generator=_g(2), device="cuda") * 4
    gu[7, : I // 2] = -120.0                                 # e^-gate overflows: silu is 0
    gu[9, 0] = float("inf")                                  # infinite scale: 0, and 0 for inf / inf
    gu = gu.to(dt)
    y, q, s = glue.silu_mul(gu, quantize=True)
    g32, u32 = gu[:, :I].double(), gu[:, I:].float()
    act = (g32 * torch.sigmoid(g32)).to(dt)
    want = (act.float() * u32).to(dt)
    # the first rounding may fall the other way (one unit: a relative 2 eps at most), and then the second as well
    eps = 2.0 ** (-10 if dt == torch.float16 else -7)
    tiny = 2.0 ** -22 if dt == torch.float16 else 1e-30
    ok = (y.float() - want.float()).abs() <= 2.02 * eps * want.float().abs() + tiny * (1 + u32.abs())
    assert bool((ok | ~torch.isfinite(want)).all())
    rows = [r for r in range(300) if r != 9]
    qr, sr = oq.quantize_int8(y[rows].cpu(), per_token=True)
    assert torch.equal(q[rows].cpu(), qr) and torch.equal(s[rows].cpu(), sr.float().reshape(-1))
    assert torch.isinf(s[9]) and not q[9].any()


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_silu_of_every_gate(dt):
    """All 65536 gates: every variant gives the bits of the staged one, which divides by 1 + e^-gate, and those are within
    a rounding of 64 bits as long as e^-gate is finite in fp32 (beyond, the result is a zero)."""
    from llmqrt_b200 import glue
    gates = torch.arange(-2 ** 15, 2 ** 15, device="cuda", dtype=torch.int32).to(torch.int16).view(dt).reshape(16, 4096)
    rows = torch.cat([gates, torch.ones_like(gates)], 1)
    staged = torch.zeros(16, 8192 + 8, dtype=dt, device="cuda")              # rows off a 16-byte boundary
    staged[:, 1:8193] = rows
    want = glue.silu_mul(staged[:, 1:8193])[0]
    many = glue.silu_mul(rows.repeat(20, 1))[0]                               # one block per row
    for got in (glue.silu_mul(rows)[0], many[:16], many[-16:]):
        assert torch.equal(got.isnan(), want.isnan())
        ok = ~want.isnan()
        assert torch.equal(got[ok].view(torch.int16), want[ok].view(torch.int16))
    g = gates.double()
    assert torch.equal(want.isnan(), g.isnan() | (g == -float("inf")))
    exact, y = g * torch.sigmoid(g), want.double()
    ok = g.isfinite() & (g > -88.7)                                          # e^88.7 is the last below the largest fp32
    half = torch.finfo(dt).eps / 2
    tiny = torch.finfo(dt).smallest_normal * torch.finfo(dt).eps              # spacing of the subnormals
    # one rounding to 16 bits after a relative error of a few 2^-24
    assert bool(((y - exact).abs() <= half * 1.01 * exact.abs() + tiny * 0.51)[ok].all())
    assert bool((y[(g < -90) & g.isfinite()] == 0).all()) and bool((y[g == float("inf")] == float("inf")).all())


@pytest.mark.parametrize("M,K", [(1, 8), (3, 1032), (3, 18944), (2, 65536), (2, 65544), (300, 1016), (300, 1024), (300, 2056),
                                 (300, 4104), (296, 8200), (1200, 896)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_quantizers_match_oracle_bits(M, K, dt):
    """Every unit count per thread and both row splits, a zero row and an infinite one; flat per-tensor passes."""
    from llmqrt_b200 import ops
    from oracle import quant as oq
    x = torch.randn(M, K, generator=_g(3), device="cuda")
    x = (x * torch.exp(4 * torch.randn(M, 1, generator=_g(4), device="cuda"))).clamp(-60000, 60000).to(dt)
    if M > 2:
        x[1] = 0
    c = x.cpu()
    q, _, s = ops.quantize_int8(x, True)
    qr, sr = oq.quantize_int8(c, True)
    assert torch.equal(q.cpu(), qr) and torch.equal(s.cpu(), sr.float().reshape(-1))
    q, s = ops.quantize_fp8(x, True)
    qr, sr = oq.quantize_fp8(c, True)
    nan = qr.float().isnan()
    assert torch.equal(q.cpu().float().isnan(), nan) and torch.equal(s.cpu().reshape(-1), sr.float().reshape(-1))
    assert torch.equal(q.cpu().view(torch.uint8)[~nan], qr.view(torch.uint8)[~nan])
    q, _, s = ops.quantize_int8(x, False)
    qr, sr = oq.quantize_int8(c, False)
    assert torch.equal(q.cpu(), qr) and float(s) == float(sr)
    q, s = ops.quantize_fp8(x, False)
    qr, sr = oq.quantize_fp8(c, False)
    assert torch.equal(q.cpu().view(torch.uint8), qr.view(torch.uint8)) and float(s) == float(sr)
    scale = torch.tensor([0.37], device="cuda")
    q = ops.quantize_fp8_static(x, scale)
    assert torch.equal(q.cpu().view(torch.uint8), oq.quantize_fp8_static(c, scale.cpu()).view(torch.uint8))
    if M > 2:
        x[2, 0] = float("inf")
        q, _, s = ops.quantize_int8(x[2:3], True)
        assert torch.isinf(s).all() and not q.any()


@pytest.mark.parametrize("H", [8, 1016, 1024, 1032, 3584, 4104, 8192])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_rmsnorm_small_blocks(H, dt):
    """300 rows: one small block each, one to eight units per thread."""
    from llmqrt_b200 import glue
    from oracle import quant as oq
    x, r = (torch.randn(300, H, generator=_g(5 + i), device="cuda").to(dt) for i in range(2))
    w = (1 + 0.1 * torch.randn(H, generator=_g(7), device="cuda")).to(dt)
    y, h, q, s = glue.rmsnorm(x, w, 1e-6, residual=r, quantize=True)
    want_h = (x.float() + r.float()).to(dt)
    assert torch.equal(h, want_h)
    n = (want_h.double() * (want_h.double().square().mean(-1, keepdim=True) + 1e-6).rsqrt()).float().to(dt)
    want = (n.float() * w.float()).to(dt)
    eps = 2.0 ** (-10 if dt == torch.float16 else -7)        # one unit in the last place of the first rounding, passed on
    assert bool(((y.float() - want.float()).abs() <= 2.02 * eps * want.float().abs()).all())
    qr, sr = oq.quantize_int8(y.cpu(), True)
    assert torch.equal(q.cpu(), qr) and torch.equal(s.cpu(), sr.float().reshape(-1))
    y2, _, _, _ = glue.rmsnorm(want_h, w, 1e-6)
    assert torch.equal(y2, y)


@pytest.mark.parametrize("H", [8, 264, 1016, 1032, 2056, 3584, 4104, 8192])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_rmsnorm_bits_do_not_depend_on_the_batch(H, dt):
    """Many rows take small blocks with several units per thread, few rows one unit per thread: one order of the sum."""
    from llmqrt_b200 import glue
    x, r = (torch.randn(600, H, generator=_g(8 + i), device="cuda").to(dt) for i in range(2))
    w = (1 + 0.1 * torch.randn(H, generator=_g(10), device="cuda")).to(dt)
    many = glue.rmsnorm(x, w, 1e-6, residual=r, quantize=True)
    for i in range(0, 600, 200):
        few = glue.rmsnorm(x[i:i + 200], w, 1e-6, residual=r[i:i + 200], quantize=True)
        for a, b in zip(many, few):
            a = a[i:i + 200]
            assert torch.equal(a.view(torch.int16), b.view(torch.int16)) if a.dtype == dt else torch.equal(a, b)


@pytest.mark.parametrize("M,N", [(1, 1), (3, 7), (2, 4096), (64, 8200), (5, 9001), (64, 152064), (300, 1024)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_argmax_rows(M, N, dt):
    """Ties (16-bit values repeat), signed zeros, infinities and NaN; one CTA and a cluster of them; odd rows."""
    from llmqrt_b200 import glue
    x = torch.randn(M, N, generator=_g(11), device="cuda").to(dt)
    if N > 4:
        x[0] = -1.0
        x[0, 2], x[0, N - 1] = 0.0, 0.0                      # a tie far apart
        x[0, 1] = -0.0                                       # equal to +0: the lowest index wins
        x[M - 1, N // 2] = float("inf")
        if M > 1:
            x[1] = float("-inf")
        if M > 2:
            x[2, 5 % N], x[2, N - 1] = float("nan"), float("nan")
    val, idx = glue.argmax_rows(x, 100)
    f = x.float()
    for m in range(M):
        nan = x[m].isnan().nonzero()
        want = int(nan[0]) if len(nan) else int((f[m] == f[m].max()).nonzero()[0])
        assert int(idx[m]) == 100 + want and torch.equal(val[m].view(torch.int16), x[m, want].view(torch.int16))
