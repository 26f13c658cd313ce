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
