"""A few-token 4-bit decoder block runs its additions and SiLU inside the GEMMs.  Whoever watches, replaces or
differentiates one of its modules must see the calls that the plain composition makes, and the same numbers."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu

H, HQ, HKV, D, I, G = 128, 2, 1, 64, 256, 32


def _layer(n, k, g, group=G):
    from llmqrt_b200.linear import WQLinear_GEMM
    layer = WQLinear_GEMM(4, group, k, n, False, "cuda")
    layer.qweight.random_(-2 ** 31, 2 ** 31 - 1, generator=g)
    layer.qzeros.random_(-2 ** 31, 2 ** 31 - 1, generator=g)
    layer.scales.uniform_(0.001, 0.01, generator=g)
    return layer


def _block(rows=16):
    from llmqrt_b200.fused_utils import FusedGateUpMLP
    from llmqrt_b200.nonlinear import LlamaLikeBlock, RMSNorm
    g = torch.Generator(device="cuda").manual_seed(3)
    mlp = FusedGateUpMLP(_layer(I, H, g), _layer(I, H, g), _layer(H, I, g))
    norms = [RMSNorm((1 + 0.1 * torch.randn(H, generator=g, device="cuda")).half()) for _ in range(2)]
    return LlamaLikeBlock(H, HQ, HKV, _layer((HQ + 2 * HKV) * D, H, g), None, None, None, _layer(H, HQ * D, g), mlp, *norms,
                          dev="cuda", max_seq_len=rows)


def _plain(block, x):
    """The block as a composition of calls, each one its module's own."""
    h = x + block.attn(block.norm_1(x))[0]
    return h + block.mlp.forward(block.norm_2(h))


def _run(block, f, x):
    block.attn.start_pos = 3
    return f(block, x)


@contextlib.contextmanager
def _watch(block, name, how, seen):
    """Puts a witness on the module `name`; it adds 1 to what the module gives, so passing it by also shows."""
    from torch.nn.modules import module as M
    target = block.get_submodule(name)
    cls, forward = type(target), type(target).forward

    def hook(module, *args):
        if module is target:
            seen.append(name)
            return args[-1] + 1

    def replaced(*args):
        seen.append(name)
        return forward(*(args if args[0] is target else (target, *args))) + 1

    if how == "hook":
        handle = target.register_forward_hook(hook)
    elif how == "pre-hook":
        handle = target.register_forward_pre_hook(lambda m, a: (seen.append(name), (a[0] + 1,))[1])
    elif how == "global":
        handle = M.register_module_forward_hook(hook)
    elif how == "instance":
        target.forward = replaced
    else:
        cls.forward = lambda self, *a: replaced(self, *a) if self is target else forward(self, *a)
    try:
        yield
    finally:
        if how in ("hook", "pre-hook", "global"):
            handle.remove()
        elif how == "instance":
            del target.forward
        else:
            cls.forward = forward


@pytest.mark.parametrize("how", ["hook", "pre-hook", "global", "instance", "class"])
@pytest.mark.parametrize("name", ["mlp.gate_up", "mlp.down_proj", "norm_2", "mlp"])
def test_witnesses_see_their_calls(name, how):
    if name == "mlp" and how in ("hook", "pre-hook", "global"):
        pytest.skip("the block takes the MLP's forward, not its call")
    block, x = _block(), torch.randn(1, 1, H, device="cuda").half()
    want = _run(block, _plain, x)
    assert torch.equal(_run(block, lambda b, t: b(t), x), want)          # the fused form rounds as the plain one
    seen = []
    with _watch(block, name, how, seen):
        got = _run(block, lambda b, t: b(t), x)
        assert seen == [name]
        assert torch.equal(got, _run(block, _plain, x)) and not torch.equal(got, want)
    assert torch.equal(_run(block, lambda b, t: b(t), x), want)


def test_gradients_reach_the_residual():
    """The layers have no backward; the residual stream around them has one."""
    block, g = _block(), torch.Generator(device="cuda").manual_seed(5)
    h, y = (torch.randn(1, 1, H, generator=g, device="cuda").half() for _ in range(2))
    want = h + block.mlp.forward(y)
    h.requires_grad_()
    out = block.mlp.add_to(h, y)
    assert torch.equal(out, want)
    out.sum().backward()
    assert torch.equal(h.grad, torch.ones_like(h))
    a, b = h.detach(), y.clone().requires_grad_()
    s, n = block.norm_2.add(a, b)
    assert s.requires_grad and torch.equal(s, a + y) and torch.equal(n, block.norm_2(a + y))
    s.sum().backward()
    assert torch.equal(b.grad, torch.ones_like(b))


def test_full_cache():
    """A token beyond the cache's last row: attended over the whole cache, neither rotated nor written."""
    rows = 16
    block = _block(rows)
    a, g = block.attn, torch.Generator(device="cuda").manual_seed(7)
    a.cache.k.normal_(generator=g)
    a.cache.v.normal_(generator=g)
    kept = a.cache.k.clone(), a.cache.v.clone()
    x = torch.randn(1, 1, H, generator=g, device="cuda").half()
    q = a.qkv_proj(x).view(HQ + 2 * HKV, D)[:HQ].double()
    for pos in (rows, rows + 5):
        a.start_pos = pos
        _, weight, _ = a(x)
        p = (q @ kept[0][0, :, 0].double().t() * D ** -0.5).softmax(-1)
        want = (p @ kept[1][0, :, 0].double()).reshape(1, 1, HQ * D)
        assert float((weight.double() - want).norm() / want.norm()) < 1e-3     # P and the result in fp16: 2^-11 each
        assert torch.equal(a.cache.k, kept[0]) and torch.equal(a.cache.v, kept[1]) and a.start_pos == pos + 1


@pytest.mark.parametrize("B", [1, 2, 16])
def test_step_in_one_call(B):
    """The block's native step against the composition of its modules: outputs, caches and positions, over several steps, up
    to the cache's last row, with weights changed in place and replaced on the way."""
    from llmqrt_b200._lib import fast
    rows, g = 12, torch.Generator(device="cuda").manual_seed(B)
    blocks = [_block(rows) for _ in range(2)]
    for block in blocks:
        block.attn.cache.increase_batch_size(B)
        block.attn.cache_batch_size = B
        block.attn.start_pos = 7
    for step in range(7):
        x = torch.randn(B, 1, H, generator=g, device="cuda").half()
        if step == 1:
            for block in blocks:
                block.attn.o_proj.qweight.add_(1)
        if step == 2:
            for block in blocks:
                block.mlp.down_proj.scales = block.mlp.down_proj.scales * 0.5
        if step == 3:
            for block in blocks:
                block.attn.REFERENCE_DOUBLE_APPEND = False
        want = _plain(blocks[0], x)
        native = fast.awq_block_step(blocks[1], x)
        # (a layer whose buffers changed is packed again by its own code, a full cache is that code's as well)
        assert (native is None) == (step in (0, 1, 2) or 7 + step >= rows)
        got = native if native is not None else blocks[1](x)
        assert torch.equal(got, want)
        for name in ("k", "v"):
            assert torch.equal(getattr(blocks[0].attn.cache, name), getattr(blocks[1].attn.cache, name))
        assert blocks[0].attn.start_pos == blocks[1].attn.start_pos == 8 + step


@pytest.mark.parametrize("B", [9, 12, 16])
@pytest.mark.parametrize("H,I", [(1536, 8960), (3584, 18944)])
def test_step_of_a_large_block(B, H, I):
    """The native step against every layer's plain call and the separate additions and SiLU, where the layers are large."""
    from llmqrt_b200 import glue
    from llmqrt_b200._lib import fast
    from llmqrt_b200.fused_utils import FusedGateUpMLP
    from llmqrt_b200.nonlinear import LlamaLikeBlock, RMSNorm
    g = torch.Generator(device="cuda").manual_seed(B)
    mlp = FusedGateUpMLP(_layer(I, H, g, 128), _layer(I, H, g, 128), _layer(H, I, g, 128))
    norms = [RMSNorm((1 + 0.1 * torch.randn(H, generator=g, device="cuda")).half()) for _ in range(2)]
    block = LlamaLikeBlock(H, 2, 1, _layer(4 * 64, H, g, 128), None, None, None, _layer(H, 2 * 64, g, 128), mlp, *norms,
                           dev="cuda", max_seq_len=16, head_dim=64)
    for layer in (block.attn.qkv_proj, block.attn.o_proj, mlp.gate_up, mlp.down_proj):
        layer.packed()
    block.attn.cache.increase_batch_size(B)
    block.attn.cache_batch_size = B
    x = torch.randn(B, 1, H, generator=g, device="cuda").half()
    h = _run(block, lambda b, t: t + b.attn(b.norm_1(t))[0], x)
    want = h + mlp.down_proj(glue.silu_mul(mlp.gate_up(block.norm_2(h)))[0])
    got = _run(block, fast.awq_block_step, x)
    assert got is not None and torch.equal(got, want)
    assert torch.equal(_run(block, lambda b, t: b(t), x), want)


@pytest.mark.parametrize("how", ["hook", "pre-hook", "global", "instance", "class"])
@pytest.mark.parametrize("name", ["norm_1", "attn", "attn.qkv_proj", "attn.o_proj"])
def test_witnesses_of_the_attention_see_their_calls(name, how):
    if name == "attn" and (how in ("hook", "pre-hook", "global") or how == "class"):
        pytest.skip("the block takes the attention's forward, not its call; its result is a triple")
    block, x = _block(), torch.randn(1, 1, H, device="cuda").half()
    want = _run(block, lambda b, t: b(t), x)
    assert torch.equal(_run(block, lambda b, t: b(t), x), want)
    seen = []
    if name == "attn":
        forward = type(block.attn).forward
        block.attn.forward = lambda *a, **k: (seen.append(name), forward(block.attn, *a, **k))[1]
        assert torch.equal(_run(block, lambda b, t: b(t), x), want) and seen == [name]
        return
    with _watch(block, name, how, seen):
        got = _run(block, lambda b, t: b(t), x)
        assert seen == [name]
        assert torch.equal(got, _run(block, _plain, x)) and not torch.equal(got, want)
    assert torch.equal(_run(block, lambda b, t: b(t), x), want)


def test_step_declines_what_it_does_not_cover():
    from llmqrt_b200._lib import fast
    block, x = _block(), torch.randn(1, 1, H, device="cuda").half()
    block.attn.start_pos = 3
    block(x)
    takes = lambda t: fast.awq_block_step(block, t) is not None
    assert takes(x)
    pos = block.attn.start_pos
    assert not takes(x.bfloat16()) and not takes(x.expand(1, 2, H)) and not takes(x.expand(2, 1, H)) and not takes(x[0])
    assert not takes(x.cpu()) and not takes(x.clone().requires_grad_()) and fast.awq_block_step(torch.nn.Linear(2, 2), x) is None
    block.attn.cache.k = block.attn.cache.k.bfloat16()
    assert not takes(x)
    block.attn.cache.k = block.attn.cache.k.half()
    block.norm_2.weight = block.norm_2.weight.float()
    assert not takes(x)
    block.norm_2.weight = block.norm_2.weight.half()
    block.attn.q_norm = torch.nn.Identity()
    assert not takes(x)
    assert block.attn.start_pos == pos


@pytest.mark.parametrize("on", ["instance", "class"])
@pytest.mark.parametrize("owner,name", [
    ("norm_2", "add"), ("mlp", "add_to"), ("mlp", "_hidden"), ("mlp.gate_up", "packed"), ("mlp.gate_up", "takes_tail"),
    ("mlp.gate_up", "silu_halves"), ("mlp.down_proj", "add_to"), ("attn.o_proj", "packed"), ("norm_1", "__call__"),
    ("attn.qkv_proj", "__call__"), ("attn.cache", "to")])
def test_replaced_functions_are_called(owner, name, on):
    """The native step stands for functions beside `forward` as well: whoever replaces one sees it called."""
    import operator
    block, x = _block(), torch.randn(1, 1, H, device="cuda").half()
    want = _run(block, lambda b, t: b(t), x)
    target, seen = operator.attrgetter(owner)(block), []
    cls, own = type(target), name in vars(type(target))
    function = getattr(cls, name)
    if on == "instance" and name == "__call__":
        pytest.skip("a call looks up its class")
    if on == "instance":
        setattr(target, name, lambda *a: (seen.append(name), function(target, *a))[1])
    else:
        setattr(cls, name, lambda self, *a: (seen.append(name) if self is target else None, function(self, *a))[1])
    try:
        assert torch.equal(_run(block, lambda b, t: b(t), x), want) and seen
    finally:
        if on == "instance":
            delattr(target, name)
        elif own:
            setattr(cls, name, function)
        else:
            delattr(cls, name)
    seen.clear()
    assert torch.equal(_run(block, lambda b, t: b(t), x), want) and not seen


def test_a_cache_of_another_class_is_asked():
    """A cache that converts itself on its own terms (as one that lives elsewhere would) does so before every step."""
    block, x, seen = _block(), torch.randn(1, 1, H, device="cuda").half(), []
    want = _run(block, lambda b, t: b(t), x)

    class Cache(type(block.attn.cache)):
        def to(self, like):
            seen.append(like.shape)
            super().to(like)

    block.attn.cache.__class__ = Cache
    assert torch.equal(_run(block, lambda b, t: b(t), x), want) and seen
