"""The native host path (csrc/fastpath.cpp) on the CPU: what it takes for numbers and what it refuses before a launch.

The arguments are read before the tensors' devices are looked at, so a call with CPU tensors that gets as far as the
device check has had its numbers accepted."""
import pytest
import torch

from llmqrt_b200 import attention, glue


class Whole:
    """A number by conversion only, as a configuration object may hand one over."""

    def __int__(self):
        return 3

    def __float__(self):
        return 3.0


@pytest.mark.parametrize("number", [3, 3.0, torch.tensor(3), torch.tensor(3.0), Whole()])
def test_numbers_are_what_converts_to_one(number):
    x = torch.zeros(1, 1, 2, 64, dtype=torch.float16)
    cache, lens = torch.zeros(1, 8, 2, 64, dtype=torch.float16), torch.zeros(1, dtype=torch.int32)
    table = torch.zeros(8, 32)
    for call in (lambda: glue.rope_kv_write(x, x, x, table, table, pos0=number),
                 lambda: attention.kv_append(cache, cache, x, x, start_pos=number),
                 lambda: attention.attn_decode(x[:, 0], cache, cache, lens, number, softcap=number),
                 lambda: attention.flash_attn_func(x, x, x, softcap=number),
                 lambda: glue.rmsnorm(x, torch.ones(64, dtype=torch.float16), number)):
        with pytest.raises(RuntimeError, match="no CPU path"):
            call()


def test_what_is_no_number_is_refused():
    x, table = torch.zeros(1, 1, 2, 64, dtype=torch.float16), torch.zeros(8, 32)
    for pos0 in (None, [1], "three"):
        with pytest.raises((TypeError, ValueError)):
            glue.rope_kv_write(x, x, x, table, table, pos0=pos0)


def test_what_counts_as_a_plain_call():
    """Hooks of the module and of all modules, a forward replaced on the instance or on the class, a subclass."""
    from torch.nn.modules import module as M

    from llmqrt_b200.linear.linear_base import calls_plainly

    class Layer(torch.nn.Module):
        def forward(self, x):
            return x

    forward, layer = Layer.forward, Layer()

    def plain():
        return calls_plainly(layer, Layer, forward)

    assert plain() and not calls_plainly(type("Sub", (Layer,), {})(), Layer, forward)
    for register in (layer.register_forward_hook, layer.register_forward_pre_hook, layer.register_full_backward_hook,
                     layer.register_full_backward_pre_hook, M.register_module_forward_hook,
                     M.register_module_forward_pre_hook, M.register_module_full_backward_hook,
                     M.register_module_full_backward_pre_hook):
        handle = register(lambda *a: None)
        assert not plain(), register
        handle.remove()
        assert plain()
    layer.forward = lambda x: x
    assert not plain()
    del layer.forward
    Layer.forward = lambda self, x: x
    assert not plain()
    Layer.forward = forward
    assert plain()


def _step(q, kc, vc, k=None, v=None, lens=None, add=1, bound=8):
    from llmqrt_b200._lib import fast
    return fast.attn_decode_step(q, kc, vc, k, v, lens, add, bound, 0.0, None, None, False)


def test_caches_and_lengths_of_too_few_sequences_are_refused():
    """The kernels read lengths and read and write cache rows for every sequence of the query: nothing is launched unless
    they are there.  (The checks come before the device check, so CPU tensors show them.)"""
    def zeros(*shape, dtype=torch.float16):
        return torch.zeros(*shape, dtype=dtype)

    q, new = zeros(3, 1, 4, 64), zeros(3, 1, 2, 64)
    kc, vc, lens = zeros(3, 8, 2, 64), zeros(3, 8, 2, 64), zeros(3, dtype=torch.int32)
    calls = {
        "step": lambda kc=kc, vc=vc, lens=lens: _step(q, kc, vc, new, new, lens),
        "decode": lambda kc=kc, vc=vc, lens=lens: attention.attn_decode(q[:, 0], kc, vc, lens, 8),
        "append": lambda kc=kc, vc=vc, lens=lens: attention.kv_append(kc, vc, new, new, cache_seqlens=lens)}
    for name, call in calls.items():
        with pytest.raises(RuntimeError, match="no CPU path"):           # sound: only the device is wrong
            call()
        with pytest.raises(RuntimeError, match="no CPU path"):           # one cache shorter than the other
            call(vc=zeros(3, 8, 2, 64)[:, :6])
        for bad in ({"kc": kc[:2]}, {"vc": vc[:2]}, {"lens": lens[:2]}, {"kc": zeros(3, 8, 2, 32)}, {"kc": zeros(8, 2, 64)},
                    {"vc": vc.transpose(1, 2)}, {"lens": lens.long()}):
            with pytest.raises((RuntimeError, TypeError)) as e:
                call(**bad)
            assert "no CPU path" not in str(e.value), (name, bad)
    with pytest.raises(RuntimeError, match="no CPU path"):               # a number for all lengths
        _step(q, kc, vc, new, new)
    for bad in (zeros(3, 2, 4, 64), zeros(3, 4, 64)):
        with pytest.raises(RuntimeError, match="q must be"):
            _step(bad, kc, vc)
    with pytest.raises(RuntimeError, match="k and v must be"):
        attention.kv_append(kc, vc, new, new[:2])
    with pytest.raises(TypeError, match="one dtype"):
        attention.kv_append(kc, vc, new.float(), new)


def test_prompt_attention_of_mixed_types_is_refused():
    x = torch.zeros(1, 4, 2, 64, dtype=torch.float16)
    with pytest.raises(TypeError, match="one dtype"):
        attention.flash_attn_func(x, x.bfloat16(), x)
    with pytest.raises(TypeError, match="one dtype"):
        attention.flash_attn_func(x, x, x.bfloat16())


@pytest.mark.parametrize("name", ["gemm_tc.cu", "awq.cu"])
def test_schedules_ask_the_device_once(name):
    """Small calls are bound by the host: an estimate that asks the runtime for the device (or takes a lock) for every size
    it tries shows in them.  Read off the source: no loop's header does, and no loop calls what does."""
    import os
    import re
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = re.sub(r"//[^\n]*", "", open(os.path.join(root, "llmqrt_b200", "csrc", name)).read())
    host = src[src.rindex("__global__"):]
    for loop in re.finditer(r"\b(?:for|while) \((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)", host):
        body = host[loop.end():].split("\n  }\n")[0] if host[loop.end():].lstrip().startswith("{") else ""
        assert "sm_count()" not in loop.group(0), loop.group(0)
        assert not re.search(r"\bactive(?:_clusters)?(?:<[^;]*>)?\(", body), loop.group(0)
