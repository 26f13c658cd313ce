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
