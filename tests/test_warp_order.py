"""Source checks, on the CPU, of what a warp's asynchronous instructions need: violations are races or hangs that hardly ever
show, so the order is read off the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmqrt_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_columns_stored_again_are_waited_for():
    """Prefill attention stores the first half of P once more where the reference moves.  Two tcgen05.st to one column are not
    ordered by themselves: the first has to be waited for."""
    src = _source("attn_prefill.cu")
    redo = re.search(r"again = __any_sync\(.*?start\(\);\s*exp_of\(0\);\s*exp_of\(1\);", src, re.S)
    assert redo and "tmem_st_wait()" in redo.group(0)
