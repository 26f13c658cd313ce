"""Source checks, on the CPU, of what a warp's asynchronous instructions need: violations are races or hangs that hardly ever
show, so the order is read off the sources."""
import os
import re

import pytest

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


def _headers(src, at):
    """What stands ahead of the opening brace of every block around position `at`."""
    out, depth, i = [], 0, at
    while i > 0:
        i -= 1
        if src[i] == "}":
            depth += 1
        elif src[i] == "{":
            if depth == 0:
                out.append(re.split(r"[;{}]", src[:i])[-1].strip())
            else:
                depth -= 1
    return out


@pytest.mark.parametrize("name", ["gemm_tc.cu", "attn_prefill.cu"])
def test_a_warp_leaves_together(name):
    """Lanes that read the abort flag for themselves may see it raised at different moments and part; ahead of votes, elections
    and .sync.aligned accesses that every lane has to reach, the failing block would never end.  Only a role that is one
    lane reads the flag itself (a loader lambda is called by one lane)."""
    src = _source(name)
    start = src.index("__global__")
    for m in re.finditer(r"\*abort\b|\babort_flag\s*[=!]=", src[start:]):
        at = start + m.start()
        assert any("lane == 0" in h or "awq_load" in h for h in _headers(src, at)), src[at - 60:at + 40]
