"""Source check, on the CPU: a kernel reaches into another CTA's shared memory only behind a cluster barrier.

Distributed shared memory may be accessed once the CTA that owns it is known to have started.  The blocks of a cluster
are scheduled together, which is not that promise: a kernel has to have waited on a cluster barrier first.  A violation
is a race that hardly ever shows, so the order is read off the sources."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "llmqrt_b200", "csrc", "*.cu")))
REMOTE = re.compile(r"(?:st|ld|red|atom)[a-z.]*\.shared::cluster|map_shared_rank\(|mbar_arrive_remote\(|bulk_copy_to_cta\(|"
                    r"cluster_addr\(")
BARRIER = re.compile(r"barrier\.cluster\.wait|cluster_sync_all\(\)|cluster_wait\(\)|\.sync\(\)")


def _functions(path):
    """(name, body) of every kernel of a file, up to the next one, and of every reduction helper."""
    src = re.sub(r"//[^\n]*", "", open(path).read())
    parts = re.split(r"(?=__global__|__device__ __forceinline__ float cluster_reduce)", src)[1:]
    for part in parts:
        yield re.search(r"(\w+)\s*\((?=[^()]*?[*\w]+ \w+)", part.split("__launch_bounds__")[-1]).group(1), part


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_remote_shared_memory_is_reached_behind_a_barrier(path):
    for name, body in _functions(path):
        remote = REMOTE.search(body)
        if remote is None:
            continue
        wait = BARRIER.search(body)
        assert wait and wait.start() < remote.start(), f"{os.path.basename(path)}: {name} reaches a peer before any cluster barrier"
