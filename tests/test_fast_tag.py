"""The native host path is loaded only if it was built from the present source for the present interpreter and torch."""
import os
import sys

import pytest
import torch

from llmqrt_b200 import _lib, build


def test_tag_names_everything_the_binary_depends_on(tmp_path, monkeypatch):
    tags = {build.fast_tag()}
    assert build.fast_tag() in tags
    for i, name in enumerate(("FAST_SRC", "INCLUDE")):
        other = tmp_path / str(i)
        other.mkdir()
        for src in (build.FAST_SRC, os.path.join(build.INCLUDE, "llmqrt_b200.h")):
            (other / os.path.basename(src)).write_bytes(open(src, "rb").read())
        target = other / ("fastpath.cpp" if name == "FAST_SRC" else "llmqrt_b200.h")
        target.write_bytes(target.read_bytes() + b"\n")
        with monkeypatch.context() as m:
            m.setattr(build, name, str(target) if name == "FAST_SRC" else str(other))
            tags.add(build.fast_tag())
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0")
        tags.add(build.fast_tag())
    with monkeypatch.context() as m:
        m.setattr(sys, "implementation", type("Impl", (), {"cache_tag": "other-1"}))
        tags.add(build.fast_tag())
    assert len(tags) == 5


def test_a_file_of_another_tag_is_not_loaded(monkeypatch):
    """As after a host compiler that failed behind the library's own build, or a torch upgrade."""
    class Built(Exception):
        pass

    def rebuild():
        raise Built

    assert os.path.exists(build.fast_path()) and _lib.fast.__file__ == build.fast_path()
    monkeypatch.setattr(build, "fast_tag", lambda: "0" * 12)
    monkeypatch.setattr(build, "build", rebuild)
    with pytest.raises(Built):
        _lib._load_fast()
