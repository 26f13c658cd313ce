"""Build recipe of libllmqrt_b200.so (sm_100a only).

    python -m llmqrt_b200.build            # incremental
    python -m llmqrt_b200.build --force    # rebuild everything
    python -m llmqrt_b200.build --verbose  # adds -Xptxas -v (registers / spills per kernel)

Every .cu under llmqrt_b200/csrc is compiled with nvcc to an object file and the objects are
linked into llmqrt_b200/lib/libllmqrt_b200.so.  nvcc cross-compiles, so no GPU is needed.
csrc/fastpath.cpp becomes the Python extension llmqrt_b200/lib/_fast.<tag>.so (g++, ATen), which calls that library; the
tag names what the file was made from and for (see fast_tag), so a stale one is never taken for the present one.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import glob
import hashlib
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIBDIR = os.path.join(PKG, "lib")
OBJDIR = os.path.join(LIBDIR, "obj")
LIB = os.path.join(LIBDIR, "libllmqrt_b200.so")
FAST_SRC = os.path.join(CSRC, "fastpath.cpp")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
    "-I", INCLUDE,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA kernels of llmqrt_b200 cannot be built")
    return exe


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def fast_tag() -> str:
    """What the host path's binary depends on: its source, the C ABI it calls, the interpreter and ATen."""
    import torch
    h = hashlib.sha256()
    for path in (FAST_SRC, os.path.join(INCLUDE, "llmqrt_b200.h")):
        with open(path, "rb") as f:
            h.update(f.read() + b"\0")
    h.update(repr((sys.implementation.cache_tag, torch.__version__, torch._C._GLIBCXX_USE_CXX11_ABI)).encode())
    return h.hexdigest()[:12]


def fast_path() -> str:
    return os.path.join(LIBDIR, "_fast.%s.so" % fast_tag())


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJDIR, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + sorted(glob.glob(os.path.join(INCLUDE, "*.h")))
    nvcc = _nvcc()
    jobs = []
    for src in sources:
        obj = os.path.join(OBJDIR, os.path.basename(src)[:-3] + ".o")
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc, *NVCC_FLAGS, *os.environ.get("LLMQRT_NVCC_FLAGS", "").split(), "-c", src, "-o", obj]
            if verbose:
                cmd[1:1] = ["-Xptxas", "-v"]
            jobs.append((src, cmd))

    def run(job):
        src, cmd = job
        p = subprocess.run(cmd, capture_output=True, text=True)
        return src, p.returncode, p.stdout + p.stderr

    failed = False
    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for src, rc, out in ex.map(run, jobs):
            if out.strip() and (verbose or rc != 0):
                print(f"--- {os.path.basename(src)}\n{out}", file=sys.stderr)
            failed |= rc != 0
    if failed:
        raise RuntimeError("nvcc failed; see messages above")

    objs = [os.path.join(OBJDIR, os.path.basename(s)[:-3] + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError("link failed:\n" + p.stdout + p.stderr)
    if force or not os.path.exists(fast_path()):
        _build_fast()
    return LIB


def _build_fast() -> None:
    import sysconfig

    import torch
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    target = fast_path()
    tmp = target + ".tmp%d" % os.getpid()
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(tdir, "include"),
           "-I" + os.path.join(tdir, "include", "torch", "csrc", "api", "include"), "-I" + os.path.join(cuda, "include"),
           "-I" + INCLUDE, FAST_SRC, "-o", tmp, "-L" + LIBDIR, "-lllmqrt_b200", "-L" + os.path.join(tdir, "lib"), "-lc10",
           "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    p = subprocess.run(cmd, capture_output=True, text=True)
    if p.returncode != 0:
        raise RuntimeError("building the host path failed:\n" + p.stdout + p.stderr)
    os.replace(tmp, target)
    for old in glob.glob(os.path.join(LIBDIR, "_fast*.so")):
        if old != target:
            os.remove(old)


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
