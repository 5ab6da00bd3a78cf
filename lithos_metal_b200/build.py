"""Builds the CUDA library in-tree: ``lithos_metal_b200/_lib/liblithos_b200.so`` for sm_100a with nvcc.

``python -m lithos_metal_b200.build`` (or :func:`build`). The shared object has a plain C ABI (include/lithos_b200.h) and is loaded with
ctypes: it needs neither Python's headers nor torch's. Beside it ``lithos_host.<Python>-torch<version>.so``, a CPython extension
(csrc/host_ext.cpp, g++ with the headers of both): the Python layer's calls without the cost of ctypes. It is built for one Python and one torch,
and every call works without it.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from importlib import metadata

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC_DIR = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "_lib", "liblithos_b200.so")
# the native call path of the Python layer: named for what it was compiled against, so that another Python or torch never loads it
HOST_OUT = os.path.join(HERE, "_lib", f"lithos_host.{sys.implementation.cache_tag}-torch{metadata.version('torch')}.so")
HOST_SOURCE = "host_ext.cpp"
SOURCES = ["lithos_b200.cu", "cluster.cu"]
# (No -split-compile: with it ptxas made one of two different kernels from the same cluster.cu, as its threads happened to finish, and the one --
# five builds in eight -- was up to 17 % slower: 32 FP32 rows of 151,936 without a filter 28.8 us instead of 24.8.)
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC,-fvisibility=hidden",
              "--fmad=true", "-Xptxas", "-v", "-cudart", "shared"]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA library cannot be built")


def _host_command():
    """g++ on the CPython extension: it reads tensors through torch's headers and links against the torch that is installed."""
    import torch
    base = os.path.join(os.path.dirname(torch.__file__))
    inc = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
           os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    return [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[f"-isystem{d}" for d in inc], "-o", HOST_OUT, os.path.join(SRC_DIR, HOST_SOURCE), "-L", os.path.join(base, "lib"),
            "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10"]


def _stale(path: str) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    deps = [os.path.join(SRC_DIR, f) for f in os.listdir(SRC_DIR)] + [os.path.join(ROOT, "include", "lithos_b200.h"), os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def _run(cmd):
    return subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _finish(log: str, cmds, done, verbose: bool) -> None:
    text = "".join(" ".join(c) + "\n" + r.stdout for c, r in zip(cmds, done))
    with open(os.path.join(os.path.dirname(OUT), log), "w") as f:
        f.write(text)
    failed = any(r.returncode != 0 for r in done)
    if verbose or failed:
        print(text)
    if failed:
        raise RuntimeError(f"the build failed; see {os.path.join(os.path.dirname(OUT), log)}")


def build_library(force: bool = False, verbose: bool = False) -> str:
    """The CUDA library."""
    if not force and not _stale(OUT):
        return OUT
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    cmds = [[_nvcc(), *NVCC_FLAGS, "-I", os.path.join(ROOT, "include"), "-c", "-o", os.path.join(os.path.dirname(OUT), os.path.splitext(src)[0] + ".o"),
             os.path.join(SRC_DIR, src)] for src in SOURCES]
    with ThreadPoolExecutor(len(cmds)) as pool:                             # the translation units side by side
        done = list(pool.map(_run, cmds))
    cmds.append([_nvcc(), "-shared", "-cudart", "shared", "-o", OUT, *[c[c.index("-o") + 1] for c in cmds]])
    if all(r.returncode == 0 for r in done):
        done.append(_run(cmds[-1]))
    _finish("build.log", cmds, done, verbose)
    return OUT


def build_host(force: bool = False, verbose: bool = False) -> str:
    """The native call path of the Python layer, for the Python that runs and the torch that is installed."""
    if not force and not _stale(HOST_OUT):
        return HOST_OUT
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    cmd = _host_command()
    _finish("build_host.log", [cmd], [_run(cmd)], verbose)
    return HOST_OUT


def build(force: bool = False, verbose: bool = False) -> str:
    with ThreadPoolExecutor(2) as pool:
        both = [pool.submit(f, force, verbose) for f in (build_library, build_host)]
    for f in both:
        f.result()
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
