"""Builds the CUDA library in-tree: ``lithos_metal_b200/_lib/liblithos_b200.so`` for sm_100a with nvcc.

``python -m lithos_metal_b200.build`` (or :func:`build`). The shared object has a plain C ABI (include/lithos_b200.h);
it is loaded with ctypes, so no Python headers and no torch headers are involved.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC_DIR = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "_lib", "liblithos_b200.so")
SOURCES = ["lithos_b200.cu", "cluster.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC,-fvisibility=hidden",
              "--fmad=true", "-Xptxas", "-v", "-cudart", "shared"]


# The cluster sampler's phases are functions called from one kernel: split compilation allocates their registers function by function,
# which leaves the kernel 50-350 bytes of stack instead of 270-700 (its stack lives in L2). The other kernels are compiled whole.
EXTRA_FLAGS = {"cluster.cu": ["-split-compile=0"]}


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA library cannot be built")


def _stale() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = [os.path.join(SRC_DIR, f) for f in os.listdir(SRC_DIR)] + [os.path.join(ROOT, "include", "lithos_b200.h"), os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def _run(cmd):
    return subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return OUT
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    cmds = [[_nvcc(), *NVCC_FLAGS, *EXTRA_FLAGS.get(src, []), "-I", os.path.join(ROOT, "include"), "-c", "-o", os.path.join(os.path.dirname(OUT), os.path.splitext(src)[0] + ".o"),
             os.path.join(SRC_DIR, src)] for src in SOURCES]
    with ThreadPoolExecutor(len(cmds)) as pool:                             # the translation units side by side
        done = list(pool.map(_run, cmds))
    cmds.append([_nvcc(), "-shared", "-cudart", "shared", "-o", OUT, *[c[c.index("-o") + 1] for c in cmds]])
    if all(r.returncode == 0 for r in done):
        done.append(_run(cmds[-1]))
    log = os.path.join(os.path.dirname(OUT), "build.log")
    text = "".join(" ".join(c) + "\n" + r.stdout for c, r in zip(cmds, done))
    with open(log, "w") as f:
        f.write(text)
    failed = any(r.returncode != 0 for r in done)
    if verbose or failed:
        print(text)
    if failed:
        raise RuntimeError(f"nvcc failed; see {log}")
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
