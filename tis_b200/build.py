"""Builds the in-tree CUDA library tis_b200/libtis_b200.so for sm_100a.

    python -m tis_b200.build          (or __graft_entry__.build())

nvcc compiles the .cu files under tis_b200/csrc side by side (the variants of
the split kernel take over a minute each) and links them into one shared
object; the library is loaded from the package directory by
tis_b200.abi.load_library.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libtis_b200.so")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr",
         "-Xcompiler", "-fPIC,-ffp-contract=off"]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def nvcc():
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def needs_build() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = sources() + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    deps.append(os.path.join(HERE, "..", "include", "tis_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return OUT
    exe = nvcc()

    def run(cmd):
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        subprocess.run(cmd, check=True)

    with tempfile.TemporaryDirectory() as tmp:
        objs = [os.path.join(tmp, os.path.basename(f) + ".o") for f in sources()]
        with ThreadPoolExecutor(max(1, os.cpu_count() or 1)) as pool:
            list(pool.map(lambda fo: run([exe] + ARCH + FLAGS + ["-c", "-o", fo[1], fo[0]]), zip(sources(), objs)))
        run([exe] + ARCH + ["-shared", "-o", OUT + ".tmp"] + objs)
    os.replace(OUT + ".tmp", OUT)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
