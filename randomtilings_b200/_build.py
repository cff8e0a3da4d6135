"""In-tree build of the native library (librt_b200.so) for sm_100a.

nvcc cross-compiles without a GPU, so this runs on any machine with CUDA 12.9.
The library lands next to this file so that it travels with the source tree.
"""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "librt_b200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    # IEEE single-precision division and no FMA contraction surprises: the
    # rect-triangle acceptance test must match the host CPU bit for bit.
    "-prec-div=true", "-fmad=false",
]


def sources() -> list[str]:
    return sorted(
        os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp"))
    )


def headers() -> list[str]:
    out = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    inc = os.path.join(HERE, "..", "include")
    out += [os.path.join(inc, f) for f in os.listdir(inc) if f.endswith(".h")]
    return out


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(f) > t for f in sources() + headers())


def nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    tmp = LIB + ".tmp"

    def run(cmd: list[str]) -> None:
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        subprocess.run(cmd, check=True, cwd=CSRC)

    # One compiler per source file, on all cores: on eight they take a minute, one
    # after the other three and a half.
    with tempfile.TemporaryDirectory() as objs:
        todo = [(f, os.path.join(objs, os.path.basename(f) + ".o")) for f in sources()]
        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
            list(pool.map(lambda x: run([nvcc(), *NVCC_FLAGS, "-c", "-o", x[1], x[0]]), todo))
        run([nvcc(), *NVCC_FLAGS, "-shared", "-o", tmp, *[o for _, o in todo], "-lcudart"])
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
