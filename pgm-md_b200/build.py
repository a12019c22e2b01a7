"""Builds the engine library in-tree: pgm-md_b200/libpgm_b200.so (sm_100a, nvcc, cuFFT).

    python pgm-md_b200/build.py            (or __graft_entry__.build())

The library exports the C ABI of include/pgm_b200.h.  It is built for sm_100a only.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB = PKG / "libpgm_b200.so"
SOURCES = [CSRC / "engine.cu", CSRC / "transforms.cu", CSRC / "transforms64.cu", CSRC / "persistent.cu",
           CSRC / "capi.cpp"]
HEADERS = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + [ROOT / "include" / "pgm_b200.h"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def cuda_lib_dir() -> str:
    return str(Path(nvcc()).resolve().parent.parent / "lib64")


def needs_build() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    return any(p.stat().st_mtime > t for p in SOURCES + HEADERS)


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return LIB
    tmp = LIB.with_suffix(".so.tmp")

    def run(cmd):
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + r.stdout + r.stderr)

    with tempfile.TemporaryDirectory() as d:   # the sources side by side, then the link
        objects = [str(Path(d) / (p.stem + ".o")) for p in SOURCES]
        flags = [*ARCH, "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC,-O2"]
        with ThreadPoolExecutor() as pool:
            list(pool.map(run, [[nvcc(), *flags, "-c", "-o", o, str(p)] for p, o in zip(SOURCES, objects)]))
        run([nvcc(), *ARCH, "-shared", "-o", str(tmp), *objects, "-lcufft", f"-L{cuda_lib_dir()}",
             "-Xlinker", f"-rpath,{cuda_lib_dir()}"])
    tmp.replace(LIB)
    return LIB


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose=True)
    print(p)
