"""Builds libkfb200.so (the C-ABI library, nvcc for sm_100a) and kernelforge._host (its caller on torch tensors) in-tree.

    python kernel-forge_b200/build.py [--force] [--verbose]

Each csrc/*.cu is compiled to build/<name>.o (in parallel, skipped when up to date) and the
objects are linked into kernelforge/libkfb200.so.  ptxas resource usage (registers, spills,
shared memory) of every kernel is kept in build/<name>.ptxas.txt.  The library uses no torch headers;
csrc/host.cpp does and becomes the CPython extension kernelforge/_host.so next to it.
"""

from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_ROOT = Path(__file__).resolve().parent
CSRC = PKG_ROOT / "csrc"
BUILD = PKG_ROOT / "build"
LIB = PKG_ROOT / "kernelforge" / "libkfb200.so"
HOST = PKG_ROOT / "kernelforge" / "_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v", "--expt-relaxed-constexpr",
]


# per-source extra flags
EXTRA_FLAGS: dict[str, list[str]] = {}


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the kfb200 library needs the CUDA 12.8+ toolkit")
    return exe


def _deps_mtime() -> float:
    hdrs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + [PKG_ROOT.parent / "include" / "kfb200.h", Path(__file__)]
    return max(p.stat().st_mtime for p in hdrs if p.exists())


def _compile(src: Path, force: bool, verbose: bool) -> Path:
    obj = BUILD / (src.stem + ".o")
    if not force and obj.exists() and obj.stat().st_mtime >= max(src.stat().st_mtime, _deps_mtime()):
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, *EXTRA_FLAGS.get(src.name, []), "-c", str(src), "-o", str(obj)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    (BUILD / (src.stem + ".ptxas.txt")).write_text(res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src.name}:\n{res.stdout}\n{res.stderr}")
    if verbose:
        print(res.stderr)
    return obj


def _build_host(force: bool) -> Path:
    """csrc/host.cpp -> kernelforge/_host.so, linked to libkfb200.so beside it and to the installed torch."""
    src = CSRC / "host.cpp"
    newest = max(src.stat().st_mtime, (PKG_ROOT.parent / "include" / "kfb200.h").stat().st_mtime, Path(__file__).stat().st_mtime)
    if not force and HOST.exists() and HOST.stat().st_mtime >= newest:
        return HOST
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include", sysconfig.get_paths()["include"]]
    cmd = [shutil.which("g++") or "c++", "-shared", "-fPIC", "-O2", "-std=c++17", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(arg for i in includes for arg in ("-isystem", str(i))), str(src), "-o", str(HOST), f"-L{LIB.parent}", "-l:libkfb200.so",
           f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
           "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{root / 'lib'}"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed on {src.name}:\n{res.stdout}\n{res.stderr}")
    return HOST


def build(force: bool = False, verbose: bool = False) -> Path:
    BUILD.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    with ThreadPoolExecutor(max_workers=min(8, len(sources))) as pool:
        objs = list(pool.map(lambda s: _compile(s, force, verbose), sources))
    if force or not LIB.exists() or LIB.stat().st_mtime < max(o.stat().st_mtime for o in objs):
        cmd = [_nvcc(), "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a",
               "-Xcompiler", "-fPIC", "-cudart", "static"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _build_host(force)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
    sys.exit(0)
