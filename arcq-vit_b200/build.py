"""Build recipe for the CUDA shared library (sm_100a only) and the host extension, in-tree.

``python arcq-vit_b200/build.py`` or ``build_library()``: one nvcc call that compiles ``csrc/arcq_b200.cu`` into
``libarcq_b200.so`` and one g++ call that compiles ``csrc/host_ext.cpp`` (torch tensors in, library calls out) into
``_arcq_host.so``, both next to this file.  nvcc cross-compiles, so no GPU is needed to build.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libarcq_b200.so"
HOST_SOURCE = CSRC / "host_ext.cpp"
HOST_PATH = PKG_DIR / "_arcq_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--shared", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put /usr/local/cuda/bin on PATH")


def sources():
    return sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")) + [PKG_DIR.parent / "include" / "arcq_b200.h"]


def _older(target: Path, srcs) -> bool:
    return not target.exists() or any(src.stat().st_mtime > target.stat().st_mtime for src in srcs)


def is_stale() -> bool:
    return _older(LIB_PATH, sources()) or _older(HOST_PATH, [HOST_SOURCE, PKG_DIR.parent / "include" / "arcq_b200.h"])


def _run(cmd, verbose: bool = False) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)


def _host_command():
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-w",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f"-I{root / 'include'}", f"-I{root / 'include' / 'torch' / 'csrc' / 'api' / 'include'}", f"-I{cuda / 'include'}",
            f"-I{sysconfig.get_paths()['include']}", "-o", str(HOST_PATH), str(HOST_SOURCE),
            f"-L{root / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
            f"-L{PKG_DIR}", "-larcq_b200", "-Wl,-rpath,$ORIGIN"]


def build_library(force: bool = False, verbose: bool = False) -> Path:
    """Compile what is missing or older than its sources."""
    if force or _older(LIB_PATH, sources()):
        _run([_nvcc(), *(["-Xptxas", "-v"] if verbose else []), *NVCC_FLAGS, "-o", str(LIB_PATH), str(CSRC / "arcq_b200.cu")], verbose)
    if force or _older(HOST_PATH, [HOST_SOURCE, PKG_DIR.parent / "include" / "arcq_b200.h"]):
        _run(_host_command())
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
