"""Build libb200fp8.so (sm_100a only) next to this file with nvcc, and _torch_call.so beside it with g++.

    python -m hf_kernels_helion_b200.build [--force] [--verbose]

The shared library has a plain C ABI (include/b200fp8.h) and links the CUDA runtime
statically, so it loads on a machine without a GPU as well (it just cannot launch).
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from pathlib import Path

from . import _lib

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libb200fp8.so"
SOURCES = [CSRC / "b200fp8.cu"]
NATIVE_PATH = PKG_DIR / "_torch_call.so"   # host side of the Python calls: links torch, has no kernels
NATIVE_SOURCES = [CSRC / "torch_call.cpp", PKG_DIR.parent / "include" / "b200fp8.h"]
HEADERS = sorted(CSRC.glob("*.cuh")) + [PKG_DIR.parent / "include" / "b200fp8.h"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; set CUDA_HOME")
    return nvcc


def _is_stale(target: Path, sources) -> bool:
    return not target.exists() or any(p.stat().st_mtime > target.stat().st_mtime for p in sources)


def _native_is_stale() -> bool:
    """Older than its sources, or built for another torch or Python (it carries the names of its own as a string)."""
    return _is_stale(NATIVE_PATH, NATIVE_SOURCES) or _lib.native_tag().encode() + b"\0" not in NATIVE_PATH.read_bytes()


def is_stale() -> bool:
    return _is_stale(LIB_PATH, SOURCES + HEADERS) or _native_is_stale()


def _native_command() -> list[str]:
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    root = str(Path(find_nvcc()).resolve().parent.parent)
    includes = cpp_extension.include_paths() + [sysconfig.get_path("include"), os.path.join(root, "include")]
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DB200FP8_BUILT_FOR="{_lib.native_tag()}"']
    for d in includes:
        cmd += ["-isystem", d]
    cmd += [str(NATIVE_SOURCES[0]), "-o", str(NATIVE_PATH)]
    for d in cpp_extension.library_paths():
        cmd += ["-L", d]
    return cmd + ["-lc10", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-lc10_cuda"]


def _run(cmd, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{Path(cmd[0]).name} failed with exit code {res.returncode}")


def build(force: bool = False, verbose: bool = False) -> Path:
    if force or _is_stale(LIB_PATH, SOURCES + HEADERS):
        cmd = [find_nvcc(), *NVCC_FLAGS]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        _run(cmd + ["-o", str(LIB_PATH), *map(str, SOURCES)], verbose)
    if force or _native_is_stale():
        _run(_native_command(), verbose)
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
