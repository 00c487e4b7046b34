"""Builds ``libb200attn.so`` in-tree with nvcc for sm_100a, and ``_host.so`` (the operators' host path, plain C++
against torch's headers) with the host compiler.

``python -m flagattention_b200.build`` compiles every ``csrc/*.cu`` (in parallel, one object per
file, skipping objects newer than all sources) and links the shared library next to this file.
nvcc cross-compiles without a GPU, so this also works on a CPU-only machine.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
OBJ_DIR = CSRC / "build"
LIB_PATH = PKG_DIR / "libb200attn.so"
HOST_SRC = CSRC / "torch_host.cpp"
HOST_PATH = PKG_DIR / "_host.so"     # Python extension module: the operators' host path

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libb200attn.so")
    return exe


def _newest_header_mtime() -> float:
    hdrs = list(CSRC.glob("*.cuh")) + list((PKG_DIR.parent / "include").glob("*.h"))
    return max(h.stat().st_mtime for h in hdrs)


def _compile_one(src: Path, force: bool, verbose: bool, hdr_mtime: float) -> Path:
    obj = OBJ_DIR / (src.stem + ".o")
    if not force and obj.exists() and obj.stat().st_mtime > max(src.stat().st_mtime, hdr_mtime):
        return obj
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
    if verbose:
        sys.stderr.write(res.stderr)
    return obj


def _build_host(force: bool) -> None:
    """Compiles the host path against torch's C++ headers and libraries."""
    newest = max(HOST_SRC.stat().st_mtime, (PKG_DIR.parent / "include" / "b200attn.h").stat().st_mtime)
    if not force and HOST_PATH.exists() and HOST_PATH.stat().st_mtime > newest:
        return
    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    cuda_include = Path(_nvcc()).resolve().parent.parent / "include"
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{p}" for p in include_paths()], f"-I{cuda_include}", f"-I{sysconfig.get_paths()['include']}",
           str(HOST_SRC), "-o", str(HOST_PATH), *[f"-L{p}" for p in library_paths()],
           "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed for {HOST_SRC.name}:\n{res.stdout}\n{res.stderr}")


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile and link the library; returns its path."""
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    hdr_mtime = _newest_header_mtime()
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as pool:
        host = pool.submit(_build_host, force)
        objs = list(pool.map(lambda s: _compile_one(s, force, verbose, hdr_mtime), sources))
        host.result()
    if force or not LIB_PATH.exists() or any(o.stat().st_mtime > LIB_PATH.stat().st_mtime for o in objs):
        cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", str(LIB_PATH),
               *[str(o) for o in objs]]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
