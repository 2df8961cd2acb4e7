"""Build libbob_sm100.so (nvcc, sm_100a) and bob_torch.so (g++, PyTorch's headers) in-tree.

    python -m flashbob_b200.build

nvcc cross-compiles without a GPU.  Both land next to this file so that they are found by
`flashbob_b200._lib` and `flashbob_b200._native` without any install step.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libbob_sm100.so"
TORCH_MODULE = PKG / "bob_torch.so"
SOURCES = ("api.cu", "selftest.cu", "noalloc.cu")
HEADERS = ("ptx.cuh", "sweep.cuh", "decode.cuh", "tmap.h", "internal.h")


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")
    return cand


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in (*deps, PKG.parent / "include" / "bob_sm100.h"))


def build_torch_module(force: bool = False) -> Path:
    """Compile the operator's native host path into bob_torch.so (skipped when up to date)."""
    src = CSRC / "torch_binding.cpp"
    if not force and not _stale(TORCH_MODULE, [src]):
        return TORCH_MODULE
    import sysconfig

    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parents[1]
    cmd = [
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
        f"-I{root / 'include'}", f"-I{root / 'include' / 'torch' / 'csrc' / 'api' / 'include'}",
        f"-I{sysconfig.get_paths()['include']}", f"-I{cuda / 'include'}", str(src), "-o", str(TORCH_MODULE),
        f"-L{root / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
    ]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed:\n{res.stdout}\n{res.stderr}")
    return TORCH_MODULE


def build_library(force: bool = False, verbose: bool = False) -> Path:
    """Compile the CUDA sources into libbob_sm100.so (skipped when up to date), and the native host path."""
    build_torch_module(force)
    if not force and not _stale(LIB, [CSRC / s for s in SOURCES + HEADERS if (CSRC / s).exists()]):
        return LIB
    srcs = [str(CSRC / s) for s in SOURCES if (CSRC / s).exists()]
    cmd = [
        _nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-shared", "-Xcompiler", "-fPIC", "-o", str(LIB), *srcs,
    ]
    if verbose:
        cmd[1:1] = ["-Xptxas", "-v"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed:\n{res.stdout}\n{res.stderr}")
    if verbose:
        print(res.stderr)
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
