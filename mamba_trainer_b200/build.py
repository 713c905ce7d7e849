"""Build libm3scan.so (the C-ABI library) in-tree with nvcc for sm_100a, and beside it _m3torch.so, the autograd nodes
over it.

    python -m mamba_trainer_b200.build [--force] [--verbose]

The library has no PyTorch dependency: it is plain CUDA behind `extern "C"`; _m3torch.so is a torch extension that links
to it.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libm3scan.so"
EXT = PKG / "_m3torch.so"
SOURCES = ["m3_api.cu", "m3_generic_fwd.cu", "m3_generic_bwd.cu", "m3_noalloc.cu", "m3_rows_fwd.cu", "m3_rows_bwd.cu", "m3_tc_fwd.cu", "m3_tc_bwd.cu", "m3_tc_ahead.cu", "m3_step.cu", "m3_mixer_call.cu", "m3_front.cu",
           "m3_host_pipe.cu", "m3_conv.cu", "m3_mixer.cu", "m3_reduce.cu"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; libm3scan cannot be built")


def _stale() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))
    deps.append(PKG.parent / "include" / "m3scan.h")
    return any(p.stat().st_mtime > t for p in deps)


def _build_extension(force: bool) -> None:
    src, header = CSRC / "m3_torch.cpp", PKG.parent / "include" / "m3scan.h"
    if not force and EXT.exists() and EXT.stat().st_mtime > max(src.stat().st_mtime, header.stat().st_mtime):
        return
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    inc = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", Path(sysconfig.get_paths()["include"]),
           Path(_nvcc()).resolve().parent.parent / "include"]
    tmp = EXT.with_suffix(".tmp")   # a process that has the old one loaded keeps its file
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_m3torch",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{i}" for i in inc], str(src), "-o", str(tmp),
           f"-L{root / 'lib'}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-Wl,-rpath,{root / 'lib'}",
           f"-L{PKG}", "-l:libm3scan.so", "-Wl,-rpath,$ORIGIN"]
    subprocess.run(cmd, check=True)
    tmp.replace(EXT)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every CUDA source into one shared library, and the torch extension over it; returns the library's path."""
    _build_library(force, verbose)
    _build_extension(force)
    return LIB


def _build_library(force: bool, verbose: bool) -> None:
    if not force and not _stale():
        return
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)
    nvcc = _nvcc()
    common = [
        "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
    ]
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    objs = []
    for src in SOURCES:
        obj = objdir / (src + ".o")
        objs.append(str(obj))
        cmd = [nvcc, *common, "-c", str(CSRC / src), "-o", str(obj)]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError(f"nvcc failed on {src}")
    link = [nvcc, "-shared", "-o", str(LIB), *objs, "-lcudart"]
    subprocess.run(link, check=True)


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
