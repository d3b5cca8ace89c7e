"""Builds the C-ABI shared library ``lib/librte_b200.so`` (CUDA kernels for sm_100a) and ``lib/_rte_host.so`` (the operator
table's native autograd operators over that ABI) in-tree.

    python -m speedup_thingy_b200.build          # rebuild if sources are newer than the library

nvcc cross-compiles without a GPU, so this also runs on a CPU-only build machine.
"""
from __future__ import annotations

import os
import shlex
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB = PKG / "lib" / "librte_b200.so"
HOST_LIB = PKG / "lib" / "_rte_host.so"
SOURCES = ["gemm_tcgen05.cu", "elementwise.cu", "attention.cu", "macro_phi.cu", "router.cu", "audit.cu", "shortlist.cu", "cluster_pool.cu", "svd_ffn.cu", "gemm_small.cu", "gemm_tile.cu", "gemm_resident.cu", "codebook.cu", "allreduce.cu", "host_random.cu",
           "operator_table.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found: cannot build librte_b200.so")
    return exe


def needs_build() -> bool:
    if not LIB.exists() or not HOST_LIB.exists():
        return True
    newest = max(p.stat().st_mtime for p in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.cpp"), ROOT / "include" / "rte_b200.h",
                                             Path(__file__)])
    return newest > min(LIB.stat().st_mtime, HOST_LIB.stat().st_mtime)


def _host_compile() -> list[str]:
    import torch

    inc = Path(torch.__file__).resolve().parent / "include"
    cuda = Path(_nvcc()).resolve().parent.parent / "include"
    dirs = [ROOT / "include", inc, inc / "torch" / "csrc" / "api" / "include", cuda, sysconfig.get_paths()["include"]]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-DTORCH_EXTENSION_NAME=_rte_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{d}" for d in dirs],
            "-c", str(CSRC / "host_ops.cpp"), "-o", str(HOST_LIB.with_suffix(".o"))]


def _host_link() -> list[str]:
    import torch

    return ["g++", "-shared", "-o", str(HOST_LIB), str(HOST_LIB.with_suffix(".o")), f"-L{Path(torch.__file__).resolve().parent / 'lib'}",
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-L{LIB.parent}", "-lrte_b200",
            "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return LIB
    LIB.parent.mkdir(parents=True, exist_ok=True)
    objs = []
    procs = []
    for src in SOURCES:
        path = CSRC / src
        if not path.exists():
            continue
        obj = LIB.parent / (path.stem + ".o")
        # RTE_NVCC_EXTRA: extra compiler flags, e.g. -DRTE_GEMM_DIAG (the GEMM's timing diagnostics: with it the
        # environment variable RTE_GEMM_DIAG_FLAGS switches off stores / MMAs / loads inside the kernel)
        cmd = [_nvcc(), *NVCC_FLAGS, *shlex.split(os.environ.get("RTE_NVCC_EXTRA", "")), "-I", str(ROOT / "include"),
               "-I", str(CSRC), "-c", str(path), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(str(obj))
    procs.append(("host_ops.cpp", subprocess.Popen(_host_compile(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, proc in procs:
        out, _ = proc.communicate()
        if verbose or proc.returncode != 0:
            sys.stderr.write(out)
        if proc.returncode != 0:
            raise RuntimeError(f"compilation of {src} failed")
    link = [_nvcc(), "-shared", "-o", str(LIB), *objs, "-cudart", "static", "-Xlinker", "--exclude-libs=ALL"]
    for cmd, lib in ((link, LIB), (_host_link(), HOST_LIB)):
        res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout)
            raise RuntimeError(f"link of {lib.name} failed")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
