"""Ahead-of-time build of libb200fp4.so (sm_100a only) with nvcc.

``python cutedsl-fully-opensourced_b200/build.py`` or ``build()`` compiles every
``csrc/*.cu`` to an object file (in parallel, skipping objects that are newer
than their sources) and links them into ``lib/libb200fp4.so`` next to this
file, then the host path of the torch operators (csrc/torch_binding.cpp) into
``lib/_b200fp4_torch.so``, a CPython extension that links against it.  There is
no JIT and no fallback: the Python layer refuses to work when either is missing.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
OBJ_DIR = os.path.join(PKG_DIR, "build")
LIB_DIR = os.path.join(PKG_DIR, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libb200fp4.so")
BINDING_SRC = os.path.join(CSRC, "torch_binding.cpp")
BINDING_PATH = os.path.join(LIB_DIR, "_b200fp4_torch.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libb200fp4 can only be built with the CUDA toolkit")
    return exe


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ_DIR, exist_ok=True)
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = _nvcc()
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + sorted(
        glob.glob(os.path.join(os.path.dirname(PKG_DIR), "include", "*.h")))
    jobs = []
    objects = []
    for src in sources:
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objects.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as pool:
        for cmd, r in pool.map(run, jobs):
            if verbose or r.returncode:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode:
                raise RuntimeError(f"nvcc failed on {cmd[-3]}")
    if jobs or force or _stale(LIB_PATH, objects):
        link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *objects]
        r = subprocess.run(link, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("linking libb200fp4.so failed")
    build_binding(force, verbose)
    return LIB_PATH


def build_binding(force: bool = False, verbose: bool = False) -> str:
    """The CPython extension between torch tensors and the C-ABI (host code only: the system C++ compiler)."""
    header = os.path.join(os.path.dirname(PKG_DIR), "include", "b200fp4.h")
    if not force and not _stale(BINDING_PATH, [BINDING_SRC, header]):
        return BINDING_PATH
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    # the compiler that nvcc drives, whatever CXX says: torch's C++ runtime must be the only one in the process
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}/include",
           f"-I{sysconfig.get_path('include')}", BINDING_SRC, "-o", BINDING_PATH,
           f"-L{root}/lib", "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
           f"-L{LIB_DIR}", "-lb200fp4", "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{root}/lib"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError("compiling _b200fp4_torch.so failed")
    return BINDING_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
