"""Builds libss2d_b200.so (the C-ABI library of include/ss2d_b200.h) in-tree with nvcc for sm_100a, and _host.so, the host
extension through which Python calls it.

    python vmamba_b200/build.py [--force] [--verbose]

(run as a file: importing the package needs the library this script produces)

Each translation unit of csrc/ is compiled to an object in parallel, then linked with the
static CUDA runtime.  No torch headers are involved: the library has a plain C interface.  The host extension
(csrc/host_*.cpp, g++) is the torch side of it: argument checks, results, workspaces and autograd nodes in C++, so that
a small call does not spend its time in Python.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
OBJ_DIR = os.path.join(HERE, "build")
LIB_PATH = os.path.join(HERE, "libss2d_b200.so")
HOST_PATH = os.path.join(HERE, "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the ss2d_b200 library must be built with the CUDA toolkit")
    return exe


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime() -> float:
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, "ss2d_b200.h")]
    return max(os.path.getmtime(f) for f in files)


def is_stale() -> bool:
    return any(not os.path.exists(p) or os.path.getmtime(p) < _deps_mtime() for p in (LIB_PATH, HOST_PATH))


def host_sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.startswith("host_") and f.endswith(".cpp"))


def _host_command(src: str, obj: str):
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_API_INCLUDE_EXTENSION_H", "-DTORCH_EXTENSION_NAME=_host",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [INCLUDE, *cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    return ["g++", *flags, *(f"-I{i}" for i in inc), "-c", src, "-o", obj]


def _link_host(objs):
    from torch.utils import cpp_extension
    libs = [f"-L{p}" for p in cpp_extension.library_paths()]
    cmd = ["g++", "-shared", "-o", HOST_PATH, *objs, f"-L{HERE}", "-l:libss2d_b200.so", "-Wl,-rpath,$ORIGIN", *libs,
           "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link of the host extension failed:\n{r.stdout}{r.stderr}")


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not is_stale():
        return LIB_PATH
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    logs = {}

    def compile_one(src):
        obj = os.path.join(OBJ_DIR, os.path.splitext(os.path.basename(src))[0] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", src, "-o", obj] if src.endswith(".cu") else _host_command(src, obj)
        r = subprocess.run(cmd, capture_output=True, text=True)
        logs[src] = r.stdout + r.stderr
        if r.returncode != 0:
            raise RuntimeError(f"compilation failed for {src}:\n{logs[src]}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        built = list(ex.map(compile_one, host_sources() + sources()))
    host_objs, objs = built[:len(host_sources())], built[len(host_sources()):]
    with open(os.path.join(OBJ_DIR, "ptxas.log"), "w") as f:
        for src in sorted(logs):
            f.write(f"==== {os.path.basename(src)}\n{logs[src]}\n")
    cmd = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-cudart", "static"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}{r.stderr}")
    _link_host(host_objs)
    if verbose:
        for src in sorted(logs):
            print(logs[src])
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
