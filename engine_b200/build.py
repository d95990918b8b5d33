"""Build recipe for libhanzoquant_b200.so (plain nvcc, sm_100a only).

The library is built in-tree next to this file so the shared object travels
with the source tree; there is no JIT step at import time.  Every .cu under
csrc/ is compiled to an object of its own (in parallel, and only when it or a
header changed), then the objects are linked into one shared library.
"""
from __future__ import annotations

import os
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(HERE, "build")
LIB_PATH = os.path.join(HERE, "libhanzoquant_b200.so")
HOST_SRC = os.path.join(CSRC, "hq_torch.cpp")
HOST_PATH = os.path.join(HERE, "_hqtorch.so")
PUBLIC_HEADER = os.path.join(HERE, "..", "include", "hanzoquant_b200.h")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))] + [PUBLIC_HEADER]


def _obj(src: str) -> str:
    return os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def needs_build() -> bool:
    return _stale(LIB_PATH, sources() + _headers())


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ and link them into one shared library, then the host path's extension module;
    returns the library's path."""
    path = build_library(force, verbose)
    build_host(force)
    return path


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB_PATH
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libhanzoquant_b200.so")
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdrs = _headers()
    todo = [s for s in sources() if force or _stale(_obj(s), [s] + hdrs)]

    def compile_one(src):
        cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", _obj(src)]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        return src, subprocess.run(cmd, capture_output=True, text=True)

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(todo)))) as pool:
        for src, res in pool.map(compile_one, todo):
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed on {os.path.basename(src)}:\n" + res.stdout + res.stderr)
            if verbose:
                print(res.stderr)
    link = [nvcc, "-shared", "-o", LIB_PATH, *[_obj(s) for s in sources()], "-lcuda"]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("link failed:\n" + res.stdout + res.stderr)
    return LIB_PATH


def build_host(force: bool = False) -> str:
    """The Python layer's host path (csrc/hq_torch.cpp) as an extension module beside the library it calls."""
    if not force and not _stale(HOST_PATH, [HOST_SRC, PUBLIC_HEADER]):
        return HOST_PATH
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wno-deprecated-declarations",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", HOST_SRC, "-o", HOST_PATH,
           *[f"-I{p}" for p in cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]],
           f"-L{libs}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python",
           f"-L{HERE}", "-l:libhanzoquant_b200.so", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed on hq_torch.cpp:\n" + res.stdout + res.stderr)
    return HOST_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
