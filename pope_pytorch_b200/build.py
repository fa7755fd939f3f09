"""Builds libpope_b200.so in-tree with nvcc for sm_100a (no torch headers: the library is plain C ABI), and the torch
binding ``_host`` over it with the C++ compiler.

    python -m pope_pytorch_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libpope_b200.so")
HOST_SRC = os.path.join(CSRC, "torch_host.cpp")
HOST_PATH = os.path.join(PKG_DIR, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))
OBJ_DIR = os.path.join(PKG_DIR, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; libpope_b200.so cannot be built")
    return cand


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime() -> float:
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")]
    files.append(os.path.join(os.path.dirname(PKG_DIR), "include", "pope_b200.h"))
    files.append(os.path.abspath(__file__))
    return max(os.path.getmtime(f) for f in files)


def _build_host(force: bool) -> None:
    """The extension module: torch headers, no nvcc; finds libpope_b200.so beside itself."""
    deps = [HOST_SRC, os.path.join(os.path.dirname(PKG_DIR), "include", "pope_b200.h"), os.path.abspath(__file__)]
    if not force and os.path.exists(HOST_PATH) and os.path.getmtime(HOST_PATH) >= max(os.path.getmtime(f) for f in deps):
        return
    import torch
    from torch.utils.cpp_extension import CUDA_HOME, include_paths, library_paths
    cuda = CUDA_HOME or "/usr/local/cuda"
    inc = [*include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    tmp = HOST_PATH + ".tmp"
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-isystem{i}" for i in inc), HOST_SRC, "-o", tmp,
           *(f"-L{p}" for p in library_paths()), "-lc10", "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10_cuda",
           f"-L{PKG_DIR}", "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, HOST_PATH)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/, link the shared library and build the torch binding.  Returns the library's path."""
    lib = _build_lib(force, verbose)
    _build_host(force)
    return lib


def _build_lib(force: bool, verbose: bool) -> str:
    if not force and os.path.exists(LIB_PATH) and os.path.getmtime(LIB_PATH) >= _deps_mtime():
        return LIB_PATH
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", src, "-o", obj]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose:
            sys.stderr.write(res.stderr)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, _sources()))
    tmp = LIB_PATH + ".tmp"
    link = [nvcc, "-shared", "-o", tmp, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
