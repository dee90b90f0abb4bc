"""Builds ``liblmoe.so`` (the C-ABI CUDA library, nvcc for sm_100a) and ``_host.so`` (the layers' native host path on
PyTorch's allocator and autograd, g++) in-tree.

    python -m swamla_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  Objects go to ``swamla_b200/csrc/_obj`` and the
shared library to ``swamla_b200/liblmoe.so``.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(HERE, "liblmoe.so")
HOST = os.path.join(HERE, "_host.so")
HOST_STAMP = os.path.join(OBJ, "host_stamp.txt")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-cudart", "shared",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime() -> float:
    latest = 0.0
    for root in (CSRC, INCLUDE):
        for dirpath, _, files in os.walk(root):
            if dirpath.startswith(OBJ):
                continue
            for f in files:
                if f.endswith((".cu", ".cuh", ".h", ".cpp")):
                    latest = max(latest, os.path.getmtime(os.path.join(dirpath, f)))
    return latest


def _host_versions() -> str:
    """What ``_host.so`` is bound to besides its sources."""
    from importlib.metadata import version
    return f"torch {version('torch')}, python {sys.version.split()[0]}"


def _host_fits() -> bool:
    try:
        with open(HOST_STAMP) as f:
            return f.read() == _host_versions()
    except OSError:
        return False


def _build_host() -> None:
    """``csrc/torch_host.cpp`` -> ``_host.so``: a Python module against the installed PyTorch's headers and libraries,
    linked to ``liblmoe.so`` beside it."""
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"), INCLUDE]
    libdir = os.path.join(root, "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-isystem{i}" for i in inc],
           os.path.join(CSRC, "torch_host.cpp"), "-o", HOST, f"-L{HERE}", f"-L{libdir}", "-l:liblmoe.so", "-ltorch_python",
           "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
           f"-L{os.path.join(os.path.dirname(os.path.dirname(_nvcc())), 'lib64')}", "-lcudart", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for torch_host.cpp:\n{r.stdout}\n{r.stderr}")
    with open(HOST_STAMP, "w") as f:
        f.write(_host_versions())


def build(force: bool = False, verbose: bool = False) -> str:
    newest = _deps_mtime()
    os.makedirs(OBJ, exist_ok=True)
    if not force and all(os.path.exists(p) and os.path.getmtime(p) >= newest for p in (LIB, HOST)):
        if not _host_fits():          # PyTorch or Python has changed since
            _build_host()
        return LIB
    nvcc = _nvcc()

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, src[:-3] + ".o")
        extra = os.environ.get("LMOE_NVCC_EXTRA", "").split()     # e.g. -DLMOE_CHAIN_TRACE for a development build
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, sources()))
    cmd = [nvcc, "-shared", "-cudart", "shared", "-o", LIB, *objs, "-Xlinker", "-rpath,/usr/local/cuda/lib64"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_host()
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
