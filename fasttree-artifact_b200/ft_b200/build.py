"""Builds libfasttree_b200.so (sm_100a) and the Python call module ft_call.so in-tree, with nvcc and g++.

Usage:  python fasttree-artifact_b200/ft_b200/build.py [--force] [--verbose]
"""
import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))   # fasttree-artifact_b200/
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIB_PATH = os.path.join(PKG_DIR, "libfasttree_b200.so")

SOURCES = ["ft_api.cu", "ft_planner.cu"]

CALL_PATH = os.path.join(PKG_DIR, "ft_call.so")     # Python extension: checks, argument block and call of a decode step
CALL_SOURCE = os.path.join(CSRC, "ft_call.cpp")
CALL_STAMP = CALL_PATH + ".srchash"


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return exe


STAMP_PATH = LIB_PATH + ".srchash"


def _source_digest():
    """SHA-256 over the names and contents of every file the library is built from.  Content, not time stamps:
    a copy of the tree (another machine, a container snapshot) keeps no usable modification times."""
    import hashlib
    h = hashlib.sha256()
    for folder in (CSRC, INCLUDE):
        for name in sorted(os.listdir(folder)):
            if name.endswith((".cu", ".cuh", ".h")):
                h.update(name.encode())
                with open(os.path.join(folder, name), "rb") as fh:
                    h.update(fh.read())
    h.update(os.environ.get("FT_B200_NVCC_FLAGS", "").encode())
    return h.hexdigest()


def _stale():
    """True when the library is missing or was built from other sources than the ones in the tree."""
    if not os.path.exists(LIB_PATH) or not os.path.exists(STAMP_PATH):
        return True
    with open(STAMP_PATH) as fh:
        return fh.read().strip() != _source_digest()


def _call_digest():
    """What the call module was built from: its source, the C ABI's header, and the torch and Python it links to."""
    import hashlib
    import torch
    h = hashlib.sha256(f"{torch.__version__} {sys.version}".encode())
    for path in (CALL_SOURCE, os.path.join(INCLUDE, "fasttree_b200.h")):
        with open(path, "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()


def call_module_stale():
    if not os.path.exists(CALL_PATH) or not os.path.exists(CALL_STAMP):
        return True
    with open(CALL_STAMP) as fh:
        return fh.read().strip() != _call_digest()


def build_call_module(force=False, verbose=False):
    """Compile ft_call.cpp into a Python extension module against the installed torch."""
    if not force and not call_module_stale():
        return CALL_PATH
    import sysconfig
    import torch
    torch_dir = os.path.dirname(torch.__file__)
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        raise RuntimeError("g++ not found; the call module cannot be built")
    cuda_home = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = [cxx, "-shared", "-fPIC", "-O2", "-std=c++17", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", INCLUDE, "-I", os.path.join(torch_dir, "include"),
           "-I", os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           "-I", os.path.join(cuda_home, "include"), "-I", sysconfig.get_paths()["include"],
           CALL_SOURCE, "-o", CALL_PATH, "-L", os.path.join(torch_dir, "lib"),
           "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if verbose or res.returncode != 0:
        print(res.stdout)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + res.stdout)
    with open(CALL_STAMP, "w") as fh:
        fh.write(_call_digest() + "\n")
    return CALL_PATH


def build_library(force=False, verbose=False):
    """Compile every CUDA source for sm_100a into one shared library."""
    if not force and not _stale():
        return LIB_PATH
    digest = _source_digest()
    cmd = [_nvcc(), "-shared", "-Xcompiler", "-fPIC", "-O3", "-std=c++17", "-lineinfo",
           "-gencode", "arch=compute_100a,code=sm_100a",
           "-I", INCLUDE, "-I", CSRC, "-o", LIB_PATH]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += os.environ.get("FT_B200_NVCC_FLAGS", "").split()
    cmd += [os.path.join(CSRC, s) for s in SOURCES]
    cmd += ["-lcuda"]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if verbose or res.returncode != 0:
        print(res.stdout)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout)
    with open(STAMP_PATH, "w") as fh:
        fh.write(digest + "\n")
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_call_module(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
