"""Builds, in-tree, libmcep.so (the CUDA kernels and the C ABI, nvcc, for sm_100a only) and
_mcep_torch.so (the native part of the Python binding, g++ against torch's headers)."""
from __future__ import annotations

import fcntl
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
# MCEP_LIB points the package at a library built elsewhere (e.g. a diagnostic build)
LIB = os.environ.get("MCEP_LIB") or os.path.join(HERE, "libmcep.so")
SOURCES = ["ep_kernels.cu", "ep_runtime.cu", "ep_noalloc.cu", "ep_elastic_kernels.cu",
           "ep_elastic.cu"]
HEADERS = ["ep_kernels.cuh", "ep_device.cuh", "ep_routing.cuh", "ep_launch.cuh", "ep_elastic.cuh", "ep_runtime_internal.h",
           os.path.join("..", "..", "include", "mcep.h")]


STAMP = LIB + ".sources"  # digest of the sources the library was built from


def _digest() -> str:
    h = hashlib.sha256()
    h.update(os.environ.get("MCEP_NVCC_FLAGS", "").encode())
    for f in SOURCES + HEADERS:
        path = os.path.join(CSRC, f)
        if os.path.exists(path):
            with open(path, "rb") as fh:
                h.update(fh.read())
    return h.hexdigest()


def _stale() -> bool:
    """True when the library is missing or was built from other sources (file
    contents are compared, not times: a copy of the tree keeps no times)."""
    if not os.path.exists(LIB):
        return True
    try:
        with open(STAMP) as fh:
            return fh.read().strip() != _digest()
    except OSError:
        return True


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    # several processes of one job may import the package at once: one builds
    with open(LIB + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not _stale():
                return LIB
            return _build_locked(force, verbose)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def _build_locked(force: bool, verbose: bool) -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        if os.path.exists(LIB) and not force:
            return LIB  # a prebuilt library and no compiler: use what is there
        raise RuntimeError("mooncake_b200: nvcc not found; cannot build libmcep.so")
    cmd = [nvcc, "-std=c++17", "-O3", "-lineinfo",
           "-gencode", "arch=compute_100a,code=sm_100a",
           "-Xcompiler", "-fPIC", "-shared", "-cudart", "static",
           "-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
    cmd[1:1] = os.environ.get("MCEP_NVCC_FLAGS", "").split()  # e.g. -DMCEP_PHASE_TRACE
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    subprocess.run(cmd, check=True)
    with open(STAMP, "w") as fh:
        fh.write(_digest())
    return LIB


# ---- the torch binding ------------------------------------------------------------
BINDING = os.path.join(HERE, "_mcep_torch.so")
BINDING_STAMP = BINDING + ".sources"
BINDING_SOURCES = ["ep_py_torch.cpp", os.path.join("..", "..", "include", "mcep.h")]


def _binding_digest() -> str:
    import torch
    h = hashlib.sha256(f"{torch.__version__} {sys.version_info[:2]}".encode())
    for f in BINDING_SOURCES:
        path = os.path.join(CSRC, f)
        if os.path.exists(path):
            with open(path, "rb") as fh:
                h.update(fh.read())
    return h.hexdigest()


def _binding_stale() -> bool:
    if not os.path.exists(BINDING):
        return True
    try:
        with open(BINDING_STAMP) as fh:
            return fh.read().strip() != _binding_digest()
    except OSError:
        return True


def build_binding(force: bool = False) -> str:
    if not force and not _binding_stale():
        return BINDING
    with open(BINDING + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not force and not _binding_stale():
                return BINDING
            cxx = shutil.which("g++")
            if cxx is None:
                if os.path.exists(BINDING) and not force:
                    return BINDING  # a prebuilt binding and no compiler: use what is there
                raise RuntimeError("mooncake_b200: g++ not found; cannot build _mcep_torch.so")
            import sysconfig
            import torch
            root = os.path.dirname(torch.__file__)
            cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
            include = [os.path.join(HERE, "..", "include"), sysconfig.get_paths()["include"],
                       os.path.join(root, "include"),
                       os.path.join(root, "include", "torch", "csrc", "api", "include"),
                       os.path.join(cuda, "include")]
            cmd = [cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-fvisibility=hidden",
                   f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            cmd += [a for d in include for a in ("-isystem", d)]
            cmd += [os.path.join(CSRC, BINDING_SOURCES[0]), "-o", BINDING, "-L", os.path.join(root, "lib"),
                    "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
            subprocess.run(cmd, check=True)
            with open(BINDING_STAMP, "w") as fh:
                fh.write(_binding_digest())
            return BINDING
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build_binding(force="--force" in sys.argv))
