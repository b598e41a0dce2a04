"""Build the two shared objects of the package in-tree.

    python -m tybok_b200.build [--force] [--verbose]

``libtybok_b200.so``: the kernels and their C ABI, nvcc for sm_100a (no torch, no pybind);
``tybok_b200._lib`` loads it with ctypes, and nvcc cross-compiles without a GPU.
``_native.so``: the host path from torch tensors to that C ABI (``csrc/host``), a Python extension
built with the host compiler against this interpreter's torch.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libtybok_b200.so")
HOST_SRC = os.path.join(CSRC, "host")
NATIVE = os.path.join(HERE, "_native.so")
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]


def sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _newer(out: str, deps: list[str]) -> bool:
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in deps)


def _stale() -> bool:
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if os.path.isfile(os.path.join(CSRC, f))]
    return _newer(LIB, deps + [os.path.join(HERE, "..", "include", "tybok_b200.h")])


def build_native(force: bool = False) -> str:
    """Compile ``csrc/host/*.cpp`` into ``_native.so``, linked to ``libtybok_b200.so`` beside it; returns its path."""
    from concurrent.futures import ThreadPoolExecutor
    import sysconfig
    import tempfile

    srcs = sorted(os.path.join(HOST_SRC, f) for f in os.listdir(HOST_SRC) if f.endswith(".cpp"))
    deps = [os.path.join(HOST_SRC, f) for f in os.listdir(HOST_SRC)] + [os.path.join(HERE, "..", "include", "tybok_b200.h")]
    if not force and not _newer(NATIVE, deps):
        return NATIVE
    import torch
    from torch.utils import cpp_extension as ext

    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        raise RuntimeError("no host C++ compiler: _native.so cannot be built on this machine")
    cuda = ext.CUDA_HOME or "/usr/local/cuda"
    inc = [f"-isystem{p}" for p in ext.include_paths(device_type="cuda")] + [f"-isystem{sysconfig.get_paths()['include']}"]
    flags = ["-O2", "-fPIC", "-std=c++17", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_native", "-DTORCH_API_INCLUDE_EXTENSION_H",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *inc]
    with tempfile.TemporaryDirectory() as tmp:
        def compile_one(src: str) -> str:
            obj = os.path.join(tmp, os.path.basename(src) + ".o")
            proc = subprocess.run([cxx, *flags, "-c", src, "-o", obj], capture_output=True, text=True)
            if proc.returncode != 0:
                raise RuntimeError(f"{cxx} failed on {src}:\n{proc.stderr}")
            return obj

        with ThreadPoolExecutor() as pool:
            objs = list(pool.map(compile_one, srcs))
        libs = os.path.join(os.path.dirname(torch.__file__), "lib")
        cmd = [cxx, "-shared", "-o", NATIVE, *objs, f"-L{HERE}", "-l:libtybok_b200.so", f"-L{libs}", "-lc10", "-lc10_cuda", "-ltorch_cpu",
               "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-L{cuda}/lib64", "-lcudart", "-Wl,-rpath,$ORIGIN"]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode != 0:
            raise RuntimeError(f"link of _native.so failed:\n{' '.join(cmd)}\n{proc.stderr}")
    return NATIVE


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``csrc/*.cu`` into ``libtybok_b200.so`` and the host path into ``_native.so``; returns the library's path."""
    if not force and not _stale():
        build_native()
        return LIB
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: libtybok_b200.so cannot be built on this machine")
    cmd = [nvcc, "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-O3", "-lineinfo", *ARCH_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB, *sources()]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed:\n{' '.join(cmd)}\n{proc.stdout}\n{proc.stderr}")
    if verbose:
        print(proc.stderr)
    build_native(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
