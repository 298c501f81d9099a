"""Builds libadamas_b200.so (nvcc, sm_100a only) and the extension module _native.so (g++, csrc/binding.cpp) next to this file.

    python adamas_b200/build.py [--force] [-v]

(run it as a script: `python -m adamas_b200.build` imports the package first, which refuses to load
when the library is missing or stale)
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libadamas_b200.so")
NATIVE_PATH = os.path.join(PKG_DIR, "_native.so")
SOURCES = [os.path.join(CSRC, "adamas_b200.cu")]
NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-shared",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; adamas_b200 has no prebuilt or CPU fallback")
    return exe


def _native_command() -> list:
    """The CPython extension over torch's C++ headers; torch's libraries are loaded by `import torch` before it, the
    CUDA library is found next to it."""
    import sysconfig

    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    return [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", NATIVE_PATH,
            os.path.join(CSRC, "binding.cpp"), "-I", os.path.join(root, "include"),
            "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
            "-I", sysconfig.get_paths()["include"], "-I", os.path.join(cuda, "include"),
            "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
            "-L", PKG_DIR, "-ladamas_b200", "-Wl,-rpath,$ORIGIN"]


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    return any(os.path.getmtime(d) > built for d in deps if os.path.exists(d))


def _run(cmd, verbose: bool) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + proc.stdout + proc.stderr)
    if verbose:
        print(proc.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the CUDA sources and the Python binding where they are missing or older than a source."""
    header = os.path.join(os.path.dirname(PKG_DIR), "include", "adamas_b200.h")
    binding = os.path.join(CSRC, "binding.cpp")
    kernels = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")]
    if force or _stale(LIB_PATH, kernels + [header]):
        cmd = [_nvcc(), *NVCC_FLAGS, "-o", LIB_PATH, *SOURCES]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        _run(cmd, verbose)
    if force or _stale(NATIVE_PATH, [binding, header]):
        _run(_native_command(), verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
