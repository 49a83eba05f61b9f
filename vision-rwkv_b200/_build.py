"""Build the CUDA library in-tree with nvcc for sm_100a (no torch headers involved), and the torch extension that
calls it with g++.

    python -m vision_rwkv_b200._build        # or __graft_entry__.build()

The results, lib/libvrwkv_b200.so and lib/_native.so, are what `_lib.py` loads.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_DIR = os.path.join(PKG_DIR, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libvrwkv_b200.so")
TORCH_SRC = os.path.join(CSRC, "torch")
NATIVE_PATH = os.path.join(LIB_DIR, "_native.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _files(*dirs):
    return [os.path.join(d, f) for d in dirs for f in os.listdir(d) if os.path.isfile(os.path.join(d, f))]


def _stale(target, deps):
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def _run_all(commands, verbose):
    """Run the compilers side by side; the first failure's output is the error."""
    procs = [subprocess.Popen(c, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True) for c in commands]
    for cmd, proc in zip(commands, procs):
        out, err = proc.communicate()
        if proc.returncode != 0:
            raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + out + err)
        if verbose:
            sys.stderr.write(err)


def _nvcc():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libvrwkv_b200.so")
    return nvcc


def build_library(verbose=False):
    """Compile every .cu under csrc/ (one compiler process each) into one shared library."""
    nvcc, obj_dir = _nvcc(), os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    headers = [d for d in _files(CSRC, os.path.join(ROOT, "include")) if not d.endswith(".cu")]
    objects, commands = [], []
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src) + ".o")
        objects.append(obj)
        if _stale(obj, headers + [src, os.path.abspath(__file__)]):
            cmd = [nvcc, *NVCC_FLAGS, "-c", "-I", os.path.join(ROOT, "include"), "-I", CSRC, src, "-o", obj]
            commands.append(cmd + (["-Xptxas", "-v"] if verbose else []))
    _run_all(commands, verbose)
    _run_all([[nvcc, *NVCC_FLAGS, "-shared", *objects, "-o", LIB_PATH]], False)


def build_native():
    """Compile csrc/torch/*.cpp against torch's headers; links the library above by its place beside the extension."""
    import sysconfig
    import torch
    torch_dir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    include = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include/torch/csrc/api/include"),
               os.path.join(cuda, "include"), sysconfig.get_paths()["include"], os.path.join(ROOT, "include"), TORCH_SRC]
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    deps = _files(TORCH_SRC, os.path.join(ROOT, "include"))
    headers = [d for d in deps if d.endswith(".h")] + [os.path.abspath(__file__)]
    objects, commands = [], []
    for src in sorted(d for d in deps if d.endswith(".cpp")):
        obj = os.path.join(obj_dir, os.path.basename(src) + ".o")
        objects.append(obj)
        if _stale(obj, headers + [src]):
            commands.append(["g++", "-O2", "-std=c++17", "-fPIC", "-DTORCH_API_INCLUDE_EXTENSION_H", "-DTORCH_EXTENSION_NAME=_native",
                             *[f"-isystem{d}" for d in include], "-c", src, "-o", obj])
    _run_all(commands, False)
    _run_all([["g++", "-shared", *objects, "-L" + os.path.join(torch_dir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
               "-ltorch", "-ltorch_python", "-L" + LIB_DIR, "-lvrwkv_b200", "-Wl,-rpath,$ORIGIN", "-o", NATIVE_PATH]], False)


def build(force: bool = False, verbose: bool = False) -> str:
    """Build whatever is out of date (everything with force=True).  Returns the library's path."""
    if force:
        shutil.rmtree(os.path.join(LIB_DIR, "obj"), ignore_errors=True)
    if force or _stale(LIB_PATH, _files(CSRC, os.path.join(ROOT, "include"))):
        build_library(verbose)
    if force or _stale(NATIVE_PATH, _files(TORCH_SRC, os.path.join(ROOT, "include"))):
        build_native()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose="-v" in sys.argv))
