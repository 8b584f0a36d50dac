"""Build libmatgptq_b200.so in-tree with nvcc for sm_100a.

    python -m matgptq_b200.build [--force] [--verbose]

The library has no torch or Python dependency: it is the C-ABI boundary declared in
``include/matgptq_b200.h``.  Beside it the module ``_torch_ops.so`` (``csrc/torch_ops.cpp``) registers the torch
operators on top of that ABI.  Objects are rebuilt only when a source or header is newer, the module also when torch,
Python or its command line is another than it was built with.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")
BUILD_DIR = os.path.join(PKG_DIR, "build")
LIB_PATH = os.path.join(PKG_DIR, "libmatgptq_b200.so")

TORCH_OPS_SOURCE = os.path.join(CSRC, "torch_ops.cpp")
TORCH_OPS_PATH = os.path.join(PKG_DIR, "_torch_ops.so")
TORCH_OPS_STAMP = os.path.join(BUILD_DIR, "_torch_ops.txt")  # what the module was built with

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libmatgptq_b200")
    return nvcc


def _sources() -> list[str]:
    return sorted(name for name in os.listdir(CSRC) if name.endswith(".cu"))


def _newest_header_mtime() -> float:
    """Newest header, or source that another source includes (gemv_zp.cu compiles gemv.cu a second time)."""
    mt = 0.0
    for d in (CSRC, INCLUDE):
        for name in os.listdir(d):
            if name.endswith((".h", ".cuh")) or name == "gemv.cu":
                mt = max(mt, os.path.getmtime(os.path.join(d, name)))
    return mt


def _torch_ops_command() -> list[str]:
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    return ["g++", "-O2", "-std=c++20", "-fPIC", "-shared", TORCH_OPS_SOURCE, "-o", TORCH_OPS_PATH,
            "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
            "-I", os.path.join(cuda, "include"), "-I", sysconfig.get_paths()["include"],
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-L", os.path.join(root, "lib"), "-Wl,-rpath," + os.path.join(root, "lib"),
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]


def _torch_ops_built_with() -> str:
    import torch
    return "\n".join([torch.__version__, sys.version, *_torch_ops_command()])


def _torch_ops_stale() -> bool:
    """The module is bound to the ABI of the torch and Python that compiled it: an upgrade of either makes it stale
    although no source is newer."""
    if not os.path.exists(TORCH_OPS_PATH) or not os.path.exists(TORCH_OPS_STAMP):
        return True
    if os.path.getmtime(TORCH_OPS_PATH) < max(os.path.getmtime(TORCH_OPS_SOURCE),
                                              os.path.getmtime(os.path.join(INCLUDE, "matgptq_b200.h"))):
        return True
    with open(TORCH_OPS_STAMP) as f:
        return f.read() != _torch_ops_built_with()


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``.cu`` under ``csrc/`` and link the shared library, compile the operator module. Returns the
    library's path."""
    nvcc = _nvcc()
    os.makedirs(BUILD_DIR, exist_ok=True)
    hdr_mtime = _newest_header_mtime()
    objects = []
    procs = []
    for src in _sources():
        src_path = os.path.join(CSRC, src)
        obj = os.path.join(BUILD_DIR, src.replace(".cu", ".o"))
        objects.append(obj)
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src_path), hdr_mtime)
        if stale:
            cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-I", CSRC, "-c", src_path, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
                print(" ".join(cmd), flush=True)
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    operators = None
    if force or _torch_ops_stale():
        operators = subprocess.Popen(_torch_ops_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    failed = False
    for src, proc in procs:
        out, _ = proc.communicate()
        if proc.returncode != 0:
            failed = True
            sys.stderr.write(f"--- nvcc failed on {src} ---\n{out}\n")
        elif verbose and out:
            print(out)
    if operators is not None:
        out, _ = operators.communicate()
        if operators.returncode != 0:
            failed = True
            sys.stderr.write(f"--- g++ failed on torch_ops.cpp ---\n{out}\n")
        else:
            with open(TORCH_OPS_STAMP, "w") as f:
                f.write(_torch_ops_built_with())
    if failed:
        raise RuntimeError("compilation failed")
    relink = force or procs or not os.path.exists(LIB_PATH)
    if relink:
        cmd = [nvcc, "-shared", "-o", LIB_PATH, *objects, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        subprocess.run(cmd, check=True)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
