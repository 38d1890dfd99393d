"""Builds the C-ABI library ``lib/libb200lora.so`` from ``csrc/*.cu`` with nvcc for sm_100a, and the Python
ops' native host path ``lib/_b200host.so`` from ``csrc/host.cpp`` with g++ against the installed torch.

Both are built in-tree and never installed.  ``build()`` is a no-op when they are newer than
every source; ``force=True`` rebuilds.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libb200lora.so")
HOST_PATH = os.path.join(LIB_DIR, "_b200host.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _older(path: str, deps) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(d) > t for d in deps)


def _headers():
    return glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(INCLUDE, "*.h"))


def _stale() -> bool:
    return _older(LIB_PATH, sources() + _headers()) or _older(HOST_PATH, [HOST_SRC] + _headers())


def _host_command():
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), INCLUDE]
    return (["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-w",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + [f"-I{i}" for i in inc] +
            [HOST_SRC, "-o", HOST_PATH, LIB_PATH, "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10",
             "-lc10_cuda", "-Wl,-rpath,$ORIGIN"])


def _run(cmd, what: str, verbose: bool):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        print(res.stdout)
        print(res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"building {what} failed")
    return res


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB_PATH
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: the CUDA library cannot be built")
    os.makedirs(LIB_DIR, exist_ok=True)
    if force or _older(LIB_PATH, sources() + _headers()):
        cmd = [nvcc] + NVCC_FLAGS + ["-I", INCLUDE, "-I", CSRC] + sources() + ["-lcuda", "-Xlinker", "-soname=libb200lora.so",
                                                                            "-o", LIB_PATH]
        res = _run(cmd, "libb200lora.so", verbose)
        with open(os.path.join(LIB_DIR, "ptxas.log"), "w") as f:      # registers, spills, shared memory per kernel
            f.write("".join(l for l in res.stderr.splitlines(True) if "Compile time" not in l))
    _run(_host_command(), "_b200host.so", verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
