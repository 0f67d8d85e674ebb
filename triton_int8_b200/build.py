"""Build the native parts in-tree: libi8linear.so (CUDA, with nvcc for sm_100a, which cross-compiles without a GPU) and
_host.so (the host path of the composed calls, a torch extension module, with g++).

    python -m triton_int8_b200.build [--force]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libi8linear.so")
HOST_PATH = os.path.join(PKG_DIR, "_host.so")
SOURCES = ["quant.cu", "gemm.cu", "fused.cu", "compose.cu"]
HOST_SOURCE = os.path.join(CSRC, "host.cpp")
ABI_HEADER = os.path.join(os.path.dirname(PKG_DIR), "include", "i8linear.h")
HEADERS = [os.path.join(CSRC, "common.cuh"), os.path.join(CSRC, "ptx.cuh"), ABI_HEADER]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--shared", "-cudart", "static",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add it to PATH")


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def needs_build() -> bool:
    return _stale(LIB_PATH, [os.path.join(CSRC, s) for s in SOURCES] + HEADERS)


def host_abi() -> str:
    """What _host.so is built against: a module for another torch or Python may load all the same and then misread their
    objects."""
    import sysconfig

    import torch
    return f"torch {torch.__version__}, {sysconfig.get_config_var('SOABI')}"


def needs_host_build() -> bool:
    if _stale(HOST_PATH, [HOST_SOURCE, ABI_HEADER]):
        return True
    with open(HOST_PATH, "rb") as f:
        return host_abi().encode() + b"\0" not in f.read()


def _host_command() -> list:
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), cuda,
               sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DI8L_HOST_ABI="{host_abi()}"', *(f"-isystem{i}" for i in include),
            "-o", HOST_PATH, HOST_SOURCE, f"-L{os.path.join(root, 'lib')}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10",
            "-lc10_cuda"]


def build(force: bool = False, verbose: bool = False) -> str:
    jobs = []
    if force or needs_build():
        cmd = [_nvcc(), *NVCC_FLAGS, "-o", LIB_PATH] + [os.path.join(CSRC, s) for s in SOURCES]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        jobs.append(cmd)
    if force or needs_host_build():
        jobs.append(_host_command())
    running = [(cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)) for cmd in jobs]
    for cmd, proc in running:
        out = proc.communicate()[0]
        if verbose:
            print(" ".join(cmd) + "\n" + out)
        if proc.returncode != 0:
            raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n{out}")
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
