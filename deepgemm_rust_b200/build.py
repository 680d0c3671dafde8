"""Ahead-of-time build of libdgb200.so (the C-ABI library) with nvcc for sm_100a, and of the package's
compiled Python binding.

`python deepgemm_rust_b200/build.py` (or build()) compiles csrc/dg_api.cu, which includes the
kernel headers, into deepgemm_rust_b200/libdgb200.so (nvcc cross-compiles without a GPU), and
csrc/dg_binding.cpp with the host compiler against torch into deepgemm_rust_b200/_dg_binding.so.
"""
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libdgb200.so")
BINDING = os.path.join(HERE, "_dg_binding.so")
HEADER = os.path.join(HERE, "..", "include", "dgb200.h")
SOURCES = ["dg_api.cu"]
BINDING_SOURCE = "dg_binding.cpp"


def deps():
    """Every source the library is compiled from: all of csrc/ plus the public header."""
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))) + [HEADER]


NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-shared",
         "-Xcompiler", "-fPIC,-fvisibility=default", "--expt-relaxed-constexpr"]


def stale(target, sources) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in sources)


def needs_build() -> bool:
    return stale(OUT, deps())


def build_binding(force: bool = False) -> str:
    source = os.path.join(CSRC, BINDING_SOURCE)
    if not force and not stale(BINDING, [source, HEADER]):
        return BINDING
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    lib = os.path.join(root, "lib")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-w",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [f"-I{d}" for d in include] + [source, "-o", BINDING, f"-L{lib}", f"-Wl,-rpath,{lib}", "-ltorch_python", "-ltorch_cpu", "-lc10", "-ldl"]
    subprocess.check_call(cmd)
    return BINDING


def build(force: bool = False, verbose: bool = False) -> str:
    build_binding(force)
    if not force and not needs_build():
        return OUT
    cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", OUT] + [os.path.join(CSRC, s) for s in SOURCES]
    subprocess.check_call(cmd)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
