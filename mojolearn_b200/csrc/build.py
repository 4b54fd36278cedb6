"""Compile libb200i.so (the CUDA kernels and their C ABI) for sm_100a, in tree.

    python -m mojolearn_b200.csrc.build [--force] [--verbose]

nvcc cross-compiles without a GPU. The flags are part of the numerical
contract: no multiply-add contraction by the compiler (-fmad=false), IEEE
subnormals (-ftz=false), IEEE division and square root, no fast-math. Every
fused multiply-add in the kernels is an explicit fma.rn.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libb200i.so")
#: the negative-control build: every window admitted (-DB200I_SABOTAGE_ADMIT_ALWAYS); loaded only by the tests
SABOTAGE_LIB = os.path.join(HERE, "libb200i_sabotage_admit.so")
SOURCES = ["b200i.cu"]
HEADERS = sorted(f for f in os.listdir(HERE) if f.endswith(".cuh")) + [os.path.join("..", "..", "include", "b200i.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-fmad=false", "-ftz=false", "-prec-div=true", "-prec-sqrt=true",
    "-shared", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=default", "-cudart", "shared",
]


def stale(lib=LIB):
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    deps = [os.path.join(HERE, s) for s in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    return any(os.path.exists(d) and os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False, sabotage=False):
    lib = SABOTAGE_LIB if sabotage else LIB
    if not force and not stale(lib):
        return lib
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc] + NVCC_FLAGS + (["-DB200I_SABOTAGE_ADMIT_ALWAYS"] if sabotage else []) + (["-Xptxas", "-v"] if verbose else []) \
        + [os.path.join(HERE, s) for s in SOURCES] + ["-o", lib]
    subprocess.run(cmd, check=True)
    return lib


#: the native host side of a product call (host_call.cpp), a Python extension over torch's C++ library
HOST_LIB = os.path.join(os.path.dirname(HERE), "_host_call.so")


def build_host(force=False):
    source = os.path.join(HERE, "host_call.cpp")
    if not force and os.path.exists(HOST_LIB) and os.path.getmtime(HOST_LIB) >= os.path.getmtime(source):
        return HOST_LIB
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           "-I" + os.path.join(root, "include"), "-I/usr/local/cuda/include", "-I" + sysconfig.get_paths()["include"], source, "-L" + os.path.join(root, "lib"),
           "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-ltorch_python", "-o", HOST_LIB]
    subprocess.run(cmd, check=True)
    return HOST_LIB


if __name__ == "__main__":
    build_host("--force" in sys.argv)
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, sabotage="--sabotage" in sys.argv))
