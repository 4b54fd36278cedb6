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


def host_tag():
    """What a built host extension belongs to: torch's C++ classes and Python's objects have no stable layout."""
    import torch
    return "torch %s, python %d.%d" % ((torch.__version__,) + sys.version_info[:2])


def host_stale(lib=None):
    lib = lib or HOST_LIB
    if not os.path.exists(lib) or any(os.path.getmtime(d) > os.path.getmtime(lib) for d in (os.path.join(HERE, "host_call.cpp"), os.path.abspath(__file__))):
        return True
    with open(lib, "rb") as f:
        return host_tag().encode() + b"\0" not in f.read()  # BUILT_FOR, as host_call.cpp keeps it


def build_host(force=False):
    if not force and not host_stale():
        return HOST_LIB
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           '-DBUILT_FOR="%s"' % host_tag(), "-I" + os.path.join(root, "include"), "-I/usr/local/cuda/include", "-I" + sysconfig.get_paths()["include"],
           os.path.join(HERE, "host_call.cpp"), "-L" + os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-ltorch_python", "-o", HOST_LIB]
    subprocess.run(cmd, check=True)
    return HOST_LIB


def main(argv):
    """The CUDA library needs nvcc alone; the host extension is built where torch and a host compiler are there too."""
    print(build(force="--force" in argv, verbose="--verbose" in argv, sabotage="--sabotage" in argv))
    try:
        print(build_host("--force" in argv))
    except (ImportError, OSError, subprocess.CalledProcessError) as x:
        print("no native host side for torch products (%s); they go through ctypes" % x, file=sys.stderr)


if __name__ == "__main__":
    main(sys.argv[1:])
