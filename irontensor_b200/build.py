"""Builds, in-tree, libirontensor_b200.so with nvcc for sm_100a (cross-compiles without a GPU) and _host_ops.so, the native host
side of the Python ops, with g++ against the installed torch.

    python -m irontensor_b200.build [--force] [--verbose]
"""
import os
import subprocess
import sys

_HERE = os.path.dirname(os.path.abspath(__file__))
_CSRC = os.path.join(_HERE, "csrc")
_OUT = os.path.join(_HERE, "libirontensor_b200.so")
_INC = os.path.join(os.path.dirname(_HERE), "include")
_HOST_SRC = os.path.join(_CSRC, "host_ops.cpp")
_HOST_OUT = os.path.join(_HERE, "_host_ops.so")


def _sources():
    deps = [os.path.join(_CSRC, f) for f in sorted(os.listdir(_CSRC)) if f.endswith((".cu", ".cuh"))]
    deps.append(os.path.join(_INC, "irontensor_b200.h"))
    return deps


def up_to_date():
    if not os.path.exists(_OUT):
        return False
    t = os.path.getmtime(_OUT)
    return all(os.path.getmtime(s) <= t for s in _sources())


def _host_up_to_date():
    return os.path.exists(_HOST_OUT) and all(os.path.getmtime(s) <= os.path.getmtime(_HOST_OUT)
                                             for s in (_HOST_SRC, os.path.join(_INC, "irontensor_b200.h")))


def build_host(force=False):
    """_host_ops.so: links libirontensor_b200.so (next to it) and torch's libraries (loaded by `import torch` beforehand)."""
    if not force and _host_up_to_date():
        return _HOST_OUT
    import sysconfig
    import torch
    from torch.utils import cpp_extension as ext
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-Wno-missing-field-initializers",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I" + sysconfig.get_paths()["include"]]
    cmd += ["-isystem" + p for p in ext.include_paths() + ["/usr/local/cuda/include"]]
    cmd += [_HOST_SRC, "-o", _HOST_OUT, "-L" + _HERE, "-l:libirontensor_b200.so", "-Wl,-rpath,$ORIGIN"]
    cmd += ["-L" + p for p in ext.library_paths()] + ["-lc10", "-ltorch_cpu", "-ltorch_python", "-lc10_cuda", "-ltorch_cuda"]
    subprocess.run(cmd, check=True)
    return _HOST_OUT


def build(force=False, verbose=False):
    if not force and up_to_date():
        build_host()
        return _OUT
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "-shared", "-Xcompiler", "-fPIC", "-o", _OUT, os.path.join(_CSRC, "it_capi.cu")]
    if verbose:
        cmd[1:1] = ["-Xptxas", "-v"]
    subprocess.run(cmd, check=True)
    build_host(force)
    return _OUT


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(_OUT)
