"""Compile the CUDA library and the host module in-tree for sm_100a:  python -m medvision_b200.build

libmvr.so    the kernels behind the C ABI (nvcc; no torch)
_native.so   the Python package's host path on torch tensors (g++; links libmvr.so and torch)
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmvr.so")
NATIVE = os.path.join(HERE, "_native.so")
SOURCES = ["mvr_api.cu"]
HEADERS = ["mvr_arith.cuh", "mvr_geom.cuh", "mvr_generic.cuh", "mvr_stream3d.cuh", "mvr_tma3d.cuh", "mvr_brick3d.cuh", "mvr_bwd3d.cuh", "mvr_offset.cuh", "mvr_cubic3d.cuh", "mvr_flat.cuh", "mvr_label.cuh", "mvr_plane2d.cuh", "mvr_elastic.cuh", "mvr_head.cuh",
           os.path.join("..", "..", "include", "mvr.h")]
NATIVE_SOURCES = ["mvr_torch.cpp"]
NATIVE_HEADERS = [os.path.join("..", "..", "include", "mvr.h")]

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-shared"]
CXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-w"]


def _older(target, files):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(os.path.join(CSRC, f)) > t for f in files)


def needs_build():
    return _older(LIB, SOURCES + HEADERS) or _older(NATIVE, NATIVE_SOURCES + NATIVE_HEADERS)


def _build_native():
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    includes = cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]
    # the system compiler and its shared libstdc++: a second, static copy of the C++ runtime in the module crashes in iostreams
    cmd = ["g++"] + CXX_FLAGS + ["-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI]
    for i in includes:
        cmd += ["-isystem", i]
    cmd += ["-o", NATIVE] + [os.path.join(CSRC, s) for s in NATIVE_SOURCES]
    for p in cpp_extension.library_paths("cuda"):
        cmd += ["-L" + p]
    cmd += ["-L" + HERE, "-Wl,-rpath,$ORIGIN", "-l:libmvr.so", "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
            "-lcudart"]
    subprocess.check_call(cmd)


def build(force=False, verbose=False):
    """nvcc cross-compiles without a GPU; both .so stay beside the package."""
    if force or _older(LIB, SOURCES + HEADERS):
        nvcc = os.environ.get("NVCC", "nvcc")
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + \
              ["-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
        subprocess.check_call(cmd)
    if force or _older(NATIVE, NATIVE_SOURCES + NATIVE_HEADERS):
        _build_native()
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
