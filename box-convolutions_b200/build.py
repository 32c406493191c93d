"""Builds the CUDA library for sm_100a and its PyTorch binding, in-tree:

    box-convolutions_b200/box_convolution/libboxconv_b200.so
    box-convolutions_b200/box_convolution/_torch_binding.<ABI>.so

The library: plain nvcc, no torch headers; its surface is the C ABI in include/boxconv_b200.h.
nvcc cross-compiles without a GPU.  The binding (csrc/torch_binding.cpp): g++ with torch's headers,
linked against the library beside it.  Usage: python box-convolutions_b200/build.py [--force] [-v]
"""
import argparse
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "box_convolution", "libboxconv_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17", "--threads", "0", "-Xcompiler", "-fPIC", "-shared",
]


BINDING_SRC = os.path.join(CSRC, "torch_binding.cpp")
BINDING = os.path.join(HERE, "box_convolution", "_torch_binding" + sysconfig.get_config_var("EXT_SUFFIX"))
CXX = os.environ.get("CXX", "g++")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def headers():
    return sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + [
        os.path.join(os.path.dirname(HERE), "include", "boxconv_b200.h")]


def newer(out, inputs):
    if not os.path.exists(out):
        return False
    t = os.path.getmtime(out)
    return all(os.path.getmtime(f) < t for f in inputs + [os.path.abspath(__file__)])


def run(cmd, out, verbose):
    if verbose:
        print(" ".join(cmd))
    subprocess.check_call(cmd)
    os.replace(out + ".tmp", out)


def build_library(force=False, verbose=False):
    if force or not newer(OUT, sources() + headers()):
        run([NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", OUT + ".tmp"] + sources(), OUT, verbose)
    return OUT


def build_binding(force=False, verbose=False):
    if force or not newer(BINDING, [BINDING_SRC, headers()[-1]]):
        import torch
        root = os.path.dirname(torch.__file__)
        cuda = os.path.dirname(os.path.dirname(NVCC))
        dirs = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
        libs = os.path.join(root, "lib")
        run([CXX, "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
             "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI] + ["-isystem" + d for d in dirs] +
            ["-o", BINDING + ".tmp", BINDING_SRC, "-L" + os.path.dirname(OUT), "-lboxconv_b200", "-L" + libs, "-lc10", "-lc10_cuda",
             "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + libs],
            BINDING, verbose)
    return BINDING


def build(force=False, verbose=False):
    out = build_library(force, verbose)
    build_binding(force, verbose)
    return out


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-v", "--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
    sys.exit(0)
