"""How the integral image's tiles are dealt out to CTAs and clusters (csrc/scan_shape.cuh), compiled for the host: every launch covers its
planes within 16 warps a CTA and 8 CTAs a cluster, and only planes that a cluster reads twice are shared by fewer than eight.  CPU only."""
import ctypes
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_launches_cover_their_planes(tmp_path):
    out = str(tmp_path / "libscan.so")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                           "-I", os.path.join(PKG_DIR, "csrc"), "-o", out, os.path.join(ROOT, "tests", "host_emulation", "scan.cu")])
    assert ctypes.CDLL(out).scan_shapes(160, 400, 16) > 0
