"""The dispatch rules of the whole-plane kernels (csrc/box_plane_kernels.cuh and what it includes), compiled for the host and
walked over all sizes: what a rule sends to a kernel is a launch that this kernel can run.  CPU only (nvcc compiles without a
GPU; no kernel is instantiated)."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG_DIR, ROOT


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rules") / "librules.so")
    src = os.path.join(ROOT, "tests", "host_emulation", "rules.cu")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                           "-I", os.path.join(PKG_DIR, "csrc"), "-o", out, src])
    lib = ctypes.CDLL(out)
    lib.rule_pair_backward.argtypes = [ctypes.c_int64] + [ctypes.c_int] * 4 + [ctypes.POINTER(ctypes.c_int)] * 2
    return lib


def test_pair_backward_launches_fit_their_kernels(rules):
    bound, columns = ctypes.c_int(), ctypes.c_int()
    served = set()
    for h in range(1, 321):
        for w in range(60, 321):
            if (h % 8 or w % 4) and (h + w) % 17:      # unaligned sizes are refused before anything else: a sample of them
                continue
            for F in (1, 4, 32):
                for planes in (1, 149, 5000):
                    for wide in (0, 1):
                        threads = rules.rule_pair_backward(planes, F, h, w, wide, ctypes.byref(bound), ctypes.byref(columns))
                        if threads:
                            served.add(((h + 7) // 8) * ((w + 127) // 128))
                            assert h % 8 == 0 and w % 4 == 0
                            assert threads <= bound.value, (planes, F, h, w, wide)
                            assert columns.value <= 512, (planes, F, h, w, wide)
    assert served == {14, 16, 18, 20, 22, 24, 26, 28, 30, 32}
