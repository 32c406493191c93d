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
    lib.rule_backward.argtypes = [ctypes.c_int64] + [ctypes.c_int] * 4
    lib.rule_slabs_backward.argtypes = [ctypes.c_int64] + [ctypes.c_int] * 3
    lib.rule_tmem_forward.argtypes = [ctypes.c_int64] + [ctypes.c_int] * 3 + [ctypes.POINTER(ctypes.c_int)] * 3
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


def test_tensor_memory_forward_launches_fit_their_kernels(rules):
    tiles, warps, columns = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    served = set()
    for h in range(1, 321):
        for w in range(60, 321):
            if (h % 8 or w % 4) and (h + w) % 17:
                continue
            for F in (2, 3, 4, 32):
                for planes in (74, 148, 223, 5000):
                    if rules.rule_tmem_forward(planes, F, h, w, ctypes.byref(tiles), ctypes.byref(warps), ctypes.byref(columns)):
                        served.add(tiles.value)
                        assert h % 8 == 0 and w % 4 == 0 and columns.value <= 512
                        # one tile a building warp in the streaming kernels, two in the other, which one column of tiles does not have
                        assert tiles.value <= 8 and warps.value == 8 or warps.value == 16 and tiles.value <= (16 if w <= 128 else 32)
    assert {1, 2, 8, 9, 16, 18, 32} <= served


# Planes, filters, rows, columns (and whether float32) on both sides of the rules' lines, as measured: where other kernels are faster,
# and where these are.
FORWARD_ELSEWHERE = [(2878, 4, 96, 160), (340, 6, 80, 160), (217, 4, 120, 160), (1171, 3, 128, 172), (1799, 3, 8, 216), (191, 3, 24, 228), (2332, 6, 24, 84),
                     (470, 3, 64, 168), (1405, 3, 64, 88), (1299, 6, 128, 80), (228, 2, 8, 188), (188, 4, 8, 208), (2114, 2, 8, 216), (184, 2, 16, 244), (1157, 4, 16, 212)]
FORWARD_HERE = [(512, 4, 64, 128), (8192, 4, 64, 128), (128, 4, 128, 256), (101, 3, 56, 116), (147, 3, 104, 72), (500, 3, 64, 128), (123, 16, 8, 80), (967, 4, 8, 128),
                (260, 16, 8, 256), (604, 6, 16, 164), (104, 4, 104, 164), (84, 2, 72, 172), (682, 4, 40, 184)]
PAIR_ELSEWHERE = [(1471, 1, 88, 156, 0), (725, 4, 72, 132, 1), (748, 2, 80, 132, 1), (1992, 2, 72, 140, 0), (969, 2, 96, 148, 1), (550, 4, 96, 156, 1), (564, 4, 88, 140, 0), (272, 4, 88, 160, 1)]
PAIR_HERE = [(722, 16, 88, 136, 1), (592, 16, 72, 140, 0), (360, 8, 80, 152, 1), (425, 6, 80, 160, 1), (383, 4, 88, 140, 0), (128, 4, 128, 256, 1), (128, 4, 96, 160, 1), (110, 16, 112, 132, 1), (991, 4, 128, 156, 1), (1482, 4, 112, 160, 1), (1583, 6, 104, 164, 1), (1400, 4, 72, 164, 1), (149, 4, 128, 128, 1)]


def test_sizes_that_other_kernels_are_faster_on_go_there(rules):
    n = [ctypes.byref(ctypes.c_int()) for _ in range(3)]
    assert not [c for c in FORWARD_ELSEWHERE if rules.rule_tmem_forward(*c, *n)]
    assert all(rules.rule_tmem_forward(*c, *n) for c in FORWARD_HERE)
    assert not [c for c in PAIR_ELSEWHERE if rules.rule_pair_backward(*c, *n[:2])]
    assert all(rules.rule_pair_backward(*c, *n[:2]) for c in PAIR_HERE)


# 14 and 16 tiles of 8 x 128: strips where a third of the lanes would idle, with three filters or more, for any number of planes
STRIPS_HERE = [(575, 4, 128, 72, 1), (593, 4, 56, 140, 1), (37, 3, 64, 164, 1), (148, 8, 112, 84, 0), (1300, 4, 80, 144, 1), (722, 16, 88, 136, 1)]
STRIPS_ELSEWHERE = [(148, 6, 56, 176, 0), (37, 6, 64, 200, 1), (1500, 8, 112, 92, 1), (149, 8, 64, 200, 1), (148, 2, 128, 76, 0), (300, 2, 128, 72, 1)]


def test_backward_tiles_do_not_depend_on_the_number_of_planes(rules):
    """Tiles of 8 x 128 add up alike one or two a warp, all others differently.  One or two filters on planes of 17 to 32 tiles that 16
    square ones hold are the exception."""
    assert all(rules.rule_backward(*c) == 3 for c in STRIPS_HERE)
    assert not [c for c in STRIPS_ELSEWHERE if rules.rule_backward(*c) not in (0, 1)]
    seen = set()
    for h in list(range(8, 289, 8)) + [1, 33, 93]:
        for w in list(range(4, 289, 4)) + [1, 65, 157]:
            for F in (1, 2, 3, 4, 6, 8, 32):
                if F <= 2 and 72 <= h <= 96 and 132 <= w <= 160:
                    continue
                for wide in (0, 1):
                    kinds = [rules.rule_backward(planes, F, h, w, wide) for planes in (1, 37, 74, 148, 149, 296, 297, 444, 445, 5000)]
                    assert len({max(k, 1) for k in kinds}) == 1, (F, h, w, wide, kinds)
                    seen |= set(kinds)
    assert seen == {0, 1, 2, 3}


# Backward from the input's integral image, planes of 13 to 16 tiles of strips: planes, filters, rows, columns.
SLABS_HERE = [(10, 32, 72, 184), (37, 16, 32, 492), (37, 8, 75, 194), (50, 6, 152, 96), (50, 32, 95, 134), (64, 6, 48, 284), (34, 4, 190, 78), (74, 6, 72, 208), (90, 8, 25, 446), (160, 8, 88, 144),
              (160, 16, 38, 356), (200, 4, 48, 284), (250, 32, 26, 395), (1 << 40, 4, 48, 284)]
SLABS_ELSEWHERE = [(1, 8, 40, 328), (8, 8, 104, 144), (10, 16, 203, 64), (20, 8, 80, 188), (50, 4, 120, 132), (64, 4, 96, 160), (128, 4, 96, 160), (256, 4, 96, 160), (1024, 4, 96, 160), (256, 6, 104, 144),
                   (148, 6, 48, 340), (90, 8, 105, 136), (900, 6, 88, 144)]


def test_slabs_where_strips_would_leave_the_gpu_idle(rules):
    assert all(rules.rule_slabs_backward(*c) for c in SLABS_HERE)
    assert not [c for c in SLABS_ELSEWHERE if rules.rule_slabs_backward(*c)]
