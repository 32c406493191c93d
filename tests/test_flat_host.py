"""The whole-plane kernels that deal out strips (csrc/bc_flat.cuh), compiled for the host: what a launch asks for is what the device and the
packed fields of a strip hold, every plane that the kernel's predecessor took still fits, rows are where the kernels' clamped sums of offsets say,
and neighbouring strips fall into neighbouring banks across row groups and planes.  CPU only."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG_DIR, ROOT

NAMES = "warps tiles_a_warp planes split columns smem strips groups plane last row sub group_bank plane_bank tiles image".split()


@pytest.fixture(scope="module")
def flat(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("flat") / "libflat.so")
    src = os.path.join(ROOT, "tests", "host_emulation", "flat.cu")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                           "-I", os.path.join(PKG_DIR, "csrc"), "-o", out, src])
    return ctypes.CDLL(out)


def plan(flat, N, C, F, h, w, write_gin=1):
    v = (ctypes.c_int64 * 16)()
    flat.flat_backward(N, C, F, h, w, write_gin, v)
    return dict(zip(NAMES, v))


def served():
    """Sizes of at most 32 tiles of 32 x 32 whose padded integral image and two rows of sums a tile take at most 200 KB."""
    for h in list(range(1, 41)) + list(range(41, 1025, 13)) + [63, 64, 65, 127, 128, 255, 256, 952, 960, 1000, 1023, 1024]:
        for w in list(range(1, 41)) + list(range(41, 1025, 17)) + [63, 64, 65, 127, 128, 255, 256, 1000, 1023, 1024]:
            tiles = -(-h // 32) * -(-w // 32)
            if tiles <= 32 and ((h + 1) * (w + 9) + h // 8 + 7 + 64 * tiles) * 4 <= 200 * 1024:
                yield h, w


def test_launches_fit(flat):
    for h, w in served():
        for N, C, F in ((1, 1, 1), (1, 3, 4), (7, 1, 8), (33, 4, 2), (150, 1, 32), (3000, 2, 4)):
            for gin in (0, 1):
                p = plan(flat, N, C, F, h, w, gin)
                at = (N, C, F, h, w, p)
                assert p["warps"] <= (24 if p["tiles_a_warp"] == 1 else 16), at
                assert p["warps"] * p["tiles_a_warp"] * 32 >= p["strips"] * p["groups"] * p["planes"] and p["tiles"] == p["warps"] * p["tiles_a_warp"], at
                assert p["smem"] <= 227 * 1024 - 64 and p["image"] + p["tiles"] * 544 < p["smem"], at
                assert 1 <= p["planes"] <= min(255, N) and p["strips"] < 1024 and p["groups"] < 1024, at
                each = -(-F // p["split"]) if p["split"] > 1 else 1
                assert 1 <= p["split"] <= min(F, 8) and p["columns"] in (64, 128, 256, 512), at
                assert 64 * p["tiles_a_warp"] * -(-p["warps"] // 4) * each <= p["columns"], at
                if gin and p["split"] > 1:
                    assert p["tiles"] * 4096 * each <= p["smem"], at


def test_forward_launches_fit(flat):
    for h, w in served():
        for N, C, F in ((1, 1, 1), (1, 3, 4), (7, 1, 6), (150, 1, 32), (3000, 2, 4)):
            v = (ctypes.c_int64 * 9)()
            flat.flat_forward(N, C, F, h, w, v)
            warps, planes, fsplit, tsplit, smem, strips, groups, image, tight = v
            at = (N, C, F, h, w, list(v))
            assert warps <= 32 and strips * groups * planes <= warps * 32 and planes <= N, at
            assert smem <= 227 * 1024 - 64 and 1 <= fsplit <= F and F % fsplit == 0 and tsplit in (1, 2, 4), at
            assert smem >= image + warps * 544 + 48 * F + (0 if tight else warps * 1152) and (not tight or image >= warps * 1152), at


def test_layout(flat):
    for h, w in list(served())[::7]:
        p = plan(flat, 1, 1, 1, h, w)
        assert p["group_bank"] == p["plane_bank"] == 0, (h, w)
        assert p["row"] == 4 * p["sub"] and p["sub"] == 4 * (p["strips"] + 4)
        assert p["last"] == flat.flat_row(h, w, h) and p["last"] + p["row"] <= p["plane"]
        for group in {0, p["groups"] - 1}:
            for a in (-h - 17, -9, -8, -1, 0, 1, 5, 7, 8, h, h + 16):
                for j in range(9):
                    row = min(max(group * 8 + a + j, 0), h)
                    assert flat.flat_offset(h, w, group, a, j) == flat.flat_row(h, w, row), (h, w, group, a, j)
