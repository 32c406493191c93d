"""The whole-plane kernels that deal out strips (csrc/bc_flat.cuh), compiled for the host: what a launch asks for is what the device and the
packed fields of a strip hold, every plane that the kernel's predecessor took still fits, rows are where the kernels' clamped sums of offsets say,
neighbouring strips fall into neighbouring banks across row groups and planes, and scans need no order among lanes but that of their own
barriers.  CPU only."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
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


# Planes with an SM to a CTA: (planes, filters, CTAs of a cluster) on both sides of what a GPU runs at once: 74 clusters of two, 45 of three, 33 of four, 15 of eight
@pytest.mark.parametrize("planes,F,split", [(74, 4, 2), (75, 4, 1), (45, 3, 3), (46, 3, 2), (33, 4, 4), (34, 4, 2), (15, 8, 8), (16, 8, 4), (33, 8, 4)])
@pytest.mark.parametrize("h,w", [(96, 144), (112, 132)])
def test_clusters_run_at_once(flat, planes, F, split, h, w):
    assert plan(flat, planes, 1, F, h, w)["split"] == split


def test_small_ctas_share_an_sm_by_four(flat):
    for h, w, warps in ((22, 20, 1), (39, 19, 1), (37, 60, 3), (70, 24, 2)):
        for planes in (74, 141, 147, 272, 296, 510):
            p = plan(flat, planes, 1, 8, h, w)
            assert p["warps"] == warps and (p["split"] == 1 or planes * p["split"] <= 148 * (8 // warps if warps > 2 else 4)), (planes, p)


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


# samples, channels, filters: around one and two CTAs an SM, and around the numbers of clusters that run at once
@pytest.mark.parametrize("N,C,F", [(1, 1, 1), (1, 1, 32), (1, 3, 4), (7, 1, 8), (15, 1, 8), (16, 1, 8), (33, 1, 4), (9, 4, 6), (37, 2, 2), (148, 1, 32), (149, 1, 32), (33, 4, 2), (297, 1, 3), (3000, 2, 4)])
def test_every_launch_fits(flat, N, C, F):
    at, sizes = (ctypes.c_int64 * 2)(), ctypes.c_int64()
    for gin in (0, 1):
        assert not flat.flat_walk_backward(N, C, F, gin, at, ctypes.byref(sizes)), list(at)
    assert not flat.flat_walk_forward(N, C, F, at, ctypes.byref(sizes)), list(at)
    assert sizes.value > 100000


def test_every_layout(flat):
    at, sizes = (ctypes.c_int64 * 2)(), ctypes.c_int64()
    assert not flat.flat_walk_layout(at, ctypes.byref(sizes)), list(at)


@pytest.fixture(scope="module")
def warp(tmp_path_factory):
    at = tmp_path_factory.mktemp("warp")
    shutil.copy(os.path.join(PKG_DIR, "csrc", "bc_flat.cuh"), at)
    for name in ("bc_quad.cuh", "bc_tile_io.cuh", "bc_tmem.cuh"):
        (at / name).write_text("")
    out = str(at / "libwarp.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", str(at), "-o", out,
                           os.path.join(ROOT, "tests", "host_emulation", "flat_warp.cpp")])
    return ctypes.CDLL(out)


# tiles a warp, rows, columns: strips that divide a tile (no barrier of the CTA between the scan and what follows it) and rows over two tiles
@pytest.mark.parametrize("T,h,w", [(2, 512, 4), (2, 256, 8), (2, 128, 16), (2, 64, 32), (2, 32, 64), (2, 16, 128), (2, 63, 31), (2, 32, 60), (2, 24, 77), (2, 8, 250),
                                   (1, 32, 32), (1, 15, 64), (1, 24, 40), (1, 8, 125)])
@pytest.mark.parametrize("backwards", [0, 1])
def test_scans_with_lanes_one_after_the_other(warp, T, h, w, backwards):
    """Between two barriers lanes may run in any order: whole numbers, so that sums are exact."""
    plane = np.random.RandomState(h + w).randint(-99, 100, (h, w)).astype(np.float32)
    out, published = np.full((32 * T, 8, 4), np.nan, np.float32), np.full((32 * T, 4), np.nan, np.float32)
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in (plane, out, published)]
    warp.flat_warp(T, backwards, h, w, *p)
    strips, groups = -(-w // 4), -(-h // 8)
    assert 32 * (T - 1) < strips * groups <= 32 * T
    padded = np.zeros((groups * 8, strips * 4), np.float32)
    padded[:h, :w] = plane
    want = padded.reshape(groups, 8, strips * 4).cumsum(1).cumsum(2).reshape(groups, 8, strips, 4).transpose(0, 2, 1, 3).reshape(-1, 8, 4)
    assert np.array_equal(out[:len(want)], want)
    assert np.array_equal(published[:len(want)], want[:, 7])
