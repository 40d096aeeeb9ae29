"""CPU: the rules that share work out (icbc_gb300/csrc/bc1_shares.h): blocks
per task of a batch, blocks per warp of an image, bands of a host-buffer call."""
import ctypes
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 152
BYTE_WARPS, FLOAT_WARPS = 16 * SMS, 12 * SMS  # resident warps of the byte-row and the float-row batch kernels


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("shares") / "shares.so")
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "shares_check.cpp"), "-o", out],
                   check=True)
    lib = ctypes.CDLL(out)
    lib.bands.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    lib.image.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int]
    return lib


def shape(rules, levels, blocks, warps, level_kernels):
    lv, bl = np.array(levels, np.int32), np.array(blocks, np.int64)
    sizes, ctas = np.zeros(10, np.int32), np.zeros(10, np.int32)
    rules.batch(ctypes.c_void_p(lv.ctypes.data), ctypes.c_void_p(bl.ctypes.data), len(lv), ctypes.c_int64(warps),
                int(level_kernels), ctypes.c_void_p(sizes.ctypes.data), ctypes.c_void_p(ctas.ctypes.data))
    return sizes, ctas


def tasks(levels, blocks, sizes):
    return sum(-(-b // int(sizes[lv])) for lv, b in zip(levels, blocks))


@pytest.mark.parametrize("level", range(10))
@pytest.mark.parametrize("byte_rows", (True, False))
def test_small_tasks_fit_in_one_round(rules, level, byte_rows):
    """Tasks smaller than 32 blocks never make a second round: every task has a warp of its own."""
    warps = BYTE_WARPS if byte_rows else FLOAT_WARPS
    for total in (1, 40, 1000, 20000, 41000, 44000, 50000, 58000, 70000, 77000, 300000):
        for images in (1, 7, 60):
            blocks = [max(1, total // images)] * images
            sizes, ctas = shape(rules, [level] * images, blocks, warps, byte_rows)
            assert 1 <= sizes[level] <= 32 and ctas[level] in (4, 8)
            assert sizes[level] == 32 or tasks([level] * images, blocks, sizes) <= warps
            if not byte_rows:
                assert ctas[level] == 4


def test_light_levels_keep_whole_warps(rules):
    """Levels 0-1 take 32 blocks a task; levels 2-5 less only while that leaves most warps without a task, and never
    beside others' work that already fills them."""
    rng = random.Random(3)
    for _ in range(300):
        n = rng.randrange(1, 80)
        levels = [rng.randrange(10) for _ in range(n)]
        blocks = [int(10 ** rng.uniform(0, 4)) for _ in range(n)]
        for warps, byte_rows in ((BYTE_WARPS, True), (FLOAT_WARPS, False)):
            sizes, _ = shape(rules, levels, blocks, warps, byte_rows)
            assert sizes[0] == sizes[1] == 32
            assert len(set(sizes[2:6])) == len(set(sizes[6:8])) == len(set(sizes[8:10])) == 1
            for size in sizes:
                assert 1 <= size <= 32
            if sizes[3] < 32 and any(2 <= lv <= 5 for lv in levels):
                assert tasks(levels, blocks, sizes) <= 3 * warps // 8
            if sizes[7] < 32 and any(lv in (6, 7) for lv in levels):
                lights32 = [32 if 2 <= lv <= 5 else s for lv, s in enumerate(sizes)]
                assert tasks(levels, blocks, lights32) <= warps


def test_image_share(rules):
    """Below level 4 an image of more than a round takes whole warps; from level 4 on rounds are shared out evenly."""
    for n in (1, 500, 20000, 58368, 58369, 75625, 116000, 500000):
        for workers in (FLOAT_WARPS, BYTE_WARPS):
            for level in range(2, 10):
                share = rules.image(n, workers, level)
                assert 1 <= share <= 32
                if level < 4:
                    assert share == 32 if n > 32 * workers else share >= 16
                else:
                    rounds = -(-n // (32 * workers))
                    assert -(-n // share) <= rounds * workers


@pytest.mark.parametrize("level", range(10))
def test_host_bands(rules, level):
    """Bands follow the number of blocks, whatever the image's sides: a low, wide image is cut as a square one is."""
    last = 1
    for k in (1, 16, 47, 64, 95, 128, 156, 200, 256, 352, 512, 706, 1024, 4096):
        bands = rules.bands(level, k * 1024, SMS)
        assert 1 <= bands <= 8
        if k <= 16:
            assert bands == 1
        if k >= 512:
            assert bands >= 3  # the upload overlaps
        last = bands
    assert last >= 3
