"""GPU: which kernels an image takes follows its size and launch shape
(icbc_gpu_launch_plan).  Each route on the images where it can go wrong --
nothing listed, everything listed, a ragged mixture -- at sizes derived from
the SM count, against the oracle, bit for bit."""
import numpy as np
import pytest

from icbc_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def sides(blocks):
    """(width, height) of a whole-block image of about `blocks` blocks, at most that many."""
    bw = int(blocks ** 0.5)
    return 4 * bw, 4 * (blocks // bw)


def check(ig, img, level, decoder=1):
    import torch
    cw = (0.299, 0.587, 0.114)
    b, e = ig.compress_image(torch.from_numpy(img).cuda(), level, decoder, cw, ig.WEIGHTS_ALPHA, with_errors=True)
    ob, oe = O.encode_image(img, level, decoder, cw, 1, None, True, True, nthreads=16)
    assert np.array_equal(b.cpu().numpy(), ob)
    assert np.array_equal(e.cpu().numpy().view(np.uint32), oe.view(np.uint32))


def contents(w, h, seed, noise=True):
    yield np.full((h, w, 4), 200, np.uint8)  # nothing to list
    if noise:  # everything listed: five colours a block, so that the oracle's search stays short
        img = np.random.default_rng(seed).integers(0, 5, (h, w, 1), dtype=np.uint8) * np.uint8(60)
        img = np.repeat(img, 4, 2)
        img[..., 3] = 255
        img[::4, ::4, :3], img[1::4, 1::4, :3] = 0, 240
        yield img
    yield synth.quality_sweep_image(w - 1, h - 2, seed=seed)


# Blocks an SM either side of the limits 96, 512 and 900, and the plan there by level.
SIZES = {"below 96": 95, "from 96": 97, "below 512": 510, "from 512": 514, "below 900": 898, "from 900": 902}


def expected(level, size):
    per_sm = SIZES[size]
    if per_sm < (96 if level >= 4 else 512):
        return 1, 4
    if level >= 4 and per_sm < {4: 512, 5: 512, 6: 900, 7: 900}.get(level, 0):
        return 1, 16 if level >= 6 and per_sm >= 512 else 8
    return 2, 4 if level < 4 else 8 if level < 6 or per_sm < 512 else 16


@pytest.mark.parametrize("size", sorted(SIZES))
@pytest.mark.parametrize("level", range(2, 10))
def test_sizes(gpu_lib, level, size):
    ig = gpu_lib
    sms = ig.load().icbc_gpu_sm_count()
    w, h = sides(sms * SIZES[size] + (15 if SIZES[size] % 2 else 0))
    assert ig.launch_plan(level, w, h, ig.WEIGHTS_ALPHA)[:2] == expected(level, size)
    large = SIZES[size] > 800
    for img in contents(w, h, level, noise=not large):
        check(ig, img, level)


@pytest.mark.parametrize("level", range(4, 10))
def test_four_warp_listed_pass(gpu_lib, level):
    """cta_warps 4 at levels 4-9: the warp-wide listed kernel, partial and whole rounds."""
    ig = gpu_lib
    sms = ig.load().icbc_gpu_sm_count()
    saved = ig.get_launch_config(level)
    try:
        ig.set_launch_config(level, 2, 0, 4)
        for per_sm in (97, 600):
            w, h = sides(sms * per_sm)
            assert ig.launch_plan(level, w, h, ig.WEIGHTS_ALPHA)[:2] == (2, 4)
            for img in contents(w, h, level + per_sm, noise=per_sm < 100):
                check(ig, img, level, decoder=2)
    finally:
        ig.set_launch_config(level, *saved)


@pytest.mark.parametrize("level", (0, 3, 5, 8, 9))
def test_launch_shapes_that_differ(gpu_lib, level):
    """Every launch shape the autotuner may pick, on an image large enough that they make different launches."""
    import torch
    ig = gpu_lib
    sms = ig.load().icbc_gpu_sm_count()
    w, h = sides(sms * 1100)
    img = torch.from_numpy(synth.quality_sweep_image(w - 3, h - 1, seed=4)).cuda()
    saved = ig.get_launch_config(level)
    plans = set()
    try:
        ref = ig.compress_image(img, level, 0, (1, 1, 1), ig.WEIGHTS_ALPHA)
        for g, p in ig.TUNE_CANDIDATES:
            for c in (ig.TUNE_CTA_WARPS if level >= 2 else (0,)):
                ig.set_launch_config(level, g, p, c)
                plans.add(ig.launch_plan(level, w - 3, h - 1, ig.WEIGHTS_ALPHA))
                assert torch.equal(ig.compress_image(img, level, 0, (1, 1, 1), ig.WEIGHTS_ALPHA), ref), (g, p, c)
    finally:
        ig.set_launch_config(level, *saved)
    assert len(plans) >= (8 if level >= 2 else 3), plans


def test_autotune_keeps_what_it_cannot_measure(gpu_lib):
    """On an image too small for a setting to reach its launch, autotune times it once and keeps the setting in force
    (the level's default CTA size)."""
    import torch
    ig = gpu_lib
    img = torch.from_numpy(synth.quality_sweep_image(320, 200, seed=4)).cuda()
    saved = {lv: ig.get_launch_config(lv) for lv in (3, 5, 8)}
    try:
        for lv, cta in ((3, 4), (5, 8), (8, 16)):
            ig.set_launch_config(lv, 3, 1, 0)
            t = ig.autotune(img, levels=(lv,), candidates=[(1, 0), (3, 1), (8, 0)], repeats=2)[lv]
            assert (t["groups_per_warp"], t["persistent"], t["cta_warps"]) == (3, 1, cta)
            assert len(set(t["candidates"].values())) == 1
            assert ig.get_launch_config(lv) == (3, 1, cta)
    finally:
        for lv, c in saved.items():
            ig.set_launch_config(lv, *c)
