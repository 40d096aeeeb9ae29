"""GPU: the number of blocks a warp or CTA takes follows the size of the work
(balanced_share in bc1_level.cu).  Sizes at its edges -- one block, one block
more or less than a round of the resident warps, a round and a second nearly
empty one -- must give the oracle's blocks and errors, bit for bit."""
import numpy as np
import pytest

from icbc_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# Blocks per side pair: 1, 31-33, 608 = 152 x 4, one round of 152 x 12 and 152 x 16 warps and one more,
# and just over 32 blocks for each of 152 x 12 (float rows) and 152 x 16 (byte rows) warps.
SHAPES = ((1, 1), (31, 1), (33, 1), (19, 32), (48, 38), (32, 76), (35, 70), (243, 241), (280, 278))


def check(ig, img, level, mode, plane):
    import torch
    t = torch.from_numpy(img).cuda()
    kw = {"weight_plane": torch.from_numpy(plane).cuda()} if mode == ig.WEIGHTS_PLANE else {}
    b, e = ig.compress_image(t, level, 2, (0.299, 0.587, 0.114), mode, with_errors=True, **kw)
    ob, oe = O.encode_image(img, level, 2, (0.299, 0.587, 0.114), mode, plane, True, True, nthreads=16)
    assert np.array_equal(b.cpu().numpy(), ob)
    assert np.array_equal(e.cpu().numpy().view(np.uint32), oe.view(np.uint32))


@pytest.mark.parametrize("level", (2, 5, 8, 9))
@pytest.mark.parametrize("bw,bh", SHAPES)
def test_image_sizes(gpu_lib, level, bw, bh):
    img = synth.hard_mixture_image(4 * bw - bw % 3, 4 * bh, seed=bw * 7 + level)
    plane = synth.uniform(9, level, img.shape[:2]).astype(np.float32)
    for mode in (0, 1, 2):
        check(gpu_lib, img, level, mode, plane if mode == 2 else None)


@pytest.mark.parametrize("level", (3, 8, 9))
@pytest.mark.parametrize("n", (1, 5, 1823, 1825, 3649, 58369))
def test_block_counts(gpu_lib, level, n):
    cols, w = synth.mixed_blocks(n, seed=n + level)
    b, e = gpu_lib.compress_blocks(cols, w, level, 1, (1, 1, 1), True, True)
    ob, oe = O.compress_blocks(cols, w, level, 1, (1, 1, 1), True, True, nthreads=16)
    assert np.array_equal(b, ob) and np.array_equal(e.view(np.uint32), oe.view(np.uint32))


@pytest.mark.parametrize("level", (4, 8, 9))
@pytest.mark.parametrize("bh", (305, 608, 610))
def test_cta_rounds(gpu_lib, level, bh):
    """Images of the 16-warp CTAs: the listed blocks just under and over whole rounds of 152 x 512."""
    img = synth.quality_sweep_image(4 * 512, 4 * bh, seed=bh)
    check(gpu_lib, img, level, 1, None)


@pytest.mark.parametrize("level", (3, 4, 6, 8, 9))
@pytest.mark.parametrize("bw,bh", ((14591, 1), (96, 152), (305, 255), (304, 256), (303, 452), (300, 456)))
def test_cta_sizes(gpu_lib, level, bw, bh):
    """Either side of 96 blocks an SM (8-warp CTAs from there), of 512 (16-warp ones, and at levels 2-5 a list of the
    blocks to search) and of 900 (the list at levels 6-7)."""
    check(gpu_lib, synth.hard_mixture_image(4 * bw, 4 * bh, seed=bw + level), level, 1, None)


@pytest.mark.parametrize("n,decoders", ((1, (0, 1, 2, 3)), (700, (0, 1, 2, 3)), (8191, (1,)), (8193, (2,)),
                                        (98303, (1,)), (98305, (0,))))
def test_refinement_counts(gpu_lib, n, decoders):
    """32 lanes a block below 8,192 blocks, 8 below 98,304, 4 from there on."""
    cols, w = synth.mixed_blocks(n, seed=n)
    for dec in decoders:
        for tc, tcb in ((True, True), (False, False)):
            b, e = gpu_lib.compress_blocks(cols, w, 9, dec, (0.299, 0.587, 0.114), tc, tcb)
            ob, oe = O.compress_blocks(cols, w, 9, dec, (0.299, 0.587, 0.114), tc, tcb, nthreads=16)
            assert np.array_equal(b, ob) and np.array_equal(e.view(np.uint32), oe.view(np.uint32))


@pytest.mark.parametrize("sides", ((4, 9, 1), (40, 64, 33, 8), (300, 500, 260, 410, 77)))
def test_small_batches(gpu_lib, sides):
    """Batches below 32 blocks for every warp take smaller tasks: some past a list's end, ragged images, mixed
    levels, decoders and colour weights in one CTA's round."""
    import torch
    ig = gpu_lib
    keep, descs, cases = [], [], []
    for k, side in enumerate(sides):
        for level in range(10):
            img = synth.quality_sweep_image(side + level, side, seed=k) if side >= 33 else synth.hard_mixture_image(
                side + level, side, seed=k)
            t, n = torch.from_numpy(img).cuda(), ig.blocks_of(side + level, side)
            out, err = torch.zeros((n, 8), dtype=torch.uint8, device="cuda"), torch.zeros(n, device="cuda")
            cw = (1.0, 1.0, 1.0) if level % 2 else (0.299, 0.587, 0.114)
            keep += [t, out, err]
            descs.append(ig.image_desc(t, level, out, err, (k + level) % 4, cw, level % 2))
            cases.append((img, level, (k + level) % 4, cw, level % 2, out, err))
    b = ig.Batch(descs, keepalive=keep)
    b.launch()
    torch.cuda.synchronize()
    for img, level, dec, cw, mode, out, err in cases:
        ob, oe = O.encode_image(img, level, dec, cw, mode, None, True, True, nthreads=16)
        assert np.array_equal(out.cpu().numpy(), ob), (img.shape, level)
        assert np.array_equal(err.cpu().numpy().view(np.uint32), oe.view(np.uint32))
    b.close()
