"""GPU: a batch's task sizes and kernels follow its levels and block counts
(batch_shape in bc1_shares.h).  Batches on each side of the rule's limits --
with a weight-plane image, of one level, mixed -- give each image's own
launch's blocks and errors, which other tests hold to the oracle."""
import numpy as np
import pytest

from icbc_gb300 import synth

pytestmark = pytest.mark.gpu


def run(ig, images):
    """images: (array, level, decoder, colour weights, weight mode); the batch against compress_image, twice."""
    import torch
    keep, descs, want, got = [], [], [], []
    for img, level, dec, cw, mode in images:
        t = torch.from_numpy(img).cuda()
        kw = {}
        if mode == ig.WEIGHTS_PLANE:
            kw["weight_plane"] = torch.from_numpy(synth.uniform(level, 7, img.shape[:2]).astype(np.float32)).cuda()
        b, e = ig.compress_image(t, level, dec, cw, mode, with_errors=True, **kw)
        out, err = torch.zeros_like(b), torch.zeros_like(e)
        descs.append(ig.image_desc(t, level, out, err, dec, cw, mode, **kw))
        keep += [t, out, err, *kw.values()]
        want.append((b, e))
        got.append((out, err))
    batch = ig.Batch(descs, keepalive=keep)
    for _ in range(2):
        for out, err in got:
            out.zero_()
            err.zero_()
        batch.launch()
        torch.cuda.synchronize()
        for k, ((b, e), (out, err)) in enumerate(zip(want, got)):
            assert torch.equal(b, out), (k, images[k][1:])
            assert torch.equal(e.view(torch.int32), err.view(torch.int32)), (k, images[k][1:])
    batch.close()


def image(k, blocks):
    side = max(1, int(blocks ** 0.5))
    w, h = 4 * side - k % 3, 4 * max(1, blocks // side)
    return synth.hard_mixture_image(w, h, seed=k) if k % 2 else synth.quality_sweep_image(max(w, 4), max(h, 4), seed=k)


@pytest.mark.parametrize("level", (1, 3, 8, 9))
@pytest.mark.parametrize("total", (700, 20000, 46000, 59000))
def test_one_level_with_a_weight_plane(gpu_lib, level, total):
    """Float rows, 12 warps an SM: task sizes either side of what fits in a round."""
    ig = gpu_lib
    run(ig, [(image(k, total // 4 + 3 * k), level, k % 4, (0.299, 0.587, 0.114), ig.WEIGHTS_PLANE if k == 1 else k % 2)
             for k in range(4)])


@pytest.mark.parametrize("level", (2, 5, 6, 8, 9))
@pytest.mark.parametrize("total", (300, 5000, 20000, 80000))
def test_one_level(gpu_lib, level, total):
    ig = gpu_lib
    run(ig, [(image(k, total // 6 + 3 * k), level, k // 3, (1, 1, 1) if k < 4 else (0.299, 0.587, 0.114), k % 2)
             for k in range(6)])


@pytest.mark.parametrize("total", (600, 6000, 60000, 200000))
@pytest.mark.parametrize("levels", (range(10), range(3, 7), range(6, 10)))
@pytest.mark.parametrize("plane", (False, True))
def test_mixed_levels(gpu_lib, total, levels, plane):
    ig = gpu_lib
    levels = list(levels)
    run(ig, [(image(k, total // 20 + k), levels[k % len(levels)], k % 3, (1, 1, 1), ig.WEIGHTS_PLANE if plane and k == 5 else 1)
             for k in range(20)])
