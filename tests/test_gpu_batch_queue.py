"""GPU: the batched form's CTA-wide kernels draw tasks until a round has one
for every warp; tasks past the end of an image's list have nothing to do."""
import numpy as np
import pytest

from icbc_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", (2, 6, 8, 9))
def test_lists_empty_and_short(gpu_lib, level):
    """Images of which the first pass leaves nothing, one block or everything, in one queue: a round draws on past the
    tasks that have nothing left.  Against the oracle."""
    import torch
    ig = gpu_lib
    flat = np.full((4 * 60, 4 * 60, 4), 77, np.uint8)
    one = flat.copy()
    one[100:104, 40:44] = synth.hard_mixture_image(4, 4, seed=1)
    full = np.random.default_rng(level).integers(0, 256, (4 * 50, 4 * 51, 4), dtype=np.uint8)
    imgs = [flat, one, full, flat, flat, one, flat, full, flat, one, flat]
    keep, descs, outs = [], [], []
    for img in imgs:
        t = torch.from_numpy(img).cuda()
        n = ig.blocks_of(img.shape[1], img.shape[0])
        out, err = torch.zeros((n, 8), dtype=torch.uint8, device="cuda"), torch.zeros(n, device="cuda")
        descs.append(ig.image_desc(t, level, out, err, 0, (1, 1, 1), 0))
        keep += [t, out, err]
        outs.append((out, err))
    saved = ig.get_batch_cta_warps(level)
    try:
        for cta in (0, 4, 8, 16):
            ig.set_batch_cta_warps(level, cta)
            batch = ig.Batch(descs, keepalive=keep)
            for out, err in outs:
                out.zero_()
            batch.launch()
            torch.cuda.synchronize()
            for img, (out, err) in zip(imgs, outs):
                ob, oe = O.encode_image(img, level, 0, (1, 1, 1), 0, None, True, True, nthreads=16)
                assert np.array_equal(out.cpu().numpy(), ob)
                assert np.array_equal(err.cpu().numpy().view(np.uint32), oe.view(np.uint32))
            batch.close()
    finally:
        ig.set_batch_cta_warps(level, saved)
