"""GPU: at levels 8-9 the first pass over RGBA8 images tells blocks of one
colour by their bytes.  Every byte value as a single-colour block under
varied weights (some texels without any), the same with one texel one step
away in one channel, and blocks without weight, against the oracle, bit for
bit, through the two-pass image call and a batch."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def blocks_image(seed):
    """256 x 80 blocks: column = byte value, row = kind."""
    rng = np.random.default_rng(seed)
    bh, bw = 80, 256
    img = np.zeros((bh, 4, bw, 4, 4), np.uint8)
    v = np.arange(256)
    colour = np.stack([v, v[::-1], rng.permutation(256)], -1).astype(np.uint8)
    img[..., :3] = colour[None, None, :, None, :]
    alpha = rng.integers(0, 256, (bh, 4, bw, 4))
    alpha[rng.random(alpha.shape) < 0.3] = 0
    alpha[::7] = rng.integers(0, 2, alpha[::7].shape)  # the least weights
    alpha[5::11] = 0
    img[..., 3] = alpha
    for row in range(40, 80):  # one texel one step away
        y, x, c = row % 4, (row // 4) % 4, row % 3
        t = img[row, y, :, x, c].astype(int)
        img[row, y, :, x, c] = np.where(t < 255, t + 1, t - 1)
    return img.reshape(4 * bh, 4 * bw, 4)


@pytest.mark.parametrize("level", (8, 9))
@pytest.mark.parametrize("mode", (0, 1))
def test_bytes_decide(gpu_lib, level, mode):
    import torch
    ig = gpu_lib
    img = blocks_image(level + mode)
    ob, oe = O.encode_image(img, level, 0, (0.299, 0.587, 0.114), mode, None, True, True, nthreads=16)
    t = torch.from_numpy(img).cuda()
    b, e = ig.compress_image(t, level, 0, (0.299, 0.587, 0.114), mode, with_errors=True)
    assert np.array_equal(b.cpu().numpy(), ob)
    assert np.array_equal(e.cpu().numpy().view(np.uint32), oe.view(np.uint32))
    out, err = torch.zeros_like(b), torch.zeros_like(e)
    batch = ig.Batch([ig.image_desc(t, level, out, err, 0, (0.299, 0.587, 0.114), mode)], keepalive=(t, out, err))
    batch.launch()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), ob)
    assert np.array_equal(err.cpu().numpy().view(np.uint32), oe.view(np.uint32))
    batch.close()
