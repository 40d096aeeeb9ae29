"""GPU: levels 2-4 rebuild the sums of a block's colours without the black
ones at the width that the warp needs: blocks of up to 4, 8 and 12 colours of
which some are near black, through the small-image, listed and batch kernels,
against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", (2, 3, 4))
@pytest.mark.parametrize("dark", (3, 7, 11))
def test_rebuild_without_black(gpu_lib, level, dark):
    import torch
    ig = gpu_lib
    rng = np.random.default_rng(level * 100 + dark)
    sms = ig.load().icbc_gpu_sm_count()
    for per_sm in (20, 520):
        bw = int((sms * per_sm) ** 0.5)
        w, h = 4 * bw, 4 * (sms * per_sm // bw)
        colours = rng.integers(0, 256, (h // 4, w // 4, dark + 1, 3), dtype=np.uint8)
        colours[:, :, : 1 + dark // 3] = rng.integers(0, 31, (h // 4, w // 4, 1 + dark // 3, 3), dtype=np.uint8)
        pick = rng.integers(0, dark + 1, (h // 4, w // 4, 16))
        tex = np.take_along_axis(colours, pick[..., None], 2).reshape(h // 4, w // 4, 4, 4, 3)
        img = np.full((h // 4, 4, w // 4, 4, 4), 255, np.uint8)
        img[..., :3] = tex.transpose(0, 2, 1, 3, 4)
        img = img.reshape(h, w, 4)
        t = torch.from_numpy(img).cuda()
        ref, err = ig.compress_image(t, level, 0, (1, 1, 1), 0, with_errors=True)
        ob, oe = O.encode_image(img, level, 0, (1, 1, 1), 0, None, True, True, nthreads=16)
        assert np.array_equal(ref.cpu().numpy(), ob)
        assert np.array_equal(err.cpu().numpy().view(np.uint32), oe.view(np.uint32))
        out = torch.zeros_like(ref)
        b = ig.Batch([ig.image_desc(t, level, out, None, 0, (1, 1, 1), 0)], keepalive=(t, out))
        b.launch()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
        b.close()
