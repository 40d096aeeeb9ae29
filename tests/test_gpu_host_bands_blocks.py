"""GPU: the host-buffer call cuts an image into bands by its number of blocks
(host_bands in bc1_shares.h), so low, wide images have bands too.  Images
either side of the rule's limits, ragged sides, every weight source, against
the device call (itself held to the oracle)."""
import numpy as np
import pytest

from icbc_gb300 import synth

pytestmark = pytest.mark.gpu


def wide(w, h, seed):
    """A tile of the mixture repeated (at an odd period, so that its blocks differ)."""
    return np.ascontiguousarray(np.tile(synth.hard_mixture_image(1001, h, seed=seed), (1, w // 1001 + 1, 1))[:, :w])


@pytest.mark.parametrize("level,thousands", ((0, (47, 49, 191, 520)), (3, (79, 81, 260, 700)), (4, (75, 79, 300, 400, 500)),
                                             (6, (75, 79, 300, 420)), (8, (95, 97, 250)), (9, (97, 330))))
def test_low_wide_images(gpu_lib, level, thousands):
    import torch
    ig = gpu_lib
    for k in thousands:
        bh = 40 + k % 7
        h, w = 4 * bh - 1, 4 * (k * 1024 // bh) - 3
        img = wide(w, h, seed=level + k)
        mode = (level + k) % 3
        plane = synth.uniform(3, k, (h, w)).astype(np.float32)
        kw = {"weight_plane": plane} if mode == 2 else {}
        dev = {"weight_plane": torch.from_numpy(plane).cuda()} if mode == 2 else {}
        errors = np.zeros(ig.blocks_of(w, h), np.float32)
        got = ig.compress_image_host(img, level, 1, (0.299, 0.587, 0.114), mode, errors=errors, **kw)
        out, err = ig.compress_image(torch.from_numpy(img).cuda(), level, 1, (0.299, 0.587, 0.114), mode,
                                     with_errors=True, **dev)
        assert np.array_equal(got, out.cpu().numpy())
        assert np.array_equal(errors.view(np.uint32), err.cpu().numpy().view(np.uint32))


def test_fewer_rows_than_bands(gpu_lib):
    """One or two block rows of a very wide image: no more bands than rows."""
    import torch
    ig = gpu_lib
    for level in (1, 6):
        for h in (3, 8):
            img = wide(4 * 150000, h, seed=level)
            got = ig.compress_image_host(img, level, 0, (1, 1, 1), 1)
            assert np.array_equal(got, ig.compress_image(torch.from_numpy(img).cuda(), level, 0, (1, 1, 1), 1).cpu().numpy())
