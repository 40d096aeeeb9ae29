"""GPU: the host-buffer call cuts an image into bands of whole block rows by
level and height.  Heights either side of each band count, ragged sides and
every weight source, against the device call (itself held to the oracle)."""
import numpy as np
import pytest

from icbc_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,rows", ((1, 128), (4, 200), (6, 128), (8, 170), (9, 170)))
@pytest.mark.parametrize("bands", (1, 2, 3))
@pytest.mark.parametrize("extra", (-1, 0, 3))
def test_bands(gpu_lib, level, rows, bands, extra):
    import torch
    ig = gpu_lib
    h, w = 4 * rows * bands + extra, 4 * 37 - bands
    img = synth.hard_mixture_image(w, h, seed=level + bands)
    plane = synth.uniform(3, bands, (h, w)).astype(np.float32)
    for mode in (0, 1, 2):
        kw = {"weight_plane": plane} if mode == 2 else {}
        dev = {"weight_plane": torch.from_numpy(plane).cuda()} if mode == 2 else {}
        errors = np.zeros(ig.blocks_of(w, h), np.float32)
        got = ig.compress_image_host(img, level, 1, (0.299, 0.587, 0.114), mode, errors=errors, **kw)
        out, err = ig.compress_image(torch.from_numpy(img).cuda(), level, 1, (0.299, 0.587, 0.114), mode,
                                     with_errors=True, **dev)
        assert np.array_equal(got, out.cpu().numpy())
        assert np.array_equal(errors.view(np.uint32), err.cpu().numpy().view(np.uint32))


def test_overlapped_rounds(gpu_lib):
    """Bands of more than a round of 16-warp CTAs each, evenly shared or not."""
    import torch
    ig = gpu_lib
    img = synth.quality_sweep_image(2048, 4 * 1024, seed=2)
    for level in (6, 8):
        got = ig.compress_image_host(img, level, 0, (1, 1, 1), 1)
        out = ig.compress_image(torch.from_numpy(img).cuda(), level, 0, (1, 1, 1), 1)
        assert np.array_equal(got, out.cpu().numpy())
