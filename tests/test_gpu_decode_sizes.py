"""GPU: decode and evaluate move texels a block row per lane, 32 blocks a warp.
Block counts at and around whole warps and CTAs, random bytes as blocks (both
palette orders, every index), against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (1, 7, 8, 31, 32, 33, 255, 256, 257, 1000))
def test_decode_and_evaluate(gpu_lib, n):
    import torch
    rng = np.random.default_rng(n)
    blocks = rng.integers(0, 256, (n, 8), dtype=np.uint8)
    blocks[:: 3, :4] = 0  # equal endpoints
    texels = rng.integers(0, 256, (n, 64), dtype=np.uint8)
    texels[0], blocks[0] = 255, 0  # the largest error: 16 texels of 3 * 255^2
    b, t = torch.from_numpy(blocks).cuda(), torch.from_numpy(texels).cuda()
    for dec in range(4):
        assert np.array_equal(gpu_lib.decode_blocks(b, dec).cpu().numpy(), O.decode_bc1(blocks, dec).reshape(n, 64))
        e = gpu_lib.evaluate_errors(t, b, dec).cpu().numpy()
        assert np.array_equal(e.view(np.uint32), O.evaluate_bc1_error(texels, blocks, dec).view(np.uint32))
        b3 = np.concatenate([rng.integers(0, 256, (n, 8), dtype=np.uint8), blocks], 1)
        got = gpu_lib.decode_bc3_blocks(torch.from_numpy(b3).cuda(), dec).cpu().numpy()
        assert np.array_equal(got, O.decode_bc3(b3, dec).reshape(n, 64))
