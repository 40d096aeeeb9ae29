"""GPU: the bounded arithmetic of float rows at levels 8-9 (tame_colors in
bc1_encode.cuh) on blocks whose search really runs with the least and the
greatest products of its domain, against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

WEIGHTS = {"least": (2.0 ** -20, 2.0 ** -18), "greatest": (2.0 ** 9, 2.0 ** 10), "both": None}


@pytest.mark.parametrize("level", (8, 9))
@pytest.mark.parametrize("weights", sorted(WEIGHTS))
@pytest.mark.parametrize("small", (0, 1, 2))
def test_products(gpu_lib, level, weights, small):
    """One channel keeps the colours apart, the other two lie at the least of the domain (and once one at 0)."""
    rng = np.random.default_rng(level * 10 + small)
    n = 512
    cols = rng.uniform(2.0 ** -50, 2.0 ** -44, (n, 16, 4)).astype(np.float32)
    steps = rng.integers(2, 17, n)
    apart = (small + 1) % 3
    cols[:, :, apart] = rng.integers(0, 1 << 20, (n, 16)) % steps[:, None] / np.float32(16)
    cols[::5, :, apart] *= 2.0
    cols[::7, :, small] = 0.0
    if WEIGHTS[weights]:
        w = rng.uniform(*WEIGHTS[weights], (n, 16)).astype(np.float32)
    else:  # prefix sums that round the least weights away
        w = np.where(rng.random((n, 16)) < 0.5, 2.0 ** -20, 2.0 ** 10).astype(np.float32)
    kept = np.array([len(np.unique(c)) for c in cols[:, :, apart]])  # apart by 1/16 at least: none of them merge
    assert (kept >= 2).mean() > 0.95 and kept.max() > 8
    for dec, cw, tc in ((0, (1, 1, 1), True), (2, (0.299, 0.587, 0.114), True), (1, (1, 1, 1), False)):
        b, e = gpu_lib.compress_blocks(cols, w, level, dec, cw, tc, True)
        ob, oe = O.compress_blocks(cols, w, level, dec, cw, tc, True, nthreads=16)
        assert np.array_equal(b, ob) and np.array_equal(e.view(np.uint32), oe.view(np.uint32))
