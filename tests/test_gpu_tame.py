"""GPU: float rows at levels 8-9 take the bounded rows' fused arithmetic when a
warp's colours and weights lie in its domain (tame_colors in bc1_encode.cuh).
Values at and past the edges of that domain, alone and beside ordinary blocks
of the same warp, against the oracle, bit for bit."""
import numpy as np
import pytest

from icbc_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

EDGES = {
    "least colour": (2.0 ** -50, 1.0), "below it": (np.nextafter(np.float32(2.0 ** -50), np.float32(0)), 1.0),
    "denormal colour": (2.0 ** -140, 1.0), "greatest colour": (2.0, 1.0),
    "above it": (np.nextafter(np.float32(2.0), np.float32(3)), 1.0), "negative colour": (-0.25, 1.0),
    "least weight": (0.5, 2.0 ** -20), "weight below": (0.5, np.nextafter(np.float32(2.0 ** -20), np.float32(0))),
    "greatest weight": (0.5, 2.0 ** 10), "weight above": (0.5, np.nextafter(np.float32(2.0 ** 10), np.float32(1e9))),
    "tiny weight": (0.5, 2.0 ** -100), "zero": (0.0, 0.0),
}


@pytest.mark.parametrize("level", (8, 9))
@pytest.mark.parametrize("edge", sorted(EDGES))
@pytest.mark.parametrize("alone", (False, True))
def test_edges(gpu_lib, level, edge, alone):
    value, weight = EDGES[edge]
    cols, w = synth.mixed_blocks(192, seed=5)
    cols, w = cols.copy(), w.copy()
    some = slice(None) if alone else slice(3, None, 40)  # every block of the warps, or one or two of a warp
    cols[some, 2:13:5, 1] = value
    cols[some, 7, :3] = value
    w[some, 1:16:4] = weight
    for dec, tc in ((0, True), (2, True), (3, False)):
        b, e = gpu_lib.compress_blocks(cols, w, level, dec, (0.299, 0.587, 0.114), tc, True)
        ob, oe = O.compress_blocks(cols, w, level, dec, (0.299, 0.587, 0.114), tc, True)
        assert np.array_equal(b, ob) and np.array_equal(e.view(np.uint32), oe.view(np.uint32))


def test_products_at_the_edge(gpu_lib):
    """Every colour and weight at the least of the domain, and at the greatest."""
    rng = np.random.default_rng(1)
    for lo, hi, wlo, whi in ((2.0 ** -50, 2.0 ** -44, 2.0 ** -20, 2.0 ** -18), (1.5, 2.0, 2.0 ** 9, 2.0 ** 10)):
        cols = rng.uniform(lo, hi, (512, 16, 4)).astype(np.float32)
        w = rng.uniform(wlo, whi, (512, 16)).astype(np.float32)
        b, e = gpu_lib.compress_blocks(cols, w, 8, 0, (1, 1, 1), True, True)
        ob, oe = O.compress_blocks(cols, w, 8, 0, (1, 1, 1), True, True)
        assert np.array_equal(b, ob) and np.array_equal(e.view(np.uint32), oe.view(np.uint32))
