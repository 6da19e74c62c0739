"""The requantizer's symbol histogram decides its trellis: blocks of single coefficients at the edges of the groups of eight it
walks, runs of 15, 16, 17 and 48 zeros, a last coefficient at 63, the largest sizes and empty blocks, over one and several CTAs
of 128 blocks, against the oracle. Coefficients are integers: equal."""

import numpy as np
import pytest

import rcg

pytestmark = pytest.mark.gpu

_SPOTS = [[], [1], [7], [8], [15, 16], [16], [17], [1, 17], [1, 18], [1, 19], [63], [1, 63], [14, 62], [15, 32, 49],
          list(range(1, 64)), list(range(8, 64, 8))]


@pytest.mark.parametrize("blocks_w,blocks_h", [(1, 1), (16, 1), (127, 1), (43, 3), (64, 9)])
@pytest.mark.parametrize("largest", [3, 2047])
def test_histogram_edges(ctx, oracle, blocks_w, blocks_h, largest):
    rng = np.random.default_rng(blocks_w + largest)
    n, w, h = blocks_w * blocks_h, blocks_w * 8, blocks_h * 8
    coefs = np.zeros((n, 64), np.int16)
    for b in range(n):
        for k in _SPOTS[b % len(_SPOTS)]:
            coefs[b, k] = rng.integers(1, largest + 1) * rng.choice([-1, 1])
        coefs[b, 0] = rng.integers(-200, 200)
    coefs = coefs.ravel()
    q4 = np.zeros((4, 64), np.uint8)
    q4[0] = 2
    present = np.array([1, 0, 0, 0], np.uint8)
    ci = rcg.CoefImage(w, h, [rcg.CoefComponent(1, 1, 1, 0, blocks_w, blocks_h, coefs)], q4, present)
    _, _, lay = oracle.build_coefs(np.zeros((h, w), np.uint8), 50, 3, False)
    for quality in (10, 60, 90):
        got = ctx.requantize(ci, quality, True)
        want = oracle.requantize(oracle.GeneralCoefs(w, h, lay, [0], q4, present, coefs), quality, True)
        assert np.array_equal(got.flat(), want.coefs), quality
