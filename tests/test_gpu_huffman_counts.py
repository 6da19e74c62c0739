"""Code lengths from counts that add up in 32 bits and from counts past 2^23 (added in 64), against the oracle's planner: the
baseline's size and every scan's cost follow from the lengths. Whole numbers: equal."""

import numpy as np
import pytest

import rcg

pytestmark = pytest.mark.gpu


# (0, 1) is by far the commonest AC symbol, about 62.9 in a block: 136900 blocks give 8.6 million (2^23 is 8.39 million).
@pytest.mark.parametrize("side", [8, 370])
def test_lengths_from_small_and_large_counts(ctx, oracle, side):
    rng = np.random.default_rng(side)
    n = side * side
    coefs = np.where(rng.random(n * 64) < 0.5, 1, -1).astype(np.int16)
    other = rng.random(n * 64) < 0.0015
    coefs[other] = rng.choice([0, 2, -3, 5, 17, -130, 900], int(other.sum()))
    ci = rcg.CoefImage(side * 8, side * 8, [rcg.CoefComponent(1, 1, 1, 0, side, side, coefs)], np.ones((2, 64), np.uint8))
    _, _, lay = oracle.build_coefs(np.zeros((side * 8, side * 8), np.uint8), 50, 3, False)
    got = ctx.plan(ci)
    progressive, baseline, best, distinct = oracle.plan(side * 8, side * 8, lay, coefs)
    assert got.baseline_bytes == baseline
    assert got.progressive_bytes == progressive
    assert list(got.distinct) == list(distinct)
    assert got.scans == best
