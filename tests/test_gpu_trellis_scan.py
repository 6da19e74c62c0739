"""The trellis's bounded scan over earlier nodes against the oracle's full scan: equal coefficients.

The kernel scans a position's predecessors from the newest and stops at a bound. These inputs are the ones where the
scan is long, where costs tie and where the bound does not hold: blocks with every coefficient a candidate, sparse
blocks with long runs (zero-run codes), few distinct values (equal costs), and caller weights that are negative, zero
or NaN (a cost relative to dropping everything may then rise again).
"""

import numpy as np
import pytest

import rcg

pytestmark = pytest.mark.gpu

W, H = 136, 104


def _image(kind, channels=3):
    rng = np.random.default_rng(11)
    if kind == "dense":
        img = rng.integers(0, 256, (H, W, channels))
    elif kind == "two_values":
        img = 255 * rng.integers(0, 2, (H, W, channels))
    elif kind == "sparse":  # one bright pixel per block: coefficients of similar size over the whole block
        img = np.full((H, W, channels), 90)
        for by in range(0, H, 8):
            for bx in range(0, W, 8):
                img[by + rng.integers(8), bx + rng.integers(8)] += rng.integers(10, 160)
    else:  # "stripes": equal blocks, equal costs
        img = np.where((np.arange(W) // 3 % 2 == 0)[None, :, None], 60, 190) * np.ones((H, W, channels))
    return np.clip(img, 0, 255).astype(np.uint8)


@pytest.mark.parametrize("kind", ["dense", "two_values", "sparse", "stripes"])
@pytest.mark.parametrize("q", [2, 40, 75, 92, 99])
def test_plain_trellis(ctx, oracle, kind, q):
    img = _image(kind)
    got = ctx.build_coefs(img, rcg.EncodeOptions(q, rcg.Subsampling.S444, True)).flat()
    want, _, _ = oracle.build_coefs(img, q, int(rcg.Subsampling.S444), True)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("kind", ["dense", "sparse"])
@pytest.mark.parametrize("q", [30, 80])
def test_requantized(ctx, oracle, kind, q):
    img = _image(kind)
    coefs, qt, lay = oracle.build_coefs(img, 95, int(rcg.Subsampling.S420), True)
    g = oracle.general_from_encoder(W, H, lay, qt, coefs)
    src = ctx.decode_coefs(oracle.write_jpeg_variant(g, 0, False))
    want = oracle.requantize(g, q)
    assert np.array_equal(ctx.requantize(src, q).flat(), want.coefs)


@pytest.mark.parametrize("kind", ["dense", "two_values", "sparse"])
@pytest.mark.parametrize("weights", ["zero", "tiny", "signs", "nan"])
def test_caller_weights(ctx, oracle, kind, weights):
    img = _image(kind)
    rng = np.random.default_rng(12)
    n = oracle.build_coefs(img, 60, int(rcg.Subsampling.S444), True)[0].size
    w = rng.uniform(0.1, 3.0, n).astype(np.float32)
    if weights == "zero":
        w[rng.random(n) < 0.5] = 0.0
    elif weights == "tiny":
        w[rng.random(n) < 0.5] = 1e-30
    elif weights == "signs":
        w[rng.random(n) < 0.05] *= -1
    else:
        w[rng.random(n) < 0.002] = np.nan
    got = ctx.build_coefs_weighted(img, rcg.EncodeOptions(60, rcg.Subsampling.S444, True), w).flat()
    want, _, _ = oracle.build_coefs(img, 60, int(rcg.Subsampling.S444), True, weights=w)
    assert np.array_equal(got, want)
