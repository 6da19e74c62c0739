"""Requantization of coefficients at the ends of 16 bits, where the source's table entry is 255 and so stays: -32768 is a
value of 16 bits, one more than any other, and the trellis prices it with the same rate model (jpeg/src/rdo.rs:47-52). Equal
to the oracle's, coefficient for coefficient."""

import numpy as np
import pytest

import rcg
import rcg.synth as synth

from test_gpu_requantize import _check, _source

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.02, 0.2, 0.9])
@pytest.mark.parametrize("gray", [False, True])
def test_16_bit_values_match_the_oracle(ctx, oracle, share, gray):
    img = synth.image(131, 90, 61, sensor_sigma=2.0)
    src, lay = _source(oracle, np.ascontiguousarray(img[:, :, 0]) if gray else img, 90, rcg.Subsampling.S444)
    rng = np.random.default_rng(62)
    # A table of two kinds of entries: 255, never raised, and 1, raised by every quality asked for.
    table = np.where(rng.random(64) < 0.5, 255, 1).astype(np.uint8)
    comps = []
    for c in src.comps:
        a = rng.integers(-40, 41, c.coefs.size).astype(np.int16)
        ends = rng.random(a.size) < share
        a[ends] = rng.choice(np.array([-32768, -32767, 32767, -16384, 16384], np.int16), int(ends.sum()))
        comps.append(rcg.CoefComponent(c.id, c.h, c.v, 0, c.blocks_w, c.blocks_h, a))
    q4 = np.zeros((4, 64), np.uint8)
    q4[0] = table
    ends_src = rcg.CoefImage(src.width, src.height, comps, q4, np.array([1, 0, 0, 0], np.uint8))
    for q in (20, 75, 95):
        _check(ctx, oracle, ends_src, lay, q, True)
