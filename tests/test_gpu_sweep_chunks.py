"""A sweep encodes an image's candidates together, as many at a time as its coefficient buffer (512 MB) holds: scores equal those
of one-quality sweeps, below, at and past the edge of a chunk, in layouts of different size."""

import numpy as np
import pytest

import rcg
import rcg.synth as synth

pytestmark = pytest.mark.gpu


# 12 MP candidates have 36 MB (4:2:0) or 72 MB (4:4:4) of coefficients: 14 or 7 at a time; 17x33 fit in any number.
@pytest.mark.parametrize("w,h,sub,qs", [(17, 33, rcg.Subsampling.Auto, [1, 100]), (4000, 3000, rcg.Subsampling.S444, [30, 50, 95, 60, 80, 70, 90]),
                                        (4000, 3000, rcg.Subsampling.Auto, [20, 95, 40, 91, 60, 89, 80, 90, 50])])
def test_chunks_of_candidates(ctx, w, h, sub, qs):
    img = np.tile(synth.image(512, 384, 75, sensor_sigma=3.0), (h // 384 + 1, w // 512 + 1, 1))[:h, :w].copy()
    opts = rcg.EncodeOptions(90, sub, True)
    got = ctx.sweep_qualities([img], qs, opts)[0]
    for k, q in enumerate(qs):
        assert got[k] == ctx.sweep_qualities([img], [q], opts)[0, 0], q
