"""Near ties of a lockstep batch, the last candidate's among them: with every candidate a tie (band infinity), each image's
result is that of its own search, which reports every candidate's exact score."""

import math

import numpy as np
import pytest

import rcg
import rcg.synth as synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_q", [1, 2, 60, 100])
def test_every_tie_is_decided_and_reported(max_q):
    opts = rcg.EncodeOptions(90, rcg.Subsampling.S420, True)
    images = [synth.image(64, 48, 71), synth.image(131, 67, 72, sensor_sigma=3.0), synth.image(200, 96, 73)[:, :, 0].copy()]
    with rcg.Context(0) as c:
        c.set_tie_band(math.inf)
        for targets in ([-50.0, 20.0, 60.0], [60.0, 75.0, 85.0]):
            want = [c.find_quality_ssimulacra2(im, t, max_q, opts) for im, t in zip(images, targets)]
            for _ in range(2):  # the second time from a stored graph or its capture
                got = c.search_batch(images, targets, max_q, opts, lockstep=True)
                for a, b in zip(got, want):
                    assert a.trace == b.trace and (a.quality, a.score) == (b.quality, b.score)
                    assert np.array_equal(a.coefs.flat(), b.coefs.flat())
