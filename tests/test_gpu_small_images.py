"""Small images take forms of their own in the scorer: a launch of few bands scores one channel per CTA, and an image of few
64x64 blocks is built by 32x32 blocks. Neither changes a sample or a sum, so a score has the same bits as in a work-list
large enough to take the forms of large images."""

import numpy as np
import pytest

import rcg.synth as synth

pytestmark = pytest.mark.gpu


def _pair(w, h, gray, seed):
    ref = synth.image(max(w, 8), max(h, 8), seed, sensor_sigma=4.0)[:h, :w].copy()
    if gray:
        ref = ref[:, :, 1].copy()
    noise = np.random.default_rng(seed).integers(-12, 13, ref.shape)
    return ref, np.clip(ref.astype(int) + noise, 0, 255).astype(np.uint8)


# Single samples and pairs at the last scales; one 32 block and its neighbours; 152 blocks of 64 and one more; 1024 bands
# (768 + 192 + 48 + 12 + 3 + 1) and a few more.
@pytest.mark.parametrize("w,h", [(8, 8), (9, 31), (32, 32), (33, 65), (64, 64), (65, 31), (97, 161), (240, 180), (512, 512),
                                 (1216, 512), (1217, 512), (1024, 768), (1030, 769)])
@pytest.mark.parametrize("gray", [False, True])
def test_small_forms_give_the_same_bits(ctx, w, h, gray):
    ref, dist = _pair(w, h, gray, w + h)
    filler = _pair(1600, 1200, False, 5)
    want = ctx.ssimulacra2_batch([(ref, dist), filler])[0]
    assert ctx.ssimulacra2(ref, dist) == want
    # a work-list of few bands, gray images among those of three channels
    small = _pair(40, 40, not gray, 6)
    assert ctx.ssimulacra2_batch([(ref, dist), small])[0] == want
