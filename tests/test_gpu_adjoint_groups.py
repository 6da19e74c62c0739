"""The gradient where the moments of all planes do not fit: the planes go through the blurs in groups, blurred again for the
backward pass, down to one plane at a time, and the result is the same bits. The workspace is limited more and more."""

import ctypes

import numpy as np
import pytest

import rcg
import rcg.synth as synth

pytestmark = pytest.mark.gpu


def _limit(c, bytes_):
    f = rcg._lib.rcg_internal_limit_workspace
    f.restype, f.argtypes = None, [ctypes.c_void_p, ctypes.c_uint64]
    f(c._ptr, int(bytes_))


def _shrink(call, want, most):
    """The least limit, in steps of 3%, that `call` succeeds under, where its result is `want`."""
    limit, least = most, None
    while True:
        with rcg.Context(0) as c:
            _limit(c, limit)
            try:
                got = call(c)
            except rcg.RcgError as e:
                assert e.status == rcg.RCG_NO_MEMORY
                return least
            for a, b in zip(got, want):
                assert np.array_equal(a, b)
        least, limit = limit, int(limit * 0.97)


# Images are copied to buffers of 39 bytes a pixel (both images, the gradient); small buffers come to less than 1 MB.
SLACK = 1 << 20


@pytest.mark.parametrize("w,h", [(640, 480), (387, 521)])
def test_gradient_fp64(w, h):
    img = synth.image(w, h, 91, sensor_sigma=2.0)
    dist = np.clip(img.astype(np.float32) + np.random.default_rng(92).normal(0, 4, img.shape).astype(np.float32), 0, 255)
    with rcg.Context(0) as c:
        want = c.ssimulacra2_grad(img, dist)
    least = _shrink(lambda c: c.ssimulacra2_grad(img, dist), want, w * h * 600 + SLACK)
    # One launch per plane needed 37 planes of doubles; one group needs 64 of them.
    assert least is not None and least <= w * h * (39 + 37 * 8) + SLACK, least / (w * h)


def test_weights_fp32():
    w, h = 640, 480
    opts = rcg.EncodeOptions(60, rcg.Subsampling.S420, True)
    img = synth.image(w, h, 93, sensor_sigma=2.0)
    with rcg.Context(0) as c:
        dec = c.reconstruct(c.build_coefs(img, opts))
        lay = c.coef_layout(w, h, 3, opts)
        want = c.perceptual_weights(img, dec, lay)
    least = _shrink(lambda c: c.perceptual_weights(img, dec, lay), want, w * h * 400 + SLACK)
    # Beside the pass: the images (6 bytes a pixel), the distorted one and the gradient (36), weights (6), block energies.
    assert least is not None and least <= w * h * (50 + 37 * 4) + SLACK, least / (w * h)
