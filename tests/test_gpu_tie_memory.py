"""A near tie needs no memory beyond the exact scorer's own: its pyramids of both images and its working planes. The
workspace is limited to what a search without ties needs and that, for whole quads of columns and odd widths, gray and in
colour, and the tied search then gives the result it gives without a limit."""

import ctypes
import math

import numpy as np
import pytest

import rcg
import rcg.synth as synth

pytestmark = pytest.mark.gpu


def _limited(bytes_, band, img):
    f = rcg._lib.rcg_internal_limit_workspace
    f.restype, f.argtypes = None, [ctypes.c_void_p, ctypes.c_uint64]
    with rcg.Context(0) as c:
        f(c._ptr, int(bytes_))
        c.set_tie_band(band)
        try:
            return c.find_quality_ssimulacra2(img, 60.0, 100, rcg.EncodeOptions(90, rcg.Subsampling.S420, True))
        except rcg.RcgError as e:
            assert e.status == rcg.RCG_NO_MEMORY
            return None


@pytest.mark.parametrize("w,h", [(640, 480), (643, 477)])
@pytest.mark.parametrize("gray", [False, True])
def test_tied_search_fits(w, h, gray):
    img = synth.image(w, h, 95, sensor_sigma=2.0)
    if gray:
        img = np.ascontiguousarray(img[:, :, 1])
    lo, hi = 0, 1 << 30
    while hi - lo > 1 << 17:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if _limited(mid, 0.0, img) else (mid, hi)
    # XYB of both images, five blurred quantities and 18 maps in doubles; four levels of two pyramids in floats (8 B/px).
    exact = w * h * ((11 + 18) * 8 + 8.3) + (1 << 20)
    want, got = _limited(0, math.inf, img), _limited(hi + exact, math.inf, img)
    assert got is not None
    assert got.trace == want.trace and np.array_equal(got.coefs.flat(), want.coefs.flat())
