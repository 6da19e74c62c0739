"""The launch from an image's pixels to its FDCT caches (256 x 16 pixels a CTA) at the edges of its tiles, against the oracle's
encoder, and from device buffers of every alignment. Coefficients are integers: equal."""

import numpy as np
import pytest

import rcg
import rcg.synth as synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (3, 250), (5, 2), (255, 15), (256, 16), (257, 17), (249, 9), (513, 33), (1026, 24)])
@pytest.mark.parametrize("sub", [rcg.Subsampling.S420, rcg.Subsampling.S422, rcg.Subsampling.S444, None])
def test_coefficients_at_tile_edges(ctx, oracle, w, h, sub):
    img = synth.image(max(w, 8), max(h, 8), w + h, sensor_sigma=20.0)[:h, :w].copy()
    if sub is None:
        img, sub = img[:, :, 0].copy(), rcg.Subsampling.S420
    for trellis in (False, True):
        ci = ctx.build_coefs(img, rcg.EncodeOptions(90, sub, trellis))
        coefs, _, _ = oracle.build_coefs(img, 90, int(sub), trellis)
        assert np.array_equal(ci.flat(), coefs)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_device_images_of_any_alignment(ctx, channels, offset):
    import torch

    w, h = 261, 35  # the image's last bytes end a quad short of a word
    img = np.ascontiguousarray(synth.image(w, h, 9)[:, :, :channels])
    buf = torch.zeros(img.size + 8, dtype=torch.uint8, device="cuda")
    opts = rcg.EncodeOptions(90, rcg.Subsampling.S420, True)
    found = []
    for at in (0, offset):
        buf[at: at + img.size] = torch.from_numpy(img.ravel())
        out = torch.zeros(4 * w * h, dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        r = ctx.search_device(buf.data_ptr() + at, w, h, channels, 70.0, 100, opts, out.data_ptr(), out.numel())
        ctx.synchronize()
        found.append((r, out.cpu().numpy()))
    assert found[0][0] == found[1][0]
    assert np.array_equal(found[0][1], found[1][1])
