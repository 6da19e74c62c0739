"""Block grids wider or taller than the MCU grid, not the same for both chroma components: a caller's layout may hold them
(jpeg/src/decode.rs:1345-1358 asks only that they cover the MCU grid), and the blocks outside change nothing. Every
sampling that the pyramid builder reads directly, widths that are and are not whole quads: a search over the padded image
visits the same qualities with the same scores, bit for bit, and its result holds the same coefficients."""

import numpy as np
import pytest

import rcg
import rcg.synth as synth

from test_gpu_requantize import _source, _to_oracle

pytestmark = pytest.mark.gpu


def _padded(c, dw, dh):
    """Component c with dw more columns and dh more rows of blocks, of coefficients that would show if they were read."""
    grid = np.full((c.blocks_h + dh, c.blocks_w + dw, 64), 100, np.int16)
    grid[: c.blocks_h, : c.blocks_w] = c.coefs.reshape(c.blocks_h, c.blocks_w, 64)
    return rcg.CoefComponent(c.id, c.h, c.v, c.tq, c.blocks_w + dw, c.blocks_h + dh, grid.reshape(-1))


@pytest.mark.parametrize("sub", [rcg.Subsampling.S444, rcg.Subsampling.S422, rcg.Subsampling.S420])
@pytest.mark.parametrize("w,h", [(96, 64), (203, 77)])
@pytest.mark.parametrize("pad", [((0, 0), (0, 0), (3, 0)), ((0, 0), (3, 2), (0, 0)), ((2, 1), (1, 0), (4, 3))])
def test_grids_of_different_widths_score_as_the_plain_ones(ctx, oracle, sub, w, h, pad):
    src, lay = _source(oracle, synth.image(w, h, 41, sensor_sigma=3.0), 95, sub)
    wide = rcg.CoefImage(src.width, src.height, [_padded(c, *p) for c, p in zip(src.comps, pad)], src.qtables,
                         src.present)
    want = ctx.find_quality_requantize(src, 70.0)
    got = ctx.find_quality_requantize(wide, 70.0)
    assert got.trace == want.trace and (got.quality, got.score) == (want.quality, want.score)
    for a, b in zip(got.coefs.comps, want.coefs.comps):
        inside = a.coefs.reshape(a.blocks_h, a.blocks_w, 64)[: b.blocks_h, : b.blocks_w]
        assert np.array_equal(inside.reshape(-1), b.coefs)
    q, s, _, trace = oracle.search_requantize(_to_oracle(oracle, src, lay), 70.0)
    assert want.quality == q and [t[0] for t in want.trace] == [t[0] for t in trace]
