"""The pyramid builder: every source it reads gives the same samples, at the edges of its 64x64 blocks too.

A search scores candidates from their decoded planes; the single scorer reads interleaved pixels (of any alignment), a
batch builds a shared reference apart from its pairs. The linear samples are the same in all of them, so the scores must
be the same bits, and the oracle's within the scorer's 1e-4 on small images. Sizes lie around the block and level edges
(64, 32, 16 samples), at the smallest images of one scale and at widths that are no multiple of four.
"""

import ctypes

import numpy as np
import pytest

import rcg
import rcg.synth as synth

pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (15, 9), (16, 16), (17, 33), (63, 65), (64, 64), (66, 127), (129, 67), (191, 130), (258, 31)]
S = rcg.Subsampling


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("sub,gray", [(S.S420, False), (S.S422, False), (S.S444, False), (S.S420, True)])
def test_candidates_from_planes_and_from_pixels(ctx, oracle, w, h, sub, gray):
    img = synth.image(max(w, 16), max(h, 16), 50, 4.0)[:h, :w]
    img = np.ascontiguousarray(img[:, :, 1] if gray else img)
    f = ctx.find_quality_ssimulacra2(img, 60.0, 100, rcg.EncodeOptions(90, sub, True))
    for q, score in f.trace:
        rec = ctx.reconstruct(ctx.build_coefs(img, rcg.EncodeOptions(q, sub, True)))
        s = ctx.ssimulacra2(img, rec)
        assert s == score, (q, s, score)
        assert abs(s - oracle.ssimulacra2(img, rec)) <= 1e-4
    # the same pairs through the batch: one reference shared by all, and one with a reference of its own
    recs = [ctx.reconstruct(ctx.build_coefs(img, rcg.EncodeOptions(q, sub, True))) for q, _ in f.trace]
    own = img.copy()
    b = ctx.ssimulacra2_batch([(img, r) for r in recs] + [(own, recs[0])])
    assert list(b) == [s for _, s in f.trace] + [f.trace[0][1]]


@pytest.mark.parametrize("w,h", [(8, 8), (61, 40), (64, 65), (130, 70)])
def test_images_at_any_alignment(ctx, w, h):
    """Device images that start 0..3 bytes past a word: the same score."""
    import torch

    ref = synth.image(max(w, 16), max(h, 16), 51, 2.0)[:h, :w].copy()
    dist = synth.image(max(w, 16), max(h, 16), 51, 7.0)[:h, :w].copy()
    want = ctx.ssimulacra2(ref, dist)
    n = ref.size
    for a in range(4):
        for b in range(4):
            buf = torch.zeros(2 * n + 64, dtype=torch.uint8, device="cuda")
            pa, pb = a, (n + 16) // 4 * 4 + b
            buf[pa:pa + n] = torch.from_numpy(ref.reshape(-1)).cuda()
            buf[pb:pb + n] = torch.from_numpy(dist.reshape(-1)).cuda()
            torch.cuda.synchronize()
            assert ctx.ssimulacra2_device(buf.data_ptr() + pa, buf.data_ptr() + pb, w, h, 3) == want, (a, b)


@pytest.mark.parametrize("channels,dtype", [(1, np.uint8), (2, np.uint8), (4, np.uint8), (1, np.uint16), (3, np.uint16),
                                            (4, np.uint16)])
@pytest.mark.parametrize("w,h", [(9, 70), (67, 65)])
def test_other_formats_match_the_oracle(ctx, oracle, channels, dtype, w, h):
    rng = np.random.default_rng(13)
    top = np.iinfo(dtype).max
    base = synth.image(max(w, 16), max(h, 16), 52, 3.0)[:h, :w, :1].astype(np.float64) / 255
    ref = np.clip(base * top + rng.uniform(-0.02, 0.02, (h, w, channels)) * top, 0, top).astype(dtype)
    dist = np.clip(ref + rng.uniform(-0.03, 0.03, ref.shape) * top, 0, top).astype(dtype)
    assert abs(ctx.ssimulacra2(ref, dist) - oracle.ssimulacra2(ref, dist)) <= 1e-4


def test_requantize_search_of_a_layout_outside_the_encoder(ctx, oracle):
    """4:4:0 (chroma halved down only) goes through the general upsampling; near ties rescore from the planes again."""
    img = synth.image(150, 101, 53, 3.0)
    coefs, qt, lay = oracle.build_coefs(np.ascontiguousarray(img.transpose(1, 0, 2)), 95, int(S.S422), True)
    g = oracle.general_from_encoder(101, 150, lay, qt, coefs)
    lay440 = dict(lay, h=lay["v"].copy(), v=lay["h"].copy(), blocks_w=lay["blocks_h"].copy(),
                  blocks_h=lay["blocks_w"].copy())
    flat = []
    off = 0
    zz = [0, 1, 8, 16, 9, 2, 3, 10, 17, 24, 32, 25, 18, 11, 4, 5, 12, 19, 26, 33, 40, 48, 41, 34, 27, 20, 13, 6, 7, 14,
          21, 28, 35, 42, 49, 56, 57, 50, 43, 36, 29, 22, 15, 23, 30, 37, 44, 51, 58, 59, 52, 45, 38, 31, 39, 46, 53, 60,
          61, 54, 47, 55, 62, 63]
    perm = [zz.index((n % 8) * 8 + n // 8) for n in zz]  # the zigzag position of each block's transpose
    for c in range(3):
        bw, bh = int(lay["blocks_w"][c]), int(lay["blocks_h"][c])
        b = coefs[off: off + bw * bh * 64].reshape(bh, bw, 64)
        off += bw * bh * 64
        flat.append(np.ascontiguousarray(b.transpose(1, 0, 2)[:, :, perm]).reshape(-1))
    g440 = oracle.GeneralCoefs(150, 101, lay440, g.tq, g.qtables4, g.has_q, np.concatenate(flat))
    src = ctx.decode_coefs(oracle.write_jpeg_variant(g440, 0, False))
    assert [c.v for c in src.comps] == [2, 1, 1] and [c.h for c in src.comps] == [1, 1, 1]
    q, _, want, trace = oracle.search_requantize(g440, 70.0)
    for target in (70.0, trace[2][1] + 1e-9):
        q, _, want, otrace = oracle.search_requantize(g440, target)
        f = ctx.find_quality_requantize(src, target)
        assert [t[0] for t in f.trace] == [t[0] for t in otrace]
        assert f.quality == q and np.array_equal(f.coefs.flat(), want.coefs)
