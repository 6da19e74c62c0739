"""Huffman streams at the edges of the span decoder, against the oracle's decoder: codes of every length (the lookup holds
10 bits), DC sizes past what a lookup entry holds, coefficients up to the last index, restart segments shorter than a
span, streams that end at and past a CTA's last span, and streams that never resynchronize (every start is found from the
one before it; past the bound on rounds a serial pass takes over). Coefficients are integers: equal.
"""

import numpy as np
import pytest

import rcg

pytestmark = pytest.mark.gpu


class _Bits:
    def __init__(self):
        self.s = []

    def put(self, v, n):
        if n:
            self.s.append(format(v, f"0{n}b"))

    def bytes(self):
        s = "".join(self.s)
        s += "1" * (-len(s) % 8)
        b = int(s, 2).to_bytes(len(s) // 8, "big") if s else b""
        return b.replace(b"\xff", b"\xff\x00")


def _codes(bits, vals):
    out, code, k = {}, 0, 0
    for length in range(1, 17):
        for _ in range(bits[length - 1]):
            out.setdefault(vals[k], (code, length))
            code, k = code + 1, k + 1
        code <<= 1
    return out


def _jpeg(blocks_w, blocks_h, dc, ac, segments, ri):
    """Gray baseline file; dc, ac: (counts per length, symbols); segments: entropy-coded bytes of each restart segment."""
    def seg(marker, body):
        return bytes([0xFF, marker]) + (len(body) + 2).to_bytes(2, "big") + body

    out = b"\xff\xd8" + seg(0xDB, b"\x00" + bytes([1] * 64))
    out += seg(0xC0, b"\x08" + (blocks_h * 8).to_bytes(2, "big") + (blocks_w * 8).to_bytes(2, "big") + b"\x01\x01\x11\x00")
    out += seg(0xC4, b"\x00" + bytes(dc[0]) + bytes(dc[1])) + seg(0xC4, b"\x10" + bytes(ac[0]) + bytes(ac[1]))
    if ri:
        out += seg(0xDD, ri.to_bytes(2, "big"))
    out += seg(0xDA, b"\x01\x01\x00\x00\x3f\x00")
    for i, s in enumerate(segments):
        out += s + (bytes([0xFF, 0xD0 + i % 8]) if i + 1 < len(segments) else b"")
    return out + b"\xff\xd9"


def _same(ctx, oracle, data):
    g, _ = oracle.decode_sequential(data)
    assert np.array_equal(ctx.decode_coefs(data).flat(), g.coefs)


@pytest.mark.parametrize("blocks_w,blocks_h,ri", [(1, 1, 0), (9, 5, 1), (40, 30, 0), (40, 30, 7), (61, 47, 0)])
def test_codes_of_every_length(ctx, oracle, blocks_w, blocks_h, ri):
    rng = np.random.default_rng(blocks_w * 100 + ri)
    dc = ([1] * 16, [3, 0, 1, 2, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 16])
    ac = ([0, 1] + [1] * 13 + [6], [0x01, 0x00, 0x11, 0x02, 0x21, 0x03, 0xF0, 0x12, 0x0A, 0x31, 0x41, 0x51, 0x04, 0x0F,
                                    0xE1, 0x61, 0x71, 0xF1, 0x2F, 0x05])
    dcc, acc = _codes(*dc), _codes(*ac)
    n, segments = blocks_w * blocks_h, []
    for at in range(0, n, ri or n):
        w = _Bits()
        for _ in range(min(ri or n, n - at)):
            size = int(rng.choice(dc[1], p=[0.4] + [0.04] * 15))
            w.put(*dcc[size])
            w.put(int(rng.integers(0, 1 << size)), size)
            k = 1
            while k < 64:
                sym = int(rng.choice(ac[1]))
                run, size = sym >> 4, sym & 15
                if size and k + run > 63:
                    continue
                w.put(*acc[sym])
                w.put(int(rng.integers(0, 1 << size)), size)
                if sym == 0:
                    break
                k += run + 1
        segments.append(w.bytes())
    _same(ctx, oracle, _jpeg(blocks_w, blocks_h, dc, ac, segments, ri))


# A CTA's spans hold 24576 bytes; a block here is 127, and 48 rounds settle 48 CTAs.
@pytest.mark.parametrize("blocks_w,blocks_h,rounds", [(193, 1, 1), (194, 1, 2), (97, 8, None), (128, 80, -1)])
def test_streams_that_never_resynchronize(ctx, oracle, blocks_w, blocks_h, rounds):
    """All codes and values end on whole bytes, one bit off (the first DC has 9 bits, the others 8): a decoder that starts
    at a byte never meets the stream's own boundaries."""
    rng = np.random.default_rng(blocks_w)
    dc, ac = ([0, 0, 2] + [0] * 13, [5, 6]), ([0] * 7 + [1] + [0] * 8, [0x08])
    w = _Bits()
    for b in range(blocks_w * blocks_h):
        w.put(b == 0, 3)
        w.put(int(rng.integers(0, 32)), 6 if b == 0 else 5)
        for v in rng.integers(0, 256, 63):
            w.put(int(v), 16)
    _same(ctx, oracle, _jpeg(blocks_w, blocks_h, dc, ac, [w.bytes()], 0))
    if rounds is not None:
        assert ctx.last_decode_rounds == rounds
