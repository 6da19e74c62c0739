"""The work that users of this framework have it do, as cases that can be timed and whose outputs can be compared.

A case is a dict of plain values; its "kind" names the entry points one pass goes through:

  search      Context.find_quality_ssimulacra2: the `--target-ssimulacra2` search of one host image
  score       Context.ssimulacra2 (host arrays) or Context.ssimulacra2_device (images already on the GPU)
  sweep       Context.sweep_qualities: a rate-quality curve
  batch       Context.search_batch: a folder of images of mixed sizes, each with its own target
  transcode   Context.decode_coefs + find_quality_requantize: JPEG bytes in, requantized coefficients out
  perceptual  Context.find_quality_perceptual(_fast): the search with gradient-weighted trellis
  encode      Context.build_coefs + plan + reconstruct: one encode at a fixed quality, its file size, its pixels
  grad        Context.ssimulacra2_grad: the FP64 score and its derivative

Images are synthetic photographs (no dataset is shipped): colour gradients, two octaves of value noise, flat
rectangles with hard edges and Gaussian sensor noise, the content of rcg.synth, drawn on the GPU so that a 12 MP
image takes milliseconds. Distorted images of a score are the 8x8 DCT blocks of the image, quantized.
"""

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "rust-compress_gb300")
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

import rcg  # noqa: E402
import rcg.synth as synth  # noqa: E402

S444, S422, S420, AUTO = 1, 2, 3, 0


def listed():
    return [
        # a thumbnail or avatar: the smallest searches, where launches and latency count
        {"name": "search_thumb", "kind": "search", "w": 240, "h": 180, "channels": 3, "sub": S444, "target": 70.0,
         "reuse": False},
        # a picture of a web page, odd sides, the encoder's own choice of subsampling
        {"name": "search_web", "kind": "search", "w": 1283, "h": 857, "channels": 3, "sub": AUTO, "target": 74.0,
         "reuse": False},
        # the benchmark's workload: a 12 MP photograph, pinned input and a reused output buffer, as a service has them
        {"name": "search_12mp", "kind": "search", "w": 4000, "h": 3000, "channels": 3, "sub": S420, "target": 70.0,
         "reuse": True},
        # a gray A4 scan at 200 dpi
        {"name": "search_gray", "kind": "search", "w": 1653, "h": 2339, "channels": 1, "sub": S420, "target": 78.0,
         "reuse": False},
        # comparing two small pictures from host memory
        {"name": "score_512", "kind": "score", "w": 512, "h": 512, "channels": 3, "depth": 8, "device": False,
         "step": 14.0},
        # the scorer workload: a 3840x2160 pair that is on the GPU already
        {"name": "score_4k", "kind": "score", "w": 3840, "h": 2160, "channels": 3, "depth": 8, "device": True,
         "step": 20.0},
        # a rate-quality curve of one picture
        {"name": "sweep_2mp", "kind": "sweep", "w": 1600, "h": 1200, "sub": S420, "qualities": 8, "q_lo": 30,
         "q_hi": 95},
        # a folder of eight pictures of mixed sizes
        {"name": "batch_8", "kind": "batch", "images": 8, "sizes_seed": 2, "lo_mp": 0.3, "hi_mp": 6.0, "sub": S420},
        # a camera's baseline JPEG made smaller at a target quality
        {"name": "transcode_6mp", "kind": "transcode", "w": 3000, "h": 2000, "source_q": 92, "sub": S420,
         "target": 75.0},
        # the perceptual trellis
        {"name": "perceptual_2mp", "kind": "perceptual", "w": 1620, "h": 1080, "sub": S420, "target": 70.0,
         "fast": False},
        # one encode at a fixed quality with its planned size and decoded pixels
        {"name": "encode_512", "kind": "encode", "w": 512, "h": 512, "channels": 3, "sub": S420, "quality": 75},
        # the derivative of the score, FP64
        {"name": "grad_half_mp", "kind": "grad", "w": 768, "h": 512, "step": 24.0},
    ]


def _log_size(rng, lo_mp, hi_mp, smallest=8):
    """(w, h) of a log-uniform area and one of the usual aspect ratios, odd sides among them."""
    area = math.exp(rng.uniform(math.log(lo_mp * 1e6), math.log(hi_mp * 1e6)))
    aspect = rng.choice((4 / 3, 3 / 2, 16 / 9, 1.0, 3 / 4, 2 / 3))
    w = max(smallest, int(math.sqrt(area * aspect)) - rng.randint(0, 7))
    return w, max(smallest, min(int(area / w), int(hi_mp * 1e6 / w)))


def draw(rng):
    kind = rng.choice(("search", "search", "search", "score", "sweep", "batch", "transcode", "perceptual", "encode",
                       "grad"))
    sub = rng.choice((S420, S420, S422, S444))
    if kind == "search":
        w, h = _log_size(rng, 0.03, 11.5)
        return {"kind": kind, "w": w, "h": h, "channels": rng.choice((3, 3, 3, 1)), "sub": rng.choice((S420, S420, AUTO)),
                "target": round(rng.uniform(55, 85), 2), "reuse": rng.random() < 0.5}
    if kind == "score":
        w, h = _log_size(rng, 0.05, 8.2)
        device = rng.random() < 0.5
        channels, depth = (rng.choice((3, 1)), 8) if device else rng.choice(((3, 8), (4, 8), (3, 16), (1, 8)))
        return {"kind": kind, "w": w, "h": h, "channels": channels, "depth": depth, "device": device,
                "step": round(rng.uniform(4, 60), 1)}
    if kind == "sweep":
        w, h = _log_size(rng, 0.1, 2.0)
        return {"kind": kind, "w": w, "h": h, "sub": sub, "qualities": rng.randint(4, 8), "q_lo": rng.randint(10, 50),
                "q_hi": rng.randint(80, 98)}
    if kind == "batch":
        return {"kind": kind, "images": rng.randint(3, 8), "sizes_seed": rng.randint(3, 10000), "lo_mp": 0.3,
                "hi_mp": round(rng.uniform(0.5, 2.0), 2), "sub": S420}
    if kind == "transcode":
        w, h = _log_size(rng, 0.1, 6.0)
        return {"kind": kind, "w": w, "h": h, "source_q": rng.randint(85, 97), "sub": sub,
                "target": round(rng.uniform(60, 80), 2)}
    if kind == "perceptual":
        w, h = _log_size(rng, 0.1, 1.7)
        return {"kind": kind, "w": w, "h": h, "sub": sub, "target": round(rng.uniform(55, 82), 2),
                "fast": rng.random() < 0.5}
    if kind == "encode":
        w, h = _log_size(rng, 0.03, 4.0)
        return {"kind": kind, "w": w, "h": h, "channels": rng.choice((3, 3, 1)), "sub": sub,
                "quality": rng.randint(30, 95)}
    w, h = _log_size(rng, 0.05, 0.4)
    return {"kind": kind, "w": w, "h": h, "step": round(rng.uniform(8, 60), 1)}


# ---- images


def _noise(g, h, w, cell):
    lattice = torch.rand((1, 3, h // cell + 2, w // cell + 2), generator=g, device="cuda") * 2 - 1
    return torch.nn.functional.interpolate(lattice, size=(h, w), mode="bilinear", align_corners=False)[0]


def _image(w, h, seed, sigma=2.0, channels=3):
    """A (h, w, channels) uint8 image on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + 17)
    u = torch.rand(64, generator=g, device="cuda").cpu().numpy()
    ys = ((torch.arange(h, device="cuda", dtype=torch.float32) + 0.5) / h - 0.5)[:, None]
    xs = ((torch.arange(w, device="cuda", dtype=torch.float32) + 0.5) / w - 0.5)[None, :]
    img = torch.zeros((3, h, w), device="cuda")
    for k in range(3):
        th = 2 * math.pi * float(u[k * 7 + 6])
        t = (xs * math.cos(th) + ys * math.sin(th) + 0.5).clamp(0, 1)
        for c in range(3):
            c0, c1 = 255.0 * float(u[k * 7 + c]), 255.0 * float(u[k * 7 + 3 + c])
            img[c] += (c0 + (c1 - c0) * t) / 3
    cell = max(8, min(w, h) // 16)
    img += 16.0 * _noise(g, h, w, cell) + 8.0 * _noise(g, h, w, max(4, cell // 2))
    for k in range(6):
        r = u[21 + k * 7:28 + k * 7]
        x0, y0 = int(r[0] * w), int(r[1] * h)
        x1, y1 = x0 + max(1, int((0.05 + 0.25 * r[2]) * w)), y0 + max(1, int((0.05 + 0.25 * r[3]) * h))
        img[:, y0:y1, x0:x1] = torch.tensor([float(x) * 255 for x in r[4:7]], device="cuda")[:, None, None]
    img += sigma * torch.randn((3, h, w), generator=g, device="cuda")
    img = img.round().clamp(0, 255).to(torch.uint8)
    if channels == 1:
        img = img[1:2]
    return img.permute(1, 2, 0).contiguous()


def _dct_matrix(dtype):
    k = torch.arange(8, dtype=torch.float64)
    m = torch.cos((2 * k[None, :] + 1) * k[:, None] * math.pi / 16) * math.sqrt(2 / 8)
    m[0] /= math.sqrt(2)
    return m.to(dtype).cuda()


def _distort(img, step):
    """The image with every 8x8 DCT coefficient quantized by a step that grows with frequency."""
    h, w, c = img.shape
    x = img.permute(2, 0, 1).float()[None]
    x = torch.nn.functional.pad(x, (0, -w % 8, 0, -h % 8), mode="replicate")[0] - 128
    hh, ww = x.shape[1:]
    b = x.reshape(c, hh // 8, 8, ww // 8, 8).permute(0, 1, 3, 2, 4)
    m = _dct_matrix(torch.float32)
    k = torch.arange(8, device="cuda", dtype=torch.float32)
    q = step * (1 + 0.35 * (k[:, None] + k[None, :]))
    y = m @ b @ m.T
    y = m.T @ ((y / q).round() * q) @ m
    y = y.permute(0, 1, 3, 2, 4).reshape(c, hh, ww)[:, :h, :w] + 128
    return y.round().clamp(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous()


def _score_pair(case, seed):
    """(reference, distorted) of a score case on the GPU: uint8, or int32 holding 16-bit samples."""
    w, h, ch = case["w"], case["h"], case["channels"]
    ref = _image(w, h, seed, channels=1 if ch == 1 else 3)
    dist = _distort(ref, case["step"])
    if case["depth"] == 16:
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed) + 5)
        low = torch.randint(0, 200, ref.shape, generator=g, device="cuda", dtype=torch.int32)
        return ref.int() * 256 + low, dist.int() * 256 + low
    if ch == 4:  # a soft vignette as the alpha channel of both
        ys = torch.linspace(-1, 1, h, device="cuda")[:, None]
        xs = torch.linspace(-1, 1, w, device="cuda")[None, :]
        a = (255 * (1.6 - ys * ys - xs * xs).clamp(0, 1)).to(torch.uint8)[:, :, None]
        return torch.cat([ref, a], 2), torch.cat([dist, a], 2)
    return ref, dist


def _host(t):
    a = t.cpu().numpy()
    return a.astype(np.uint16) if a.dtype == np.int32 else a


# ---- a baseline JPEG file (ITU-T T.81) around given coefficients, as a camera writes it

_DC_BITS = [(0, 1, 5, 1, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0), (0, 3, 1, 1, 1, 1, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0)]


def _flat_ac():
    """A fixed AC table: every run/size symbol, short codes for the common ones (EOB, small sizes, short runs)."""
    order = sorted([0x00, 0xF0] + [r << 4 | s for r in range(16) for s in range(1, 11)],
                   key=lambda v: (0 if v == 0 else (v >> 4) * 1.1 + (v & 15) if v != 0xF0 else 9, v))
    lengths = [2, 2, 3, 4, 4, 5, 5, 6, 6, 6, 7, 7, 7, 7, 8, 8, 8, 8, 9, 9, 9, 9, 10, 10, 10, 10]
    lengths += [12] * 8 + [14] * 24
    lengths += [16] * (len(order) - len(lengths))
    return [lengths.count(n) for n in range(1, 17)], order


def _codes(bits, symbols):
    code, size = torch.zeros(256, dtype=torch.int64), torch.zeros(256, dtype=torch.int64)
    c = k = 0
    for n in range(1, 17):
        for _ in range(bits[n - 1]):
            code[symbols[k]], size[symbols[k]] = c, n
            c, k = c + 1, k + 1
        if c > 1 << n:
            raise ValueError("overfull Huffman table")
        c <<= 1
    return code.cuda(), size.cuda()


def _bits_of(v):
    """JPEG magnitude category of int64 values."""
    return torch.frexp(v.abs().double())[1].long()


def _jpeg(ci):
    """Baseline JPEG bytes of an encoder CoefImage (zigzag coefficients, blocks padded to whole MCUs)."""
    ac_bits, ac_syms = _flat_ac()
    ac_code, ac_size = _codes(ac_bits, ac_syms)
    hm, vm = max(c.h for c in ci.comps), max(c.v for c in ci.comps)
    mw, mh = -(-ci.width // (8 * hm)), -(-ci.height // (8 * vm))
    blocks, comp_of = [], []
    for k, c in enumerate(ci.comps):
        v, h = (c.v, c.h) if len(ci.comps) > 1 else (1, 1)
        b = torch.from_numpy(np.array(c.coefs)).cuda().long().reshape(mh, v, mw, h, 64)
        blocks.append(b.permute(0, 2, 1, 3, 4).reshape(mh * mw, v * h, 64))
        comp_of += [k] * (v * h)
    z = torch.cat(blocks, 1)
    per = z.shape[1]
    z = z.reshape(-1, 64)
    comp = torch.tensor(comp_of, device="cuda").repeat(mh * mw)
    n = z.shape[0]
    diff = torch.zeros(n, dtype=torch.int64, device="cuda")
    for k in range(len(ci.comps)):
        at = (comp == k).nonzero()[:, 0]
        dc = z[at, 0]
        diff[at] = dc - torch.cat([dc.new_zeros(1), dc[:-1]])
    dcs = [_codes(b, list(range(12))) for b in _DC_BITS]
    chroma = (comp > 0).long()
    s = _bits_of(diff)
    dc_code = torch.stack([dcs[0][0], dcs[1][0]])[chroma, s]
    dc_size = torch.stack([dcs[0][1], dcs[1][1]])[chroma, s]
    extra = torch.where(diff < 0, diff + (1 << s) - 1, diff)
    keys, vals, lens = [torch.arange(n, device="cuda") * 1024], [dc_code << s | extra], [dc_size + s]
    # AC: a token for each nonzero coefficient, up to three ZRLs before it, an EOB after the last one
    ac = z[:, 1:].nonzero()
    blk, pos = ac[:, 0], ac[:, 1] + 1
    v = z[blk, pos]
    first = torch.ones_like(blk, dtype=torch.bool)
    first[1:] = blk[1:] != blk[:-1]
    prev = torch.where(first, torch.zeros_like(pos), torch.cat([pos.new_zeros(1), pos[:-1]]))
    run = pos - prev - 1
    s = _bits_of(v)
    sym = (run % 16) << 4 | s
    extra = torch.where(v < 0, v + (1 << s) - 1, v)
    keys.append(blk * 1024 + pos * 8 + 7)
    vals.append(ac_code[sym] << s | extra)
    lens.append(ac_size[sym] + s)
    for j in range(3):
        at = (run // 16 > j).nonzero()[:, 0]
        keys.append(blk[at] * 1024 + pos[at] * 8 + j)
        vals.append(ac_code[0xF0].expand(at.numel()))
        lens.append(ac_size[0xF0].expand(at.numel()))
    eob = (z[:, 63] == 0).nonzero()[:, 0]
    keys.append(eob * 1024 + 1023)
    vals.append(ac_code[0].expand(eob.numel()))
    lens.append(ac_size[0].expand(eob.numel()))
    keys, vals, lens = torch.cat(keys), torch.cat(vals), torch.cat(lens)
    o = torch.argsort(keys)
    vals, lens = vals[o], lens[o]
    ends = torch.cumsum(lens, 0)
    total = int(ends[-1])
    which = torch.repeat_interleave(torch.arange(vals.numel(), device="cuda"), lens)
    bit = ends[which] - 1 - torch.arange(total, device="cuda")
    bits = (vals[which] >> bit & 1).to(torch.uint8)
    packed = np.packbits(np.concatenate([bits.cpu().numpy(), np.ones(-total % 8, np.uint8)]))
    packed = np.insert(packed, np.nonzero(packed == 0xFF)[0] + 1, 0)

    def seg(marker, body):
        return bytes([0xFF, marker]) + (len(body) + 2).to_bytes(2, "big") + bytes(body)

    zz = sorted(range(64), key=lambda i: (i // 8 + i % 8, i // 8 if (i // 8 + i % 8) % 2 else i % 8))
    q = np.asarray(ci.qtables, np.uint8).reshape(-1, 64)
    out = b"\xff\xd8"
    for t in range(2 if len(ci.comps) > 1 else 1):
        out += seg(0xDB, [t] + [int(q[t][i]) for i in zz])
    body = [8] + list(ci.height.to_bytes(2, "big")) + list(ci.width.to_bytes(2, "big")) + [len(ci.comps)]
    for k, c in enumerate(ci.comps):
        body += [k + 1, c.h << 4 | c.v, min(k, 1)]
    out += seg(0xC0, body)
    for t in range(2):
        out += seg(0xC4, [t] + list(_DC_BITS[t]) + list(range(12)))
        out += seg(0xC4, [0x10 | t] + ac_bits + ac_syms)
    body = [len(ci.comps)]
    for k in range(len(ci.comps)):
        body += [k + 1, min(k, 1) * 0x11]
    out += seg(0xDA, body + [0, 63, 0])
    assert per == len(comp_of)
    return out + packed.tobytes() + b"\xff\xd9"


# ---- the cases


def _options(case, quality=90):
    return rcg.EncodeOptions(quality, rcg.Subsampling(case["sub"]), True)


def _batch_sizes(case):
    lo, hi = case["lo_mp"] * 1e6, case["hi_mp"] * 1e6
    return synth.log_uniform_sizes(case["sizes_seed"], case["images"], (lo, 1), (hi, 1))


def prepare(case, seed):
    ctx = rcg.default_context()  # one context for the program's life, as a service keeps it
    kind = case["kind"]
    s = {"kind": kind, "case": case, "ctx": ctx}
    if kind == "search":
        img = _host(_image(case["w"], case["h"], seed, 3.0, case["channels"]))
        s["opts"] = _options(case)
        if case["reuse"]:
            s["keep"] = torch.from_numpy(img).pin_memory()
            img = s["keep"].numpy()
            n = ctx.coef_capacity(case["w"], case["h"], case["channels"], s["opts"])
            s["out"] = torch.zeros(n, dtype=torch.int16).pin_memory().numpy()
        s["img"] = img
    elif kind == "score":
        ref, dist = _score_pair(case, seed)
        s["ref"], s["dist"] = (ref, dist) if case["device"] else (_host(ref), _host(dist))
    elif kind == "sweep":
        s["img"] = _host(_image(case["w"], case["h"], seed, 3.0))
        s["opts"] = _options(case)
        n = case["qualities"]
        s["qualities"] = [round(case["q_lo"] + (case["q_hi"] - case["q_lo"]) * i / (n - 1)) for i in range(n)]
    elif kind == "batch":
        sizes = _batch_sizes(case)
        s["imgs"] = [_host(_image(w, h, seed * 64 + i, 1.5)) for i, (w, h) in enumerate(sizes)]
        u = synth.uniforms(case["sizes_seed"], 40, len(sizes))
        s["targets"] = [55.0 + 30.0 * float(x) for x in u]
        s["opts"] = _options(case)
    elif kind == "transcode":
        img = _host(_image(case["w"], case["h"], seed, 6.0))
        s["jpeg"] = _jpeg(ctx.build_coefs(img, _options(case, case["source_q"])))
    elif kind in ("perceptual", "encode"):
        s["img"] = _host(_image(case["w"], case["h"], seed, 3.0, case.get("channels", 3)))
        s["opts"] = _options(case, case.get("quality", 90))
    else:
        ref = _image(case["w"], case["h"], seed)
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed) + 9)
        # off the whole numbers, where the edge terms have a kink
        dist = _distort(ref, case["step"]).float() + 0.5 * torch.rand(ref.shape, generator=g, device="cuda") - 0.25
        s["ref"], s["dist"] = _host(ref), dist.clamp(0, 255).cpu().numpy()
    torch.cuda.synchronize()
    return s


def _trace(t):
    """The evaluated qualities and scores, padded to the eight steps of the longest bisection."""
    t = list(t) + [(0, 0.0)] * (8 - len(t))
    return {"q": np.array([q for q, _ in t], dtype=np.int64), "score": [s for _, s in t]}


def _found(f):
    return {"quality": f.quality, "score": f.score, "coefs": [c.coefs for c in f.coefs.comps],
            "qtables": f.coefs.qtables, "trace": _trace(f.trace)}


def run(state):
    ctx, case, kind = state["ctx"], state["case"], state["kind"]
    if kind == "search":
        return _found(ctx.find_quality_ssimulacra2(state["img"], case["target"], 100, state["opts"],
                                                   out=state.get("out")))
    if kind == "score":
        if case["device"]:
            return ctx.ssimulacra2_device(state["ref"].data_ptr(), state["dist"].data_ptr(), case["w"], case["h"],
                                          case["channels"])
        return ctx.ssimulacra2(state["ref"], state["dist"])
    if kind == "sweep":
        return ctx.sweep_qualities([state["img"]], state["qualities"], state["opts"])[0].tolist()
    if kind == "batch":
        res = ctx.search_batch(state["imgs"], state["targets"], 100, state["opts"])
        return [{"quality": f.quality, "score": f.score, "coefs": [c.coefs for c in f.coefs.comps]} for f in res]
    if kind == "transcode":
        ci = ctx.decode_coefs(state["jpeg"])
        return {"source": [c.coefs for c in ci.comps], "found": _found(ctx.find_quality_requantize(ci, case["target"]))}
    if kind == "perceptual":
        if case["fast"]:
            probe, found, _ = ctx.find_quality_perceptual_fast(state["img"], case["target"], 100, state["opts"],
                                                               want_weights=False)
            return {"probe": _trace(probe.trace), "found": _found(found)}
        r = ctx.find_quality_perceptual(state["img"], case["target"], 100, state["opts"], want_weights=False)
        return {"found": _found(r.found), "plain": [r.plain.quality, r.plain.score],
                "bytes": [r.plain_bytes, r.perceptual_bytes]}
    if kind == "encode":
        ci = ctx.build_coefs(state["img"], state["opts"])
        plan = ctx.plan(ci)
        return {"coefs": [c.coefs for c in ci.comps], "qtables": ci.qtables, "pixels": ctx.reconstruct(ci),
                "bytes": [plan.progressive_bytes, plan.baseline_bytes],
                "scans": np.array([b for _, b in plan.distinct], dtype=np.int64)}
    score, grad = ctx.ssimulacra2_grad(state["ref"], state["dist"])
    return {"score": score, "grad": grad}


# ---- what a pass cannot do without

# Operations of one score per full-resolution pixel: the two images' XYB, 3 channels x 5 moments x 22 taps of
# multiply-add and the error maps, over the 4/3 pixels of the pyramid.
_SCORE_OPS = 4 / 3 * (2 * 60 + 3 * (5 * 22 * 2 + 30))
# Operations of one candidate besides its score: quantization with the trellis, the IDCT and the colour conversion.
_CODEC_OPS = 200
_STEPS = 7  # candidates of a bisection over 1..100: the maximum and six or seven halvings


def _coefs(case, w=None, h=None):
    ch = case.get("channels", 3)
    lay = rcg.default_context().coef_layout(w or case["w"], h or case["h"], ch, _options(case, case.get("quality", 80)))
    return int(lay.ncoefs)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = _batch_sizes(case)
        px = sum(w * h for w, h in sizes)
        return {"bytes": 3 * px + 2 * sum(_coefs(case, w, h) for w, h in sizes),
                "flops": _STEPS * (_SCORE_OPS + _CODEC_OPS) * px}
    px = case["w"] * case["h"]
    if kind == "search":
        return {"bytes": case["channels"] * px + 2 * _coefs(case), "flops": _STEPS * (_SCORE_OPS + _CODEC_OPS) * px}
    if kind == "score":
        return {"bytes": 2 * px * case["channels"] * case["depth"] // 8, "flops": _SCORE_OPS * px}
    if kind == "sweep":
        return {"bytes": 3 * px, "flops": case["qualities"] * (_SCORE_OPS + _CODEC_OPS) * px}
    if kind == "transcode":
        return {"bytes": px // 5 + 2 * 2 * _coefs(case), "flops": _STEPS * (_SCORE_OPS + _CODEC_OPS) * px}
    if kind == "perceptual":
        steps = 12 if case["fast"] else 2 * _STEPS
        return {"bytes": 3 * px + 2 * _coefs(case), "flops": (steps * (_SCORE_OPS + _CODEC_OPS) + 3 * _SCORE_OPS) * px}
    if kind == "encode":
        return {"bytes": 2 * case["channels"] * px + 2 * _coefs(case), "flops": 2 * _CODEC_OPS * px}
    return {"bytes": (3 + 12 + 24) * px, "flops": 3 * _SCORE_OPS * px}


# ---- SSIMULACRA 2 in 64 bits, in plain torch

_WEIGHTS = [
    0.0, 0.0007376606707406586, 0.0, 0.0, 0.0007793481682867309, 0.0,
    0.0, 0.0004371155730107379, 0.0, 1.1041726426657346, 0.00066284834129271, 0.00015231632783718752,
    0.0, 0.0016406437456599754, 0.0, 1.8422455520539298, 11.441172603757666, 0.0,
    0.0007989109436015163, 0.000176816438078653, 0.0, 1.8787594979546387, 10.94906990605142, 0.0,
    0.0007289346991508072, 0.9677937080626833, 0.0, 0.00014003424285435884, 0.9981766977854967, 0.00031949755934435053,
    0.0004550992113792063, 0.0, 0.0, 0.0013648766163243398, 0.0, 0.0,
    0.0, 0.0, 0.0, 7.466890328078848, 0.0, 17.445833984131262,
    0.0006235601634041466, 0.0, 0.0, 6.683678146179332, 0.00037724407979611296, 1.027889937768264,
    225.20515300849274, 0.0, 0.0, 19.213238186143016, 0.0011401524586618361, 0.001237755635509985,
    176.39317598450694, 0.0, 0.0, 24.43300999870476, 0.28520802612117757, 0.0004485436923833408,
    0.0, 0.0, 0.0, 34.77906344483772, 44.835625328877896, 0.0,
    0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0008680556573291698, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0005313191874358747, 0.0, 0.00016533814161379112, 0.0, 0.0,
    0.0, 0.0, 0.0, 0.0004179171803251336, 0.0017290828234722833, 0.0,
    0.0020827005846636437, 0.0, 0.0, 8.826982764996862, 23.19243343998926, 0.0,
    95.1080498811086, 0.9863978034400682, 0.9834382792465353, 0.0012286405048278493, 171.2667255897307, 0.9807858872435379,
    0.0, 0.0, 0.0, 0.0005130064588990679, 0.0, 0.00010854057858411577]


def _linear64(img, top):
    """(3, h, w) linear light of samples in 0..top, (h, w, 1|3|4)."""
    if img.shape[2] == 4:  # over mid-gray, in whole numbers
        x, a = img[:, :, :3].long(), img[:, :, 3:].long()
        img = (x * a + 128 * (255 - a) + 127) // 255
    v = img.double().permute(2, 0, 1) / top
    v = torch.where(v <= 0.04045, v / 12.92, ((v.clamp(min=0.04) + 0.055) / 1.055) ** 2.4)
    return v.expand(3, -1, -1)


def _xyb64(p):
    m02, m00, m12, m10, m20, m21 = 0.078, 0.30, 0.078, 0.23, 0.2434226892454782, 0.2047674442449682
    bias = 0.0037930732552754493
    rows = ((m00, 1 - m02 - m00, m02), (m10, 1 - m12 - m10, m12), (m20, m21, 1 - m20 - m21))
    c = [(a * p[0] + b * p[1] + d * p[2] + bias) ** (1 / 3) - bias ** (1 / 3) for a, b, d in rows]
    y = (c[0] + c[1]) / 2
    return [7 * (c[0] - c[1]) + 0.42, y + 0.01, c[2] - y + 0.55]


def _blur64(x):
    k = [math.exp(-0.5 / 2.25 * (i - 5) ** 2) for i in range(11)]
    k = [v / sum(k) for v in k]
    h, w = x.shape
    z = torch.nn.functional.pad(x[None], (5, 5))[0]
    z = sum(k[t] * z[:, t:t + w] for t in range(11))
    idx = torch.arange(-5, h + 5, device=x.device)
    z = z[torch.where(idx < 0, -idx - 1, torch.where(idx >= h, 2 * h - 1 - idx, idx))]
    return sum(k[t] * z[t:t + h] for t in range(11))


def _half64(p):
    h, w = p.shape[1:]
    oh, ow = (h + 1) // 2, (w + 1) // 2
    z = torch.nn.functional.pad(p, (0, 2 * ow - w, 0, 2 * oh - h)).reshape(3, oh, 2, ow, 2).sum((2, 4))
    ny = torch.full((oh, 1), 2.0, dtype=torch.float64, device=p.device)
    nx = torch.full((1, ow), 2.0, dtype=torch.float64, device=p.device)
    ny[-1] -= h % 2
    nx[:, -1] -= w % 2
    return z / (ny * nx)


def _score64(a, b):
    """SSIMULACRA 2 of two (3, h, w) float64 linear images, as a tensor that autograd goes through."""
    stats = []
    for scale in range(6):
        if min(a.shape[1:]) < 8:
            break
        row = []
        for x, y in zip(_xyb64(a), _xyb64(b)):
            m1, m2 = _blur64(x), _blur64(y)
            s11, s22, s12 = _blur64(x * x), _blur64(y * y), _blur64(x * y)
            num_s = 2 * (s12 - m1 * m2) + 0.0009
            den = (s11 - m1 * m1) + (s22 - m2 * m2) + 0.0009
            d = (1 - (1 - (m1 - m2) ** 2) * num_s / den).clamp(min=0)
            e = (1 + (y - m2).abs()) / (1 + (x - m1).abs()) - 1
            maps = (d, e.clamp(min=0), (-e).clamp(min=0))
            row.append([[m.mean() for m in maps], [(m ** 4).mean() ** 0.25 for m in maps]])
            del m1, m2, s11, s22, s12, num_s, den, d, e, maps
        stats.append(row)
        if scale < 5:
            a, b = _half64(a), _half64(b)
    terms = [v for c in range(3) for row in stats for norm in row[c] for v in norm]
    s = 0.9562382616834844 * sum(w * t.abs() for w, t in zip(_WEIGHTS, terms))
    s = 2.326765642916932 * s - 0.020884521182843837 * s * s + 6.248496625763138e-05 * s * s * s
    return 100 - 10 * s ** 0.6276336467831387


def exact(case, seed):
    """run()'s outputs in 64 bits for the cases whose outputs are computed numbers: a score, and its derivative. The
    searches' scores belong to coefficients that the framework chooses, which are whole numbers."""
    if case["kind"] == "score":
        ref, dist = _score_pair(case, seed)
        top = 65535 if case["depth"] == 16 else 255
        with torch.no_grad():
            return float(_score64(_linear64(ref, top), _linear64(dist, top)))
    if case["kind"] == "grad":
        s = prepare(case, seed)
        ref = torch.from_numpy(s["ref"]).cuda()
        dist = torch.from_numpy(s["dist"]).cuda().double().requires_grad_(True)
        score = _score64(_linear64(ref, 255), _linear64(dist, 255))
        score.backward()
        return {"score": float(score.detach()), "grad": dist.grad}
    return None
