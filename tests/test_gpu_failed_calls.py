"""A call that fails after it has queued its uploads returns only when they are done: the caller may free its images then.
The stream is kept busy ahead of the call, and its workspace is limited so that it fails later and later; the last of these
failures comes after the uploads."""

import ctypes

import numpy as np
import pytest

import rcg
import rcg.synth as synth

pytestmark = pytest.mark.gpu

OPTS = rcg.EncodeOptions(80, rcg.Subsampling.S444, True)
W, H = 320, 240


def _calls(img, other, dist, coefs):
    return {
        "score": lambda c: c.ssimulacra2(img, other),
        "batch": lambda c: c.ssimulacra2_batch([(img, other), (other, img)]),
        "metric": lambda c: c.ssimulacra2_exact(img, other),
        "search": lambda c: c.find_quality_ssimulacra2(img, 70.0, 100, OPTS),
        "sweep": lambda c: c.sweep_qualities([img], [80, 50], OPTS),
        "encode": lambda c: c.build_coefs(img, OPTS),
        "plan": lambda c: c.plan(coefs),
        "gradient": lambda c: c.ssimulacra2_grad(img, dist),
    }


@pytest.mark.parametrize("what", list(_calls(None, None, None, None)))
def test_uploads_are_done_when_a_failed_call_returns(what):
    torch = pytest.importorskip("torch")
    keep = []

    def pinned(a):
        t = torch.from_numpy(np.ascontiguousarray(a)).pin_memory()  # the GPU reads it when the copy's turn comes
        keep.append(t)
        return t.numpy()

    base = synth.image(W, H, 81, sensor_sigma=2.0)
    img, other, dist = pinned(base), pinned(base[::-1]), pinned(base[::-1].astype(np.float32))
    with rcg.Context(0) as c:
        ci = c.build_coefs(img, OPTS)
    flat, at = pinned(ci.flat()), 0
    for comp in ci.comps:
        comp.coefs, at = flat[at: at + comp.coefs.size], at + comp.coefs.size
    call = _calls(img, other, dist, ci)[what]
    limit = rcg._lib.rcg_internal_limit_workspace
    limit.restype, limit.argtypes = None, [ctypes.c_void_p, ctypes.c_uint64]
    stream = torch.cuda.Stream()
    idle, bytes_ = [], 1 << 16
    while True:
        assert bytes_ < 1 << 32
        with rcg.Context(0) as c:
            c.set_stream(stream.cuda_stream)
            limit(c._ptr, bytes_)
            with torch.cuda.stream(stream):
                torch.cuda._sleep(40_000_000)  # 20 ms
            try:
                call(c)
                done = True
            except rcg.RcgError as e:
                assert e.status == rcg.RCG_NO_MEMORY
                idle.append(stream.query())
                done = False
            stream.synchronize()
        if done:
            break
        bytes_ += bytes_ // 8
    assert len(idle) >= 2 and idle[-1], idle
