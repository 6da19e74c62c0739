"""The adjoint's job tables: every scale and channel in one launch per step, each CTA finding its plane.

Sizes around the runs (4 columns, 8 and 16 rows) and the CTAs (256 threads) of the plane kernels, narrow and flat images
among them, against the FP64 CPU gradient.
"""

import numpy as np
import pytest

import rcg.synth as synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(8, 8), (255, 17), (257, 33), (31, 259), (1023, 40), (16, 515)])
def test_gradient_at_job_edges(ctx, oracle, w, h):
    ref = synth.image(w, h, 84, 3.0)
    rng = np.random.default_rng(w * 1000 + h)
    dist = np.clip(ref + rng.uniform(-12, 12, ref.shape), 0, 255).astype(np.float32)
    s, g = ctx.ssimulacra2_grad(ref, dist)
    s_cpu, g_cpu = oracle.grad64(ref.astype(np.float64), dist.astype(np.float64))
    scale = np.abs(g_cpu).max()
    assert abs(s - s_cpu) < 1e-9
    err = np.abs(g - g_cpu)
    # as the full-size test: equal to rounding but where a map sits on a kink and rounding picks the side
    assert (err > 1e-12 * scale + 1e-9 * np.abs(g_cpu)).mean() <= 1e-3
    assert err.max() <= 1e-5 * scale

