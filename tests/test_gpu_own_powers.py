"""The library's own powers (score_power.cuh, curve_power.cuh) over their ranges against 60-digit decimals: the score's power
within 0.504 ulp (0.5 of rounding and 7 units of 2^-63 of truncations, 2048 of them to an ulp), the curve's within 0.501
(its terms below the rounded sum are kept to 2^-104). Powers of two and their neighbours, both sides of 1, mantissas at the
ends of the logarithm's steps, random ones."""

import ctypes
import decimal
import math
import os
import subprocess

import numpy as np
import pytest

import build as rcg_build
import rcg  # noqa: F401  (the library's directory is on the path)

pytestmark = pytest.mark.gpu

CSRC = rcg_build.CSRC
SOURCE = """
#include <cuda_runtime.h>
#include "score_power.cuh"
#include "curve_power.cuh"
__global__ void k_powers(const double* x, double* out, int n, int which) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = which == 0 ? rcg::score_power(x[i]) : which == 1 ? rcg::pow24(x[i]) : rcg::pow14(x[i]);
}
extern "C" int powers(const double* x, double* out, int n, int which) {
  double *dx = nullptr, *dy = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  cudaMalloc(&dx, b);
  cudaMalloc(&dy, b);
  cudaMemcpy(dx, x, b, cudaMemcpyHostToDevice);
  k_powers<<<(n + 127) / 128, 128>>>(dx, dy, n, which);
  cudaMemcpy(out, dy, b, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def powers(tmp_path_factory):
    d = tmp_path_factory.mktemp("powers")
    src, so = os.path.join(d, "powers.cu"), os.path.join(d, "powers.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([rcg_build.nvcc(), *rcg_build.COMMON, "-I", CSRC, "-shared", "-o", so, src], check=True)
    lib = ctypes.CDLL(so)

    def call(x, which):
        x = np.ascontiguousarray(x, np.float64)
        out = np.empty_like(x)
        assert lib.powers(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data), x.size, which) == 0
        return out

    return call


def _worst(x, got, power):
    """The largest error in ulps of the result."""
    decimal.getcontext().prec = 60
    decimal.getcontext().Emin, decimal.getcontext().Emax = -9999, 9999
    p = decimal.Decimal(power)
    worst = (0.0, None)
    for a, g in zip(x, got):
        exact = (decimal.Decimal(float(a)).ln() * p).exp()
        err = abs(float((decimal.Decimal(float(g)) - exact) / decimal.Decimal(math.ulp(float(exact)))))
        worst = max(worst, (err, float(a)), key=lambda t: t[0])
    return worst


def _values(lo, hi, seed, n=1500):
    """Of each kind, those in [lo, hi]: around powers of two, around 1, at steps of 2^-20 of the logarithm, random."""
    rng = np.random.default_rng(seed)
    e0, e1 = math.frexp(lo)[1], math.frexp(hi)[1]
    two = np.array([math.ldexp(1.0, int(e)) for e in np.linspace(e0, e1 - 1, min(e1 - e0, 200)).round()])
    one = 1.0 + np.concatenate([np.arange(-40, 41) * 2.0**-53, rng.normal(0, 2.0**-20, 100), rng.normal(0, 0.02, 100)])
    l = np.concatenate([[0.5, 1.5, 2.0**20 - 1.5, 2.0**20 - 0.5], rng.integers(0, 2**20, 200) + 0.5]) / 2.0**20
    steps = np.exp2(l) * (1 + rng.integers(-3, 4, l.size) * 2.0**-24)  # where the rounded logarithm changes
    steps = np.clip(np.concatenate([steps, np.array([1.0, 2.0 - 2.0**-52])]), 1.0, 2.0 - 2.0**-52)
    steps = steps * np.exp2(rng.integers(e0, max(e1 - 1, e0 + 1), steps.size).astype(float))
    wide = np.exp2(rng.uniform(math.log2(lo), math.log2(hi) - 1e-9, n))
    x = np.concatenate([two, np.nextafter(two, 0), np.nextafter(two, np.inf), one, steps, wide, [lo, hi]])
    return x[(x >= lo) & (x <= hi)]


@pytest.mark.parametrize("lo,hi", [(2.2250738585072014e-308, 1.7976931348623157e308), (1e-6, 400.0), (0.5, 2.0)])
def test_score_power(powers, lo, hi):
    x = _values(lo, hi, 101)
    err, at = _worst(x, powers(x, 0), 0.6276336467831387)
    assert err <= 0.504, (err, at)


def test_score_power_outside_its_range_is_pow(powers):
    x = np.array([0.0, 5e-324, 1e-310, np.inf, np.nan, -1.0])
    got = powers(x, 0)
    assert got[0] == 0.0 and got[3] == np.inf and np.isnan(got[4]) and np.isnan(got[5])
    err, at = _worst(x[1:3], got[1:3], 0.6276336467831387)
    assert err <= 2.0, (err, at)


@pytest.mark.parametrize("which,power", [(1, 2.4), (2, 1.4)])
@pytest.mark.parametrize("lo,hi", [(0.0904, 1.0), (0.99, 1.01), (0.0904, 1e6), (1.1e-15, 9e14)])
def test_curve_powers(powers, which, power, lo, hi):
    x = _values(lo, hi, 103 + which)
    err, at = _worst(x, powers(x, which), power)
    assert err <= 0.501, (err, at)


@pytest.mark.parametrize("which,power", [(1, 2.4), (2, 1.4)])
def test_curve_powers_outside_their_range_are_pow(powers, which, power):
    x = np.array([1e-17, 1e17, 1e30, 1e120])
    err, at = _worst(x, powers(x, which), power)
    assert err <= 2.0, (err, at)
    assert powers(np.array([np.inf]), which)[0] == np.inf and np.isnan(powers(np.array([np.nan]), which)[0])
