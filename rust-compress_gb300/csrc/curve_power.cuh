// The sRGB curve's powers in FP64.
#pragma once

namespace rcg {

// x^0.4 = y + lo for x > 0, the fifth root of x^2 = a + ea: r = a^(-1/5) from an f32 seed by two steps of Newton's
// iteration for the inverse root (r <- r (6 - a r^5) / 5; an error e becomes 3 e^2, 1e-6 -> 3e-12 -> 3e-23), then y = a
// r^4 and one Newton step on y^5 = a + ea whose residual carries the rounding errors of a, y^2 and y^4, kept apart as lo.
// About 30 FP64 operations where pow takes some two hundred; products formed with y and lo round once more, so the powers
// below are within 0.501 ulp (tests/test_gpu_own_powers.py). False for values outside the f32 range (those go to pow).
__device__ __forceinline__ bool pow04(double x, double& a, double& ea, double& y, double& lo) {
  a = x * x;
  ea = fma(x, x, -a);
  if (!(a > 1e-30 && a < 1e30)) return false;
  const float l2 = log2f((float)a);
  double r = (double)exp2f(-0.2f * l2);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double r2 = r * r, r5 = r2 * r2 * r;
    r = r * fma(-0.2 * a, r5, 1.2);
  }
  const double r2 = r * r, r4 = r2 * r2;
  y = a * r4;
  const double y2 = y * y, e2 = fma(y, y, -y2);
  const double y4 = y2 * y2, e4 = fma(2.0 * y2, e2, fma(y2, y2, -y4));
  lo = (fma(-y4, y, a) + fma(-e4, y, ea)) * 0.2 * r4;  // y = 1 / r, so 1 / (5 y^4) = r^4 / 5
  // The curve's exponents 2.4 and 1.4 are f64 values, both 8.88e-17 below the decimals: x^-8.88e-17 = 1 - 8.88e-17 ln x.
  lo = fma(y, -8.881784197001252e-17 * 0.34657359027997264 * (double)l2, lo);
  return true;
}

// x^2.4 and x^1.4 (the f64 exponents).
__device__ __forceinline__ double pow24(double x) {
  double a, ea, y, lo;
  return pow04(x, a, ea, y, lo) ? fma(a, y, fma(a, lo, ea * y)) : pow(x, 2.4);
}
__device__ __forceinline__ double pow14(double x) {
  double a, ea, y, lo;
  return pow04(x, a, ea, y, lo) ? fma(x, y, x * lo) : pow(x, 1.4);
}

}  // namespace rcg
