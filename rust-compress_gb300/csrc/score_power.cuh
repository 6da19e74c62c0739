// The score's power in 64-bit fixed point.
#pragma once

namespace rcg {

// x^0.6276336467831387 for the score (core/src/ssimulacra2.rs:509) by one thread, in 64-bit fixed point: an FP64
// instruction occupies its quarter of an SM for 64 cycles, so pow and the polynomial before it took 6650, more than a third
// of what the reduction's last CTA needs; with this 2430 (240x180 search 541 -> 514 us, 512x512 score 90 -> 85). Method: x =
// 2^e m; a float logarithm rounded to 20 bits, l, leaves m 2^-l = 1 + r with |r| < 2^-19, whose logarithm is three terms of
// its series; 2^f is a 16-entry table of 2^(i/16) and nine terms of e^u. Fractions have 60 bits or more throughout. The
// truncations add up to at most 7 units of the result's 63 bits, 11 more than a double's: within 0.504 ulp over 2.3e-308 ..
// 1.8e308 (tests/test_gpu_own_powers.py); pow's stated bound is 2.
__device__ const unsigned long long d_exp2_16[16] = {  // 2^(i/16), 63 fraction bits
    0x8000000000000000ull, 0x85aac367cc487b15ull, 0x8b95c1e3ea8bd6e7ull, 0x91c3d373ab11c336ull,
    0x9837f0518db8a96full, 0x9ef5326091a111aeull, 0xa5fed6a9b15138eaull, 0xad583eea42a14ac6ull,
    0xb504f333f9de6484ull, 0xbd08a39f580c36bfull, 0xc5672a115506daddull, 0xce248c151f8480e4ull,
    0xd744fccad69d6af4ull, 0xe0ccdeec2a94e111ull, 0xeac0c6e7dd24392full, 0xf5257d152486cc2cull};

// 2^(f / 2^64) with 63 fraction bits.
__device__ __forceinline__ unsigned long long exp2_fixed(unsigned long long f) {
  constexpr unsigned long long kFact[8] = {  // 1 / (k + 1)!, 63 fraction bits
      0x8000000000000000ull, 0x4000000000000000ull, 0x1555555555555555ull, 0x0555555555555555ull,
      0x0111111111111111ull, 0x002d82d82d82d82eull, 0x0006806806806807ull, 0x0000d00d00d00d01ull};
  const unsigned long long t = d_exp2_16[f >> 60];
  const unsigned long long u = __umul64hi(f << 4, 0xb17217f7d1cf79acull);  // the rest times ln 2, 68 fraction bits
  unsigned long long q = 0x0000171de3a556c7ull;                           // 1 / 9!
#pragma unroll
  for (int k = 7; k >= 0; k--) q = kFact[k] + (__umul64hi(u, q) >> 4);
  return t + (__umul64hi(t, __umul64hi(u, q)) >> 3);
}

__device__ __forceinline__ double score_power(double x) {
  if (!(x >= 2.2250738585072014e-308 && x <= 1.7976931348623157e308)) return pow(x, 0.6276336467831387);
  const unsigned long long b = (unsigned long long)__double_as_longlong(x), m = (b << 11) | (1ull << 63);
  const int e = (int)(b >> 52) - 1023;
  const float mf = __uint_as_float((unsigned)((b >> 29) & 0x7fffff) | 0x3f800000u);
  const unsigned l = (unsigned)(log2f(mf) * 1048576.0f + 0.5f);  // 0 .. 2^20
  // r with 63 fraction bits; m 2^-l as half of m 2^(1 - l).
  const unsigned long long g = l == 0 ? 0ull : exp2_fixed((unsigned long long)(1048576u - l) << 44);
  const long long rr = (long long)((l == 0 ? m : __umul64hi(m, g)) - (1ull << 63));
  const long long r = (long long)((unsigned long long)rr << 16);  // 79 fraction bits
  const long long r2 = __mul64hi(r, r), r3 = __mul64hi(r2, r);
  // log2 (1 + r) with 64: r, r^2 / 2 and r^3 / 3 over ln 2.
  const long long part = (__mul64hi(r, 0x5c551d94ae0bf85ell) >> 13) - (__mul64hi(r2, 0x2e2a8eca5705fc2fll) >> 28) +
                         (__mul64hi(r3, 0x1ec709dc3a03fd75ll) >> 43);
  const unsigned long long base = (unsigned long long)l << 44, frac = base + (unsigned long long)part;
  int whole = e + (int)(l >> 20);
  if (part < 0) whole -= frac > base;
  else whole += frac < base;
  // times the exponent, 64 fraction bits.
  constexpr unsigned long long kP = 0xa0ac9942cd841000ull;
  const unsigned long long a = (unsigned long long)abs(whole);
  unsigned long long hi = __umul64hi(a, kP), lo = a * kP;
  if (whole < 0) {
    hi = ~hi + (lo == 0);
    lo = 0ull - lo;
  }
  const unsigned long long f = lo + __umul64hi(frac, kP);
  const long long n = (long long)(hi + (f < lo));
  const unsigned long long y = exp2_fixed(f);
  return __longlong_as_double((long long)(((unsigned long long)(n + 1022) << 52) + (y >> 11) + ((y >> 10) & 1)));
}

}  // namespace rcg
