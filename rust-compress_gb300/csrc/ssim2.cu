// SSIMULACRA2 scorer kernels (K8-K10): the reference's core/src/ssimulacra2.rs on one GPU.
//
// Pipeline per score: one launch that takes both images (or a decoded candidate and a reference's linear pyramid) to the
// reference's XYB and the two images' XYB differences at every scale (f32, channel-planar; the 2x2 pyramid, scales 1..5,
// in shared memory) -> one launch that covers every tile of every scale (five moments, 11-tap blur, error maps, six
// partial sums per channel) -> a deterministic f64 reduction and the final 108-weight mapping.
//
// Arithmetic. The reference holds the planes in f32 and computes XYB, the blur, the maps and the sums in f64
// (:18, :345-346, :361). GB300's FP64 rate is a small fraction of its FP32 rate, so here:
//   * planes: f32 exactly as the reference (LUT values; the 2x2 average is a compensated sum that rounds like the
//     reference's f64 sum nearly always);
//   * XYB, blur and maps: f32, arranged so that nothing cancels catastrophically. Each pixel carries the reference
//     image's XYB and the XYB *difference* of the two images, both computed from cube-root difference identities
//     (see dsq2()); both are offset by their value at the tile centre, so the five blurred moments (mu_a, mu_(a-b),
//     E[a^2], E[b^2], E[(a-b)^2]) are small where the image is smooth. The variances and mu1 - mu2 are recovered
//     exactly from them (the offsets cancel wherever the blur taps sum to 1 and are corrected with the in-image tap
//     sum within 5 columns of the zero left/right border, :34-40). The SSIM term is evaluated as
//     (sigma_(a-b)^2 + (mu1-mu2)^2 num_s) / denom_s and the edge term from r1 = a - mu1 and its difference, forms
//     that equal the reference's expressions algebraically but keep full relative precision for similar images;
//   * cube roots: 2^(log2(x) / 3) from the hardware's approximate log2 and exp2 (relative error a few 1e-7; the
//     differences between the two images never go through them, only through the identity below);
//   * sums: f32 over the 8 pixels of a thread (in registers, then added to the thread's running sums of its band),
//     f32 across a warp, f64 from there on, in a fixed order (bit-reproducible from run to run, as the reference's
//     test :630 requires). What they round does not show in a score: against the FP64 scorer, over 25 pairs (flat, ramps,
//     photographs at four noise levels and four qualities, noise, gray; 23 of 9.4 MP), the error is 1.22e-6 on average and
//     8.3e-6 at most with bands of 1, 8 or 64 chunks; with half the pixels per thread and warp 1.24e-6 and 8.2e-6.
// Identical images give exactly 100: every difference term is exactly 0, so every map value is exactly 0.
#include <type_traits>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "rcg_internal.cuh"
#include "planes_quad.cuh"
#include "score_power.cuh"
#include "step_tables.cuh"

namespace rcg {

__constant__ float c_gauss[2 * kRadius + 1];
__constant__ float c_lut8s[256];
__constant__ double c_weights[108];

// core/src/ssimulacra2.rs:42-52 (opsin absorbance matrix and bias), as f32
constexpr double kM02 = 0.078, kM00 = 0.30, kM01 = 1.0 - kM02 - kM00;
constexpr double kM12 = 0.078, kM10 = 0.23, kM11 = 1.0 - kM12 - kM10;
constexpr double kM20 = 0.2434226892454782, kM21 = 0.2047674442449682, kM22 = 1.0 - kM20 - kM21;
constexpr double kBias = 0.0037930732552754493;

// Cube root of x > 0 as 2^(log2(x) / 3) with the hardware's approximate log2 and exp2 (a few ulp). The flush-to-zero
// forms: every argument here is at least the opsin bias (0.0038) and every result at least its cube root, so no
// subnormal can occur, and the forms without .ftz only add a range check and rescaling around each operation
// (measured: the tile kernel 608 -> 556 us per 12 MP score with these and the division below).
__device__ __forceinline__ float cbrt_fast(float x) {
  float l, y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
  l *= (1.0f / 3.0f);
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(l));
  return y;
}

// a / b as a * approximate(1 / b) (2 ulp), flush-to-zero form; the divisors below are normal and well inside the
// range where the reciprocal is defined.
__device__ __forceinline__ float fdiv_ftz(float a, float b) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// x^2 + x*y + y^2 = D(x, y) (dsq2): cbrt(u) - cbrt(v) = (u - v) / D(cbrt(u), cbrt(v)).
// Per pixel the scorer needs the reference image's XYB without its constants (`a`, core/src/ssimulacra2.rs:249-258 less
// kXyb0*) and XYB(reference) - XYB(distorted) (`d`). Every quantity that is a small difference of nearly equal cube
// roots is formed from the identity above, so it keeps its relative precision in f32: X - 0.42 = 7 (c0 - c1), B - 0.55 =
// ((c2 - c0) + (c2 - c1)) / 2, each c_i - c_j from the difference of two opsin-matrix rows applied to (r, g, b); and
// the per-pixel differences between the two images from the linear differences (r_a - r_b, ...).
// The constants of X, Y and B that `a` leaves out.
constexpr float kXyb0X = 0.42f, kXyb0Y = 0.01f, kXyb0B = 0.55f;

// Two pixels at a time, every step one packed two-lane operation: the conversion is bound by instruction issue, and this
// halves it but for the special functions. A difference a - b is fma(b, -1, a), which rounds once, as it does. The opsin
// sums are at least the bias: linear samples and the rows are not negative.
__device__ __forceinline__ float2 two(float k) { return make_float2(k, k); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, two(-1.0f), a); }
__device__ __forceinline__ float2 cbrt2(float2 x) {
  float2 l, y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l.x) : "f"(x.x));
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l.y) : "f"(x.y));
  l = __fmul2_rn(l, two(1.0f / 3.0f));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(l.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(l.y));
  return y;
}
__device__ __forceinline__ float2 div2(float2 a, float2 b) { return make_float2(fdiv_ftz(a.x, b.x), fdiv_ftz(a.y, b.y)); }
__device__ __forceinline__ float2 dsq2(float2 x, float2 y) {
  return __ffma2_rn(x, x, __ffma2_rn(x, y, __fmul2_rn(y, y)));
}
// m0 r + m1 g + m2 b + c, and without c.
__device__ __forceinline__ float2 row2(float m0, float m1, float m2, float2 r, float2 g, float2 b, float c) {
  return __ffma2_rn(two(m0), r, __ffma2_rn(two(m1), g, __ffma2_rn(two(m2), b, two(c))));
}
__device__ __forceinline__ float2 row2(float m0, float m1, float m2, float2 r, float2 g, float2 b) {
  return __ffma2_rn(two(m0), r, __ffma2_rn(two(m1), g, __fmul2_rn(two(m2), b)));
}

// The three opsin rows and the exact differences of rows, rounded once. Every row sums to one, so a difference of rows
// sums to zero: applied to (r, g, b) it is applied to (r - b, g - b) with its first two entries, which is exactly zero
// for a gray pixel, as the difference of its cube roots is.
constexpr float M00 = (float)kM00, M01 = (float)kM01, M02 = (float)kM02;
constexpr float M10 = (float)kM10, M11 = (float)kM11, M12 = (float)kM12;
constexpr float M20 = (float)kM20, M21 = (float)kM21, M22 = (float)kM22;
constexpr float L20r = (float)(kM20 - kM00), L20g = (float)(kM21 - kM01);
constexpr float L21r = (float)(kM20 - kM10), L21g = (float)(kM21 - kM11);

__device__ __forceinline__ float2 diff_row2(float m0, float m1, float2 rb, float2 gb) {
  return __ffma2_rn(two(m0), rb, __fmul2_rn(two(m1), gb));
}

// `a` of two pixels.
__device__ __forceinline__ void pix_xyb2(float2 r, float2 g, float2 b, float2 (&a)[3]) {
  const float bias = (float)kBias;
  const float2 c0 = cbrt2(row2(M00, M01, M02, r, g, b, bias)), c1 = cbrt2(row2(M10, M11, M12, r, g, b, bias)),
               c2 = cbrt2(row2(M20, M21, M22, r, g, b, bias));
  a[0] = __fmul2_rn(two(7.0f), div2(__fmul2_rn(two(0.07f), sub2(r, g)), dsq2(c0, c1)));
  a[1] = sub2(__fmul2_rn(two(0.5f), __fadd2_rn(c0, c1)), two(cbrt_fast(bias)));
  const float2 rb = sub2(r, b), gb = sub2(g, b);
  a[2] = __fmul2_rn(two(0.5f), __fadd2_rn(div2(diff_row2(L20r, L20g, rb, gb), dsq2(c2, c0)),
                                          div2(diff_row2(L21r, L21g, rb, gb), dsq2(c2, c1))));
}

// `d` of two pixels. The quotient difference q_a/D_a - q_b/D_b of a row pair is formed without cancellation as
// (dq D_b - q_b dD) / (D_a D_b), dq = q_a - q_b and dD = D_a - D_b from the cube roots' differences.
__device__ __forceinline__ void pix_diff2(float2 ra, float2 ga, float2 ba, float2 rb, float2 gb, float2 bb,
                                          float2 (&d)[3]) {
  const float bias = (float)kBias;
  const float2 ca0 = cbrt2(row2(M00, M01, M02, ra, ga, ba, bias)), cb0 = cbrt2(row2(M00, M01, M02, rb, gb, bb, bias));
  const float2 ca1 = cbrt2(row2(M10, M11, M12, ra, ga, ba, bias)), cb1 = cbrt2(row2(M10, M11, M12, rb, gb, bb, bias));
  const float2 ca2 = cbrt2(row2(M20, M21, M22, ra, ga, ba, bias)), cb2 = cbrt2(row2(M20, M21, M22, rb, gb, bb, bias));
  const float2 dr = sub2(ra, rb), dg = sub2(ga, gb), db = sub2(ba, bb);
  const float2 dc0 = div2(row2(M00, M01, M02, dr, dg, db), dsq2(ca0, cb0));
  const float2 dc1 = div2(row2(M10, M11, M12, dr, dg, db), dsq2(ca1, cb1));
  const float2 dc2 = div2(row2(M20, M21, M22, dr, dg, db), dsq2(ca2, cb2));
  d[1] = __fmul2_rn(two(0.5f), __fadd2_rn(dc0, dc1));
  const float2 s0 = __fadd2_rn(ca0, cb0), s1 = __fadd2_rn(ca1, cb1), s2 = __fadd2_rn(ca2, cb2);
  // nq = -q of image b; D(x, y) of image a minus of image b: dx (xa + xb) + dx ya + xb dy + dy (ya + yb)
  auto qd = [&](float2 nq, float2 dq, float2 cax, float2 cbx, float2 dcx, float2 sx, float2 cay, float2 cby, float2 dcy,
                float2 sy) {
    const float2 Da = dsq2(cax, cay), Db = dsq2(cbx, cby);
    const float2 dD = __ffma2_rn(dcx, sx, __ffma2_rn(dcx, cay, __ffma2_rn(cbx, dcy, __fmul2_rn(dcy, sy))));
    return div2(__ffma2_rn(dq, Db, __fmul2_rn(nq, dD)), __fmul2_rn(Da, Db));
  };
  const float2 q01 = qd(__fmul2_rn(two(0.07f), sub2(gb, rb)), __fmul2_rn(two(0.07f), sub2(dr, dg)), ca0, cb0, dc0, s0, ca1,
                        cb1, dc1, s1);
  d[0] = __fmul2_rn(two(7.0f), q01);
  const float2 rbb = sub2(rb, bb), gbb = sub2(gb, bb), drb = sub2(dr, db), dgb = sub2(dg, db);
  const float2 q20 = qd(diff_row2(-L20r, -L20g, rbb, gbb), diff_row2(L20r, L20g, drb, dgb), ca2, cb2, dc2, s2, ca0, cb0, dc0,
                        s0);
  const float2 q21 = qd(diff_row2(-L21r, -L21g, rbb, gbb), diff_row2(L21r, L21g, drb, dgb), ca2, cb2, dc2, s2, ca1, cb1, dc1,
                        s1);
  d[2] = __fmul2_rn(two(0.5f), __fadd2_rn(q20, q21));
}

// Gray pixels (r = g = b = l): X and B are constants without a difference between two gray images, which the conversions
// above give as exact zeros, so a gray image has only its Y; the steps are theirs, so it scores as its RGB copy does.
__device__ __forceinline__ float2 gray_root2(int row, float2 l) {
  const float bias = (float)kBias;
  return cbrt2(row ? row2(M10, M11, M12, l, l, l, bias) : row2(M00, M01, M02, l, l, l, bias));
}
__device__ __forceinline__ float2 gray_xyb2(float2 l) {
  return sub2(__fmul2_rn(two(0.5f), __fadd2_rn(gray_root2(0, l), gray_root2(1, l))), two(cbrt_fast((float)kBias)));
}
__device__ __forceinline__ float2 gray_diff2(float2 la, float2 lb) {
  const float2 d = sub2(la, lb);
  const float2 dc0 = div2(row2(M00, M01, M02, d, d, d), dsq2(gray_root2(0, la), gray_root2(0, lb)));
  const float2 dc1 = div2(row2(M10, M11, M12, d, d, d), dsq2(gray_root2(1, la), gray_root2(1, lb)));
  return __fmul2_rn(two(0.5f), __fadd2_rn(dc0, dc1));
}

// Row index under the top/bottom mirror rule (core/src/ssimulacra2.rs:385-397); -1 for rows no valid output reads.
__device__ __forceinline__ int mirror_row(int yy, int h) {
  if (yy < -kRadius || yy > h - 1 + kRadius) return -1;
  if (yy < 0) return -yy - 1;
  if (yy >= h) return 2 * h - 1 - yy;
  return yy;
}

// Shared-memory layout of one channel of a chunk: its `a` and its `d` samples of the 42 halo rows, columns x0 - 8 ..
// x0 + 39 (whole quads around the 42 that count). A row is 52 floats, 13 16-byte slots: odd, so the two rows that eight
// lanes of the horizontal pass read (16 bytes each, 32 apart) fall in each other's gaps.
constexpr int kIW = 52;
constexpr int kIH = kTileH + 2 * kRadius;  // 42
constexpr int kLead = 8;                   // columns left of x0 in a row
constexpr int kQuads = (kLead + kTileW + 8) / 4;  // 12 quads per row
constexpr int kXs = kIH * kIW;                    // floats of one of the two
// Blurred moments: the reading form keeps three per sample (one plane of pairs, one of singles), the others five.
constexpr int pair_planes(int ref_mode) { return ref_mode == kRefRead ? 1 : 2; }
constexpr size_t tile_smem(int ref_mode) {
  return (size_t)(2 * kXs + (2 * pair_planes(ref_mode) + 1) * kIH * kTileW) * sizeof(float);
}
constexpr int tile_ctas(int ref_mode) { return ref_mode == kRefRead ? kTileCtasRead : kTileCtas; }  // per SM
constexpr int kVy = kTileH / (kTileThreads / 32);  // vertical-pass outputs per thread

// Where the blurred planes' rows keep a column (a multiple of 4 and the three after it stay together): the permutation
// that puts the 16-byte stores of eight lanes (four items of each of two rows) in distinct banks.
__device__ __forceinline__ constexpr int hb_pair(int c, int r) { return c ^ (c >> 3 & 2) ^ (4 * (r & 1)); }
__device__ __forceinline__ constexpr int hb_one(int c, int r) { return c ^ (4 * (r & 1)); }

// 16 bytes from global to shared memory without passing through registers.
__device__ __forceinline__ void copy_quad(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// One tap of a blur chain; the first is the product alone (what fma gives with a zero sum).
__device__ __forceinline__ void tap_pair(float2& s, float2 k, float2 v, bool first) {
  s = first ? __fmul2_rn(k, v) : __ffma2_rn(k, v, s);
}
__device__ __forceinline__ void tap_one(float& s, float k, float v, bool first) {
  s = first ? __fmul_rn(k, v) : fmaf(k, v, s);
}

// One CTA = one band of 32 output columns and nch chunks of 32 output rows of one scale, walked top to bottom, from the
// reference's XYB planes (`a`) and the XYB differences (`d`). Per chunk and channel: the halo's samples are copied
// to shared memory asynchronously, the horizontal pass takes off the chunk's offsets and blurs the 42 halo rows, the
// vertical pass blurs the columns and evaluates the error maps while the next halo is on its way. The blurs run the
// moment pairs that share a tap weight as packed two-lane f32 FMAs, each lane exactly fmaf.
// Offsets: every chunk takes the XYB and XYB difference at its own centre.
// Band `local` of scale `sd` (sd.tiles_x bands across; sd.nch chunks each); the band's 18 sums go to out[i * stride],
// i < 18. one: the channel to score (its six sums are written), -1: all; every thread of the CTA passes the same.
// Reference moments (kRef). The offsets a chunk subtracts from `a` come from the reference alone, so the blurred a' and
// a'^2 of every output pixel depend on the reference and the band layout only. A search scores every candidate against
// one reference: its first candidate runs kRef = kRefWrite, which also stores (blur a', blur a'^2) per output pixel and
// channel; the later ones run kRef = kRefRead, which blur only (b'^2, d'^2) as a packed pair and d', and read the other
// two. Each blurred moment is the same chain of per-lane fmaf in every mode, so the scores are bit-identical to
// kRefNone. The store keeps each chunk's 3 x 32 x 32 pairs contiguous (24 KB, [channel][row][column]); a reading CTA
// asks for the whole block in L2 with one bulk prefetch per channel as the chunk starts and reads it in its vertical
// pass.
// What bounds it: instruction issue (79% active, the FP32 pipes 62%). Measured per 12 MP score, against a kernel that
// read both linear pyramids and converted every halo sample to XYB itself (1.5 conversions per pixel and half of its
// instructions): reading form 538 -> 277 us, storing 597 -> 361; plain 4K score 397 -> 239. Of that, the planes of XYB
// alone gave 420; loads by quads with the next channel's in registers beside the passes, and the maps without their edge
// cases inside the image, 349; eight outputs per thread in both passes with the halo copied asynchronously into one
// buffer 276 (387 with two buffers of converted pairs, which left room for 16 warps per SM). CTAs per SM: 6 reading (5
// measured 282, 4 287), 4 for the other forms (5 faster at 4K by 1%, slower in a batch by 4%). Quad offsets kept over a
// chunk's channels measured 278, the maps of two rows as packed operations 273 but 242 plain: neither was kept.
template <int kRef>
__device__ __forceinline__ void ssim2_band(const ScaleDesc sd, const int local, const int one,
                                           const float* __restrict__ xa, const float* __restrict__ xd,
                                           double* __restrict__ out, const size_t stride, float2* __restrict__ refm) {
  extern __shared__ float4 smem4[];
  float* const xs = reinterpret_cast<float*>(smem4);  // the channel's a, then its d
  // Horizontally blurred moments, [kIH][kTileW]: one plane of pairs (reading form) or two, then one of singles.
  float* const hb = xs + 2 * kXs;
  constexpr int kOnes = 2 * pair_planes(kRef) * kIH * kTileW;  // where the plane of singles starts
  __shared__ float s_red[kTileThreads / 32][kScoreSums];

  const int tx = local % sd.tiles_x, ty = local / sd.tiles_x;
  const int nch = sd.nch;
  const int x0 = tx * kTileW, ybeg = ty * kTileH * nch;
  const int w = sd.w, h = sd.h, pitch = sd.pitch;
  const size_t np = (size_t)pitch * h;
  // Channels to score: all, or Y alone (ScaleDesc::planes), which is then the only plane, or channel `one` of three.
  const bool split = one >= 0 && sd.planes != 1;
  if (one > 0 && !split) return;
  const int ch0 = sd.planes == 1 ? 1 : split ? one : 0, ch1 = sd.planes == 1 ? 2 : split ? one + 1 : 3;
  const float* pa = xa + sd.off + (split ? one * np : 0);  // the planes of channel ch0
  const float* pd = xd + sd.off + (split ? one * np : 0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  float sums[kScoreSums];
#pragma unroll
  for (int i = 0; i < kScoreSums; i++) sums[i] = 0.0f;
  // The blur's six distinct taps as (k, k) pairs, held in registers for the packed FMAs (the taps are symmetric:
  // tap t and tap 2 kRadius - t are the same f32 value).
  float2 g2[kRadius + 1];
#pragma unroll
  for (int t = 0; t <= kRadius; t++) g2[t] = make_float2(c_gauss[t], c_gauss[t]);
  auto tap = [&](int t) { return g2[t <= kRadius ? t : 2 * kRadius - t]; };

  const int col = lane, rg = warp;  // vertical pass: column, group of kVy output rows
  const int gx = x0 + col;
  // In-image tap sum of this column (1 except within kRadius of the left/right edge).
  const bool edge = gx < kRadius || gx >= w - kRadius;
  float K = 1.0f;
  if (edge) {
    K = 0.0f;
#pragma unroll
    for (int t = 0; t < 2 * kRadius + 1; t++) {
      int xx = gx + t - kRadius;
      if (xx >= 0 && xx < w) K += c_gauss[t];
    }
  }
  const float omk = 1.0f - K;

  const int nrun = min(nch, (h - ybeg + kTileH - 1) / kTileH);  // chunks of this band that lie in the image
  // The halo of one channel of a chunk: 42 rows x 12 quads. Rows follow the mirror rule; outside the left and right
  // border a' and d' are zero, so those samples hold the offsets themselves.
  auto centre_of = [&](int y0) {  // a plane has fewer than 2^32 samples
    return (unsigned)min(y0 + kTileH / 2, h - 1) * (unsigned)pitch + (unsigned)min(x0 + kTileW / 2, w - 1);
  };
  auto fetch = [&](int ch, int y0, float oa, float od) {
    const float* ca = pa + (ch - ch0) * np;
    const float* cd = pd + (ch - ch0) * np;
#pragma unroll
    for (int it = 0; it < (kIH * kQuads + kTileThreads - 1) / kTileThreads; it++) {
      const int e = tid + it * kTileThreads;
      if (e >= kIH * kQuads) break;
      const int r = e / kQuads, q = e - r * kQuads;
      const int gy = mirror_row(y0 - kRadius + r, h), gq = x0 - kLead + 4 * q;
      float* dst = xs + r * kIW + 4 * q;
      const unsigned at = (unsigned)gy * (unsigned)pitch + (unsigned)gq;
      if (gy >= 0 && gq >= 0 && gq + 4 <= w) {
        copy_quad(dst, ca + at);
        copy_quad(dst + kXs, cd + at);
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const bool in = gy >= 0 && gq >= 0 && gq + k < w;
          dst[k] = in ? __ldg(ca + at + k) : oa;
          dst[kXs + k] = in ? __ldg(cd + at + k) : od;
        }
      }
    }
  };

  float oa = __ldg(pa + centre_of(ybeg)), od = __ldg(pd + centre_of(ybeg));
  fetch(ch0, ybeg, oa, od);
#pragma unroll 1
  for (int chunk = 0; chunk < nrun; chunk++) {
    const int y0 = ybeg + chunk * kTileH;
    const unsigned centre = centre_of(y0);
    // Chunks whose halo and outputs all lie inside the image take the maps without their edge cases.
    const bool inner = x0 >= kRadius && x0 + kTileW + kRadius <= w && y0 + kTileH <= h;
    float2* rchunk = nullptr;  // this chunk's block of reference moments (kRefChunk float2)
    if constexpr (kRef != kRefNone) rchunk = refm + (size_t)(sd.chunk0 + local * nch + chunk) * kRefChunk;
    if constexpr (kRef == kRefRead) {
      // 8 KB per channel (16-byte aligned, as the bulk prefetch requires: blocks are 24 KB apart from an aligned base).
      if (tid >= ch0 && tid < ch1) {
        const float2* p = rchunk + tid * kTileH * kTileW;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(kTileH * kTileW * 8) : "memory");
      }
    }
#pragma unroll 1
    for (int ch = ch0; ch < ch1; ch++) {
      // The next halo: the next channel's, or the next chunk's first.
      const bool same = ch + 1 < ch1, more = same || chunk + 1 < nrun;
      const int nch_ = same ? ch + 1 : ch0, ny0 = same ? y0 : y0 + kTileH;
      float noa = 0.f, nod = 0.f;
      if (more) {
        const unsigned nc = centre_of(ny0);
        noa = __ldg(pa + (nch_ - ch0) * np + nc);
        nod = __ldg(pd + (nch_ - ch0) * np + nc);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // this halo is in place; the previous vertical pass is done with hb
      // Horizontal pass: NX adjacent outputs of row r from column c0 on. Moments a', d', a'^2, b'^2 (b' = a' - d'), d'^2
      // (reading form: (b'^2, d'^2) and d'). The row's pairs come in as 16-byte loads of two; every output's chain
      // takes its taps in ascending order.
      auto hitem = [&](auto nx, const int r, const int c0) {
        // Quads of columns c0 - 8 .. : tap position t (output o takes it as tap t - o) is sample t + 3.
        constexpr int NX = decltype(nx)::value, NT = NX + 2 * kRadius;
        static_assert(kLead - kRadius == 3, "samples before the first tap");
        const float4* xr = reinterpret_cast<const float4*>(xs + r * kIW + c0);
        [[maybe_unused]] float2 s0[NX];
        float2 s1[NX];
        float s4[NX];
#pragma unroll
        for (int g = 0; g < (NT + 3 + 3) / 4; g++) {
          const float4 qa = xr[g], qd = xr[kXs / 4 + g];
          const float va[4] = {qa.x, qa.y, qa.z, qa.w}, vd[4] = {qd.x, qd.y, qd.z, qd.w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const int t = 4 * g + k - 3;
            if (t < 0 || t >= NT) continue;
            const float2 ad = make_float2(__fsub_rn(va[k], oa), __fsub_rn(vd[k], od));
            const float bp = __fsub_rn(ad.x, ad.y);
            float2 sq;
            [[maybe_unused]] float bb = 0.f;
            if constexpr (kRef == kRefRead) {
              sq = __fmul2_rn(make_float2(bp, ad.y), make_float2(bp, ad.y));
            } else {
              sq = __fmul2_rn(ad, ad);
              bb = __fmul_rn(bp, bp);
            }
#pragma unroll
            for (int o = 0; o < NX; o++) {
              if (t - o < 0 || t - o > 2 * kRadius) continue;
              const float2 kk = tap(t - o);
              tap_pair(s1[o], kk, sq, t == o);
              if constexpr (kRef == kRefRead) {
                tap_one(s4[o], kk.x, ad.y, t == o);
              } else {
                tap_pair(s0[o], kk, ad, t == o);
                tap_one(s4[o], kk.x, bb, t == o);
              }
            }
          }
        }
        auto put_pairs = [&](float* plane, const float2* s) {
          float* d = plane + r * kTileW * 2;
#pragma unroll
          for (int o = 0; o < NX; o += 2)
            *reinterpret_cast<float4*>(d + 2 * hb_pair(c0 + o, r)) = make_float4(s[o].x, s[o].y, s[o + 1].x, s[o + 1].y);
        };
        if constexpr (kRef == kRefRead) {
          put_pairs(hb, s1);
        } else {
          put_pairs(hb, s0);
          put_pairs(hb + 2 * kIH * kTileW, s1);
        }
        float* h4 = hb + kOnes + r * kTileW;
#pragma unroll
        for (int o = 0; o < NX; o += 4)
          *reinterpret_cast<float4*>(h4 + hb_one(c0 + o, r)) = make_float4(s4[o], s4[o + 1], s4[o + 2], s4[o + 3]);
      };
      static_assert(kTileThreads == 128 && kTileH == 32 && kTileW == 32 && kIH - kTileH == 10, "item layout");
      // Rows 0..31: one item of 8 outputs per thread; eight lanes take the 4 items of each of 2 rows.
      hitem(std::integral_constant<int, 8>(), warp * 8 + (lane >> 2), 8 * (lane & 3));
      // The 10 halo rows below: 80 items of 4 outputs (eight lanes take 4 items of each of 2 rows).
      if (tid < (kIH - kTileH) * (kTileW / 4))
        hitem(std::integral_constant<int, 4>(), kTileH + warp * 4 + ((lane >> 2) & 1) + 2 * (lane >> 4),
              4 * ((lane & 3) + 4 * ((lane >> 3) & 1)));
      float ca0[kVy], cd0[kVy];  // this thread's samples, for the edge maps
#pragma unroll
      for (int o = 0; o < kVy; o++) {
        const float* x = xs + (rg * kVy + o + kRadius) * kIW + col + kLead;
        ca0[o] = __fsub_rn(x[0], oa);
        cd0[o] = __fsub_rn(x[kXs], od);
      }
      __syncthreads();
      if (more) fetch(nch_, ny0, noa, nod);
      // Vertical pass + error maps: kVy output rows of one column per thread, the same pairs packed.
      float2* rrow = nullptr;  // this thread's row 0 in the chunk's block
      if constexpr (kRef != kRefNone) rrow = rchunk + (ch * kTileH + rg * kVy) * kTileW + col;
      float2 rm[kVy];  // the reference moments: their loads overlap the blur
      if constexpr (kRef == kRefRead) {
#pragma unroll
        for (int o = 0; o < kVy; o++) {
          rm[o] = make_float2(0.f, 0.f);
          if (inner || (gx < w && y0 + rg * kVy + o < h)) rm[o] = __ldg(rrow + o * kTileW);
        }
      }
      [[maybe_unused]] float2 s0[kVy];
      float2 s1[kVy];
      float s4[kVy];
      {
        const float2* hp = reinterpret_cast<const float2*>(hb) + rg * kVy * kTileW;
        const float* h4 = hb + kOnes + rg * kVy * kTileW;
#pragma unroll
        for (int t = 0; t < kVy + 2 * kRadius; t++) {
          const float2* row = hp + t * kTileW + hb_pair(col, t);  // rg * kVy is even
          const float2 v0 = row[0];
          float2 v1 = v0;
          if constexpr (kRef != kRefRead) v1 = row[kIH * kTileW];
          const float v4 = h4[t * kTileW + hb_one(col, t)];
#pragma unroll
          for (int o = 0; o < kVy; o++) {
            if (t - o < 0 || t - o > 2 * kRadius) continue;
            const float2 kk = tap(t - o);
            tap_pair(s1[o], kk, v1, t == o);
            if constexpr (kRef != kRefRead) tap_pair(s0[o], kk, v0, t == o);
            tap_one(s4[o], kk.x, v4, t == o);
          }
        }
        if constexpr (kRef == kRefWrite) {
#pragma unroll
          for (int o = 0; o < kVy; o++)
            if (inner || (gx < w && y0 + rg * kVy + o < h)) rrow[o * kTileW] = make_float2(s0[o].x, s1[o].x);
        }
      }
      // The chunk's offsets with the constants of the channel (kXyb0*), for the corrections at the zero border.
      const float cd = od;
      const float ca = oa + (ch == 0 ? kXyb0X : ch == 1 ? kXyb0Y : kXyb0B), cbv = ca - cd;
      float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      auto maps = [&](auto inside) {
        constexpr bool kInside = decltype(inside)::value;
#pragma unroll
        for (int o = 0; o < kVy; o++) {
          int ry = rg * kVy + o;
          int gy = y0 + ry;
          if (kInside || (gx < w && gy < h)) {
            // Blurred primed moments -> sigma_1^2, sigma_2^2, sigma_(a-b)^2, mu1 - mu2 (exactly, given K).
            float m1, dmp, e11, e22, edd;
            if constexpr (kRef == kRefRead) {
              m1 = rm[o].x;
              e11 = rm[o].y;
              dmp = s4[o];
              e22 = s1[o].x;
              edd = s1[o].y;
            } else {
              m1 = s0[o].x;
              dmp = s0[o].y;
              e11 = s1[o].x;
              edd = s1[o].y;
              e22 = s4[o];
            }
            const float m2 = m1 - dmp;
            float v1 = fmaf(-m1, m1, e11);
            float v2 = fmaf(-m2, m2, e22);
            float vd = fmaf(-dmp, dmp, edd);
            float dmu;
            if (!kInside && edge) {
              v1 = fmaf(omk * ca, fmaf(ca, K, 2.0f * m1), v1);
              v2 = fmaf(omk * cbv, fmaf(cbv, K, 2.0f * m2), v2);
              vd = fmaf(omk * cd, fmaf(cd, K, 2.0f * dmp), vd);
              dmu = fmaf(cd, K, dmp);
            } else {
              dmu = dmp + cd;
            }
            // SSIM error (core/src/ssimulacra2.rs:427-430) as (sigma_(a-b)^2 + dmu^2 num_s) / denom_s, which equals
            // 1 - (1 - dmu^2) num_s / denom_s since num_s = denom_s - sigma_(a-b)^2.
            float den = (v1 + v2) + 0.0009f;
            float num_s = den - vd;
            float d = fmaxf(fdiv_ftz(fmaf(dmu * dmu, num_s, vd), den), 0.0f);
            // Edge maps (:431-433): d1 = (|r2| - |r1|) / (1 + |r1|) with r1 = a - mu1, r2 = b - mu2 = r1 - rd.
            float r1 = ca0[o] - m1, rd = cd0[o] - dmp;
            if (!kInside && edge) {
              r1 = fmaf(ca, omk, r1);
              rd = fmaf(cd, omk, rd);
            }
            // t is 0 (then so is the numerator) or far above the subnormal range: the residuals are differences of
            // f32 values of order 1e-3..1 and their blurs, so the flush-to-zero division sees a normal divisor.
            float t = fabsf(r1 - rd) + fabsf(r1);
            float d1 = t > 0.0f ? fdiv_ftz(-rd * (2.0f * r1 - rd), t * (1.0f + fabsf(r1))) : 0.0f;
            float art = fmaxf(d1, 0.0f), det = fmaxf(-d1, 0.0f);
            float d2 = d * d, a2 = art * art, e2 = det * det;
            acc[0] += d;
            acc[1] += d2 * d2;
            acc[2] += art;
            acc[3] += a2 * a2;
            acc[4] += det;
            acc[5] += e2 * e2;
          }
        }
      };
      if (inner) maps(std::true_type());
      else maps(std::false_type());
#pragma unroll
      for (int i = 0; i < 6; i++) sums[ch * 6 + i] += acc[i];
      oa = noa;
      od = nod;
    }
  }
  // Warp sums (f32, 32 threads x kVy pixels per chunk), then the warps in f64 in a fixed order. Sums 0..15 by a
  // reduce-scatter butterfly: at each exchange (lane distance 16, 8, 4, 2) a lane keeps half of the values it carries and adds its
  // partner's copy of that half, then distance 1 adds the pair; lane l ends with sum l >> 1. The additions are those
  // of a full butterfly per sum, so every sum has the same bits, in 16 shuffles instead of 80. Sums 16 and 17 by full
  // butterflies.
  {
    float a[16];
#pragma unroll
    for (int i = 0; i < 16; i++) a[i] = sums[i];
#pragma unroll
    for (int m = 8, off = 16; m >= 1; m >>= 1, off >>= 1) {
      const bool upper = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < m; i++) {
        const float keep = upper ? a[i + m] : a[i];
        const float send = upper ? a[i] : a[i + m];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    }
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    if ((lane & 1) == 0) s_red[warp][lane >> 1] = a[0];
  }
#pragma unroll
  for (int i = 16; i < kScoreSums; i++) {
    float v = sums[i];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0) s_red[warp][i] = v;
  }
  __syncthreads();
  if (tid < kScoreSums && (!split || tid / 6 == one)) {
    double acc = 0.0;
    for (int wi = 0; wi < kTileThreads / 32; wi++) acc += (double)s_red[wi][tid];
    out[(size_t)tid * stride] = acc;  // sum-major: the reduction reads each sum contiguously
  }
}

// Launches of few bands are latency-bound (a CTA's three channels one after the other): there each band is three CTAs, one
// per channel. The sums are per channel, so they are the same bits. Measured, whole bands / split: 66 bands (240x180)
// 17.9 / 10.6 us, 340 (512x512, without reference moments) 20.0 / 18.0, 977 (0.8 MP) 43.3 / 41.4, 2300 (1.7 MP) 56.5 /
// 57.5, 12 MP 278 / 304: a CTA's start and end weigh more once the bands fill the chip.
constexpr int kSplitTiles = 1024;
__device__ __forceinline__ int channel_of_cta() { return gridDim.y == 1 ? -1 : (int)blockIdx.y; }
dim3 tile_grid(long long ctas) { return dim3((unsigned)ctas, ctas <= kSplitTiles ? 3 : 1); }

template <int kRef>
__global__ void __launch_bounds__(kTileThreads, tile_ctas(kRef))
    k_ssim2_tiles(PyramidDesc pd, const float* __restrict__ ref, const float* __restrict__ dist,
                  double* __restrict__ partials, const StepDesc* __restrict__ st, float2* __restrict__ refm) {
  grid_chain();
  if (st && !st->active) return;
  const int blk = blockIdx.x;
  int s = 0;
  while (s + 1 < pd.nscales && blk >= pd.s[s + 1].tile0) s++;
  const ScaleDesc sd = pd.s[s];
  ssim2_band<kRef>(sd, blk - sd.tile0, channel_of_cta(), ref, dist, partials + blk, (size_t)pd.total_tiles, refm);
}

// Deterministic reduction of the per-tile sums: CTA (scale, sum index) of one score; the last of its nscales x 18 CTAs to
// finish computes the score (core/src/ssimulacra2.rs:457-511) and, in a search, advances the bisection
// (jpeg/src/target.rs:29-56) and fills the next step's tables.
// What bounds it: latency (partial sums, a counter, the last CTA's serial end) and FP64 operations, of which an SM starts
// a warp's only every 16 cycles or so: warps without sums or terms leave them out. What the end needs and no CTA writes
// (weights, sample counts, the search's state) is loaded at the start by every CTA, and the bisection works on a copy in
// shared memory. Measured at 240x180: 12.7 us with the next step's tables, from 12.5 and a launch of 5.0 for the tables
// (10 requantizing), whose lookups went through stack copies of the constant tables; a search 622 -> 567 us. The last CTA
// now takes 16,300 cycles: loads and sums 4900, counter 2300, terms 3050, power 2430, bisection 770, tables 2890.
__device__ __forceinline__ void reduce_scale_sum(const PyramidDesc& pd, const double* __restrict__ partials,
                                                 double* __restrict__ scale_sums, unsigned* __restrict__ counter,
                                                 double* __restrict__ score_out, SearchState* __restrict__ ss,
                                                 StepDesc* __restrict__ st, const NextStep& next) {
  constexpr int kStateWords = sizeof(SearchState) / 4;
  static_assert(kStateWords <= 256 && sizeof(SearchState) % 4 == 0, "copied a word per thread");
  __shared__ double red[8];
  __shared__ bool last;
  __shared__ __align__(8) int state[kStateWords];
  const int s = blockIdx.x, i = blockIdx.y, t = threadIdx.x;
  const ScaleDesc sd = pd.s[s];
  const int n = sd.tiles_x * sd.tiles_y;
  if (ss && t < kStateWords) state[t] = reinterpret_cast<const int*>(ss)[t];
  // Term t follows the reference's weight order: channel, scale, norm (mean, 4-norm), then (ssim, artifact, detail)
  // (core/src/ssimulacra2.rs:491-506).
  const int ns = pd.nscales, nterms = 3 * ns * 6;
  int from = 0, nrm = 0;
  double weight = 0.0, count = 1.0;
  if (t < nterms) {
    const int c = t / (ns * 6), rem = t % (ns * 6), sc = rem / 6, r2 = rem % 6, k = r2 % 3;
    nrm = r2 / 3;
    from = sc * kScoreSums + c * 6 + 2 * k + nrm;
    weight = c_weights[t];
    count = (double)pd.s[sc].w * (double)pd.s[sc].h;
  }
  StepPre pre = {};
  if (next.kind != kNextNone) pre = step_prepare(st, next);
  double acc = 0.0;
  const double* col = partials + (size_t)i * pd.total_tiles + sd.tile0;
  for (int u = t; u < n; u += 256) acc += col[u];
  const int warps = min(8, (n + 31) / 32);  // those that hold sums
  if ((t >> 5) < warps) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((t & 31) == 0) red[t >> 5] = acc;
  }
  __syncthreads();
  if (t == 0) {
    double tot = 0.0;
    for (int wi = 0; wi < warps; wi++) tot += red[wi];
    scale_sums[s * kScoreSums + i] = tot;
    __threadfence();
    unsigned prev = atomicAdd(counter, 1u);
    last = prev == (unsigned)(pd.nscales * kScoreSums) - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // The last CTA maps the per-scale sums to the score: one thread per term, then the terms summed by a fixed pairwise
  // tree (neighbours first; deterministic).
  double term = 0.0;
  if (t < nterms) {
    double v = reinterpret_cast<const volatile double*>(scale_sums)[from] / count;
    if (nrm == 1) v = sqrt(sqrt(v));  // (sum of 4th powers / count)^0.25 (:462)
    term = weight * fabs(v);
  }
  if (t < 128) {  // 108 terms at most
#pragma unroll
    for (int span = 1; span < 32; span *= 2) term += __shfl_down_sync(0xffffffffu, term, span);
    if ((t & 31) == 0) red[t >> 5] = term;
  }
  __syncthreads();
  SearchState* const copy = reinterpret_cast<SearchState*>(state);
  if (t == 0) {
    *counter = 0;
    double ssim = (red[0] + red[1]) + (red[2] + red[3]);
    ssim *= 0.9562382616834844;
    ssim = 2.326765642916932 * ssim - 0.020884521182843837 * ssim * ssim + 6.248496625763138e-05 * ssim * ssim * ssim;
    double score = ssim > 0.0 ? 100.0 - 10.0 * score_power(ssim) : 100.0;
    // A non-finite score is the reference's Err, which the search maps to f64::MIN (cli/src/pipeline.rs:218).
    bool finite = isfinite(score);
    *score_out = finite ? score : NAN;
    if (ss) search_record(copy, finite ? score : -1.7976931348623157e308);
  }
  if (!ss) return;
  __syncthreads();
  if (t < kStateWords) reinterpret_cast<int*>(ss)[t] = state[t];
  if (next.kind != kNextNone) step_tables_body(*copy, st, next, pre);
}

__global__ void __launch_bounds__(256) k_ssim2_reduce(const __grid_constant__ PyramidDesc pd,
                                                      const double* __restrict__ partials,
                                                      double* __restrict__ scale_sums, unsigned* __restrict__ counter,
                                                      double* __restrict__ score_out, SearchState* __restrict__ ss,
                                                      StepDesc* __restrict__ st, const NextStep next) {
  grid_chain();
  if (st && !st->active) return;
  reduce_scale_sum(pd, partials, scale_sums, counter, score_out, ss, st, next);
}

// ------------------------------------------------------------------------------------------------ planes, pyramid

// An interleaved image's samples (core/src/ssimulacra2.rs:177-221, with core/src/image.rs:143-190 for alpha: 16-bit
// samples rounded to 8 bits, then composited onto mid-grey 128).
struct ImageSrc {
  const uint8_t* img;
  int w, h, channels, depth;
  const float* lut16;  // 65536-entry table for 16-bit samples without alpha
};

// Linear light of four consecutive pixels of row y (columns x0 .. x0+3, zero beyond the row). lut8: the 8-bit table in
// shared memory.
__device__ __forceinline__ void image_quad(const ImageSrc& im, int x0, int y, const float* lut8, float (&v)[3][4]) {
  const uint8_t* img = im.img;
  const int w = im.w, channels = im.channels, depth = im.depth;
  const float* lut16 = im.lut16;
  const size_t i0 = (size_t)y * w + x0;
  const int n = min(4, w - x0);
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int k = 0; k < 4; k++) v[c][k] = 0.f;
  const bool alpha = channels == 2 || channels == 4;
  const uintptr_t at = (uintptr_t)(img + i0 * 3);
  const int mis = (int)(at & 3);
  // 12 bytes of any alignment: the aligned words that hold them and a funnel shift; the fourth word only where the
  // image goes on past it (the image may end, or start, at any byte of a caller's buffer).
  if (depth == 8 && channels == 3 && n == 4 && i0 * 3 >= (size_t)mis &&
      (mis == 0 || i0 * 3 + 16 - mis <= (size_t)w * im.h * 3)) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(at - mis);
    const uint32_t w0 = p[0], w1 = p[1], w2 = p[2], w3 = mis ? p[3] : 0u;
    const uint32_t q0 = __funnelshift_r(w0, w1, 8 * mis), q1 = __funnelshift_r(w1, w2, 8 * mis),
                   q2 = __funnelshift_r(w2, w3, 8 * mis);
    uint32_t b[12] = {q0 & 0xFF, (q0 >> 8) & 0xFF, (q0 >> 16) & 0xFF, q0 >> 24, q1 & 0xFF, (q1 >> 8) & 0xFF,
                      (q1 >> 16) & 0xFF, q1 >> 24, q2 & 0xFF, (q2 >> 8) & 0xFF, (q2 >> 16) & 0xFF, q2 >> 24};
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int c = 0; c < 3; c++) v[c][k] = lut8[b[3 * k + c]];
  } else {
    for (int k = 0; k < n; k++) {
      size_t i = i0 + k;
      if (depth == 8 && !alpha) {
        if (channels == 1) {
          v[0][k] = v[1][k] = v[2][k] = lut8[img[i]];
        } else {
          v[0][k] = lut8[img[i * 3]];
          v[1][k] = lut8[img[i * 3 + 1]];
          v[2][k] = lut8[img[i * 3 + 2]];
        }
      } else if (!alpha) {
        auto s16 = [&](int c) -> unsigned {
          const uint8_t* p = img + (i * channels + c) * 2;
          return ((unsigned)p[0] << 8) | p[1];
        };
        if (channels == 1) {
          v[0][k] = v[1][k] = v[2][k] = lut16[s16(0)];
        } else {
          v[0][k] = lut16[s16(0)];
          v[1][k] = lut16[s16(1)];
          v[2][k] = lut16[s16(2)];
        }
      } else {
        unsigned sm[4];
        for (int c = 0; c < channels; c++) {
          if (depth == 8) {
            sm[c] = img[i * channels + c];
          } else {
            const uint8_t* p = img + (i * channels + c) * 2;
            unsigned u = ((unsigned)p[0] << 8) | p[1];
            sm[c] = (u * 255 + 32767) / 65535;
          }
        }
        unsigned a = sm[channels - 1];
        auto blend = [&](unsigned c) -> unsigned { return (c * a + 128u * (255 - a) + 127) / 255; };
        if (channels == 2) {
          v[0][k] = v[1][k] = v[2][k] = lut8[blend(sm[0])];
        } else {
          v[0][k] = lut8[blend(sm[0])];
          v[1][k] = lut8[blend(sm[1])];
          v[2][k] = lut8[blend(sm[2])];
        }
      }
    }
  }
}

// Linear planes [3][h][pitch] of an image (the reference-order scorer's input).
__global__ void __launch_bounds__(256) k_to_linear(const ImageSrc im, int pitch, float* __restrict__ out) {
  grid_chain();
  // The table lives in shared memory: per-thread indices differ, which would serialize constant-memory reads.
  __shared__ float lut8[256];
  lut8[threadIdx.x] = c_lut8s[threadIdx.x];
  __syncthreads();
  const int groups = (im.w + 3) / 4;
  const long long g = (long long)blockIdx.x * 256 + threadIdx.x, y = g / groups;
  if (y >= im.h) return;
  const int x0 = 4 * (int)(g - y * groups);
  float v[3][4];
  image_quad(im, x0, (int)y, lut8, v);
  const size_t np = (size_t)pitch * im.h, o = (size_t)y * pitch + x0;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (x0 + k < im.w)
#pragma unroll
      for (int c = 0; c < 3; c++) out[c * np + o + k] = v[c][k];
}

// Error-free transform: s + e == a + b exactly (Knuth's TwoSum).
__device__ __forceinline__ float two_sum(float a, float b, float& e) {
  float s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return s;
}

// Mean of a 2x2 block (q0 q1 above q2 q3) of which the right column and the lower row may lie outside the image, as
// downsample (core/src/ssimulacra2.rs:223-247) computes it: the reference sums in f64, which is exact for these inputs,
// then rounds once to f32; the compensated sum here (TwoSum, in the reference's order) rounds the same exact sum once, so
// the planes agree with the reference's except in rare double-rounding cases. The scaling is exact.
__device__ __forceinline__ float block_mean(float q0, float q1, float q2, float q3, bool right, bool below) {
  float e0 = 0.f, e1 = 0.f, e2 = 0.f;
  float s = q0;
  if (right) s = two_sum(s, q1, e0);
  if (below) s = two_sum(s, q2, e1);
  if (right && below) s = two_sum(s, q3, e2);
  return __fadd_rn(s, (e0 + e1) + e2) * (right ? (below ? 0.25f : 0.5f) : (below ? 0.5f : 1.0f));
}

// ---- pyramid builder
//
// One launch takes an image (or two) from its source to everything the scorer reads, at every scale: one CTA per 64x64
// block of scale 0 and the 32x32 .. 2x2 blocks of scales 1-5 below it, which nest exactly because each level halves the
// one above. Sixteen rows of the block at a time, each thread converts a quad (four samples of a row) to linear light,
// writes what the scorer needs of it and passes the linear samples on: a row pair sits in one warp, whose halves exchange
// two samples per channel and make one scale-1 sample each, kept in shared memory. Every coarser level is made from the
// one above in shared memory and written by quads. Linear planes exist in memory only where a later launch reads them
// (a search's reference).
// What bounds it: instruction issue in the colour conversion (69% active; packed in pairs of pixels), then the latency of
// a quad's loads. Measured per 12 MP candidate of a 4:2:0 search: 133 us, the tile kernel then 276 (62 us when this step
// wrote linear planes and the tile kernel converted them to XYB in every halo, 538); 154 us with one thread per 4x4
// block converting its four rows in turn, each waiting for the reference's samples; 168 us with each level written as it
// was made, its few threads' loads between two barriers; 142 us at 3 CTAs per SM instead of 4. A 4K pair: 130 us where
// linear planes, pyramids and their conversion took 228 (two launches each of the first two); 151 us at 2 CTAs per SM
// instead of 3. Layouts other than 4:2:0 with a width divisible by 4 took two launches: 1283x857, mostly 4:4:4,
// 44 -> 24 us per candidate, gray 1653x2339 76 -> 55.
enum BuildSrc { kFromPlanes, kFromLinear, kFromImage };
enum BuildOut {
  kOutDiff,  // differences against ref (linear) -> out
  kOutRef,   // linear -> out, XYB -> xyb
  kOutPair   // two images: XYB of the first -> xyb, differences -> out
};
struct BuildArgs {
  float* out;
  float* xyb;
  const float* ref;
  const uint8_t* planes;  // kFromPlanes: decoded components of the layout in st
  const StepDesc* st;
  ImageSrc im[2];         // kFromImage
};

constexpr int kPyrT = 64;       // scale-0 block of a CTA
constexpr int kPyrTSmall = 32;  // of a small image (kSmallBuild)
constexpr int kPyrThreads = 256;
// Rows of a level's block in shared memory, padded so that quads stay 16-byte aligned; where each level starts.
__device__ __forceinline__ constexpr int lev_pitch(int T, int L) { return (T >> L) + 4; }
__device__ __forceinline__ constexpr int lev_off(int T, int L) {
  int o = 0;
  for (int k = 1; k < L; k++) o += lev_pitch(T, k) * (T >> k);
  return o;
}
constexpr int kLevFloats = 36 * 32 + 20 * 16 + 12 * 8 + 8 * 4 + 6 * 2;  // one channel's levels 1-5 (of the larger block)

static int blocks_of(const PyramidDesc& pd, int t) { return ((pd.s[0].w + t - 1) / t) * ((pd.s[0].h + t - 1) / t); }

int pyramid_ctas(const PyramidDesc& pd) { return blocks_of(pd, kPyrT); }

__device__ __forceinline__ void put4(float* __restrict__ p, size_t np, const float2 (&v)[2][3]) {
#pragma unroll
  for (int c = 0; c < 3; c++)
    *reinterpret_cast<float4*>(p + c * np) = make_float4(v[0][c].x, v[0][c].y, v[1][c].x, v[1][c].y);
}

// The reference's linear samples of quad (x, y) of a scale (kOutDiff), asked for before the image's own are converted.
template <int kOut, bool kGray>
__device__ __forceinline__ void ref_quad(const BuildArgs& g, const ScaleDesc& sd, int x, int y, float4 (&r)[3]) {
  if constexpr (kOut == kOutDiff) {
    const size_t np = (size_t)sd.pitch * sd.h, i = (size_t)sd.off + (size_t)y * sd.pitch + x;
#pragma unroll
    for (int c = 0; c < (kGray ? 1 : 3); c++) r[c] = __ldg(reinterpret_cast<const float4*>(g.ref + c * np + i));
  }
}

// Write quad (x, y) of a scale: l the linear samples of the image (kOutPair: of the first, l2 of the second), rq its
// ref_quad.
template <int kOut, bool kGray>
__device__ __forceinline__ void emit_quad(const BuildArgs& g, const ScaleDesc& sd, int x, int y, const float4 (&rq)[3],
                                          const float (&l)[3][4], const float (&l2)[3][4]) {
  const size_t np = (size_t)sd.pitch * sd.h, i = (size_t)sd.off + (size_t)y * sd.pitch + x;
  auto at = [](const float (&v)[3][4], int c, int k) { return make_float2(v[c][2 * k], v[c][2 * k + 1]); };
  if constexpr (kGray) {
    auto put = [&](float* p, auto f) {
      const float2 a = f(0), b = f(1);
      *reinterpret_cast<float4*>(p + i) = make_float4(a.x, a.y, b.x, b.y);
    };
    if constexpr (kOut == kOutDiff) {
      put(g.out, [&](int k) {
        return gray_diff2(k ? make_float2(rq[0].z, rq[0].w) : make_float2(rq[0].x, rq[0].y), at(l, 0, k));
      });
    } else {
      put(g.xyb, [&](int k) { return gray_xyb2(at(l, 0, k)); });
      if constexpr (kOut == kOutRef) put(g.out, [&](int k) { return at(l, 0, k); });
      else put(g.out, [&](int k) { return gray_diff2(at(l, 0, k), at(l2, 0, k)); });
    }
    return;
  }
  float2 o[2][3];
  if constexpr (kOut == kOutDiff) {
    float r[3][4];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      r[c][0] = rq[c].x;
      r[c][1] = rq[c].y;
      r[c][2] = rq[c].z;
      r[c][3] = rq[c].w;
    }
#pragma unroll
    for (int k = 0; k < 2; k++)
      pix_diff2(at(r, 0, k), at(r, 1, k), at(r, 2, k), at(l, 0, k), at(l, 1, k), at(l, 2, k), o[k]);
    put4(g.out + i, np, o);
  } else {
#pragma unroll
    for (int k = 0; k < 2; k++) pix_xyb2(at(l, 0, k), at(l, 1, k), at(l, 2, k), o[k]);
    put4(g.xyb + i, np, o);
    if constexpr (kOut == kOutRef) {
#pragma unroll
      for (int c = 0; c < 3; c++)
        *reinterpret_cast<float4*>(g.out + c * np + i) = make_float4(l[c][0], l[c][1], l[c][2], l[c][3]);
    } else {
#pragma unroll
      for (int k = 0; k < 2; k++)
        pix_diff2(at(l, 0, k), at(l, 1, k), at(l, 2, k), at(l2, 0, k), at(l2, 1, k), at(l2, 2, k), o[k]);
      put4(g.out + i, np, o);
    }
  }
}

// The two samples of a row of a level's 2x2 block, or its only one (`single`).
template <int kOut, bool kGray>
__device__ __forceinline__ void emit_pair(const BuildArgs& g, const ScaleDesc& sd, int x, int y, bool single,
                                          const float (&l)[3][4], const float (&l2)[3][4]) {
  const size_t np = (size_t)sd.pitch * sd.h, i = (size_t)sd.off + (size_t)y * sd.pitch + x;
  auto at = [](const float (&v)[3][4], int c) { return make_float2(v[c][0], v[c][1]); };
  auto put2 = [&](float* p, const float2 (&v)[3]) {
#pragma unroll
    for (int c = 0; c < (kGray ? 1 : 3); c++) {
      if (single) p[c * np + i] = v[c].x;
      else *reinterpret_cast<float2*>(p + c * np + i) = v[c];
    }
  };
  float2 o[3];
  if constexpr (kOut == kOutDiff) {
    float2 r[3];
#pragma unroll
    for (int c = 0; c < (kGray ? 1 : 3); c++) {
      const float* q = g.ref + c * np + i;
      r[c] = single ? make_float2(__ldg(q), 0.f) : __ldg(reinterpret_cast<const float2*>(q));
    }
    if constexpr (kGray) o[0] = gray_diff2(r[0], at(l, 0));
    else pix_diff2(r[0], r[1], r[2], at(l, 0), at(l, 1), at(l, 2), o);
    put2(g.out, o);
  } else {
    if constexpr (kGray) o[0] = gray_xyb2(at(l, 0));
    else pix_xyb2(at(l, 0), at(l, 1), at(l, 2), o);
    put2(g.xyb, o);
    if constexpr (kOut == kOutRef) {
      const float2 v[3] = {at(l, 0), at(l, 1), at(l, 2)};
      put2(g.out, v);
    } else {
      if constexpr (kGray) o[0] = gray_diff2(at(l, 0), at(l2, 0));
      else pix_diff2(at(l, 0), at(l, 1), at(l, 2), at(l2, 0), at(l2, 1), at(l2, 2), o);
      put2(g.out, o);
    }
  }
}

// Block `blk` of a pyramid. Every thread of the CTA calls it.
template <int kSrc, int kOut, bool kGray, int T>
__device__ __forceinline__ void build_planes(const PyramidDesc& pd, const BuildArgs& g, const int blk, float* lut,
                                             float (*lev)[3][kLevFloats]) {
  constexpr int kImgs = kOut == kOutPair ? 2 : 1, kCh = kGray ? 1 : 3;
  constexpr int kRowQuads = T / 4, kRows = kPyrThreads / kRowQuads;  // of a slab
  const int t = threadIdx.x, lane = t & 31;
  if constexpr (kSrc != kFromLinear) {
    lut[t] = c_lut8s[t];
    __syncthreads();
  }
  const ScaleDesc s0 = pd.s[0];
  const int w = s0.w, h = s0.h;
  const int bx = (w + T - 1) / T, tx = blk % bx, ty = blk / bx;
  const int quad = t % kRowQuads, x0 = tx * T + 4 * quad;
  const bool lower = (lane & kRowQuads) != 0;  // the odd row of a row pair
#pragma unroll 1
  for (int slab = 0; slab < T / kRows; slab++) {
    const int y = ty * T + slab * kRows + t / kRowQuads;
    if (ty * T + slab * kRows >= h) break;
    float l[kImgs][3][4];
    if (x0 < w && y < h) {
      float4 rq[3];
      ref_quad<kOut, kGray>(g, s0, x0, y, rq);
      if constexpr (kSrc == kFromPlanes) {
        planes_quad(g.st, g.planes, w, h, lut, x0, y, l[0]);
      } else if constexpr (kSrc == kFromLinear) {
#pragma unroll
        for (int c = 0; c < kCh; c++) {
          const float4 q = *reinterpret_cast<const float4*>(g.out + s0.off + c * (size_t)s0.pitch * h +
                                                            (size_t)y * s0.pitch + x0);
          l[0][c][0] = q.x;
          l[0][c][1] = q.y;
          l[0][c][2] = q.z;
          l[0][c][3] = q.w;
        }
      } else {
#pragma unroll
        for (int m = 0; m < kImgs; m++) image_quad(g.im[m], x0, y, lut, l[m]);
      }
      emit_quad<kOut, kGray>(g, s0, x0, y, rq, l[0], l[kImgs - 1]);
    }
    // Scale 1: the row pair's upper lane makes the quad's left sample, the lower one its right one.
    if (pd.nscales > 1) {
      const int col = x0 + (lower ? 2 : 0), top = y - (lower ? 1 : 0);
#pragma unroll
      for (int m = 0; m < kImgs; m++)
#pragma unroll
        for (int c = 0; c < kCh; c++) {
          const float p0 = __shfl_xor_sync(0xffffffffu, lower ? l[m][c][0] : l[m][c][2], kRowQuads);
          const float p1 = __shfl_xor_sync(0xffffffffu, lower ? l[m][c][1] : l[m][c][3], kRowQuads);
          const float v = lower ? block_mean(p0, p1, l[m][c][2], l[m][c][3], col + 1 < w, top + 1 < h)
                                : block_mean(l[m][c][0], l[m][c][1], p0, p1, col + 1 < w, top + 1 < h);
          lev[m][c][(slab * kRows + t / kRowQuads) / 2 * lev_pitch(T, 1) + 2 * quad + (lower ? 1 : 0)] = v;
        }
    }
  }
  // Coarser levels, each from the one above in shared memory (level 1 is in place).
#pragma unroll
  for (int L = 2; L < kMaxScales; L++) {
    __syncthreads();
    if (L >= pd.nscales) break;
    const int n = T >> L;
    if (t < n * n) {
      const int lx = t % n, ly = t / n;
      const int ax = 2 * (tx * n + lx), ay = 2 * (ty * n + ly);  // the block's origin in the level above
      const int aw = pd.s[L - 1].w, ah = pd.s[L - 1].h;
      if (ax < aw && ay < ah) {
#pragma unroll
        for (int m = 0; m < kImgs; m++)
#pragma unroll
          for (int c = 0; c < kCh; c++) {
            const float* q = &lev[m][c][lev_off(T, L - 1) + 2 * ly * lev_pitch(T, L - 1) + 2 * lx];
            lev[m][c][lev_off(T, L) + ly * lev_pitch(T, L) + lx] =
                block_mean(q[0], q[1], q[lev_pitch(T, L - 1)], q[lev_pitch(T, L - 1) + 1], ax + 1 < aw, ay + 1 < ah);
          }
      }
    }
  }
  __syncthreads();
  // Then written. Of a 64 block: the 256 quads of level 1, and in a second trip the 84 of levels 2-4 and the two pairs of
  // level 5. Of a 32 block, in one: the 84 quads of levels 1-3, the two pairs of level 4 and the sample of level 5.
#pragma unroll 1
  for (int trip = 0; trip < (T == 64 ? 2 : 1); trip++) {
    int L = 1, e = t;
    if (T == 32 || trip) {
      if (t >= (T == 64 ? 86 : 87)) break;
      const int k = t < 64 ? 0 : t < 80 ? 1 : t < 84 ? 2 : t < 86 ? 3 : 4;
      L = k + (T == 64 ? 2 : 1);
      e = t - (k == 0 ? 0 : k == 1 ? 64 : k == 2 ? 80 : k == 3 ? 84 : 86);
    }
    if (L >= pd.nscales) continue;
    const ScaleDesc sd = pd.s[L];
    const int n = T >> L, nq = n < 4 ? 1 : n / 4;  // quads of a row (a pair or a sample counts as one)
    const int lx = 4 * (e % nq), ly = e / nq;
    const int x = tx * n + lx, y = ty * n + ly;
    if (x >= sd.w || y >= sd.h) continue;
    const int at = (L == 1 ? lev_off(T, 1) : L == 2 ? lev_off(T, 2) : L == 3 ? lev_off(T, 3) : L == 4 ? lev_off(T, 4)
                                                                                                 : lev_off(T, 5)) +
                   ly * (n + 4) + lx;
    float l[kImgs][3][4];
#pragma unroll
    for (int m = 0; m < kImgs; m++)
#pragma unroll
      for (int c = 0; c < kCh; c++) {
        // a row is padded by four samples, so the quad of a pair or a single sample stays in its row
        const float2 a = *reinterpret_cast<const float2*>(&lev[m][c][at]);
        const float2 b = *reinterpret_cast<const float2*>(&lev[m][c][at + 2]);
        l[m][c][0] = a.x;
        l[m][c][1] = a.y;
        l[m][c][2] = b.x;
        l[m][c][3] = b.y;
      }
    if (n >= 4) {
      float4 rq[3];
      ref_quad<kOut, kGray>(g, sd, x, y, rq);
      emit_quad<kOut, kGray>(g, sd, x, y, rq, l[0], l[kImgs - 1]);
    } else {
      emit_pair<kOut, kGray>(g, sd, x, y, n == 1, l[0], l[kImgs - 1]);
    }
  }
}

// Of either kind (the work-lists, whose images may be mixed).
template <int kSrc, int kOut, int T>
__device__ __forceinline__ void build_block(const PyramidDesc& pd, const BuildArgs& g, const int blk) {
  __shared__ float lut[256];
  __shared__ __align__(16) float lev[kOut == kOutPair ? 2 : 1][3][kLevFloats];
  if (pd.s[0].planes == 1) build_planes<kSrc, kOut, true, T>(pd, g, blk, lut, lev);
  else build_planes<kSrc, kOut, false, T>(pd, g, blk, lut, lev);
}

// CTAs per SM: a pair's conversion keeps two images' samples in registers.
constexpr int build_ctas(int out) { return out == kOutPair ? 3 : 4; }

template <int kSrc, int kOut, bool kGray, int T>
__global__ void __launch_bounds__(kPyrThreads, build_ctas(kOut)) k_build(const __grid_constant__ PyramidDesc pd,
                                                                        const __grid_constant__ BuildArgs g,
                                                                        const StepDesc* __restrict__ gate) {
  grid_chain();
  if (gate && !gate->active) return;
  __shared__ float lut[256];
  __shared__ __align__(16) float lev[kOut == kOutPair ? 2 : 1][3][kLevFloats];
  build_planes<kSrc, kOut, kGray, T>(pd, g, blockIdx.x, lut, lev);
}

// Images of at most this many 64x64 blocks are built by 32x32 blocks: one slab of level 0 and one trip for the others per
// CTA, where a 64 block takes four and two, one after the other. The same samples either way. Measured, 64 / 32: 12 blocks
// (240x180) 16.6 / 10.7 us, 64 (512x512, a pair) 22.8 / 14.9, 294 (0.8 MP) 24.4 / 26.4, 442 (1.7 MP) 30.8 / 35.0: most
// threads of a 32 block idle while the levels above 0 are converted.
constexpr int kSmallBuild = kSms;

// Queue one builder launch (st: the step that gates it, nullable). Samples that come as linear planes are never gray
// ones: a gray layout is always read directly.
template <int kSrc, int kOut>
void launch_build(const PyramidDesc& pd, const BuildArgs& g, const StepDesc* st, cudaStream_t stream) {
  constexpr bool kGray = kSrc != kFromLinear;
  const int ctas = pyramid_ctas(pd);
  if (ctas <= kSmallBuild) {
    const int n = blocks_of(pd, kPyrTSmall);
    if (kGray && pd.s[0].planes == 1)
      launch_chained(n, kPyrThreads, 0, stream, k_build<kSrc, kOut, kGray, kPyrTSmall>, pd, g, st);
    else
      launch_chained(n, kPyrThreads, 0, stream, k_build<kSrc, kOut, false, kPyrTSmall>, pd, g, st);
  } else if (kGray && pd.s[0].planes == 1) {
    launch_chained(ctas, kPyrThreads, 0, stream, k_build<kSrc, kOut, kGray, kPyrT>, pd, g, st);
  } else {
    launch_chained(ctas, kPyrThreads, 0, stream, k_build<kSrc, kOut, false, kPyrT>, pd, g, st);
  }
}

// ------------------------------------------------------------------------------------------------ work-list scorer

// Many (reference, distorted) pairs of any sizes scored together: one launch per stage over a work-list of every
// pair's CTAs (pyramids, scorer tiles, reductions). Each stage's CTA finds its job by a binary search over the jobs'
// first-CTA indices. Pairs that name the same reference (same device pointer, size and format) share one conversion of
// it: such a reference is built first (linear and XYB), then its pairs' differences; a reference of one pair is built
// with it, without linear planes.
struct ScoreItem {
  PyramidDesc pd;
  long long tile0;  // first tile of this pair
  long long part;   // first double of this pair's [18][total_tiles] partial sums
};

// One pyramid (or pair of them) in a builder work-list.
struct BuildJob {
  PyramidDesc pd;
  BuildArgs args;
};

// One scale of one pair in the tile work-list, with everything a tile needs resolved on the host.
struct TileSeg {
  const float* ref;   // channel 0 of this scale's XYB planes
  const float* dist;  // and of its differences
  double* out;        // partial sums of the segment's first band; band k, sum i at out[i * stride + k]
  int w, h, pitch, planes, tiles_x;
  int nch;            // chunks per band
  int stride;         // bands of the pair (the sum-major stride of its partials)
};

// Last index whose first entry is <= x in an ascending array of first indices (n >= 1, first[0] = 0).
__device__ __forceinline__ int find_first(const long long* __restrict__ first, int n, long long x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(first + mid) <= x)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

template <int kSrc, int kOut, int T>
__global__ void __launch_bounds__(kPyrThreads, build_ctas(kOut)) k_build_batch(const BuildJob* __restrict__ jobs,
                                                                              const long long* __restrict__ cta0, int n) {
  grid_chain();
  const int i = find_first(cta0, n, blockIdx.x);
  const BuildJob& j = jobs[i];
  build_block<kSrc, kOut, T>(j.pd, j.args, (int)((long long)blockIdx.x - __ldg(cta0 + i)));
}

// One CTA per tile of the work-list. A persistent form (a fixed grid of k CTAs per SM striding over the list, each
// CTA reusing its shared memory tile after tile) measured slower on 64 pairs of mixed sizes: 22.7 / 25.4 / 38.9 ms
// at k = 3 / 2 / 1 against 21.1 ms here, because the block scheduler hands tiles to whichever CTA slot frees first.
__global__ void __launch_bounds__(kTileThreads, tile_ctas(kRefNone))
    k_ssim2_tiles_batch(const TileSeg* __restrict__ segs, const long long* __restrict__ seg0, int nseg) {
  grid_chain();
  const long long t = blockIdx.x;
  const int g = find_first(seg0, nseg, t);
  const TileSeg sg = segs[g];
  ScaleDesc sd;
  sd.w = sg.w;
  sd.h = sg.h;
  sd.pitch = sg.pitch;
  sd.planes = sg.planes;
  sd.tiles_x = sg.tiles_x;
  sd.tiles_y = 0;
  sd.tile0 = 0;
  sd.nch = sg.nch;
  sd.off = 0;
  const int local = (int)(t - __ldg(seg0 + g));
  ssim2_band<kRefNone>(sd, local, channel_of_cta(), sg.ref, sg.dist, sg.out + local, (size_t)sg.stride, nullptr);
}

// CTA (scale, sum, pair); scale_sums [n][kMaxScales][18], counters and scores [n].
__global__ void __launch_bounds__(256) k_ssim2_reduce_batch(const ScoreItem* __restrict__ items,
                                                            const double* __restrict__ partials,
                                                            double* __restrict__ scale_sums,
                                                            unsigned* __restrict__ counters,
                                                            double* __restrict__ scores) {
  grid_chain();
  const int p = blockIdx.z;
  const ScoreItem& it = items[p];
  if ((int)blockIdx.x >= it.pd.nscales) return;
  reduce_scale_sum(it.pd, partials + it.part, scale_sums + (size_t)p * kMaxScales * kScoreSums, counters + p,
                   scores + p, nullptr, nullptr, NextStep());
}

// ------------------------------------------------------------------------------------------------ lockstep batch

// The scoring half of one bisection step of every image of a lockstep batch (capi.cu): the candidate pyramids, the
// tiles and the reductions, each one launch over a work-list of every image's CTAs; an image whose search has
// finished skips through its StepDesc's `active`.
__global__ void __launch_bounds__(kPyrThreads, build_ctas(kOutDiff)) k_build_lock(const LockItem* __restrict__ items,
                                                                                  int n) {
  grid_chain();
  const int i = lock_find<&LockItem::p0>(items, n, blockIdx.x);
  const LockItem& it = items[i];
  if (!it.st->active) return;
  BuildArgs g;
  g.out = it.dist_pyr;
  g.xyb = nullptr;
  g.ref = it.ref_pyr;
  g.planes = it.planes;
  g.st = it.st;
  build_block<kFromPlanes, kOutDiff, kPyrT>(it.pd, g, (int)((long long)blockIdx.x - it.p0));
}

template <int kRef>
__global__ void __launch_bounds__(kTileThreads, tile_ctas(kRef))
    k_ssim2_tiles_lock(const LockItem* __restrict__ items, int n) {
  grid_chain();
  const int i = lock_find<&LockItem::t0>(items, n, blockIdx.x);
  const LockItem& it = items[i];
  if (!it.st->active) return;
  const int blk = (int)((long long)blockIdx.x - it.t0);
  int s = 0;
  while (s + 1 < it.pd.nscales && blk >= it.pd.s[s + 1].tile0) s++;
  const ScaleDesc sd = it.pd.s[s];
  ssim2_band<kRef>(sd, blk - sd.tile0, channel_of_cta(), it.ref_xyb, it.dist_pyr, it.partials + blk,
                   (size_t)it.pd.total_tiles, it.refm);
}

__global__ void __launch_bounds__(256) k_ssim2_reduce_lock(const LockItem* __restrict__ items) {
  grid_chain();
  const LockItem& it = items[blockIdx.z];
  if (!it.st->active || (int)blockIdx.x >= it.pd.nscales) return;
  reduce_scale_sum(it.pd, it.partials, it.scale_sums, it.counter, it.score, it.ss, it.st,
                   NextStep{kNextEncode, it.w, it.h, it.slots, it.slot_stride, nullptr});
}

void lock_step_score(rcg_ctx* ctx, const LockItem* d_items, int n, long long p_total, long long t_total,
                     int max_scales, int ref_mode) {
  RCG_LAUNCH(ctx, "build_lock", k_build_lock, (unsigned)p_total, kPyrThreads, 0, d_items, n);
  // Every image of the batch is at the same step: the first stores its reference moments, the later ones read them.
  if (ref_mode == kRefWrite)
    RCG_LAUNCH(ctx, "ssim2_tiles_lock", k_ssim2_tiles_lock<kRefWrite>, tile_grid(t_total), kTileThreads,
               tile_smem(kRefWrite),
               d_items, n);
  else if (ref_mode == kRefRead)
    RCG_LAUNCH(ctx, "ssim2_tiles_lock", k_ssim2_tiles_lock<kRefRead>, tile_grid(t_total), kTileThreads,
               tile_smem(kRefRead),
               d_items, n);
  else
    RCG_LAUNCH(ctx, "ssim2_tiles_lock", k_ssim2_tiles_lock<kRefNone>, tile_grid(t_total), kTileThreads,
               tile_smem(kRefNone),
               d_items, n);
  RCG_LAUNCH(ctx, "ssim2_reduce_lock", k_ssim2_reduce_lock, dim3(max_scales, kScoreSums, n), 256, 0, d_items);
}

// The source description of an image on the device; false: no memory for the 16-bit table.
static bool image_src(rcg_ctx* ctx, const uint8_t* d_img, int w, int h, int channels, int depth, ImageSrc* im) {
  *im = ImageSrc{d_img, w, h, channels, depth, nullptr};
  if (depth != 16 || channels == 2 || channels == 4) return true;
  im->lut16 = srgb_lut16_device(ctx);
  return im->lut16 != nullptr;
}

int to_linear(rcg_ctx* ctx, const uint8_t* d_img, int w, int h, int pitch, int channels, int depth, float* d_lin) {
  ImageSrc im;
  if (!image_src(ctx, d_img, w, h, channels, depth, &im)) return RCG_NO_MEMORY;
  const long long quads = (long long)((w + 3) / 4) * h;
  RCG_LAUNCH(ctx, "to_linear", k_to_linear, (unsigned)((quads + 255) / 256), 256, 0, im, pitch, d_lin);
  return RCG_OK;
}

int build_pair(rcg_ctx* ctx, const PyramidDesc& pd, const uint8_t* d_ref, const uint8_t* d_dist, int channels, int depth,
               float* d_xyb, float* d_diff) {
  BuildArgs g = {};
  if (!image_src(ctx, d_ref, pd.s[0].w, pd.s[0].h, channels, depth, &g.im[0]) ||
      !image_src(ctx, d_dist, pd.s[0].w, pd.s[0].h, channels, depth, &g.im[1]))
    return RCG_NO_MEMORY;
  g.out = d_diff;
  g.xyb = d_xyb;
  cudaEvent_t ea, eb;
  launch_begin(ctx, "build_pair", &ea, &eb);
  launch_build<kFromImage, kOutPair>(pd, g, nullptr, ctx->stream);
  launch_end(ctx, "build_pair", ea, eb);
  return RCG_OK;
}

int build_reference(rcg_ctx* ctx, const PyramidDesc& pd, const uint8_t* d_img, int channels, float* d_lin, float* d_xyb) {
  BuildArgs g = {};
  if (!image_src(ctx, d_img, pd.s[0].w, pd.s[0].h, channels, 8, &g.im[0])) return RCG_NO_MEMORY;
  g.out = d_lin;
  g.xyb = d_xyb;
  cudaEvent_t ea, eb;
  launch_begin(ctx, "build_reference", &ea, &eb);
  launch_build<kFromImage, kOutRef>(pd, g, nullptr, ctx->stream);
  launch_end(ctx, "build_reference", ea, eb);
  return RCG_OK;
}

int build_decoded(rcg_ctx* ctx, const PyramidDesc& pd, StepDesc* d_step, const uint8_t* d_planes, bool direct,
                  float* d_out, float* d_xyb, const float* d_ref) {
  BuildArgs g = {};
  g.out = d_out;
  g.xyb = d_xyb;
  g.ref = d_ref;
  g.planes = d_planes;
  g.st = d_step;
  if (!direct) upsample_color(ctx, d_step, d_planes, pd.s[0].w, pd.s[0].h, nullptr, d_out, pd.s[0].pitch,
                               (size_t)pd.s[0].pitch * pd.s[0].h);
  const char* name = d_ref ? "build_diff" : "build_reference";
  cudaEvent_t ea, eb;
  launch_begin(ctx, name, &ea, &eb);
  if (d_ref && direct)
    launch_build<kFromPlanes, kOutDiff>(pd, g, d_step, ctx->stream);
  else if (d_ref)
    launch_build<kFromLinear, kOutDiff>(pd, g, d_step, ctx->stream);
  else if (direct)
    launch_build<kFromPlanes, kOutRef>(pd, g, d_step, ctx->stream);
  else
    launch_build<kFromLinear, kOutRef>(pd, g, d_step, ctx->stream);
  launch_end(ctx, name, ea, eb);
  return RCG_OK;
}

PyramidDesc make_pyramid(int w, int h, int channels) {
  PyramidDesc pd;
  std::memset(&pd, 0, sizeof pd);
  long long off = 0;
  int tiles = 0;
  for (int s = 0; s < kMaxScales; s++) {
    if (w < kMinSide || h < kMinSide) break;
    ScaleDesc& sd = pd.s[s];
    sd.w = w;
    sd.h = h;
    sd.pitch = (w + 3) / 4 * 4;
    sd.planes = channels <= 2 ? 1 : 3;
    sd.tiles_x = (w + kTileW - 1) / kTileW;
    sd.tiles_y = (h + kTileH - 1) / kTileH;
    sd.tile0 = tiles;
    sd.nch = 1;
    sd.chunk0 = tiles;
    sd.off = off;
    tiles += sd.tiles_x * sd.tiles_y;
    off += (long long)sd.planes * sd.pitch * h;
    pd.nscales = s + 1;
    w = (w + 1) / 2;
    h = (h + 1) / 2;
  }
  pd.total_tiles = tiles;
  pd.total_chunks = tiles;
  pd.floats = off;
  return pd;
}

static std::mutex g_scorer_mu;
static bool g_scorer_ready[64];

// Upload the scorer's constant tables to the current device once (cudaMemcpyToSymbol only; nothing is allocated).
// core/src/ssimulacra2.rs:54-163 (WEIGHTS)
static const double kScorerWeights[108] = {
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
    0.0, 0.0, 0.0, 0.0005130064588990679, 0.0, 0.00010854057858411537};

const double* scorer_weights() { return kScorerWeights; }

static cudaError_t scorer_constants(int device) {
  std::lock_guard<std::mutex> lk(g_scorer_mu);
  if (device >= 0 && device < 64 && g_scorer_ready[device]) return cudaSuccess;
  // core/src/ssimulacra2.rs:260-271 (kernel): f64 taps, rounded to f32 here.
  double k[2 * kRadius + 1], sum = 0.0;
  for (int i = 0; i < 2 * kRadius + 1; i++) {
    double x = (double)i - (double)kRadius;
    k[i] = std::exp(-0.5 / (1.5 * 1.5) * x * x);
    sum += k[i];
  }
  // Taps i and 2 kRadius - i have the same x * x, hence the same f32 value: the tile kernel holds six distinct taps.
  float kf[2 * kRadius + 1];
  for (int i = 0; i < 2 * kRadius + 1; i++) kf[i] = (float)(k[i] / sum);
  float lut[256];
  srgb_lut8(lut);
  const double* W = scorer_weights();
  cudaError_t e;
  if ((e = cudaMemcpyToSymbol(c_gauss, kf, sizeof kf)) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_lut8s, lut, sizeof lut)) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_weights, W, sizeof c_weights)) != cudaSuccess) return e;
  if (int ce = codec_upload_lut(lut)) return (cudaError_t)ce;
  if ((e = cudaFuncSetAttribute(k_ssim2_tiles<kRefNone>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(kRefNone))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_ssim2_tiles<kRefWrite>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(kRefWrite))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_ssim2_tiles<kRefRead>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(kRefRead))) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute(k_ssim2_tiles_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(kRefNone))) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute(k_ssim2_tiles_lock<kRefNone>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(kRefNone))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_ssim2_tiles_lock<kRefWrite>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(kRefWrite))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_ssim2_tiles_lock<kRefRead>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(kRefRead))) != cudaSuccess)
    return e;
  if (device >= 0 && device < 64) g_scorer_ready[device] = true;
  return cudaSuccess;
}

int scorer_init(rcg_ctx* ctx) {
  cudaError_t e = scorer_constants(ctx->device);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "scorer constant tables");
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ band autotuner

// Bands pay off where a scale has enough tiles to keep every SM busy with long CTAs; smaller scales (and whole
// images below kBandMinTiles0 scale-0 tiles, which are never tuned) keep 32x32 tiles.
constexpr int kBandMinTiles = 3 * kSms;
constexpr int kBandMinTiles0 = 1024;
constexpr int kBandCandidates[] = {1, 2, 4, 8};

PyramidDesc banded(const PyramidDesc& pd, int nch0, int min_tiles) {
  PyramidDesc b = pd;
  int total = 0, chunks = 0;
  for (int s = 0; s < pd.nscales; s++) {
    ScaleDesc& sd = b.s[s];
    const int tiles = pd.s[s].tiles_x * pd.s[s].tiles_y;
    const int n = (nch0 > 1 && tiles >= min_tiles) ? std::min(nch0, pd.s[s].tiles_y) : 1;
    sd.nch = n;
    sd.tiles_y = (pd.s[s].tiles_y + n - 1) / n;
    sd.tile0 = total;
    sd.chunk0 = chunks;
    total += sd.tiles_x * sd.tiles_y;
    chunks += sd.tiles_x * sd.tiles_y * n;
  }
  b.total_tiles = total;
  b.total_chunks = chunks;
  return b;
}

// Deterministic stand-in content for the tuning runs, in place of the reference's XYB and of the differences (values in
// [0, 1], the second half like the first); the kernel's time does not depend on the values.
__global__ void k_tune_fill(float* __restrict__ p, long long n) {
  grid_chain();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    uint32_t x = (uint32_t)(i % (n / 2)) * 2654435761u;
    x ^= x >> 15;
    float v = (float)(x & 0xFFFFFF) * (1.0f / 16777216.0f);
    p[i] = i < n / 2 ? v : fminf(1.0f, v * 0.98f + 0.01f);
  }
}

static std::mutex g_band_mu;
static std::map<std::pair<int, int>, int> g_band_choice;  // (device, size class) -> chunks per band

// Size class: scale-0 tiles in half-octave steps, gray images (one channel's work per tile) apart.
static int band_class(const PyramidDesc& pd) {
  const double t = (double)pd.s[0].tiles_x * pd.s[0].tiles_y;
  return (int)std::floor(2.0 * std::log2(std::max(1.0, t))) + (pd.s[0].planes == 1 ? 1000 : 0);
}

// Time k_ssim2_tiles for each candidate on a stand-in pair of this geometry (own allocation, freed after); the
// fastest by the best of three launches wins.
static int tune_bands(rcg_ctx* ctx, const PyramidDesc& pd) {
  float* pyr = nullptr;
  double* part = nullptr;
  const long long n = 2 * pd.floats;
  if (cudaMalloc(&pyr, (size_t)n * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&part, (size_t)pd.total_tiles * kScoreSums * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    if (pyr) cudaFree(pyr);
    return 1;  // no room to tune: tiles
  }
  k_tune_fill<<<4 * kSms, 256, 0, ctx->stream>>>(pyr, n);
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  int best = 1;
  float best_ms = 1e30f;
  for (int nch0 : kBandCandidates) {
    const PyramidDesc pb = banded(pd, nch0, kBandMinTiles);
    float t = 1e30f;
    for (int rep = 0; rep < 4; rep++) {
      cudaEventRecord(a, ctx->stream);
      k_ssim2_tiles<kRefNone><<<pb.total_tiles, kTileThreads, tile_smem(kRefNone), ctx->stream>>>(pb, pyr, pyr + pd.floats,
                                                                                        part, nullptr, nullptr);
      cudaEventRecord(b, ctx->stream);
      cudaEventSynchronize(b);
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, a, b);
      if (rep > 0) t = std::min(t, ms);  // the first launch warms up
    }
    if (t < best_ms * 0.99f) {  // a longer band must win by more than noise
      best_ms = t;
      best = nch0;
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(pyr);
  cudaFree(part);
  cudaGetLastError();
  return best;
}

PyramidDesc plan_bands(rcg_ctx* ctx, const PyramidDesc& pd) {
  // A fixed choice applies at every scale; a tuned one only where a scale has tiles enough to fill the GPU.
  return banded(pd, band_chunks(ctx, pd), ctx->band_chunks > 0 ? 0 : kBandMinTiles);
}

int band_chunks(rcg_ctx* ctx, const PyramidDesc& pd) {
  if (ctx->band_chunks > 0) return ctx->band_chunks;
  if (pd.nscales == 0 || pd.s[0].tiles_x * pd.s[0].tiles_y < kBandMinTiles0) return 1;
  const auto key = std::make_pair(ctx->device, band_class(pd));
  std::lock_guard<std::mutex> lk(g_band_mu);
  auto it = g_band_choice.find(key);
  if (it != g_band_choice.end()) return it->second;
  const int best = tune_bands(ctx, pd);
  g_band_choice[key] = best;
  return best;
}

int score_workspace(rcg_ctx* ctx, const PyramidDesc& pd) {
  double* partials = (double*)workspace(ctx, "score_partials", (size_t)pd.total_tiles * kScoreSums * sizeof(double));
  double* scale_sums = (double*)workspace(ctx, "score_scale_sums", kMaxScales * kScoreSums * sizeof(double));
  unsigned* counter = (unsigned*)workspace(ctx, "score_counter", 256);
  return partials && scale_sums && counter ? RCG_OK : RCG_NO_MEMORY;
}

int score_pyramids(rcg_ctx* ctx, const PyramidDesc& pd, const float* d_ref, const float* d_dist, double* d_score,
                   SearchState* search, StepDesc* step, float2* refm, int ref_mode, const NextStep& next) {
  if (score_workspace(ctx, pd) != RCG_OK) return RCG_NO_MEMORY;
  double* partials = (double*)ctx->bufs["score_partials"].ptr;
  double* scale_sums = (double*)ctx->bufs["score_scale_sums"].ptr;
  unsigned* counter = (unsigned*)ctx->bufs["score_counter"].ptr;
  const PyramidDesc pb = plan_bands(ctx, pd);
  if (!refm || ref_mode == kRefNone)
    RCG_LAUNCH(ctx, "ssim2_tiles", k_ssim2_tiles<kRefNone>, tile_grid(pb.total_tiles), kTileThreads,
               tile_smem(kRefNone), pb, d_ref, d_dist, partials, step, nullptr);
  else if (ref_mode == kRefWrite)
    RCG_LAUNCH(ctx, "ssim2_tiles_store", k_ssim2_tiles<kRefWrite>, tile_grid(pb.total_tiles), kTileThreads,
               tile_smem(kRefWrite), pb, d_ref, d_dist, partials, step, refm);
  else
    RCG_LAUNCH(ctx, "ssim2_tiles_cached", k_ssim2_tiles<kRefRead>, tile_grid(pb.total_tiles), kTileThreads,
               tile_smem(kRefRead), pb, d_ref, d_dist, partials, step, refm);
  dim3 rg(pb.nscales, kScoreSums);
  RCG_LAUNCH(ctx, "ssim2_reduce", k_ssim2_reduce, rg, 256, 0, pb, partials, scale_sums, counter, d_score, search,
             step, next);
  return RCG_OK;
}

int score_batch(rcg_ctx* ctx, int n, const uint8_t* const* d_refs, const uint8_t* const* d_dists,
                const uint32_t* widths, const uint32_t* heights, const int* channels, const int* depths,
                double** d_scores, const Decoded* decoded) {
  std::vector<ScoreItem> items((size_t)n);
  std::map<std::tuple<const uint8_t*, uint32_t, uint32_t, int, int>, int> first_ref;
  std::vector<int> ref_of((size_t)n), uses((size_t)n, 0);
  long long tiles = 0, parts = 0, floats = 0;
  int max_scales = 1;
  bool need16 = false;
  for (int i = 0; i < n; i++) {
    ScoreItem& it = items[(size_t)i];
    std::memset(&it, 0, sizeof it);
    it.pd = plan_bands(ctx, make_pyramid((int)widths[i], (int)heights[i], channels[i]));
    const int depth = depths ? depths[i] : 8;
    const auto found =
        first_ref.emplace(std::make_tuple(d_refs[i], widths[i], heights[i], channels[i], depth), i).first;
    ref_of[(size_t)i] = found->second;
    uses[(size_t)found->second]++;
    it.tile0 = tiles;
    tiles += it.pd.total_tiles;
    it.part = parts;
    parts += (long long)kScoreSums * it.pd.total_tiles;
    max_scales = std::max(max_scales, it.pd.nscales);
    need16 |= depth == 16 && channels[i] != 2 && channels[i] != 4;
  }
  auto alloc = [&](const PyramidDesc& pd) {
    const long long at = floats;
    floats = (floats + pd.floats + 63) / 64 * 64;  // 256-byte plane starts (vector stores)
    return at;
  };
  // Per pair the offsets of its reference's XYB and of its differences; per shared reference its linear pyramid.
  std::vector<long long> off_xyb((size_t)n), off_lin((size_t)n, -1), off_diff((size_t)n);
  for (int i = 0; i < n; i++) {
    const int r = ref_of[(size_t)i];
    if (r == i) {
      off_xyb[(size_t)i] = alloc(items[(size_t)i].pd);
      if (uses[(size_t)i] > 1 || decoded) off_lin[(size_t)i] = alloc(items[(size_t)i].pd);
    }
    off_diff[(size_t)i] = alloc(items[(size_t)i].pd);
  }
  if (tiles > INT32_MAX) return fail(ctx, RCG_INVALID, "batch too large for one launch");
  float* base = (float*)workspace(ctx, "batch_pyr", (size_t)floats * sizeof(float));
  double* partials = (double*)workspace(ctx, "batch_partials", (size_t)parts * sizeof(double));
  double* sums = (double*)workspace(ctx, "batch_sums", (size_t)n * kMaxScales * kScoreSums * sizeof(double));
  unsigned* counters = (unsigned*)workspace(ctx, "batch_counters", (size_t)n * sizeof(unsigned));
  double* scores = (double*)workspace(ctx, "batch_scores", (size_t)n * sizeof(double));
  const float* lut16 = need16 ? srgb_lut16_device(ctx) : nullptr;
  if (!base || !partials || !sums || !counters || !scores || (need16 && !lut16)) return RCG_NO_MEMORY;
  // Builder jobs in three lists: the shared references, their pairs' differences, the pairs of a reference of their own.
  constexpr int kLists = 3;
  std::vector<BuildJob> jobs[kLists];
  std::vector<long long> first[kLists];
  long long ctas[kLists] = {0, 0, 0};
  auto add = [&](int list, int i, const BuildArgs& g) {
    const PyramidDesc& pd = items[(size_t)i].pd;
    jobs[list].push_back(BuildJob{pd, g});
    first[list].push_back(ctas[list]);
    ctas[list] += pyramid_ctas(pd);
  };
  for (int i = 0; i < n; i++) {
    const int r = ref_of[(size_t)i], depth = depths ? depths[i] : 8, w = (int)widths[i], h = (int)heights[i];
    const ImageSrc a = {d_refs[i], w, h, channels[i], depth, lut16},
                   b = {decoded ? nullptr : d_dists[i], w, h, channels[i], depth, lut16};
    BuildArgs g = {};
    if (uses[(size_t)r] == 1 && !decoded) {
      g.im[0] = a;
      g.im[1] = b;
      g.xyb = base + off_xyb[(size_t)i];
      g.out = base + off_diff[(size_t)i];
      add(2, i, g);
      continue;
    }
    if (r == i) {
      g.im[0] = a;
      g.xyb = base + off_xyb[(size_t)i];
      g.out = base + off_lin[(size_t)i];
      add(0, i, g);
    }
    g = {};
    if (decoded) {
      g.planes = decoded[i].planes;
      g.st = decoded[i].st;
    } else {
      g.im[0] = b;
    }
    g.ref = base + off_lin[(size_t)r];
    g.out = base + off_diff[(size_t)i];
    add(1, i, g);
  }
  // A list of few blocks is built by 32x32 ones, as one small image is (kSmallBuild).
  bool small[kLists];
  for (int k = 0; k < kLists; k++) {
    small[k] = ctas[k] <= kSmallBuild;
    if (!small[k]) continue;
    ctas[k] = 0;
    for (size_t j = 0; j < jobs[k].size(); j++) {
      first[k][j] = ctas[k];
      ctas[k] += blocks_of(jobs[k][j].pd, kPyrTSmall);
    }
  }
  // The work-list in one upload: pairs, then the tile segments (one per pair and scale) and their first tiles, then the
  // builder lists and their first CTAs.
  int nseg = 0;
  for (const ScoreItem& it : items) nseg += it.pd.nscales;
  size_t list_bytes = 0;
  auto place = [&](size_t bytes) {
    const size_t at = list_bytes;
    list_bytes = (list_bytes + bytes + 15) / 16 * 16;
    return at;
  };
  const size_t o_items = place((size_t)n * sizeof(ScoreItem)), o_seg = place((size_t)nseg * sizeof(TileSeg)),
               o_seg0 = place((size_t)nseg * 8);
  size_t o_jobs[kLists], o_first[kLists];
  for (int k = 0; k < kLists; k++) {
    if (ctas[k] > INT32_MAX) return fail(ctx, RCG_INVALID, "batch too large for one launch");
    o_jobs[k] = place(jobs[k].size() * sizeof(BuildJob));
    o_first[k] = place(first[k].size() * 8);
  }
  unsigned char* d_list = (unsigned char*)workspace(ctx, "batch_items", list_bytes);
  if (!d_list) return RCG_NO_MEMORY;
  // The context keeps the list: its copy may still read it when this returns, and every call waits for its stream.
  std::vector<unsigned char>& list = ctx->work_list;
  list.assign(list_bytes, 0);
  std::memcpy(list.data() + o_items, items.data(), (size_t)n * sizeof(ScoreItem));
  for (int k = 0; k < kLists; k++) {
    if (jobs[k].empty()) continue;
    std::memcpy(list.data() + o_jobs[k], jobs[k].data(), jobs[k].size() * sizeof(BuildJob));
    std::memcpy(list.data() + o_first[k], first[k].data(), first[k].size() * 8);
  }
  TileSeg* segs = (TileSeg*)(list.data() + o_seg);
  long long* seg0 = (long long*)(list.data() + o_seg0);
  int gseg = 0;
  for (int i = 0; i < n; i++) {
    const ScoreItem& it = items[(size_t)i];
    for (int sc = 0; sc < it.pd.nscales; sc++, gseg++) {
      const ScaleDesc& sd = it.pd.s[sc];
      TileSeg& sg = segs[gseg];
      sg.ref = base + off_xyb[(size_t)ref_of[(size_t)i]] + sd.off;
      sg.dist = base + off_diff[(size_t)i] + sd.off;
      sg.out = partials + it.part + sd.tile0;
      sg.w = sd.w;
      sg.h = sd.h;
      sg.pitch = sd.pitch;
      sg.planes = sd.planes;
      sg.tiles_x = sd.tiles_x;
      sg.nch = sd.nch;
      sg.stride = it.pd.total_tiles;
      seg0[gseg] = it.tile0 + sd.tile0;
    }
  }
  int rc = copy_to_device(ctx, d_list, list.data(), list_bytes);
  if (rc != RCG_OK) return rc;
  const ScoreItem* d_items = (const ScoreItem*)(d_list + o_items);
  const TileSeg* d_segs = (const TileSeg*)(d_list + o_seg);
  const long long* d_seg0 = (const long long*)(d_list + o_seg0);
  auto d_jobs = [&](int k) { return (const BuildJob*)(d_list + o_jobs[k]); };
  auto d_first = [&](int k) { return (const long long*)(d_list + o_first[k]); };
  int nj[kLists];
  for (int k = 0; k < kLists; k++) nj[k] = (int)jobs[k].size();
  // The launches take only the work-list's totals and this context's buffers: a later batch with the same totals
  // replays them (its own pairs come in through the work-list uploaded above).
  const std::vector<long long> key = {3,     n,     nseg,    tiles,   max_scales, nj[0],
                                      nj[1], nj[2], ctas[0], ctas[1], ctas[2], decoded != nullptr,
                                      small[0], small[1], small[2]};
  rc = run_step_loop(ctx, key, [&]() {
    auto build = [&](int k, auto big, auto little) {
      if (nj[k])
        RCG_LAUNCH(ctx, "build_batch", (small[k] ? little : big), (unsigned)ctas[k], kPyrThreads, 0, d_jobs(k), d_first(k),
                   nj[k]);
    };
    build(0, &k_build_batch<kFromImage, kOutRef, kPyrT>, &k_build_batch<kFromImage, kOutRef, kPyrTSmall>);
    if (decoded)
      build(1, &k_build_batch<kFromPlanes, kOutDiff, kPyrT>, &k_build_batch<kFromPlanes, kOutDiff, kPyrTSmall>);
    else
      build(1, &k_build_batch<kFromImage, kOutDiff, kPyrT>, &k_build_batch<kFromImage, kOutDiff, kPyrTSmall>);
    build(2, &k_build_batch<kFromImage, kOutPair, kPyrT>, &k_build_batch<kFromImage, kOutPair, kPyrTSmall>);
    RCG_LAUNCH(ctx, "ssim2_tiles_batch", k_ssim2_tiles_batch, tile_grid(tiles), kTileThreads, tile_smem(kRefNone), d_segs,
               d_seg0, nseg);
    RCG_LAUNCH(ctx, "ssim2_reduce_batch", k_ssim2_reduce_batch, dim3(max_scales, kScoreSums, n), 256, 0, d_items,
               partials, sums, counters, scores);
  });
  if (rc != RCG_OK) return rc;
  *d_scores = scores;
  return RCG_OK;
}

}  // namespace rcg

// ------------------------------------------------------------------------------------------------ no-alloc scorer

namespace rcg {

// Fixed scratch of rcg_ssimulacra2_device_noalloc: the reference's XYB pyramid and the differences, the per-tile partial
// sums, the per-scale sums and the reduction's completion counter. Sized for images of at most kNoAllocMaxPixels pixels. CUDA
// places a module's device arrays on a device when the module is first used there, so every device where any scorer
// call has run holds it (about 10 MB) until the process exits. The per-device set-up below is cached for the life of
// the process; a cudaDeviceReset invalidates it and is not supported.
constexpr long long kNoAllocMaxPixels = 512LL * 512LL;
constexpr long long kNoAllocPyrFloats = 1250000;  // one image: 3 channels x every scale in padded rows (at most 1,202,760)
constexpr int kNoAllocMaxTiles = 4096;
constexpr size_t kNoAllocPyrBytes = (size_t)kNoAllocPyrFloats * sizeof(float);
constexpr size_t kNoAllocPartialOff = 2 * kNoAllocPyrBytes;
constexpr size_t kNoAllocSumsOff = kNoAllocPartialOff + (size_t)kNoAllocMaxTiles * kScoreSums * sizeof(double);
constexpr size_t kNoAllocCounterOff = kNoAllocSumsOff + (size_t)kMaxScales * kScoreSums * sizeof(double);
constexpr size_t kNoAllocBytes = kNoAllocCounterOff + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

static std::mutex g_noalloc_mu;
static unsigned char* g_noalloc_addr[64];

// Once per device, with that device current: the device address of the scratch (host code cannot use the symbol
// itself, which names a host-side shadow) and the scorer's constant tables.
static int noalloc_setup(unsigned char** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return RCG_CUDA_ERROR;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      return RCG_CUDA_ERROR;
    }
    if (scorer_constants(dev) != cudaSuccess) {
      cudaGetLastError();
      return RCG_CUDA_ERROR;
    }
    g_noalloc_addr[dev] = (unsigned char*)p;
  }
  *out = g_noalloc_addr[dev];
  return RCG_OK;
}

}  // namespace rcg

extern "C" int rcg_ssimulacra2_device_noalloc(const uint8_t* d_reference, const uint8_t* d_distorted,
                                              uint32_t width, uint32_t height, int channels, double* d_score,
                                              void* stream) {
  using namespace rcg;
  if (!d_reference || !d_distorted || !d_score) return RCG_INVALID;
  if (channels != 1 && channels != 3) return RCG_INVALID;
  if (width < (uint32_t)kMinSide || height < (uint32_t)kMinSide) return RCG_INVALID;
  if ((long long)width * (long long)height > kNoAllocMaxPixels) return RCG_INVALID;
  const int w = (int)width, h = (int)height;
  PyramidDesc pd = make_pyramid(w, h, channels);
  if (pd.floats > kNoAllocPyrFloats || pd.total_tiles > kNoAllocMaxTiles) return RCG_INVALID;
  unsigned char* base = nullptr;
  int rc = noalloc_setup(&base);
  if (rc != RCG_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  float* pyr_ref = (float*)base;
  float* pyr_dist = (float*)(base + kNoAllocPyrBytes);
  double* partials = (double*)(base + kNoAllocPartialOff);
  double* sums = (double*)(base + kNoAllocSumsOff);
  unsigned* counter = (unsigned*)(base + kNoAllocCounterOff);
  // The scratch keeps whatever the previous call left: the completion counter must start at zero.
  if (cudaMemsetAsync(counter, 0, sizeof(unsigned), s) != cudaSuccess) {
    cudaGetLastError();
    return RCG_CUDA_ERROR;
  }
  BuildArgs g = {};
  g.im[0] = ImageSrc{d_reference, w, h, channels, 8, nullptr};
  g.im[1] = ImageSrc{d_distorted, w, h, channels, 8, nullptr};
  g.xyb = pyr_ref;
  g.out = pyr_dist;
  launch_build<kFromImage, kOutPair>(pd, g, nullptr, s);
  launch_chained(tile_grid(pd.total_tiles), kTileThreads, tile_smem(kRefNone), s, k_ssim2_tiles<kRefNone>, pd, pyr_ref,
                 pyr_dist, partials, nullptr, nullptr);
  launch_chained(dim3(pd.nscales, kScoreSums), 256, 0, s, k_ssim2_reduce, pd, partials, sums, counter, d_score, nullptr,
                 nullptr, NextStep());
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? RCG_OK : RCG_CUDA_ERROR;
}
