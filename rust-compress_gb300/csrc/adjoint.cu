// Reverse-mode derivative of SSIMULACRA2 (core/src/ssimulacra2.rs:171-512) with respect to the distorted image's
// RGB samples, taken as continuous values in [0, 255], on the GPU.
//
// Forward: linear light by the sRGB curve itself (:172-175; the reference's 8-bit table samples it), the 2x2
// pyramid, and per scale the XYB planes, the five blurred moments per channel and the six map sums. Backward, from
// the coarsest scale to the finest: d score / d map from the 108-term sum, the final mapping and the L1/L4 norms;
// through the SSIM and edge maps to the moments and the XYB samples (one-sided derivatives at the max(., 0) and |.|
// kinks); through the blurs (the zero-padded row blur is its own transpose, the mirrored column blur scatters
// back); through XYB to linear light; plus the coarser scales' gradients spread back over their 2x2 blocks; and
// finally through the sRGB curve. Every scale and channel (up to 18 planes) goes through one launch per step, each CTA
// finding its plane in a job table: the planes are independent in all steps but the pyramid and its adjoint, and most of
// them are far too small to fill the GPU alone. Where their moments fit a budget they are kept from the forward pass for
// the backward one, else the planes go in groups that are blurred again. Measured against one launch per plane (222 in
// all, the moments blurred twice): FP64 768x512 4.9 -> 2.3 ms a call, 290x250 2.2 -> 0.6 (bound by the narrow FP64 pipe
// then), FP32 inside a 1620x1080 perceptual search 2.1 -> 0.7 ms (memory). Row runs inside the row without their border
// checks measured slower (their warps diverge at every row's ends). Plane kernels, templated on the real type: FP64 (the
// checked
// gradient: it matches the FP64 CPU gradient to rounding) and FP32 (the perceptual weights, where a few significant
// digits suffice: the variances' cancellation error, ~1e-8, is small against the SSIM constant 9e-4 that bounds
// every denominator, and GB300's FP32 rate is many times its FP64 rate). Sums of the maps are f64 across threads in
// both; the final mapping runs on the host in f64.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "rcg_internal.cuh"
#include "curve_power.cuh"

namespace rcg {

namespace {

constexpr int kR = 5;  // kernel radius (:16)
constexpr double kBiasD = 0.0037930732552754493;
constexpr double kM00 = 0.30, kM02 = 0.078, kM01 = 1.0 - kM02 - kM00;
constexpr double kM10 = 0.23, kM12 = 0.078, kM11 = 1.0 - kM12 - kM10;
constexpr double kM20 = 0.2434226892454782, kM21 = 0.2047674442449682, kM22 = 1.0 - kM20 - kM21;
constexpr double kC2 = 0.0009;

// normalized Gaussian taps (sigma 1.5) in both types
__constant__ double c_k64[2 * kR + 1];
__constant__ float c_k32[2 * kR + 1];
// The curve and its derivative at the 256 integer samples, computed on the host with the same expressions (an
// 8-bit reference, and decoded candidates passed as whole-number samples, skip the pow).
__constant__ double c_lin8[256];
__constant__ double c_dlin8[256];

template <typename T> __device__ __forceinline__ T tap(int t);
template <> __device__ __forceinline__ double tap<double>(int t) { return c_k64[t]; }
template <> __device__ __forceinline__ float tap<float>(int t) { return c_k32[t]; }
__device__ __forceinline__ double cbrt_t(double x) { return cbrt(x); }
__device__ __forceinline__ float cbrt_t(float x) { return cbrtf(x); }

__device__ __forceinline__ double srgb64(double v) {
  return v <= 0.04045 ? v / 12.92 : pow24((v + 0.055) / 1.055);
}
__device__ __forceinline__ double srgb64_deriv(double v255) {
  const double v = v255 / 255.0;
  return v <= 0.04045 ? 1.0 / (12.92 * 255.0) : 2.4 * pow14((v + 0.055) / 1.055) / (1.055 * 255.0);
}

__device__ __forceinline__ long long tid1() { return (long long)blockIdx.x * blockDim.x + threadIdx.x; }

// Index of a whole-number sample in [0, 255], else -1.
__device__ __forceinline__ int sample8(float v) {
  return (v >= 0.0f && v <= 255.0f && v == rintf(v)) ? (int)v : -1;
}

// Linear planes [3][n] of the reference (8-bit samples) and of the distorted image (f32 samples), by the curve.
template <typename T>
__global__ void k_lin(const uint8_t* __restrict__ ref, const float* __restrict__ dist, long long n,
                      T* __restrict__ la, T* __restrict__ lb) {
  grid_chain();
  __shared__ T lut[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = (T)c_lin8[i];
  __syncthreads();
  for (long long i = tid1(); i < n; i += (long long)gridDim.x * blockDim.x)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      // both images through the same curve: identical inputs give identical planes (and the score 100)
      la[c * n + i] = lut[ref[i * 3 + c]];
      const float v = dist[i * 3 + c];
      const int k = sample8(v);
      lb[c * n + i] = k >= 0 ? lut[k] : (T)srgb64((double)v / 255.0);
    }
}

// One plane (a channel of a scale): its samples start at `x` in the buffers that hold a plane per channel (XYB, the
// gradient), its five moments at `m`.
struct AdjJob {
  int w, h;
  long long n, x, m;
};
constexpr int kMaxJobs = 3 * kMaxScales;
// The planes of a launch and the first CTA of each (cta0[count] is the grid's size).
struct AdjJobs {
  int count;
  unsigned cta0[kMaxJobs + 1];
  AdjJob j[kMaxJobs];
};

__device__ __forceinline__ int job_of(const AdjJobs& jobs, unsigned cta) {
  int k = 0;
  while (k + 1 < jobs.count && cta >= jobs.cta0[k + 1]) k++;
  return k;
}

// 2x2 means (:225-247), fewer samples at odd edges; 3 channels of both images (grid z).
// Grid (output columns, rows, planes): see grid_rows.
template <typename T>
__global__ void k_down(const T* __restrict__ src_a, const T* __restrict__ src_b, int w, int h, T* __restrict__ dst_a,
                       T* __restrict__ dst_b, int ow, int oh) {
  grid_chain();
  const int ox = blockIdx.x * blockDim.x + threadIdx.x;
  if (ox >= ow) return;
  const long long n = (long long)ow * oh;
  const int c = blockIdx.z % 3;
  const T* p = (blockIdx.z < 3 ? src_a : src_b) + (long long)c * w * h;
  T* dst = blockIdx.z < 3 ? dst_a : dst_b;
  const int x1 = min(2 * ox + 2, w);
  for (int oy = blockIdx.y; oy < oh; oy += gridDim.y) {
    const int y1 = min(2 * oy + 2, h);
    T s = 0;
    for (int y = 2 * oy; y < y1; y++)
      for (int x = 2 * ox; x < x1; x++) s += p[(long long)y * w + x];
    dst[c * n + (long long)oy * ow + ox] = s / (T)((y1 - 2 * oy) * (x1 - 2 * ox));
  }
}

// XYB (:249-258) of 3 linear planes: one job per scale (its first channel's), both images (grid y).
template <typename T>
__global__ void k_xyb(const __grid_constant__ AdjJobs jobs, const T* __restrict__ lin_a, const T* __restrict__ lin_b,
                      T* __restrict__ xyb_a, T* __restrict__ xyb_b) {
  grid_chain();
  const int job = job_of(jobs, blockIdx.x);
  const long long n = jobs.j[job].n, i = (long long)(blockIdx.x - jobs.cta0[job]) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const T* lin = (blockIdx.y ? lin_b : lin_a) + jobs.j[job].x;
  T* xyb = (blockIdx.y ? xyb_b : xyb_a) + jobs.j[job].x;
  const T M00 = (T)kM00, M01 = (T)kM01, M02 = (T)kM02, M10 = (T)kM10, M11 = (T)kM11, M12 = (T)kM12;
  const T M20 = (T)kM20, M21 = (T)kM21, M22 = (T)kM22, bias = (T)kBiasD;
  const T cb = cbrt_t(bias);
  {
    const T r = lin[i], g = lin[n + i], b = lin[2 * n + i];
    const T m0 = cbrt_t(fmax(M00 * r + M01 * g + M02 * b + bias, (T)0)) - cb;
    const T m1 = cbrt_t(fmax(M10 * r + M11 * g + M12 * b + bias, (T)0)) - cb;
    const T m2 = cbrt_t(fmax(M20 * r + M21 * g + M22 * b + bias, (T)0)) - cb;
    const T x = (T)0.5 * (m0 - m1), y = (T)0.5 * (m0 + m1);
    xyb[i] = x * (T)14.0 + (T)0.42;
    xyb[n + i] = y + (T)0.01;
    xyb[2 * n + i] = (m2 - y) + (T)0.55;
  }
}

// k_down's grid: a thread owns one column of one plane and strides over the rows.
dim3 grid_rows(int w, int h, int planes) {
  return dim3((unsigned)((w + 255) / 256), (unsigned)std::min(h, 65535), (unsigned)planes);
}

// Outputs per thread of the row blurs: a run of kHRun consecutive outputs reads its kHRun + 10 source samples once
// (in registers) instead of 11 per output; every output still sums its in-range taps in the same order. A plane's runs
// are numbered along its rows, so narrow planes fill their CTAs too.
constexpr int kHRun = 4;
__host__ __device__ inline long long row_runs(int w, int h) { return (long long)((w + kHRun - 1) / kHRun) * h; }

// Row blur (zero outside) of one run of a plane: the backward pass's rows (the zero-padded row blur is its own
// transpose).
template <typename T>
__device__ __forceinline__ void hblur_run(const T* __restrict__ row, int w, int x0, T (&out)[kHRun]) {
  T v[kHRun + 2 * kR];
#pragma unroll
  for (int k = 0; k < kHRun + 2 * kR; k++) {
    const int xx = x0 + k - kR;
    v[k] = xx >= 0 && xx < w ? row[xx] : (T)0;
  }
#pragma unroll
  for (int o = 0; o < kHRun; o++) {
    const int x = x0 + o;
    T s = 0;
#pragma unroll
    for (int t = 0; t <= 2 * kR; t++) {
      const int xx = x + t - kR;
      if (xx < 0 || xx >= w) continue;
      s += tap<T>(t) * v[o + t];
    }
    out[o] = s;
  }
}

// A thread's run of kHRun outputs in each of the five planes: one 16-byte store per plane (two for double) when the
// run lies in the row and the planes are 4-sample aligned, else one store per output.
template <typename T>
__device__ __forceinline__ void store_run5(T* __restrict__ dst, long long n, long long rowi, int x0, int w,
                                           const T (&out)[5][kHRun]) {
  static_assert(kHRun == 4, "vector stores of four samples");
  const long long i = rowi + x0;
  if (x0 + kHRun <= w && (w & 3) == 0 && ((uintptr_t)dst & 31) == 0) {
#pragma unroll
    for (int q = 0; q < 5; q++) {
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(dst + q * n + i) = make_float4(out[q][0], out[q][1], out[q][2], out[q][3]);
      } else {
        reinterpret_cast<double2*>(dst + q * n + i)[0] = make_double2(out[q][0], out[q][1]);
        reinterpret_cast<double2*>(dst + q * n + i)[1] = make_double2(out[q][2], out[q][3]);
      }
    }
    return;
  }
#pragma unroll
  for (int o = 0; o < kHRun; o++)
    if (x0 + o < w)
#pragma unroll
      for (int q = 0; q < 5; q++) dst[q * n + i + o] = out[q][o];
}

// The five products of the forward pass blurred along rows in one sweep: dst + q * n for q = 0 xa, 1 xb, 2 xa^2,
// 3 xb^2, 4 xa xb (each output summed over the taps in the same order as k_hblur).
template <typename T>
__global__ void __launch_bounds__(256) k_hblur5(const __grid_constant__ AdjJobs jobs, const T* __restrict__ xa_all,
                                                const T* __restrict__ xb_all, T* __restrict__ dst_all) {
  grid_chain();
  const int job = job_of(jobs, blockIdx.x);
  const AdjJob& J = jobs.j[job];
  const int w = J.w, h = J.h, runs = (w + kHRun - 1) / kHRun;
  const long long n = J.n, e = (long long)(blockIdx.x - jobs.cta0[job]) * blockDim.x + threadIdx.x;
  const long long y = e / runs;
  if (y >= h) return;
  const int x0 = (int)(e - y * runs) * kHRun;
  const T* xa = xa_all + J.x;
  const T* xb = xb_all + J.x;
  T* dst = dst_all + J.m;
  {
    const long long rowi = y * w;
    T va[kHRun + 2 * kR], vb[kHRun + 2 * kR];
#pragma unroll
    for (int k = 0; k < kHRun + 2 * kR; k++) {
      const int xx = x0 + k - kR;
      const bool in = xx >= 0 && xx < w;
      va[k] = in ? xa[rowi + xx] : (T)0;
      vb[k] = in ? xb[rowi + xx] : (T)0;
    }
    T out[5][kHRun];
#pragma unroll
    for (int o = 0; o < kHRun; o++) {
      const int x = x0 + o;
      T s0 = 0, s1 = 0, s2 = 0, s3 = 0, s4 = 0;
#pragma unroll
      for (int t = 0; t <= 2 * kR; t++) {
        const int xx = x + t - kR;
        if (xx < 0 || xx >= w) continue;
        const T a = va[o + t], b = vb[o + t], k = tap<T>(t);
        s0 += k * a;
        s1 += k * b;
        s2 += k * (a * a);
        s3 += k * (b * b);
        s4 += k * (a * b);
      }
      out[0][o] = s0;
      out[1][o] = s1;
      out[2][o] = s2;
      out[3][o] = s3;
      out[4][o] = s4;
    }
    store_run5(dst, n, rowi, x0, w, out);
  }
}

__device__ __forceinline__ int mirror64(int yy, int h) { return yy < 0 ? -yy - 1 : (yy >= h ? 2 * h - 1 - yy : yy); }

// Rows per thread of the column blurs: a run of kRun outputs reads its kRun + 10 source rows once (in registers)
// instead of 11 rows per output; every output still sums its taps in the same order. The forward blur takes runs of
// 16 (0.94 against 1.18 ms per perceptual search at 12 MP with 8), its transpose runs of 8 (0.39 against 0.47 with 16).
constexpr int kRunN = 16, kRun = 8;

// Column blur with mirrored rows (:385-397) of a job's five planes (grid y); a CTA's threads take consecutive columns of
// runs of kRunN rows, the runs one after another.
template <typename T>
__global__ void __launch_bounds__(256) k_vblur_n(const __grid_constant__ AdjJobs jobs, const T* __restrict__ src,
                                                 T* __restrict__ dst) {
  grid_chain();
  const int job = job_of(jobs, blockIdx.x);
  const AdjJob& J = jobs.j[job];
  const int w = J.w, h = J.h;
  const long long e = (long long)(blockIdx.x - jobs.cta0[job]) * blockDim.x + threadIdx.x, r = e / w;
  if (r >= (h + kRunN - 1) / kRunN) return;
  const int x = (int)(e - r * w);
  const T* sp = src + J.m + blockIdx.y * J.n + x;
  T* dp = dst + J.m + blockIdx.y * J.n + x;
  const int y0 = (int)r * kRunN;
  T v[kRunN + 2 * kR];
#pragma unroll
  for (int k = 0; k < kRunN + 2 * kR; k++) {
    const int yy = y0 + k - kR;
    v[k] = yy <= h - 1 + kR ? sp[(long long)mirror64(yy, h) * w] : (T)0;  // rows past a short last run: unused
  }
#pragma unroll
  for (int o = 0; o < kRunN; o++) {
    if (y0 + o >= h) break;
    T s = 0;
#pragma unroll
    for (int t = 0; t <= 2 * kR; t++) s += tap<T>(t) * v[o + t];
    dp[(long long)(y0 + o) * w] = s;
  }
}

// Transpose of the column blur as a gather: row y' receives tap t from the rows y whose mirrored source row is y', i.e.
// from source index y' (y = y' - t + R), -y' - 1 (mirrored at the top) and 2h - 1 - y' (at the bottom).
// A job's three gradient planes (grid y), threads as in k_vblur_n with runs of kRun rows; a run inside the interior reads
// its rows once.
template <typename T>
__global__ void __launch_bounds__(256) k_vblur_t(const __grid_constant__ AdjJobs jobs, const T* __restrict__ gsrc,
                                                 T* __restrict__ dst) {
  grid_chain();
  const int job = job_of(jobs, blockIdx.x);
  const AdjJob& J = jobs.j[job];
  const int w = J.w, h = J.h;
  const long long e = (long long)(blockIdx.x - jobs.cta0[job]) * blockDim.x + threadIdx.x, r = e / w;
  if (r >= (h + kRun - 1) / kRun) return;
  const int x = (int)(e - r * w);
  const T* g = gsrc + J.m + blockIdx.y * J.n;
  T* dp = dst + J.m + blockIdx.y * J.n;
  {
    const int y0 = (int)r * kRun;
    if (y0 >= kR && y0 + kRun - 1 < h - kR) {
      // every output row of the run is interior: row yp takes tap t from source row yp - t + kR
      T v[kRun + 2 * kR];
#pragma unroll
      for (int k = 0; k < kRun + 2 * kR; k++) v[k] = g[(long long)(y0 - kR + k) * w + x];
#pragma unroll
      for (int o = 0; o < kRun; o++) {
        T s = 0;
#pragma unroll
        for (int t = 0; t <= 2 * kR; t++) s += tap<T>(t) * v[o + 2 * kR - t];
        dp[(long long)(y0 + o) * w + x] = s;
      }
      return;
    }
    for (int yp = y0; yp < min(y0 + kRun, h); yp++) {
      T s = 0;
      if (yp >= kR && yp < h - kR) {
        // interior: only the direct source row is in range (the mirrored ones are not)
#pragma unroll
        for (int t = 0; t <= 2 * kR; t++) s += tap<T>(t) * g[(long long)(yp - t + kR) * w + x];
      } else {
#pragma unroll
        for (int t = 0; t <= 2 * kR; t++) {
          const int ys[3] = {yp - t + kR, -yp - 1 - t + kR, 2 * h - 1 - yp - t + kR};
#pragma unroll
          for (int e = 0; e < 3; e++)
            if (ys[e] >= 0 && ys[e] < h) s += tap<T>(t) * g[(long long)ys[e] * w + x];
        }
      }
      dp[(long long)yp * w + x] = s;
    }
  }
}

// The six map sums of one channel (:421-440): per-thread sums in T, then f64 per-CTA partials (parts[block][6]);
// k_sum_parts adds them in a fixed order, so the score and the gradient are the same bits on every run.
// One job's CTAs take its samples in turn.
template <typename T>
__global__ void __launch_bounds__(256) k_maps(const __grid_constant__ AdjJobs jobs, const T* __restrict__ mom_all,
                                              const T* __restrict__ xa_all, const T* __restrict__ xb_all,
                                              double* __restrict__ parts) {
  grid_chain();
  __shared__ double red[6][8];
  const int job = job_of(jobs, blockIdx.x);
  const AdjJob& J = jobs.j[job];
  const long long n = J.n, first = (long long)(blockIdx.x - jobs.cta0[job]) * blockDim.x + threadIdx.x,
                  step = (long long)(jobs.cta0[job + 1] - jobs.cta0[job]) * blockDim.x;
  const T* mom = mom_all + J.m;
  const T* xa = xa_all + J.x;
  const T* xb = xb_all + J.x;
  const T one = 1, c2 = (T)kC2;
  T acc[6] = {0, 0, 0, 0, 0, 0};
  for (long long i = first; i < n; i += step) {
    const T m1 = mom[i], m2 = mom[n + i], s11 = mom[2 * n + i], s22 = mom[3 * n + i], s12 = mom[4 * n + i];
    const T num_m = one - (m1 - m2) * (m1 - m2);
    const T num_s = (T)2 * (s12 - m1 * m2) + c2;
    const T den_s = (s11 - m1 * m1) + (s22 - m2 * m2) + c2;
    const T d = fmax(one - num_m * num_s / den_s, (T)0);
    const T d1 = (one + fabs(xb[i] - m2)) / (one + fabs(xa[i] - m1)) - one;
    const T art = fmax(d1, (T)0), det = fmax(-d1, (T)0);
    acc[0] += d;
    acc[1] += (d * d) * (d * d);
    acc[2] += art;
    acc[3] += (art * art) * (art * art);
    acc[4] += det;
    acc[5] += (det * det) * (det * det);
  }
  // Warp sums in T (the FP32 pass keeps its shuffles off this part's narrow FP64 pipe, which otherwise took half
  // of each launch), then f64 across the warps and CTAs in a fixed order.
#pragma unroll
  for (int k = 0; k < 6; k++) {
    T v = acc[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = (double)v;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double v = 0.0;
    for (int wi = 0; wi < 8; wi++) v += red[threadIdx.x][wi];
    parts[(size_t)blockIdx.x * 6 + threadIdx.x] = v;
  }
}

// sums[job][k] = the job's partials of column k, one CTA per job, one warp per column, lanes strided then a shuffle
// tree. `at`: where each job's six sums go.
struct AdjSums {
  int at[kMaxJobs];
};
__global__ void __launch_bounds__(192) k_sum_parts(const __grid_constant__ AdjJobs jobs, const __grid_constant__ AdjSums to,
                                                   const double* __restrict__ parts_all, double* __restrict__ sums_all) {
  grid_chain();
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* parts = parts_all + (size_t)jobs.cta0[blockIdx.x] * 6;
  const int nparts = (int)(jobs.cta0[blockIdx.x + 1] - jobs.cta0[blockIdx.x]);
  double* sums = sums_all + to.at[blockIdx.x];
  double v = 0.0;
  for (int i = lane; i < nparts; i += 32) v += parts[(size_t)i * 6 + k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sums[k] = v;
}

// Per sample of one channel: d score / d (m2, s22, s12) and the direct d score / d xb of the edge maps, given the
// norms' coefficients g1 (L1: weight / count) and g4 (L4: weight (S/count)^-3/4 / count) of (ssim, artifact,
// detail).
struct NormCoef {
  double g1[3], g4[3];
};
struct NormCoefs {
  NormCoef job[kMaxJobs];
};

// The three moments' gradients go to the job's first three planes of gq.
template <typename T>
__global__ void __launch_bounds__(256) k_mapgrad(const __grid_constant__ AdjJobs jobs,
                                                 const __grid_constant__ NormCoefs coefs, const T* __restrict__ mom_all,
                                                 const T* __restrict__ xa_all, const T* __restrict__ xb_all,
                                                 T* __restrict__ gq, T* __restrict__ gx) {
  grid_chain();
  const int job = job_of(jobs, blockIdx.x);
  const AdjJob& J = jobs.j[job];
  const NormCoef& ncd = coefs.job[job];
  const long long n = J.n, i = (long long)(blockIdx.x - jobs.cta0[job]) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const T* mom = mom_all + J.m;
  const T* xa = xa_all + J.x;
  const T* xb = xb_all + J.x;
  T* g_m2 = gq + J.m;
  T* g_s22 = g_m2 + n;
  T* g_s12 = g_s22 + n;
  T* g_xb = gx + J.x;
  const T one = 1, two = 2, zero = 0, c2 = (T)kC2;
  T g1[3], g4[3];
#pragma unroll
  for (int m = 0; m < 3; m++) {
    g1[m] = (T)ncd.g1[m];
    g4[m] = (T)ncd.g4[m];
  }
  {
    const T m1 = mom[i], m2 = mom[n + i], s11 = mom[2 * n + i], s22 = mom[3 * n + i], s12 = mom[4 * n + i];
    const T num_m = one - (m1 - m2) * (m1 - m2);
    const T num_s = two * (s12 - m1 * m2) + c2;
    const T den_s = (s11 - m1 * m1) + (s22 - m2 * m2) + c2;
    const T dv = one - num_m * num_s / den_s;
    T gm2 = zero, gs22 = zero, gs12 = zero;
    if (dv > zero) {
      const T gd = g1[0] + g4[0] * dv * dv * dv;
      const T g_num_m = -gd * num_s / den_s, g_num_s = -gd * num_m / den_s;
      const T g_den = gd * num_m * num_s / (den_s * den_s);
      gm2 = g_num_m * (two * (m1 - m2)) + g_num_s * (-two * m1) + g_den * (-two * m2);
      gs22 = g_den;
      gs12 = two * g_num_s;
    }
    const T a = xa[i], b = xb[i];
    const T Nn = one + fabs(b - m2), Dn = one + fabs(a - m1);
    const T d1 = Nn / Dn - one;
    const T gd1 = (d1 > zero ? g1[1] + g4[1] * d1 * d1 * d1 : zero) -
                  (d1 < zero ? g1[2] + g4[2] * (-d1) * (-d1) * (-d1) : zero);
    const T sb = b - m2 > zero ? one : (b - m2 < zero ? -one : zero);
    g_xb[i] = gd1 * sb / Dn;
    g_m2[i] = gm2 - gd1 * sb / Dn;
    g_s22[i] = gs22;
    g_s12[i] = gs12;
  }
}

// d score / d xb = direct + G^T(g_m2) + 2 xb G^T(g_s22) + xa G^T(g_s12): the row blurs of a job's three planes (already
// through the transposed column blur), combined where they are made. A thread takes one run of outputs.
template <typename T>
__global__ void __launch_bounds__(256) k_hblur_combine(const __grid_constant__ AdjJobs jobs, const T* __restrict__ src,
                                                       const T* __restrict__ xa_all, const T* __restrict__ xb_all,
                                                       T* __restrict__ gx) {
  grid_chain();
  const int job = job_of(jobs, blockIdx.x);
  const AdjJob& J = jobs.j[job];
  const int w = J.w, runs = (w + kHRun - 1) / kHRun;
  const long long n = J.n, e = (long long)(blockIdx.x - jobs.cta0[job]) * blockDim.x + threadIdx.x, y = e / runs;
  if (y >= J.h) return;
  const int x0 = (int)(e - y * runs) * kHRun;
  const T* row = src + J.m + y * w;
  T t_m2[kHRun], t_s22[kHRun], t_s12[kHRun];
  hblur_run(row, w, x0, t_m2);
  hblur_run(row + n, w, x0, t_s22);
  hblur_run(row + 2 * n, w, x0, t_s12);
  const long long i0 = J.x + y * w + x0;
#pragma unroll
  for (int o = 0; o < kHRun; o++)
    if (x0 + o < w) gx[i0 + o] += t_m2[o] + (T)2 * xb_all[i0 + o] * t_s22[o] + xa_all[i0 + o] * t_s12[o];
}

// XYB adjoint to the linear planes of this scale, plus the coarser scale's gradient spread over its 2x2 blocks.
template <typename T>
__global__ void k_xyb_adj(const T* __restrict__ lin, const T* __restrict__ g_xyb, int w, int h,
                          const T* __restrict__ g_coarse, int cw, T* __restrict__ g_lin) {
  grid_chain();
  const T M00 = (T)kM00, M01 = (T)kM01, M02 = (T)kM02, M10 = (T)kM10, M11 = (T)kM11, M12 = (T)kM12;
  const T M20 = (T)kM20, M21 = (T)kM21, M22 = (T)kM22, bias = (T)kBiasD;
  const T zero = 0, one = 1, three = 3, half = (T)0.5, seven = 7;
  const long long n = (long long)w * h, cn = (long long)cw * ((h + 1) / 2);
  for (long long i = tid1(); i < n; i += (long long)gridDim.x * blockDim.x) {
    const T r = lin[i], g = lin[n + i], b = lin[2 * n + i];
    const T u0 = M00 * r + M01 * g + M02 * b + bias, u1 = M10 * r + M11 * g + M12 * b + bias,
            u2 = M20 * r + M21 * g + M22 * b + bias;
    const T d0 = u0 > zero ? one / (three * cbrt_t(u0) * cbrt_t(u0)) : zero;
    const T d1 = u1 > zero ? one / (three * cbrt_t(u1) * cbrt_t(u1)) : zero;
    const T d2 = u2 > zero ? one / (three * cbrt_t(u2) * cbrt_t(u2)) : zero;
    const T gX = g_xyb[i], gY = g_xyb[n + i], gB = g_xyb[2 * n + i];
    const T gu0 = (seven * gX + half * gY - half * gB) * d0, gu1 = (-seven * gX + half * gY - half * gB) * d1,
            gu2 = gB * d2;
    T o[3] = {gu0 * M00 + gu1 * M10 + gu2 * M20, gu0 * M01 + gu1 * M11 + gu2 * M21,
              gu0 * M02 + gu1 * M12 + gu2 * M22};
    if (g_coarse) {
      const unsigned ui = (unsigned)i;  // within one plane: fewer than 2^32 samples
      const int y = (int)(ui / (unsigned)w), x = (int)(ui - (unsigned)y * (unsigned)w), ox = x / 2, oy = y / 2;
      const int nx = min(2 * ox + 2, w) - 2 * ox, ny = min(2 * oy + 2, h) - 2 * oy;
      const T inv = one / (T)(nx * ny);
#pragma unroll
      for (int c = 0; c < 3; c++) o[c] += g_coarse[c * cn + (long long)oy * cw + ox] * inv;
    }
#pragma unroll
    for (int c = 0; c < 3; c++) g_lin[c * n + i] = o[c];
  }
}

// Through the sRGB curve to the samples (interleaved RGB), written as f64.
template <typename T>
__global__ void k_grad_out(const T* __restrict__ g_lin, const float* __restrict__ dist, long long n,
                           double* __restrict__ grad) {
  grid_chain();
  __shared__ double dlut[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) dlut[i] = c_dlin8[i];
  __syncthreads();
  for (long long i = tid1(); i < n; i += (long long)gridDim.x * blockDim.x)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float v = dist[i * 3 + c];
      const int k = sample8(v);
      grad[i * 3 + c] = (double)g_lin[c * n + i] * (k >= 0 ? dlut[k] : srgb64_deriv((double)v));
    }
}

unsigned grid_of(long long n) {
  return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, kSms * 32));
}

// Moments of planes blurred together: their two buffers of five planes each stay within this (320 bytes a pixel in FP64:
// images of up to 80 MP go as one group, in FP32 of up to 160 MP) and within what can be allocated. Beside them the pass
// holds 24 planes (192 bytes a pixel in FP64); at the least, a plane of scale 0 at a time, 272 bytes a pixel in all.
constexpr long long kAdjBudgetBytes = 24ll << 30;

// The whole pass in real type T; workspace buffers are named per type.
template <typename T>
int grad_impl(rcg_ctx* ctx, const uint8_t* d_ref, const float* d_dist, int w, int h, double* score, double* d_grad) {
  const std::string pfx = sizeof(T) == 8 ? "adj64_" : "adj32_";
  auto ws = [&](const char* name, size_t count) { return (T*)workspace(ctx, (pfx + name).c_str(), count * sizeof(T)); };
  // constants
  double k[2 * kR + 1], sum = 0.0;
  for (int i = 0; i <= 2 * kR; i++) {
    const double x = (double)(i - kR);
    k[i] = std::exp(-0.5 / (1.5 * 1.5) * x * x);
    sum += k[i];
  }
  float k32[2 * kR + 1];
  for (int i = 0; i <= 2 * kR; i++) {
    k[i] /= sum;
    k32[i] = (float)k[i];
  }
  double lin8[256], dlin8[256], hs[kMaxScales * 18];
  CopiesDone done(ctx);
  symbol_to_device(ctx, c_k64, k, sizeof k);
  symbol_to_device(ctx, c_k32, k32, sizeof k32);
  for (int i = 0; i < 256; i++) {
    const double v = (double)i / 255.0;
    lin8[i] = v <= 0.04045 ? v / 12.92 : std::pow((v + 0.055) / 1.055, 2.4);
    dlin8[i] = v <= 0.04045 ? 1.0 / (12.92 * 255.0) : 2.4 * std::pow((v + 0.055) / 1.055, 1.4) / (1.055 * 255.0);
  }
  symbol_to_device(ctx, c_lin8, lin8, sizeof lin8);
  symbol_to_device(ctx, c_dlin8, dlin8, sizeof dlin8);
  // pyramid of both images (linear)
  struct Sc {
    int w, h;
    long long n, off;
  };
  std::vector<Sc> sc;
  long long total = 0;
  for (int s = 0, sw = w, sh = h; s < kMaxScales && sw >= kMinSide && sh >= kMinSide; s++) {
    sc.push_back({sw, sh, (long long)sw * sh, total});
    total += 3LL * sw * sh;
    sw = (sw + 1) / 2;
    sh = (sh + 1) / 2;
  }
  const int ns = (int)sc.size();
  if (ns == 0) return fail(ctx, RCG_INVALID, "SSIMULACRA 2 needs at least 8x8 pixels");
  const long long n0 = sc[0].n;
  // Every channel of every scale, and the groups of them that go through the blurs together: all, when their moments
  // (ten planes each, of which five are kept for the backward pass) fit the budget.
  struct Plane {
    int s, c;
  };
  std::vector<std::vector<Plane>> groups;
  long long most = 0, half = 0;
  auto group_by = [&](long long budget) {
    groups.clear();
    long long used = 0;
    most = 0;
    for (int s = 0; s < ns; s++)
      for (int c = 0; c < 3; c++) {
        if (groups.empty() || used + 5 * sc[s].n > budget) {
          groups.emplace_back();
          used = 0;
        }
        groups.back().push_back({s, c});
        used += 5 * sc[s].n;
        most = std::max(most, used);
      }
    half = (most + 31) / 32 * 32;  // the second buffer starts as aligned as the first
  };
  T* pa = ws("pa", total);
  T* pb = ws("pb", total);
  T* xa = ws("xa", total);
  T* xb = ws("xb", total);
  T* gx = ws("gx", total);   // d score / d xb
  T* gl = ws("gl", total);   // d score / d linear
  // The jobs of a group with `ctas` CTAs each (by plane size).
  auto jobs_of = [&](const std::vector<Plane>& g, auto ctas) {
    AdjJobs jobs;
    std::memset(&jobs, 0, sizeof jobs);
    long long m = 0, at = 0;
    for (const Plane& p : g) {
      AdjJob& j = jobs.j[jobs.count];
      j = AdjJob{sc[p.s].w, sc[p.s].h, sc[p.s].n, sc[p.s].off + p.c * sc[p.s].n, m};
      m += 5 * j.n;
      jobs.cta0[jobs.count++] = (unsigned)at;
      at += (long long)ctas(j);
    }
    jobs.cta0[jobs.count] = (unsigned)at;
    return jobs;
  };
  auto grid = [](const AdjJobs& j) { return j.cta0[j.count]; };
  auto by_samples = [](const AdjJob& j) { return (j.n + 255) / 256; };
  auto by_row_runs = [](const AdjJob& j) { return (row_runs(j.w, j.h) + 255) / 256; };
  auto by_runs = [](int rows) {
    return [rows](const AdjJob& j) { return ((long long)((j.h + rows - 1) / rows) * j.w + 255) / 256; };
  };
  auto by_grid = [](const AdjJob& j) { return (long long)grid_of(j.n); };
  double* sums = (double*)workspace(ctx, (pfx + "sums").c_str(), sizeof(double) * kMaxScales * 18);
  if (!pa || !pb || !xa || !xb || !gx || !gl || !sums) return RCG_NO_MEMORY;
  // Row-blurred products, later the gradients of the moments; the moments, later those through the transposed column
  // blur. One buffer, last: where it cannot be had, smaller groups, down to a plane at a time.
  T* hb5 = nullptr;
  double* parts = nullptr;
  for (long long budget = kAdjBudgetBytes / (2 * (long long)sizeof(T));; budget = most / 2) {
    group_by(budget);
    size_t max_parts = 0;
    for (const auto& g : groups) max_parts = std::max<size_t>(max_parts, grid(jobs_of(g, by_grid)));
    parts = (double*)workspace(ctx, (pfx + "parts").c_str(), sizeof(double) * 6 * max_parts);
    if (!parts) return RCG_NO_MEMORY;
    if ((hb5 = ws("moments", 2 * half))) break;
    if (most <= 5 * n0) return RCG_NO_MEMORY;
  }
  T* const mom = hb5 + half;
  const bool keep = groups.size() == 1;
  RCG_LAUNCH(ctx, "adj_lin", k_lin<T>, grid_of(n0), 256, 0, d_ref, d_dist, n0, pa, pb);
  for (int s = 1; s < ns; s++)
    RCG_LAUNCH(ctx, "adj_down", k_down<T>, grid_rows(sc[s].w, sc[s].h, 6), 256, 0, pa + sc[s - 1].off,
               pb + sc[s - 1].off, sc[s - 1].w, sc[s - 1].h, pa + sc[s].off, pb + sc[s].off, sc[s].w, sc[s].h);
  {
    std::vector<Plane> first;  // a scale's three channels go by its first
    for (int s = 0; s < ns; s++) first.push_back({s, 0});
    const AdjJobs jobs = jobs_of(first, by_samples);
    RCG_LAUNCH(ctx, "adj_xyb", k_xyb<T>, dim3(grid(jobs), 2), 256, 0, jobs, pa, pb, xa, xb);
  }
  // forward: the moments and map sums of every plane
  auto moments = [&](const std::vector<Plane>& g) {
    const AdjJobs rows = jobs_of(g, by_row_runs), cols = jobs_of(g, by_runs(kRunN));
    RCG_LAUNCH(ctx, "adj_hblur5", k_hblur5<T>, grid(rows), 256, 0, rows, xa, xb, hb5);
    RCG_LAUNCH(ctx, "adj_vblur", k_vblur_n<T>, dim3(grid(cols), 5), 256, 0, cols, hb5, mom);
  };
  for (const auto& g : groups) {
    moments(g);
    const AdjJobs jobs = jobs_of(g, by_grid);
    AdjSums to;
    for (size_t k = 0; k < g.size(); k++) to.at[k] = g[k].s * 18 + g[k].c * 6;
    RCG_LAUNCH(ctx, "adj_maps", k_maps<T>, grid(jobs), 256, 0, jobs, mom, xa, xb, parts);
    RCG_LAUNCH(ctx, "adj_sum_parts", k_sum_parts, (unsigned)g.size(), 192, 0, jobs, to, parts, sums);
  }
  int rc = read_back(ctx, hs, sums, sizeof hs);
  if (rc != RCG_OK) return rc;
  cudaError_t e = wait_stream(ctx);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "ssimulacra2 gradient");
  // final mapping (:491-511) and d score / d stat
  double st[kMaxScales][3][6], wst[kMaxScales][3][6];
  for (int s = 0; s < ns; s++) {
    const double count = (double)sc[s].n;
    for (int c = 0; c < 3; c++)
      for (int m = 0; m < 3; m++) {
        st[s][c][2 * m] = hs[s * 18 + c * 6 + 2 * m] / count;
        st[s][c][2 * m + 1] = std::pow(hs[s * 18 + c * 6 + 2 * m + 1] / count, 0.25);
      }
  }
  const double* W = scorer_weights();
  double wsum = 0.0;
  int i = 0;
  for (int c = 0; c < 3; c++)
    for (int s = 0; s < ns; s++)
      for (int nrm = 0; nrm < 2; nrm++)
        for (int m = 0; m < 3; m++) {
          wst[s][c][2 * m + nrm] = W[i];
          wsum += W[i] * std::fabs(st[s][c][2 * m + nrm]);
          i++;
        }
  const double kq = 0.9562382616834844, q = wsum * kq;
  const double P = 2.326765642916932 * q - 0.020884521182843837 * q * q + 6.248496625763138e-05 * q * q * q;
  const double ex = 0.6276336467831387;
  *score = P > 0.0 ? 100.0 - 10.0 * std::pow(P, ex) : 100.0;
  const long long npx = (long long)w * h;
  if (!d_grad) return RCG_OK;  // the score alone
  if (!(P > 0.0)) {
    cudaMemsetAsync(d_grad, 0, sizeof(double) * 3 * npx, ctx->stream);
    return RCG_OK;
  }
  const double dsum = -10.0 * ex * std::pow(P, ex - 1.0) *
                      (2.326765642916932 - 2.0 * 0.020884521182843837 * q + 3.0 * 6.248496625763138e-05 * q * q) *
                      kq;
  // backward: d score / d xb of every plane, then to linear light from the coarsest scale to the finest
  for (const auto& g : groups) {
    if (!keep) moments(g);
    NormCoefs coefs;
    std::memset(&coefs, 0, sizeof coefs);
    for (size_t k = 0; k < g.size(); k++) {
      const int s = g[k].s, c = g[k].c;
      const double count = (double)sc[s].n;
      for (int m = 0; m < 3; m++) {
        coefs.job[k].g1[m] = dsum * wst[s][c][2 * m] / count;
        const double mean4 = hs[s * 18 + c * 6 + 2 * m + 1] / count;
        coefs.job[k].g4[m] = mean4 > 0.0 ? dsum * wst[s][c][2 * m + 1] * std::pow(mean4, -0.75) / count : 0.0;
      }
    }
    const AdjJobs all = jobs_of(g, by_samples), cols = jobs_of(g, by_runs(kRun)), rows = jobs_of(g, by_row_runs);
    RCG_LAUNCH(ctx, "adj_mapgrad", k_mapgrad<T>, grid(all), 256, 0, all, coefs, mom, xa, xb, hb5, gx);
    // the three gradient planes through the transposed column blur, then the row blur (its own transpose)
    RCG_LAUNCH(ctx, "adj_vblur_t", k_vblur_t<T>, dim3(grid(cols), 3), 256, 0, cols, hb5, mom);
    RCG_LAUNCH(ctx, "adj_hblur", k_hblur_combine<T>, grid(rows), 256, 0, rows, mom, xa, xb, gx);
  }
  for (int s = ns - 1; s >= 0; s--)
    RCG_LAUNCH(ctx, "adj_xyb_adj", k_xyb_adj<T>, grid_of(sc[s].n), 256, 0, pb + sc[s].off, gx + sc[s].off, sc[s].w,
               sc[s].h, s + 1 < ns ? gl + sc[s + 1].off : nullptr, s + 1 < ns ? sc[s + 1].w : 0, gl + sc[s].off);
  RCG_LAUNCH(ctx, "adj_out", k_grad_out<T>, grid_of(npx), 256, 0, gl + sc[0].off, d_dist, npx, d_grad);
  return RCG_OK;
}

}  // namespace

int ssim2_grad_device(rcg_ctx* ctx, const uint8_t* d_ref, const float* d_dist, int w, int h, double* score,
                      double* d_grad, bool fp32) {
  return fp32 ? grad_impl<float>(ctx, d_ref, d_dist, w, h, score, d_grad)
              : grad_impl<double>(ctx, d_ref, d_dist, w, h, score, d_grad);
}

}  // namespace rcg
