// The tables of one search step, filled on the device by one CTA, and what they are made of (shared with the host's
// version in codec.cu, which must give the same bits).
#pragma once

#include "rcg_internal.cuh"

namespace rcg {

// The constant tables, for the host and in device memory (an array local to a function that is indexed at run time is
// written to the stack by every thread; in constant memory every lane's own index costs a turn).
#define RCG_ZIGZAG                                                                                                \
  {0,  1,  8,  16, 9,  2,  3,  10, 17, 24, 32, 25, 18, 11, 4,  5,  12, 19, 26, 33, 40, 48, 41, 34, 27, 20, 13, 6, \
   7,  14, 21, 28, 35, 42, 49, 56, 57, 50, 43, 36, 29, 22, 15, 23, 30, 37, 44, 51, 58, 59, 52, 45, 38, 31, 39,    \
   46, 53, 60, 61, 54, 47, 55, 62, 63}
#define RCG_AAN {1.0f, 1.3870398f, 1.306563f, 1.1758756f, 1.0f, 0.78569495f, 0.5411961f, 0.27589938f}
#define RCG_PERCEPTUAL_Q                                                                                       \
  {16, 16, 16,  18,  25,  37,  56,  85,  16, 17, 20,  27,  34,  40,  53,  75,                                  \
   16, 20, 24,  31,  43,  62,  91,  135, 18, 27, 31,  40,  53,  74,  106, 156,                                 \
   25, 34, 43,  53,  69,  94,  131, 189, 37, 40, 62,  74,  94,  124, 169, 238,                                 \
   56, 53, 91,  106, 131, 169, 226, 255, 85, 75, 135, 156, 189, 238, 255, 255}
static const uint8_t h_zigzag[64] = RCG_ZIGZAG;
static const float h_aan[8] = RCG_AAN;
static const uint8_t h_perceptual_q[64] = RCG_PERCEPTUAL_Q;
static __device__ const uint8_t d_zigzag[64] = RCG_ZIGZAG;
static __device__ const float d_aan[8] = RCG_AAN;
static __device__ const uint8_t d_perceptual_q[64] = RCG_PERCEPTUAL_Q;
#ifdef __CUDA_ARCH__
#define RCG_TABLE(name) d_##name
#else
#define RCG_TABLE(name) h_##name
#endif
__host__ __device__ inline int zigzag(int k) { return RCG_TABLE(zigzag)[k]; }  // jpeg/src/lib.rs:14-19
// The same where k is known at compile time (unrolled loops).
__host__ __device__ constexpr int zigzag_known(int k) {
  constexpr int Z[64] = RCG_ZIGZAG;
  return Z[k];
}
__host__ __device__ inline float aan(int i) { return RCG_TABLE(aan)[i]; }      // jpeg/src/dct.rs:8 (AAN scale factors)
__host__ __device__ inline uint8_t perceptual_q(int i) { return RCG_TABLE(perceptual_q)[i]; }  // jpeg/src/quality.rs:26-35
#undef RCG_TABLE

// Exact f32 arithmetic on host and device: round-to-nearest, never contracted.
__host__ __device__ inline float fadd(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  volatile float r = a + b;
  return r;
#endif
}
__host__ __device__ inline float fsub(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fsub_rn(a, b);
#else
  volatile float r = a - b;
  return r;
#endif
}
__host__ __device__ inline float fmul(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  volatile float r = a * b;
  return r;
#endif
}
__host__ __device__ inline float fdiv(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fdiv_rn(a, b);
#else
  volatile float r = a / b;
  return r;
#endif
}

// Sampling factors build_coefs chooses (jpeg/src/encode.rs:428-439).
__host__ __device__ inline void sampling(int channels, int subsampling, int quality, int* hmax, int* vmax) {
  if (channels == 1) {
    *hmax = 1;
    *vmax = 1;
    return;
  }
  switch (subsampling) {
    case RCG_SUB_420: *hmax = 2; *vmax = 2; break;
    case RCG_SUB_422: *hmax = 2; *vmax = 1; break;
    case RCG_SUB_444: *hmax = 1; *vmax = 1; break;
    default:
      if (quality < 90) { *hmax = 2; *vmax = 2; } else { *hmax = 1; *vmax = 1; }
  }
}

// FDCT cache slot of a component for a sampling layout: 3 caches (Y, Cb, Cr) per layout kind.
__host__ __device__ inline int layout_kind(int hmax, int vmax) { return hmax == 2 ? (vmax == 2 ? 0 : 1) : 2; }

// One entry of the per-quality tables, shared by the host (fill_step) and the device (step_tables_body) so both give
// identical bits. `q` is the quantization table (natural order).
//   quant value at a natural index whose perceptual entry is p (jpeg/src/quality.rs:6-15)
__host__ __device__ inline uint8_t quality_entry(int quality, unsigned p) {
  unsigned q = (unsigned)(quality < 1 ? 1 : (quality > 100 ? 100 : quality));
  unsigned scale = q < 50 ? 5000 / q : 200 - 2 * q;
  unsigned v = (p * scale + 50) / 100;
  return (uint8_t)(v < 1 ? 1 : (v > 255 ? 255 : v));
}
__host__ __device__ inline uint8_t qtable_entry(int quality, int n) { return quality_entry(quality, perceptual_q(n)); }
//   dequantization multiplier at natural index n = v*8+u: q[v*8+u] * AAN[u] * AAN[v] (jpeg/src/decode.rs:1316-1321)
__host__ __device__ inline float mult_of(uint8_t q, float aan_u, float aan_v) { return fmul(fmul((float)q, aan_u), aan_v); }
__host__ __device__ inline float mult_entry(const uint8_t* q, int n) { return mult_of(q[n], aan(n % 8), aan(n / 8)); }
//   fdct divisor for zigzag position k: fdct_divisors stores 1 / (q[v*8+u] * AAN[u] * AAN[v] * 8) at [u*8+v]
//   (jpeg/src/encode.rs:174-183) and quantize_plane reads it at ZZ_T[k] = (n%8)*8 + n/8 (:202), i.e. u = n%8,
//   v = n/8, q[v*8+u] = q[n]
__host__ __device__ inline float divz_entry(const uint8_t* q, int k) {
  return fdiv(1.0f, fmul(mult_entry(q, zigzag(k)), 8.0f));
}

// Block layout of a candidate (jpeg/src/encode.rs:428-443, :511-517).
__host__ __device__ inline void fill_layout(StepDesc* st, int quality, int subsampling, int channels, int trellis,
                                            int w, int h) {
  st->quality = quality;
  st->use_trellis = (trellis && quality < 100) ? 1 : 0;
  int hmax, vmax;
  sampling(channels, subsampling, quality, &hmax, &vmax);
  st->hmax = hmax;
  st->vmax = vmax;
  int pw = (w + 8 * hmax - 1) / (8 * hmax) * 8 * hmax;
  int ph = (h + 8 * vmax - 1) / (8 * vmax) * 8 * vmax;
  st->ncomp = channels == 1 ? 1 : 3;
  long long blk = 0, poff = 0;
  int kind = layout_kind(hmax, vmax);
  for (int c = 0; c < st->ncomp; c++) {
    CompDesc& cd = st->comp[c];
    cd.h = c == 0 ? hmax : 1;
    cd.v = c == 0 ? vmax : 1;
    cd.bw = c == 0 ? pw / 8 : pw / hmax / 8;
    cd.bh = c == 0 ? ph / 8 : ph / vmax / 8;
    cd.cls = c == 0 ? 0 : 1;
    cd.cache = kind * 3 + c;
    cd.blk0 = blk;
    cd.plane_off = poff;
    blk += (long long)cd.bw * cd.bh;
    poff += (long long)cd.bw * 8 * cd.bh * 8;
  }
  st->nblocks = blk;
}

// Table of one component for a requantization to `quality` (jpeg/src/encode.rs:121-126): the quality's table,
// never finer than the source's.
__host__ __device__ inline uint8_t requant_entry(const uint8_t* old, int quality, int n) {
  uint8_t t = qtable_entry(quality, n);
  return t > old[n] ? t : old[n];
}

// The candidate that the bisection state names: its quality, layout and tables, or active = 0 once the search has
// finished (or paused). kStepThreads threads, one per (component, coefficient) entry and one for the layout; the Rdo
// median is the value of rank 31 among q[1..63], the one the reference's sort yields. One CTA: bound by its own latency
// (a launch of its own took 5 us a step, 10 requantizing), so a search fills them at the end of the launch that scored the
// step before, and what does not depend on the quality is loaded before that end (step_prepare; 2.4 us of the 12.7 that
// launch took at 240x180 were spent here without it, 1.5 with).
constexpr int kStepThreads = 256;

// What a thread's entries are made of, by k: one load of 32 bytes, none of them waiting for another.
struct __align__(16) StepPre {
  float au, av, nu, nv;          // AAN factors of the natural index k and of n
  int n;                         // natural index of zigzag position k
  uint8_t pk, pn;                // perceptual entries of both
  uint8_t old_k, old_n;          // requantization: the source's entries
  int ncomp;
  int pad;
};
struct StepPreTable {
  StepPre e[64];
};
constexpr StepPreTable step_pre_table() {
  constexpr int Z[64] = RCG_ZIGZAG;
  constexpr float A[8] = RCG_AAN;
  constexpr uint8_t P[64] = RCG_PERCEPTUAL_Q;
  StepPreTable t = {};
  for (int k = 0; k < 64; k++)
    t.e[k] = StepPre{A[k % 8], A[k / 8], A[Z[k] % 8], A[Z[k] / 8], Z[k], P[k], P[Z[k]], 0, 0, 3, 0};
  return t;
}
static __device__ const StepPreTable d_step_pre = step_pre_table();
#undef RCG_ZIGZAG
#undef RCG_AAN
#undef RCG_PERCEPTUAL_Q

__device__ __forceinline__ StepPre step_prepare(const StepDesc* st, const NextStep& next) {
  const int c = threadIdx.x / 64, k = threadIdx.x % 64;
  StepPre p = d_step_pre.e[k];
  if (next.kind == kNextRequant && c < 3) {
    p.old_k = st->src_qt[c][k];
    p.old_n = st->src_qt[c][p.n];
    p.ncomp = st->ncomp;
  }
  return p;
}

// Every thread of the CTA (kStepThreads of them) calls it.
__device__ __forceinline__ void step_tables_body(const SearchState& ss, StepDesc* __restrict__ st, const NextStep& next,
                                                 const StepPre& p) {
  __shared__ __align__(16) float rq[3][64];
  __shared__ float median[3];
  const int t = threadIdx.x;
  if (ss.done) {
    if (t == 0) st->active = 0;
    return;
  }
  const int step = ss.step;
  const int q = ss.qs[step];
  const bool requant = next.kind == kNextRequant;
  const int c = t / 64, k = t % 64;
  if (t == 192) {
    st->active = 1;
    st->requant = requant ? 1 : 0;
    st->coefs = next.slots + (long long)step * next.slot_stride;
    if (requant) {
      st->quality = q;
    } else {
      fill_layout(st, q, ss.subsampling, ss.channels, ss.trellis, next.w, next.h);
      st->pweights = next.pweights;
    }
  }
  for (int i = t; i < 512; i += kStepThreads) (&st->hist[0][0])[i] = 0;
  // luma_table == chroma_table (jpeg/src/quality.rs:37-43): every component gets the same entries. A requantization
  // keeps each component's own (never finer than the source's); its components' count is the source's.
  const bool live = c < p.ncomp && c < 3;
  bool differs = false;
  if (live) {
    uint8_t qk = quality_entry(q, p.pk), qn = quality_entry(q, p.pn);
    if (requant) {  // requant_entry
      qk = max(qk, p.old_k);
      qn = max(qn, p.old_n);
      differs = qk != p.old_k;
      st->ratio[c][k] = fdiv((float)p.old_n, (float)qn);
    } else {
      st->divz[c][k] = fdiv(1.0f, fmul(mult_of(qn, p.nu, p.nv), 8.0f));
    }
    st->qt[c][k] = qk;
    st->mult[c][k] = mult_of(qk, p.au, p.av);
    rq[c][k] = (float)qn;
    st->rq[c][k] = (float)qn;
  }
  const bool changed = __syncthreads_or(differs);
  if (live && k >= 1) {
    const float rk = rq[c][k];
    int below = 0, upto = 0;
#pragma unroll 4
    for (int j = 0; j < 16; j++) {
      const float4 v = *reinterpret_cast<const float4*>(&rq[c][4 * j]);
      if (j > 0) {
        below += v.x < rk;
        upto += v.x <= rk;
      }
      below += (v.y < rk) + (v.z < rk) + (v.w < rk);
      upto += (v.y <= rk) + (v.z <= rk) + (v.w <= rk);
    }
    if (below <= 31 && upto > 31) median[c] = rk;  // several threads of one value may write it
  }
  __syncthreads();
  if (live) {
    st->rw[c][k] = k == 0 ? 1.0f : fdiv(median[c], rq[c][k]);
    if (k == 0) st->lambda[c] = fmul(fmul(0.02f, median[c]), median[c]);  // TRELLIS_KAPPA (jpeg/src/encode.rs:42)
  }
  if (requant && t == 0) {  // the trellis runs if some component's table changed (jpeg/src/encode.rs:127, :152)
    st->changed = changed ? 1 : 0;
    st->use_trellis = (ss.trellis && changed) ? 1 : 0;
  }
}

}  // namespace rcg
