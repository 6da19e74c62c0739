// JPEG encoder and decoder kernels of the quality search (K1-K7).
//
// Bit-exactness: every f32 operation the reference performs is written as an explicit round-to-nearest intrinsic
// (__fadd_rn, __fsub_rn, __fmul_rn, __fdiv_rn) in the reference's order, so no FMA contraction can change a result
// (rustc never contracts). The translation unit is also compiled with -fmad=false as a second guard. Integer steps
// (colour conversion, subsampling, upsampling, histograms) are exact by construction.
//
// Layouts in HBM:
//   FDCT cache         f32, [64][nblocks] per component: zigzag coefficient k of block b at k*nblocks + b, so a
//                      thread-per-block kernel reads one coalesced row per coefficient. Quality-independent: the
//                      reference recomputes it for every candidate (jpeg/src/encode.rs:189-196).
//   coefficients       i16, the flat CoefImage: components back to back, 64 zigzag values per block.
//   decoded planes     u8, one per component, stride blocks_w*8 (jpeg/src/decode.rs:1322-1323).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>

#include "rcg_internal.cuh"
#include "huffman.cuh"
#include "step_tables.cuh"

namespace rcg {

// ------------------------------------------------------------------------------------------------ tables

// jpeg/src/dct.rs:125-129: round half to even for |x| < 2^22; wrapping integer arithmetic beyond, as the reference.
__device__ __forceinline__ int round_f32(float x) {
  return (int)((unsigned)__float_as_int(__fadd_rn(x, 12582912.0f)) - 0x4B400000u);
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return min(max(v, lo), hi); }

// The per-quality tables of one candidate: quantization tables (jpeg/src/quality.rs), fdct divisors
// (jpeg/src/encode.rs:174-183), dequantization multipliers (jpeg/src/decode.rs:1316-1321), the Rdo parameters that
// do not depend on the rate model (jpeg/src/rdo.rs:28-45), and the block layout (jpeg/src/encode.rs:440-517).
// Host version (single calls); step_tables_body computes the same entries in parallel on the device.
inline void fill_step(StepDesc* st, int quality, int subsampling, int channels, int trellis, int w, int h) {
  const float kappa = 0.02f;  // TRELLIS_KAPPA, jpeg/src/encode.rs:42
  fill_layout(st, quality, subsampling, channels, trellis, w, h);
  // luma_table == chroma_table (jpeg/src/quality.rs:37-43): every component gets the same entries
  for (int c = 0; c < 3; c++) {
    uint8_t* qt = st->qt[c];
    for (int n = 0; n < 64; n++) qt[n] = qtable_entry(quality, n);
    for (int k = 0; k < 64; k++) st->divz[c][k] = divz_entry(qt, k);
    for (int n = 0; n < 64; n++) st->mult[c][n] = mult_entry(qt, n);
    // Rdo::new: q per zigzag position, median of q[1..] (sorted, index 31), w = (median/q)^1, lambda.
    float sorted[63];
    for (int k = 0; k < 64; k++) st->rq[c][k] = (float)qt[zigzag(k)];
    for (int k = 1; k < 64; k++) sorted[k - 1] = st->rq[c][k];
    std::sort(sorted, sorted + 63);
    float median = sorted[31];
    st->rw[c][0] = 1.0f;
    // FREQ_WEIGHT_GAMMA is 1.0 (jpeg/src/rdo.rs:12) and pow(x, 1) == x, so w = median / q exactly.
    for (int k = 1; k < 64; k++) st->rw[c][k] = fdiv(median, st->rq[c][k]);
    st->lambda[c] = fmul(fmul(kappa, median), median);
  }
}

void fill_mult(StepDesc* st, const uint8_t* qtables, int ntables) {
  for (int c = 0; c < 3; c++) {
    const uint8_t* qt = qtables + 64 * (c == 0 || ntables < 2 ? 0 : 1);
    std::memcpy(st->qt[c], qt, 64);
    for (int n = 0; n < 64; n++) st->mult[c][n] = mult_entry(qt, n);
  }
}

float mult_entry_host(const uint8_t* q, int n) { return mult_entry(q, n); }

int zigzag_natural(int k) { return zigzag(k); }

void qtables_for(int quality, uint8_t* out128) {
  for (int n = 0; n < 64; n++) out128[n] = out128[64 + n] = qtable_entry(quality, n);
}

void host_step_tables(StepDesc* st, int quality, int subsampling, int channels, int trellis, int w, int h) {
  std::memset(st, 0, sizeof *st);
  st->active = 1;
  fill_step(st, quality, subsampling, channels, trellis, w, h);
}

struct CacheSet {
  const float* p[9];
};

// Locate the component of a global block index.
__device__ __forceinline__ int comp_of(const StepDesc* st, long long gb) {
  int c = 0;
  if (st->ncomp > 1 && gb >= st->comp[1].blk0) c = gb >= st->comp[2].blk0 ? 2 : 1;
  return c;
}

// ------------------------------------------------------------------------------------------------ K1, K2 image to FDCT

// jpeg/src/dct.rs:20-57 (fdct_pass) on column j of a row-major 8x8 block held in registers.
__device__ __forceinline__ void fdct_pass(float (&d)[64]) {
#pragma unroll
  for (int j = 0; j < 8; j++) {
    float d0 = d[0 * 8 + j], d1 = d[1 * 8 + j], d2 = d[2 * 8 + j], d3 = d[3 * 8 + j];
    float d4 = d[4 * 8 + j], d5 = d[5 * 8 + j], d6 = d[6 * 8 + j], d7 = d[7 * 8 + j];
    float tmp0 = fadd(d0, d7), tmp7 = fsub(d0, d7), tmp1 = fadd(d1, d6), tmp6 = fsub(d1, d6);
    float tmp2 = fadd(d2, d5), tmp5 = fsub(d2, d5), tmp3 = fadd(d3, d4), tmp4 = fsub(d3, d4);
    float tmp10 = fadd(tmp0, tmp3), tmp13 = fsub(tmp0, tmp3), tmp11 = fadd(tmp1, tmp2), tmp12 = fsub(tmp1, tmp2);
    d[0 * 8 + j] = fadd(tmp10, tmp11);
    d[4 * 8 + j] = fsub(tmp10, tmp11);
    float z1 = fmul(fadd(tmp12, tmp13), 0.70710677f);
    d[2 * 8 + j] = fadd(tmp13, z1);
    d[6 * 8 + j] = fsub(tmp13, z1);
    float t10 = fadd(tmp4, tmp5), t11 = fadd(tmp5, tmp6), t12 = fadd(tmp6, tmp7);
    float z5 = fmul(fsub(t10, t12), 0.38268343f);
    float z2 = fadd(fmul(0.5411961f, t10), z5);
    float z4 = fadd(fmul(1.306563f, t12), z5);
    float z3 = fmul(t11, 0.70710677f);
    float z11 = fadd(tmp7, z3), z13 = fsub(tmp7, z3);
    d[5 * 8 + j] = fadd(z13, z2);
    d[3 * 8 + j] = fsub(z13, z2);
    d[1 * 8 + j] = fadd(z11, z4);
    d[7 * 8 + j] = fsub(z11, z4);
  }
}

__device__ __forceinline__ void transpose8(float (&b)[64]) {
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = i + 1; j < 8; j++) {
      float t = b[i * 8 + j];
      b[i * 8 + j] = b[j * 8 + i];
      b[j * 8 + i] = t;
    }
}

// From the image to the FDCT caches of one sampling layout. A CTA takes 256 x 16 pixels of the padded grid: the colour
// conversion with edge replication (jpeg/src/encode.rs:451-477) into shared memory, the chroma box filter
// (sum + n/2) / n (:478-499), then a thread per block: level shift (x - 128), FDCT (jpeg/src/dct.rs:59-65), stored in
// zigzag order (flat[ZZ_T[k]], jpeg/src/encode.rs:201-211) as cache[k * blocks + b], 32 blocks of a row side by side.
// What bounds it: the store of the caches (72 MB at 12 MP 4:2:0) at large sizes, its latency and launch at small ones.
// Measured against a launch each for the planes, either chroma plane and the three caches, whose planes made two trips
// through memory, converted and filtered a byte at a time: 12 MP 4:2:0 124 -> 48 us, 2 MP 56 -> 16, 240x180 4:4:4 26 -> 11.
constexpr int kFdW = 256, kFdH = 16, kFdThreads = 128;

struct FdctOut {
  float* cache[3];
  int bw[3], bh[3];
};

template <int kFx, int kFy, bool kGray>
__global__ void __launch_bounds__(kFdThreads) k_fdct_image(const uint8_t* __restrict__ src, int w, int h,
                                                           const FdctOut out) {
  grid_chain();
  constexpr bool kDown = !kGray && kFx * kFy > 1;
  constexpr int kSubW = kFdW / kFx, kSubH = kFdH / kFy;
  __shared__ __align__(16) uint8_t px[kGray ? 1 : 3][kFdH][kFdW];
  __shared__ __align__(16) uint8_t sub[2][kDown ? kSubH : 1][kDown ? kSubW : 8];
  const int t = threadIdx.x, x0 = blockIdx.x * kFdW, y0 = blockIdx.y * kFdH;
  constexpr int kBytes = kGray ? 4 : 12;  // of four pixels
  const size_t total = (size_t)w * h * (kBytes / 4);
#pragma unroll 2
  for (int e = t; e < kFdW / 4 * kFdH; e += kFdThreads) {
    const int q = e % (kFdW / 4), r = e / (kFdW / 4), gx = x0 + 4 * q;
    if (gx >= out.bw[0] * 8) continue;  // past the padded grid
    const size_t row = (size_t)min(y0 + r, h - 1) * w, at = (row + gx) * (kBytes / 4);
    uint32_t b[3] = {0, 0, 0};
    const int mis = (int)((uintptr_t)(src + at) & 3);
    // Bytes of any alignment: the aligned words that hold them and a funnel shift, where those lie in the image.
    if (gx + 4 <= w && at >= (size_t)mis && (mis == 0 || at + kBytes + 4 - mis <= total)) {
      const uint32_t* p = reinterpret_cast<const uint32_t*>(src + at - mis);
      uint32_t v[4];
#pragma unroll
      for (int k = 0; k < kBytes / 4; k++) v[k] = __ldg(p + k);
      v[kBytes / 4] = mis ? __ldg(p + kBytes / 4) : 0u;
#pragma unroll
      for (int k = 0; k < kBytes / 4; k++) b[k] = __funnelshift_r(v[k], v[k + 1], 8 * mis);
    } else {
#pragma unroll
      for (int k = 0; k < kBytes; k++) {
        const int px4 = kGray ? k : k / 3, c = kGray ? 0 : k % 3;
        const uint32_t v = src[(row + min(gx + px4, w - 1)) * (kBytes / 4) + c];
        b[k / 4] |= v << (8 * (k % 4));
      }
    }
    if (kGray) {
      *reinterpret_cast<uint32_t*>(&px[0][r][4 * q]) = b[0];
    } else {
      uint32_t yy = 0, cb = 0, cr = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        auto byte = [&](int i) { return (int)((b[i / 4] >> (8 * (i % 4))) & 0xFF); };
        const int rr = byte(3 * k), gg = byte(3 * k + 1), bb = byte(3 * k + 2);
        yy |= (uint32_t)(uint8_t)((19595 * rr + 38470 * gg + 7471 * bb + 32768) >> 16) << (8 * k);
        cb |= (uint32_t)(uint8_t)((-11059 * rr - 21709 * gg + 32768 * bb + (128 << 16) + 32767) >> 16) << (8 * k);
        cr |= (uint32_t)(uint8_t)((32768 * rr - 27439 * gg - 5329 * bb + (128 << 16) + 32767) >> 16) << (8 * k);
      }
      *reinterpret_cast<uint32_t*>(&px[0][r][4 * q]) = yy;
      *reinterpret_cast<uint32_t*>(&px[kGray ? 0 : 1][r][4 * q]) = cb;
      *reinterpret_cast<uint32_t*>(&px[kGray ? 0 : 2][r][4 * q]) = cr;
    }
  }
  __syncthreads();
  if constexpr (kDown) {
    static_assert(kFx == 2, "chroma is halved across");
    for (int e = t; e < 2 * kSubH * (kSubW / 4); e += kFdThreads) {
      const int q = e % (kSubW / 4), r = e / (kSubW / 4) % kSubH, c = e / (kSubW / 4 * kSubH);
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        unsigned sum = 0;
#pragma unroll
        for (int dy = 0; dy < kFy; dy++) {
          const uint2 p = *reinterpret_cast<const uint2*>(&px[1 + c][kFy * r + dy][8 * q]);
          const uint32_t word = k < 2 ? p.x : p.y;
          sum += ((word >> (16 * (k & 1))) & 0xFF) + ((word >> (16 * (k & 1) + 8)) & 0xFF);
        }
        v |= ((sum + kFx * kFy / 2) / (kFx * kFy)) << (8 * k);
      }
      *reinterpret_cast<uint32_t*>(&sub[c][r][4 * q]) = v;
    }
    __syncthreads();
  }
  constexpr int kLuma = kFdW / 8 * (kFdH / 8), kChroma = kGray ? 0 : kSubW / 8 * (kSubH / 8);
#pragma unroll 1
  for (int i = t; i < kLuma + 2 * kChroma; i += kFdThreads) {
    const int c = i < kLuma ? 0 : i < kLuma + kChroma ? 1 : 2;
    const int e = i - (c == 0 ? 0 : c == 1 ? kLuma : kLuma + kChroma), across = c == 0 ? kFdW / 8 : kSubW / 8;
    const int lx = e % across, ly = e / across;
    const int bx = blockIdx.x * across + lx, by = blockIdx.y * (c == 0 ? kFdH / 8 : kSubH / 8) + ly;
    if (bx >= out.bw[c] || by >= out.bh[c]) continue;
    const bool down = kDown && c > 0;
    const uint8_t* from = down ? &sub[c - 1][ly * 8][lx * 8] : &px[kGray ? 0 : c][ly * 8][lx * 8];
    float blk[64];
#pragma unroll
    for (int y = 0; y < 8; y++) {
      const uint2 v = *reinterpret_cast<const uint2*>(from + y * (down ? kSubW : kFdW));
#pragma unroll
      for (int x = 0; x < 8; x++) {
        const unsigned word = x < 4 ? v.x : v.y;
        blk[y * 8 + x] = fsub((float)((word >> (8 * (x & 3))) & 0xFF), 128.0f);
      }
    }
    fdct_pass(blk);
    transpose8(blk);
    fdct_pass(blk);
    const long long nb = (long long)out.bw[c] * out.bh[c], b = (long long)by * out.bw[c] + bx;
    float* cache = out.cache[c] + b;
#pragma unroll
    for (int k = 0; k < 64; k++) {
      constexpr int ZT[64] = {0,  8,  1,  2,  9,  16, 24, 17, 10, 3,  4,  11, 18, 25, 32, 40, 33, 26, 19, 12, 5,  6,
                              13, 20, 27, 34, 41, 48, 56, 49, 42, 35, 28, 21, 14, 7,  15, 22, 29, 36, 43, 50, 57, 58,
                              51, 44, 37, 30, 23, 31, 38, 45, 52, 59, 60, 53, 46, 39, 47, 54, 61, 62, 55, 63};
      cache[(long long)k * nb] = blk[ZT[k]];
    }
  }
}

int fdct_image(rcg_ctx* ctx, const uint8_t* d_src, int w, int h, int channels, int fx, int fy, float* const* d_caches,
               const int* bw, const int* bh) {
  FdctOut out;
  std::memset(&out, 0, sizeof out);
  for (int c = 0; c < (channels == 1 ? 1 : 3); c++) {
    out.cache[c] = d_caches[c];
    out.bw[c] = bw[c];
    out.bh[c] = bh[c];
  }
  const dim3 grid((unsigned)((bw[0] * 8 + kFdW - 1) / kFdW), (unsigned)((bh[0] * 8 + kFdH - 1) / kFdH));
  if (channels == 1)
    RCG_LAUNCH(ctx, "fdct_image", (k_fdct_image<1, 1, true>), grid, kFdThreads, 0, d_src, w, h, out);
  else if (fy == 2)
    RCG_LAUNCH(ctx, "fdct_image", (k_fdct_image<2, 2, false>), grid, kFdThreads, 0, d_src, w, h, out);
  else if (fx == 2)
    RCG_LAUNCH(ctx, "fdct_image", (k_fdct_image<2, 1, false>), grid, kFdThreads, 0, d_src, w, h, out);
  else
    RCG_LAUNCH(ctx, "fdct_image", (k_fdct_image<1, 1, false>), grid, kFdThreads, 0, d_src, w, h, out);
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ K3 quantize

__device__ __forceinline__ int bitlen(unsigned v) { return 32 - __clz(v); }

// Plain quantization (jpeg/src/encode.rs:200-205): round_f32(flat*div) clamped to +-2047. When the candidate uses
// the trellis, the plain coefficients only feed the AC symbol histogram of the rate model (jpeg/src/encode.rs:
// 221-228, :343-374: (run<<4)|size symbols, ZRL 0xF0, EOB 0x00; luma = component 0, chroma = components 1-2);
// otherwise they are the candidate's output.
// At most 128 registers: 4 CTAs per SM instead of 3 (34 -> 30 us per 12 MP candidate, small spill).
__device__ __forceinline__ void quantize_body(StepDesc* __restrict__ st, const CacheSet& cs, long long bx) {
  __shared__ unsigned int sh[2][256];
  if (!st->active) return;
  const bool hist = st->use_trellis != 0;
  if (hist) {
    for (int i = threadIdx.x; i < 512; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
  }
  const long long gb = bx * blockDim.x + threadIdx.x;
  if (gb < st->nblocks) {
    int c = comp_of(st, gb);
    const CompDesc& cd = st->comp[c];
    const long long nb = (long long)cd.bw * cd.bh;
    const float* cache = cs.p[cd.cache] + (gb - cd.blk0);
    const float* divz = st->divz[c];
    // All 64 loads are issued before any is used (fully unrolled into registers).
    int v[64];
#pragma unroll
    for (int k = 0; k < 64; k++) v[k] = clampi(round_f32(fmul(__ldg(cache + (long long)k * nb), divz[k])), -2047, 2047);
    if (!hist) {
      int16_t* out = st->coefs + gb * 64;
#pragma unroll
      for (int g = 0; g < 8; g++) {
        int4 pk;
        pk.x = (v[g * 8 + 0] & 0xFFFF) | (v[g * 8 + 1] << 16);
        pk.y = (v[g * 8 + 2] & 0xFFFF) | (v[g * 8 + 3] << 16);
        pk.z = (v[g * 8 + 4] & 0xFFFF) | (v[g * 8 + 5] << 16);
        pk.w = (v[g * 8 + 6] & 0xFFFF) | (v[g * 8 + 7] << 16);
        reinterpret_cast<int4*>(out)[g] = pk;
      }
    } else {
      unsigned* hs = sh[cd.cls];
      unsigned run = 0;
#pragma unroll
      for (int k = 1; k < 64; k++) {
        if (v[k] == 0) {
          run++;
          continue;
        }
        while (run >= 16) {
          atomicAdd(&hs[0xF0], 1u);
          run -= 16;
        }
        unsigned size = (unsigned)bitlen((unsigned)abs(v[k]));
        atomicAdd(&hs[(run << 4) | size], 1u);
        run = 0;
      }
      if (run > 0) atomicAdd(&hs[0], 1u);
    }
  }
  if (hist) {
    __syncthreads();
    for (int i = threadIdx.x; i < 512; i += blockDim.x) {
      unsigned v = (&sh[0][0])[i];
      if (v) atomicAdd(&(&st->hist[0][0])[i], v);
    }
  }
}

__global__ void __launch_bounds__(128, 4) k_quantize(StepDesc* __restrict__ st, CacheSet cs) {
  grid_chain();
  quantize_body(st + blockIdx.y, cs, blockIdx.x);  // blockIdx.y: the candidate of several encoded at once
}

int quantize(rcg_ctx* ctx, StepDesc* d_step, const float* const* d_caches, long long max_blocks, int count) {
  CacheSet cs;
  for (int i = 0; i < 9; i++) cs.p[i] = d_caches[i];
  const dim3 grid((unsigned)((max_blocks + 127) / 128), (unsigned)count);
  RCG_LAUNCH(ctx, "quantize", k_quantize, grid, 128, 0, d_step, cs);
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ K4 rate model

// Code lengths of the measured AC statistics (huff_lengths: build_lengths over the 256 symbols plus optimal_table's
// dummy), then optimal_table's sizes (jpeg/src/encode.rs:245-262), Rdo's code-length table (jpeg/src/rdo.rs:36-39)
// and the lambda*rate table (jpeg/src/rdo.rs:47-52). One CTA per component.
__device__ __forceinline__ void rate_tables_body(StepDesc* __restrict__ st, const int comp) {
  __shared__ unsigned freq[kHuffSyms];
  __shared__ unsigned char lens[kHuffSyms];
  __shared__ HuffScratch scratch;
  __shared__ float len[256];
  if (!st->active || !st->use_trellis) return;
  // the rate model is per class, lambda per component
  if (comp >= st->ncomp) return;
  const int cls = comp < 1 ? comp : 1;
  const int t = threadIdx.x;
  if (t < kHuffSyms) freq[t] = t < 256 ? st->hist[cls][t] : 1u;
  huff_lengths(freq, lens, scratch);
  // optimal_table sizes of the 256 real symbols; an empty table gets symbol 0 at length 1. Rdo: 0 -> 18 bits.
  if (t < 256) {
    const bool any = scratch.n_used > 1;  // a used symbol besides the dummy
    unsigned size = lens[t];
    if (!any && t == 0) size = 1;
    len[t] = size == 0 ? 18.0f : (float)size;
  }
  __syncthreads();
  const float lambda = st->lambda[comp];
  // rate(run, v) = zrl * len[0xF0] + len[((run % 16) << 4) | size] + size, for size = bit length of v.
  for (int i = t; i < 64 * kRateSizes; i += blockDim.x) {
    int run = i / kRateSizes, size = i % kRateSizes;
    float rate = fadd(fadd(fmul((float)(run / 16), len[0xF0]), len[((run % 16) << 4) | size]), (float)size);
    st->lr[comp][i] = fmul(lambda, rate);
  }
  // Per size, the least entry over all runs (the trellis's scan bound): 16 lanes of 4 runs each per size. The products
  // are those of the table and rounding is monotone, so the minimum is one of its entries.
  {
    const int size = t >> 4;
    float least = 3.0e38f;
    for (int run = t & 15; run < 64; run += 16) {
      float rate = fadd(fadd(fmul((float)(run / 16), len[0xF0]), len[((run % 16) << 4) | size]), (float)size);
      least = fminf(least, fmul(lambda, rate));
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, off));
    if ((t & 15) == 0 && size < kRateSizes) st->lrmin[comp][size] = least;
  }
  if (t == 0) st->eob[comp] = fmul(lambda, len[0]);
}

__global__ void __launch_bounds__(288) k_rate_tables(StepDesc* __restrict__ st) {
  grid_chain();
  rate_tables_body(st + blockIdx.y, blockIdx.x);
}

int rate_tables(rcg_ctx* ctx, StepDesc* d_step, int count) {
  RCG_LAUNCH(ctx, "rate_tables", k_rate_tables, dim3(3, (unsigned)count), 288, 0, d_step);
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ K5 trellis

// Rdo::quantize_ac (jpeg/src/rdo.rs:54-119) for one block per thread, plus the DC rounding of the trellis pass
// (jpeg/src/encode.rs:206-214). Same candidates, costs, evaluation order and strict `<` tie rule as the reference;
// both candidate values of a position scan the earlier nodes in one pass (neither sees the other: the reference
// skips nodes at the same position, :86-88). zd[i-1] is carried as a running sum, and each node keeps zd at its
// own position, so no 64-entry zd table is needed.
// kWeighted: the perceptual mode. Each coefficient's distortion weight becomes rw[k] * pweights[block][k] (one f32
// product, then the same squared-error product as the plain weight); the plain instantiation reads no weights.
// One block per thread: the DP of a block is serial, so the kernel is bound by the latency of one position and, at
// large sizes, by the per-position work every lane runs (sorting or listing blocks by their number of candidates
// measured no better). What counts is therefore the length of a position's dependency chain and the bytes a block
// keeps outside registers. Measured per candidate, full scans over nodes in local memory against the form below:
// 240x180 4:4:4 35 -> 19 us (a search's mean), 1283x857 69 -> 25, 1653x2339 gray 77 -> 38, 4000x3000 65.5 -> 55,
// a 3000x2000 requantization 154 -> 100 (its source rows as 16-byte loads among that), weighted 1620x1080 54 -> 32.
// 7 CTAs per SM (72 registers): 8 spill (58 us at 12 MP), 6 leave too few warps (68 us with 4 nodes in registers);
// the window at 2 nodes: 1, 3, 4 and 6 measured 53, 64, 66 and 71 us at 12 MP and 42, -, -, - against 38 us gray; 64
// threads a CTA 62 us. Coefficients arrive 8 at a time, the next chunk's loads in flight (deeper prefetches, through
// registers or shared memory, measured slower); scale, step and weight of a position are one 16-byte entry.
//
// The scan over earlier nodes goes from the newest to the oldest and stops when no older node can win. Keeping a
// coefficient of magnitude >= 1 lowers cost - zd (the cost relative to dropping everything so far) by far more than
// any code length differs, so the best predecessor is nearly always one of the last few nodes, where a full scan
// costs as many steps as the block has candidates so far. The bound is exact, so the coefficients are those of the
// full scan: npmin is the least cost - zd of a node and all before it, rounded down; every node's base is at least
// (npmin + zprev)(1 - 2^-23) by the two roundings of its own computation (costs and zd are sums of non-negative terms
// and zd never falls), scan_floor stays below that, and the two additions after it are the node's own, with the
// least rate of the table in place of the node's: rounding is monotone, so a bound above the best rules out every
// older node. Ties: a full ascending scan with strict < keeps the start of the block over any node and the lowest
// node of equal cost, which descending is <= among nodes and < against the start. Weights of a caller may be negative
// or NaN: such a block scans in full from there on.
__device__ __forceinline__ float scan_floor(float pmin, float zprev) {
  return __fmul_rd(__fadd_rd(pmin, zprev), 1.0f - 0x1p-22f);
}

constexpr int kWin = 2;  // nodes of the trellis scan held in registers

template <bool kWeighted>
__device__ __forceinline__ void trellis_body(StepDesc* __restrict__ st, const CacheSet& cs, long long bx) {
  // The per-position tables of every component and the lambda*rate tables of the components this CTA's blocks
  // belong to (usually one), staged in shared memory: the DP reads them at every position.
  __shared__ float lr[3][64 * kRateSizes];
  __shared__ float4 s_tab[3][64];  // per position: (scale, step, weight, -)
  if (!st->active || !st->use_trellis) return;
  const bool requant = st->requant != 0;
  const long long blk0 = bx * blockDim.x;
  const int c_lo = comp_of(st, blk0), c_hi = comp_of(st, min(blk0 + (long long)blockDim.x, st->nblocks) - 1);
  for (int i = threadIdx.x; i < (c_hi - c_lo + 1) * 64 * kRateSizes; i += blockDim.x)
    (&lr[c_lo][0])[i] = (&st->lr[c_lo][0])[i];
  for (int i = threadIdx.x; i < 3 * 64; i += blockDim.x) {
    const int c = i / 64, k = i % 64;
    s_tab[c][k] = make_float4(requant ? st->ratio[c][k] : st->divz[c][k], st->rq[c][k], st->rw[c][k], 0.0f);
  }
  __syncthreads();
  const long long gb = blk0 + threadIdx.x;
  if (gb >= st->nblocks) return;
  const int c = comp_of(st, gb);
  const CompDesc& cd = st->comp[c];
  const long long nb = (long long)cd.bw * cd.bh;
  // Encoding: a[k] = flat[ZZ_T[k]] * div[ZZ_T[k]] from the FDCT cache (jpeg/src/encode.rs:207-211).
  // Requantization: a[k] = source[k] * ratio[k] (jpeg/src/encode.rs:162-166); the DC stays the plain value.
  const float* cache = requant ? nullptr : cs.p[cd.cache] + (gb - cd.blk0);
  const int16_t* src = requant ? st->coef_src + gb * 64 : nullptr;
  const float4* tab = s_tab[c];
  const float* lrc = lr[c];
  const float* lmin = st->lrmin[c];
  const float* pw = kWeighted ? st->pweights + gb * 64 : nullptr;  // 16-byte aligned rows of 64 floats

  // Every node as (cost, zd, the least cost - zd up to it, packed position | value | predecessor): written once, read
  // by the few scans that go past the window and by the final walk back.
  float4 nodes[126];
  // The newest kWin nodes, newest first (cost infinity: none yet), and the bound for the nodes older than they.
  float wcost[kWin], wzd[kWin];
  int wrow[kWin];  // (position + 1) * kRateSizes: the rate row of position i is i * kRateSizes - wrow
#pragma unroll
  for (int n = 0; n < kWin; n++) {
    wcost[n] = __int_as_float(0x7f800000);
    wzd[n] = 0.0f;
    wrow[n] = kRateSizes;
  }
  float pm_all = __int_as_float(0x7f800000), pm_old = pm_all;
  bool prune = true;
  int nn = 0;
  int dc = 0;
  float zprev = 0.0f;  // zd[i-1]

  // The coefficients arrive 8 at a time: the next chunk's loads are in flight while this chunk's DP steps run.
  constexpr int kChunk = 8;
  // A requantization's chunk is one 16-byte load of the block's row.
  auto load_chunk = [&](int c0, float* to) {
    if (requant) {
      const int4 p = __ldg(reinterpret_cast<const int4*>(src + c0));
      const int w4[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
      for (int j = 0; j < kChunk; j++) to[j] = (float)(short)((w4[j >> 1] >> (16 * (j & 1))) & 0xFFFF);
    } else {
#pragma unroll
      for (int j = 0; j < kChunk; j++) to[j] = __ldg(cache + (long long)(c0 + j) * nb);
    }
  };
  float cur[kChunk], nxt[kChunk];
  load_chunk(0, cur);
#pragma unroll 1
  for (int c0 = 0; c0 < 64; c0 += kChunk) {
    if (c0 + kChunk < 64) load_chunk(c0 + kChunk, nxt);
    float wv[kChunk];
    if constexpr (kWeighted) {
      const float4* p4 = reinterpret_cast<const float4*>(pw + c0);
#pragma unroll
      for (int g = 0; g < kChunk / 4; g++) {
        const float4 v = __ldg(p4 + g);
        wv[4 * g] = v.x;
        wv[4 * g + 1] = v.y;
        wv[4 * g + 2] = v.z;
        wv[4 * g + 3] = v.w;
      }
    }
#pragma unroll
    for (int j = 0; j < kChunk; j++) {
      const int i = c0 + j;
      const float4 tb = tab[i];
      float a = fmul(cur[j], tb.x);
      if (i == 0) {
        dc = clampi(round_f32(a), -2047, 2047);
        continue;
      }
      float q = tb.y, w = kWeighted ? fmul(tb.z, wv[j]) : tb.z;
      if constexpr (kWeighted) prune = prune && w >= 0.0f;
      const bool neg = a < 0.0f;  // a node keeps its value with this sign
      float m = fabsf(a);
      const float rounded = fadd(m, 0.5f);
      int pushed = 0, packed[2] = {0, 0};
      float best[2] = {0.0f, 0.0f};
      if (rounded >= 1.0f) {
        const unsigned v0 = (unsigned)rounded;
        unsigned lo = v0 > 1 ? v0 - 1 : v0;
        bool two = lo != v0;
        // candidate lo (first) and v0 (second, if distinct)
        float e_lo = fmul(fsub(m, (float)lo), q);
        float dnz_lo = fmul(fmul(e_lo, e_lo), w);
        float e_hi = fmul(fsub(m, (float)v0), q);
        float dnz_hi = fmul(fmul(e_hi, e_hi), w);
        int s_lo = bitlen(lo), s_hi = bitlen(v0);
        float best_lo = fadd(fadd(zprev, lrc[(i - 1) * kRateSizes + s_lo]), dnz_lo);
        float best_hi = fadd(fadd(zprev, lrc[(i - 1) * kRateSizes + s_hi]), dnz_hi);
        int prev_lo = -1, prev_hi = -1;
        auto offer = [&](float cost, float zd, int row, int ni) {
          const float base = fadd(cost, fsub(zprev, zd));
          const float* lrow = lrc + (i * kRateSizes - row);
          const float c_lo = fadd(fadd(base, lrow[s_lo]), dnz_lo);
          const float c_hi = fadd(fadd(base, lrow[s_hi]), dnz_hi);
          if (c_lo < best_lo || (c_lo == best_lo && prev_lo >= 0)) {
            best_lo = c_lo;
            prev_lo = ni;
          }
          if (c_hi < best_hi || (c_hi == best_hi && prev_hi >= 0)) {
            best_hi = c_hi;
            prev_hi = ni;
          }
        };
#pragma unroll
        for (int n = 0; n < kWin; n++) offer(wcost[n], wzd[n], wrow[n], nn - 1 - n);
        // No node from here down can win once both bounds lie above the best (see the note on the scan above).
        auto settled = [&](float pm) {
          const float floor_base = scan_floor(pm, zprev);
          return prune && fadd(fadd(floor_base, lmin[s_lo]), dnz_lo) > best_lo &&
                 fadd(fadd(floor_base, lmin[s_hi]), dnz_hi) > best_hi;
        };
        if (nn > kWin && !settled(pm_old)) {
          for (int ni = nn - 1 - kWin; ni >= 0; ni--) {
            const float4 nd = nodes[ni];
            if (settled(nd.z)) break;
            offer(nd.x, nd.y, ((__float_as_int(nd.w) & 63) + 1) * kRateSizes, ni);
          }
        }
        best[0] = best_lo;
        best[1] = best_hi;
        const int sign = neg ? -1 : 1;
        packed[0] = i | (prev_lo & 0xff) << 6 | (sign * (int)lo) << 14;
        packed[1] = i | (prev_hi & 0xff) << 6 | (sign * (int)v0) << 14;
        pushed = two ? 2 : 1;
      }
      // zd[i] = zd[i-1] + (a*q)^2 * w; a node at position i keeps zd[i] (the reference reads zd[n.pos]).
      float e = fmul(a, q);
      float zcur = fadd(zprev, fmul(fmul(e, e), w));
#pragma unroll
      for (int n = 0; n < 2; n++) {
        if (n < pushed) {
          pm_all = fminf(pm_all, __fsub_rd(best[n], zcur));
          nodes[nn] = make_float4(best[n], zcur, pm_all, __int_as_float(packed[n]));
          nn++;
          pm_old = fminf(pm_old, __fsub_rd(wcost[kWin - 1], wzd[kWin - 1]));
#pragma unroll
          for (int k = kWin - 1; k > 0; k--) {
            wcost[k] = wcost[k - 1];
            wzd[k] = wzd[k - 1];
            wrow[k] = wrow[k - 1];
          }
          wcost[0] = best[n];
          wzd[0] = zcur;
          wrow[0] = (i + 1) * kRateSizes;
        }
      }
      zprev = zcur;
    }
#pragma unroll
    for (int j = 0; j < kChunk; j++) cur[j] = nxt[j];
  }
  // End of block (jpeg/src/rdo.rs:98-108): zprev is zd[63].
  const float eob = st->eob[c];
  float best_cost = fadd(zprev, eob);
  int best_end = -1;
  for (int ni = nn - 1; ni >= 0; ni--) {
    // Positions ascend, so once a node lies below 63 all before it do and pay the end-of-block code.
    const float4 nd = nodes[ni];
    const bool pays = (__float_as_int(nd.w) & 63) < 63;
    if (prune && pays && fadd(scan_floor(nd.z, zprev), eob) > best_cost) break;
    float cst = fadd(fadd(nd.x, fsub(zprev, nd.y)), pays ? eob : 0.0f);
    if (cst < best_cost || (cst == best_cost && best_end >= 0)) {
      best_cost = cst;
      best_end = ni;
    }
  }
  int16_t* out = st->coefs + gb * 64;
  int4 z = make_int4(0, 0, 0, 0);
  int4 first = z;
  // quantize_ac clears positions 1..63 (jpeg/src/rdo.rs:109-111); the DC is the rounded a[0] when encoding and the
  // plain requantized value (already in place) when requantizing.
  first.x = requant ? (reinterpret_cast<const int4*>(out)[0].x & 0xFFFF) : (dc & 0xFFFF);
  reinterpret_cast<int4*>(out)[0] = first;
#pragma unroll
  for (int g = 1; g < 8; g++) reinterpret_cast<int4*>(out)[g] = z;
  int node = best_end;
  while (node >= 0) {
    const int pk = __float_as_int(nodes[node].w);
    out[pk & 63] = (int16_t)(pk >> 14);
    node = (int)(signed char)(pk >> 6);
  }
}

template <bool kWeighted>
__global__ void __launch_bounds__(128, 7) k_trellis(StepDesc* __restrict__ st, CacheSet cs) {
  grid_chain();
  trellis_body<kWeighted>(st + blockIdx.y, cs, blockIdx.x);
}

int trellis(rcg_ctx* ctx, StepDesc* d_step, const float* const* d_caches, long long max_blocks, bool weighted,
            int count) {
  CacheSet cs;
  for (int i = 0; i < 9; i++) cs.p[i] = d_caches ? d_caches[i] : nullptr;
  const dim3 grid((unsigned)((max_blocks + 127) / 128), (unsigned)count);
  if (weighted)
    RCG_LAUNCH(ctx, "trellis_weighted", k_trellis<true>, grid, 128, 0, d_step, cs);
  else
    RCG_LAUNCH(ctx, "trellis", k_trellis<false>, grid, 128, 0, d_step, cs);
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ K6 IDCT

// jpeg/src/dct.rs:67-109 (idct_pass)
__device__ __forceinline__ void idct_pass(float (&d)[64]) {
  const float SQRT_2 = 1.41421356237309504880f;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    float tmp0 = d[0 * 8 + j], tmp1 = d[2 * 8 + j], tmp2 = d[4 * 8 + j], tmp3 = d[6 * 8 + j];
    float tmp10 = fadd(tmp0, tmp2), tmp11 = fsub(tmp0, tmp2), tmp13 = fadd(tmp1, tmp3);
    float tmp12 = fsub(fmul(fsub(tmp1, tmp3), SQRT_2), tmp13);
    float e0 = fadd(tmp10, tmp13), e3 = fsub(tmp10, tmp13), e1 = fadd(tmp11, tmp12), e2 = fsub(tmp11, tmp12);
    float tmp4 = d[1 * 8 + j], tmp5 = d[3 * 8 + j], tmp6 = d[5 * 8 + j], tmp7 = d[7 * 8 + j];
    float z13 = fadd(tmp6, tmp5), z10 = fsub(tmp6, tmp5), z11 = fadd(tmp4, tmp7), z12 = fsub(tmp4, tmp7);
    float o7 = fadd(z11, z13);
    float o11 = fmul(fsub(z11, z13), SQRT_2);
    float z5 = fmul(fadd(z10, z12), 1.8477591f);
    float o10 = fsub(fmul(1.0823922f, z12), z5);
    float o12 = fadd(fmul(-2.613126f, z10), z5);
    float o6 = fsub(o12, o7);
    float o5 = fsub(o11, o6);
    float o4 = fadd(o10, o5);
    d[0 * 8 + j] = fadd(e0, o7);
    d[7 * 8 + j] = fsub(e0, o7);
    d[1 * 8 + j] = fadd(e1, o6);
    d[6 * 8 + j] = fsub(e1, o6);
    d[2 * 8 + j] = fadd(e2, o5);
    d[5 * 8 + j] = fsub(e2, o5);
    d[4 * 8 + j] = fadd(e3, o4);
    d[3 * 8 + j] = fsub(e3, o4);
  }
}

// idct_planes (jpeg/src/decode.rs:1310-1343): dequantize into natural order, IDCT (jpeg/src/dct.rs:111-123),
// round_f32 + 128 clamped to 0..255. One thread per block.
__device__ __forceinline__ void dequant_idct_body(const StepDesc* __restrict__ st, const int16_t* __restrict__ coefs,
                                                  uint8_t* __restrict__ planes, long long cta) {
  if (!st->active) return;
  long long gb = cta * blockDim.x + threadIdx.x;
  if (gb >= st->nblocks) return;
  int c = comp_of(st, gb);
  const CompDesc& cd = st->comp[c];
  long long lb = gb - cd.blk0;
  int by = (int)(lb / cd.bw), bx = (int)(lb % cd.bw);
  const float* mult = st->mult[c];
  float blk[64];
  const int16_t* base = coefs ? coefs : st->coefs;
  const int4* src = reinterpret_cast<const int4*>(base + gb * 64);
#pragma unroll
  for (int g = 0; g < 8; g++) {
    int4 pk = src[g];
    int w4[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
    for (int j = 0; j < 8; j++) {
      int k = g * 8 + j;
      int v = (int)(short)((w4[j >> 1] >> (16 * (j & 1))) & 0xFFFF);
      int n = zigzag_known(k);
      blk[n] = fmul((float)v, mult[n]);
    }
  }
  idct_pass(blk);
  transpose8(blk);
  idct_pass(blk);
  transpose8(blk);
  int stride = cd.bw * 8;
  uint8_t* dst = planes + cd.plane_off + (size_t)(by * 8) * stride + bx * 8;
#pragma unroll
  for (int y = 0; y < 8; y++) {
    unsigned lo = 0, hi = 0;
#pragma unroll
    for (int x = 0; x < 8; x++) {
      unsigned p = (unsigned)clampi(round_f32(fmul(blk[y * 8 + x], 0.125f)) + 128, 0, 255);
      if (x < 4)
        lo |= p << (8 * x);
      else
        hi |= p << (8 * (x - 4));
    }
    *reinterpret_cast<uint2*>(dst + (size_t)y * stride) = make_uint2(lo, hi);
  }
}

__global__ void __launch_bounds__(128) k_dequant_idct(const StepDesc* __restrict__ st,
                                                     const int16_t* __restrict__ coefs, uint8_t* __restrict__ planes,
                                                     long long planes_stride) {
  grid_chain();
  dequant_idct_body(st + blockIdx.y, coefs, planes + blockIdx.y * planes_stride, blockIdx.x);
}

int dequant_idct(rcg_ctx* ctx, StepDesc* d_step, const int16_t* d_coefs, uint8_t* d_planes, long long max_blocks,
                 int count, long long planes_stride) {
  const dim3 grid((unsigned)((max_blocks + 127) / 128), (unsigned)count);
  RCG_LAUNCH(ctx, "dequant_idct", k_dequant_idct, grid, 128, 0, d_step, d_coefs, d_planes, planes_stride);
  return RCG_OK;
}

// The trellis and the decoding of its result by the same thread, for candidates of few blocks (the decoder's launch costs
// them more than the trellis's occupancy): the registers of the two phases do not add up, but the decoder's leave room for
// four CTAs per SM instead of seven, so the line lies at one wave of those. Measured per search, apart / together: 17 CTAs
// (240x180) 551 / 542 us, 408 (0.8 MP) 1082 / 1076, 474 (3.9 MP gray) 1280 / 1265; 1107 (6 MP, requantizing) 4877 / 5015.
constexpr int kDecodeCtas = 4;
constexpr long long kTrellisDecodeCtas = kDecodeCtas * kSms;

template <bool kWeighted>
__global__ void __launch_bounds__(128, kDecodeCtas) k_trellis_decode(StepDesc* __restrict__ st, CacheSet cs,
                                                                     uint8_t* __restrict__ planes) {
  grid_chain();
  trellis_body<kWeighted>(st, cs, blockIdx.x);
  dequant_idct_body(st, nullptr, planes, blockIdx.x);  // a thread's own block: its coefficients are its own stores
}

int trellis_decode(rcg_ctx* ctx, StepDesc* d_step, const float* const* d_caches, long long max_blocks, bool weighted,
                   uint8_t* d_planes) {
  const long long ctas = (max_blocks + 127) / 128;
  if (ctas > kTrellisDecodeCtas) {
    trellis(ctx, d_step, d_caches, max_blocks, weighted);
    return dequant_idct(ctx, d_step, nullptr, d_planes, max_blocks);
  }
  CacheSet cs;
  for (int i = 0; i < 9; i++) cs.p[i] = d_caches ? d_caches[i] : nullptr;
  if (weighted)
    RCG_LAUNCH(ctx, "trellis_decode", k_trellis_decode<true>, (unsigned)ctas, 128, 0, d_step, cs, d_planes);
  else
    RCG_LAUNCH(ctx, "trellis_decode", k_trellis_decode<false>, (unsigned)ctas, 128, 0, d_step, cs, d_planes);
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ K7 upsample+colour

__constant__ float c_lut8[256];

// upsample (jpeg/src/decode.rs:1768-1828) of one component sample at full-resolution (x, y).
__device__ __forceinline__ int up_sample(const uint8_t* p, int stride, int cw, int ch, int fx, int fy, int x, int y) {
  auto px = [&](int xx, int yy) -> int { return p[(size_t)yy * stride + xx]; };
  if (fx == 1 && fy == 1) return px(x, y);
  if (fx == 2 && fy == 1) {
    int i = x / 2;
    int nr = px(i, y);
    int fr = (x % 2 == 0) ? px(max(i - 1, 0), y) : px(min(i + 1, cw - 1), y);
    return (3 * nr + fr + ((x % 2 == 0) ? 1 : 2)) >> 2;
  }
  if (fx == 1 && fy == 2) {
    int j = y / 2;
    int fy_ = (y % 2 == 0) ? max(j - 1, 0) : min(j + 1, ch - 1);
    return (3 * px(x, j) + px(x, fy_) + ((y % 2 == 0) ? 1 : 2)) >> 2;
  }
  if (fx == 2 && fy == 2) {
    int j = y / 2;
    int fy_ = (y % 2 == 0) ? max(j - 1, 0) : min(j + 1, ch - 1);
    int i = x / 2;
    int fi = (x % 2 == 0) ? max(i - 1, 0) : min(i + 1, cw - 1);
    int nr = 3 * px(i, j) + px(i, fy_);
    int fr = 3 * px(fi, j) + px(fi, fy_);
    return (3 * nr + fr + ((x % 2 == 0) ? 8 : 7)) >> 4;
  }
  return px(x / fx, y / fy);
}

// Decoder::finish for an 8-bit YCbCr or Gray CoefImage (jpeg/src/decode.rs:1404-1444): upsample every component to
// full resolution, then the fixed-point YCbCr->RGB of :1438-1441. Writes interleaved pixels and/or the linear-light
// planes the scorer starts from (core/src/ssimulacra2.rs:192-203: Gray is replicated to three channels), np samples apart
// (0: Gray, one plane).
// 10 CTAs per SM (48 registers) instead of 7: the kernel waits on loads, so more warps hide more of it
// (51 -> 47 us per 12 MP candidate).
__device__ __forceinline__ void upsample_color_body(const StepDesc* __restrict__ st,
                                                    const uint8_t* __restrict__ planes, int w, int h,
                                                    uint8_t* __restrict__ rgb, float* __restrict__ lin,
                                                    const int pitch, const size_t np, const unsigned bx,
                                                    const unsigned by, const unsigned gy) {
  if (!st->active) return;
  const int ncomp = st->ncomp, hmax = st->hmax, vmax = st->vmax;
  const CompDesc c0 = st->comp[0];
  // The sRGB table lives in shared memory: per-thread indices differ, which would serialize constant-memory reads.
  __shared__ float lut[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = c_lut8[i];
  __syncthreads();
  // Four consecutive pixels of one row per thread, so each thread moves enough bytes per request.
  const int x0 = 4 * (bx * blockDim.x + threadIdx.x);
  if (x0 >= w) return;
  const bool vec_out = pitch % 4 == 0;    // whole quads: the last one may run into the row's padding
  for (int y = by; y < h; y += gy) {
    int yv[4], cbv[4], crv[4];
    // Luma: full resolution when it carries the maximum sampling factors (always, for this encoder's layouts).
    if (c0.h == hmax && c0.v == vmax) {
      const uint8_t* yr = planes + c0.plane_off + (size_t)y * (c0.bw * 8);
      uint32_t q = *reinterpret_cast<const uint32_t*>(yr + x0);  // x0 % 4 == 0, row stride % 8 == 0
#pragma unroll
      for (int k = 0; k < 4; k++) yv[k] = (q >> (8 * k)) & 0xFF;
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        int x = min(x0 + k, w - 1);
        yv[k] = up_sample(planes + c0.plane_off, c0.bw * 8, (w * c0.h + hmax - 1) / hmax,
                          (h * c0.v + vmax - 1) / vmax, hmax / c0.h, vmax / c0.v, x, y);
      }
    }
    if (ncomp == 3) {
#pragma unroll
      for (int c = 1; c < 3; c++) {
        const CompDesc cd = st->comp[c];
        const uint8_t* p = planes + cd.plane_off;
        const int stride = cd.bw * 8;
        const int cw = (w * cd.h + hmax - 1) / hmax, ch = (h * cd.v + vmax - 1) / vmax;
        const int fx = hmax / cd.h, fy = vmax / cd.v;
        int* out = c == 1 ? cbv : crv;
        if (fx == 2 && fy == 2) {
          // Triangle filter of jpeg/src/decode.rs:1806-1818 for x0..x0+3 (x0 even): chroma columns i-1..i+2.
          const int j = y / 2;
          const int far_y = (y % 2 == 0) ? max(j - 1, 0) : min(j + 1, ch - 1);
          const uint8_t* rn = p + (size_t)j * stride;
          const uint8_t* rf = p + (size_t)far_y * stride;
          const int i = x0 / 2;
          int vert[4];
#pragma unroll
          for (int d = 0; d < 4; d++) {
            int col = min(max(i - 1 + d, 0), cw - 1);
            vert[d] = 3 * rn[col] + rf[col];
          }
          out[0] = (3 * vert[1] + vert[0] + 8) >> 4;  // x0 even: far = i-1
          out[1] = (3 * vert[1] + vert[2] + 7) >> 4;  // x0+1 odd: far = i+1
          out[2] = (3 * vert[2] + vert[1] + 8) >> 4;  // x0+2 even: near i+1, far i
          out[3] = (3 * vert[2] + vert[3] + 7) >> 4;  // x0+3 odd: near i+1, far i+2
          // Clamping every column to [0, cw-1] is the reference's rule (saturating i-1, min(i+1, cw-1)); a near
          // column never needs it for a pixel inside the image (x < w implies x/2 < cw).
        } else {
#pragma unroll
          for (int k = 0; k < 4; k++) out[k] = up_sample(p, stride, cw, ch, fx, fy, min(x0 + k, w - 1), y);
        }
      }
    }
    float l[3][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (ncomp == 1) {
        l[0][k] = l[1][k] = l[2][k] = lut[yv[k]];
        if (rgb && x0 + k < w) rgb[(size_t)y * w + x0 + k] = (uint8_t)yv[k];
      } else {
        int cb = cbv[k] - 128, cr = crv[k] - 128;
        int r = clampi(yv[k] + ((91881 * cr + 32768) >> 16), 0, 255);
        int g = clampi(yv[k] - ((22554 * cb + 46802 * cr + 32768) >> 16), 0, 255);
        int b = clampi(yv[k] + ((116130 * cb + 32768) >> 16), 0, 255);
        l[0][k] = lut[r];
        l[1][k] = lut[g];
        l[2][k] = lut[b];
        if (rgb && x0 + k < w) {
          size_t i = ((size_t)y * w + x0 + k) * 3;
          rgb[i] = (uint8_t)r;
          rgb[i + 1] = (uint8_t)g;
          rgb[i + 2] = (uint8_t)b;
        }
      }
    }
    if (lin) {
      size_t i = (size_t)y * pitch + x0;
      if (vec_out) {
#pragma unroll
        for (int c = 0; c < 3; c++)
          *reinterpret_cast<float4*>(lin + c * np + i) = make_float4(l[c][0], l[c][1], l[c][2], l[c][3]);
      } else {
        for (int k = 0; k < 4 && x0 + k < w; k++)
#pragma unroll
          for (int c = 0; c < 3; c++) lin[c * np + i + k] = l[c][k];
      }
    }
  }
}

__global__ void __launch_bounds__(128, 10) k_upsample_color(const StepDesc* __restrict__ st,
                                                             const uint8_t* __restrict__ planes, int w, int h,
                                                             uint8_t* __restrict__ rgb, float* __restrict__ lin,
                                                             int pitch, size_t np) {
  grid_chain();
  upsample_color_body(st, planes, w, h, rgb, lin, pitch, np, blockIdx.x, blockIdx.y, gridDim.y);
}

int upsample_color(rcg_ctx* ctx, StepDesc* d_step, const uint8_t* d_planes, int w, int h, uint8_t* d_rgb,
                   float* d_lin, int pitch, size_t plane) {
  // A CTA takes every (h + 1) / 8-th row, eight in all, so that it fills its shared-memory table once for them.
  dim3 grid(((w + 3) / 4 + 127) / 128, std::min(((h + 1) / 2 + 3) / 4, 65535));
  RCG_LAUNCH(ctx, "upsample_color", k_upsample_color, grid, 128, 0, d_step, d_planes, w, h, d_rgb, d_lin, pitch,
             plane);
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ step tables

// A search's first step (and the first one after a near tie): the later ones' tables are filled where the step before is
// scored (ssim2_reduce), unless the search's metric is another.
__global__ void __launch_bounds__(kStepThreads) k_step_tables(const SearchState* __restrict__ ss,
                                                              StepDesc* __restrict__ st, const NextStep next) {
  grid_chain();
  step_tables_body(*ss, st, next, step_prepare(st, next));
}

int step_tables(rcg_ctx* ctx, SearchState* d_search, StepDesc* d_step, const NextStep& next) {
  RCG_LAUNCH(ctx, "step_tables", k_step_tables, 1, kStepThreads, 0, d_search, d_step, next);
  return RCG_OK;
}

// ------------------------------------------------------------------------------------------------ lockstep batch

// One bisection step of every image of a lockstep batch: the same kernel bodies as one search, each launch over a
// work-list of every image's CTAs (an image whose search has finished skips through its StepDesc's `active`).
__global__ void __launch_bounds__(kStepThreads) k_step_tables_lock(const LockItem* __restrict__ items) {
  grid_chain();
  const LockItem& it = items[blockIdx.x];
  const NextStep next = {kNextEncode, it.w, it.h, it.slots, it.slot_stride, nullptr};
  step_tables_body(*it.ss, it.st, next, step_prepare(it.st, next));
}

__device__ __forceinline__ CacheSet lock_caches(const LockItem& it) {
  CacheSet cs;
#pragma unroll
  for (int i = 0; i < 9; i++) cs.p[i] = it.caches[i];
  return cs;
}

__global__ void __launch_bounds__(128, 4) k_quantize_lock(const LockItem* __restrict__ items, int n) {
  grid_chain();
  const int i = lock_find<&LockItem::q0>(items, n, blockIdx.x);
  const LockItem& it = items[i];
  quantize_body(it.st, lock_caches(it), (long long)blockIdx.x - it.q0);
}

__global__ void __launch_bounds__(288) k_rate_tables_lock(const LockItem* __restrict__ items) {
  grid_chain();
  rate_tables_body(items[blockIdx.y].st, blockIdx.x);
}

__global__ void __launch_bounds__(128, 7) k_trellis_lock(const LockItem* __restrict__ items, int n) {
  grid_chain();
  const int i = lock_find<&LockItem::q0>(items, n, blockIdx.x);
  const LockItem& it = items[i];
  trellis_body<false>(it.st, lock_caches(it), (long long)blockIdx.x - it.q0);
}

__global__ void __launch_bounds__(128) k_dequant_idct_lock(const LockItem* __restrict__ items, int n) {
  grid_chain();
  const int i = lock_find<&LockItem::q0>(items, n, blockIdx.x);
  const LockItem& it = items[i];
  dequant_idct_body(it.st, nullptr, it.planes, (long long)blockIdx.x - it.q0);
}

void lock_step_codec(rcg_ctx* ctx, const LockItem* d_items, int n, long long q_total, bool first) {
  if (first) RCG_LAUNCH(ctx, "step_tables_lock", k_step_tables_lock, n, kStepThreads, 0, d_items);
  RCG_LAUNCH(ctx, "quantize_lock", k_quantize_lock, (unsigned)q_total, 128, 0, d_items, n);
  RCG_LAUNCH(ctx, "rate_tables_lock", k_rate_tables_lock, dim3(3, n), 288, 0, d_items);
  RCG_LAUNCH(ctx, "trellis_lock", k_trellis_lock, (unsigned)q_total, 128, 0, d_items, n);
  RCG_LAUNCH(ctx, "dequant_idct_lock", k_dequant_idct_lock, (unsigned)q_total, 128, 0, d_items, n);
}

int codec_upload_lut(const float* lut8) {
  cudaError_t e = cudaMemcpyToSymbol(c_lut8, lut8, 256 * sizeof(float));
  return e == cudaSuccess ? 0 : (int)e;
}

// ------------------------------------------------------------------------------------------------ requantization

// Slot assignment of jpeg/src/encode.rs:139-148: components with equal tables share a slot, a new table takes the
// first free one. Also reports whether any table changed (:127) and the slot tables.
inline int requant_slots(const StepDesc* st, int* tq, uint8_t (*slot_qt)[64], int* present) {
  int changed = 0;
  for (int sl = 0; sl < 4; sl++) present[sl] = 0;
  for (int c = 0; c < st->ncomp; c++) {
    bool same_as_old = true;
    for (int n = 0; n < 64; n++) same_as_old &= st->qt[c][n] == st->src_qt[c][n];
    changed |= same_as_old ? 0 : 1;
    int slot = -1;
    for (int sl = 0; sl < 4 && slot < 0; sl++) {
      if (!present[sl]) continue;
      bool eq = true;
      for (int n = 0; n < 64; n++) eq &= slot_qt[sl][n] == st->qt[c][n];
      if (eq) slot = sl;
    }
    if (slot < 0) {
      for (int sl = 0; sl < 4 && slot < 0; sl++)
        if (!present[sl]) slot = sl;
      for (int n = 0; n < 64; n++) slot_qt[slot][n] = st->qt[c][n];
      present[slot] = 1;
    }
    tq[c] = slot;
  }
  return changed;
}

void host_requant_tables(StepDesc* st, int quality, int trellis, int tq_out[3], uint8_t slot_qt_out[4][64],
                         int present_out[4]) {
  const float kappa = 0.02f;  // TRELLIS_KAPPA, jpeg/src/encode.rs:42
  st->quality = quality;
  st->requant = 1;
  for (int c = 0; c < st->ncomp; c++) {
    uint8_t* nt = st->qt[c];
    for (int n = 0; n < 64; n++) nt[n] = requant_entry(st->src_qt[c], quality, n);
    for (int k = 0; k < 64; k++) {
      int n = zigzag(k);
      st->ratio[c][k] = fdiv((float)st->src_qt[c][n], (float)nt[n]);
      st->rq[c][k] = (float)nt[n];
    }
    for (int n = 0; n < 64; n++) st->mult[c][n] = mult_entry(nt, n);
    float sorted[63];
    for (int k = 1; k < 64; k++) sorted[k - 1] = st->rq[c][k];
    std::sort(sorted, sorted + 63);
    float median = sorted[31];
    st->rw[c][0] = 1.0f;
    for (int k = 1; k < 64; k++) st->rw[c][k] = fdiv(median, st->rq[c][k]);
    st->lambda[c] = fmul(fmul(kappa, median), median);
  }
  st->changed = requant_slots(st, tq_out, slot_qt_out, present_out);
  st->use_trellis = (trellis && st->changed) ? 1 : 0;
  std::memset(st->hist, 0, sizeof st->hist);
}

// The AC symbols of one block, eight coefficients at a time: `sizes` their 4-bit sizes, the nonzero ones found by their
// bits (a loop over the block's nonzero coefficients instead of a branch per coefficient). Quantization keeps the branches:
// its values arrive a coefficient at a time from 64 rows, and this form measured 14.2 against 12.2 us at 0.8 MP, 31.8
// against 29.7 at 12 MP.
__device__ __forceinline__ void hist_group(uint32_t sizes, int g, int& last, unsigned* hs) {
  while (sizes) {
    const int j = (__ffs(sizes) - 1) >> 2, k = g * 8 + j;
    const unsigned size = (sizes >> (4 * j)) & 15u;
    sizes &= ~(15u << (4 * j));
    unsigned run = (unsigned)(k - last - 1);
    last = k;
    while (run >= 16) {
      atomicAdd(&hs[0xF0], 1u);
      run -= 16;
    }
    atomicAdd(&hs[(run << 4) | size], 1u);
  }
}

// Adds the CTA's symbols to the candidate's. cls: the class of this thread's block if its last coefficients are zero (an
// end-of-block symbol), else -1. Every thread of the CTA calls it.
__device__ __forceinline__ void hist_finish(StepDesc* st, unsigned (&sh)[2][256], int cls) {
  const unsigned n0 = __popc(__ballot_sync(0xffffffffu, cls == 0)), n1 = __popc(__ballot_sync(0xffffffffu, cls == 1));
  if ((threadIdx.x & 31) == 0) {
    if (n0) atomicAdd(&sh[0][0], n0);
    if (n1) atomicAdd(&sh[1][0], n1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    const unsigned v = (&sh[0][0])[i];
    if (v) atomicAdd(&(&st->hist[0][0])[i], v);
  }
}

__device__ __forceinline__ int4 pack8(const int (&v)[8]) {
  return make_int4((v[0] & 0xFFFF) | (v[1] << 16), (v[2] & 0xFFFF) | (v[3] << 16), (v[4] & 0xFFFF) | (v[5] << 16),
                   (v[6] & 0xFFFF) | (v[7] << 16));
}

// 4-bit sizes of eight coefficients (at most 2047 in magnitude: sizes to 11).
__device__ __forceinline__ uint32_t sizes8(const int (&v)[8]) {
  uint32_t w = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) w |= (uint32_t)bitlen((unsigned)abs(v[j])) << (4 * j);
  return w;
}

// Plain requantization (jpeg/src/encode.rs:132-138): round_f32(coef * old/new) clamped to +-2047, every position.
// When the trellis pass follows, also the AC symbol histogram of the result over the blocks of the MCU grid
// (ac_code_lengths, :155 -> :223-227, :376-398).
// What bounds it: the latency of its row loads between the histogram's serial steps; 28.6 -> 22.9 us per 6 MP candidate
// with hist_group and the end-of-block symbols counted per warp.
__global__ void __launch_bounds__(128) k_requant_plain(StepDesc* __restrict__ st) {
  grid_chain();
  __shared__ unsigned int sh[2][256];
  if (!st->active) return;
  const bool hist = st->use_trellis != 0;
  if (hist) {
    for (int i = threadIdx.x; i < 512; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
  }
  const long long gb = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int eob = -1;
  if (gb < st->nblocks) {
    const int c = comp_of(st, gb);
    const CompDesc& cd = st->comp[c];
    const float* ratio = st->ratio[c];
    const int4* src = reinterpret_cast<const int4*>(st->coef_src + gb * 64);
    int4* out = reinterpret_cast<int4*>(st->coefs + gb * 64);
    uint32_t sizes[8];
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const int4 pk = __ldg(src + g);
      const int w4[4] = {pk.x, pk.y, pk.z, pk.w};
      int v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int x = (int)(short)((w4[j >> 1] >> (16 * (j & 1))) & 0xFFFF);
        v[j] = clampi(round_f32(fmul((float)x, ratio[g * 8 + j])), -2047, 2047);
      }
      out[g] = pack8(v);
      sizes[g] = sizes8(v);
    }
    const long long lb = gb - cd.blk0;
    const int by = (int)(lb / cd.bw), bx = (int)(lb % cd.bw);
    if (hist && bx < st->mcus_x * cd.h && by < st->mcus_y * cd.v) {
      sizes[0] &= ~15u;  // the DC
      int last = 0;
#pragma unroll
      for (int g = 0; g < 8; g++) hist_group(sizes[g], g, last, sh[cd.cls]);
      if (last < 63) eob = cd.cls;
    }
  }
  if (hist) hist_finish(st, sh, eob);
}

int requantize_plain(rcg_ctx* ctx, StepDesc* d_step, long long max_blocks) {
  int grid = (int)((max_blocks + 127) / 128);
  RCG_LAUNCH(ctx, "requant_plain", k_requant_plain, grid, 128, 0, d_step);
  return RCG_OK;
}

}  // namespace rcg
