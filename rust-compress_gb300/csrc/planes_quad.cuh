// Decoded component planes to linear light, four pixels at a time, for the pyramid builder (ssim2.cu): the layouts of an
// encoder's own candidates. The last quad of a row whose width is no multiple of 4 runs into the row's padding: its
// samples beyond the image come from the decoded planes' own padding and are never used.
#pragma once

#include <stdint.h>

#include "rcg_internal.cuh"

namespace rcg {

// Four chroma samples of row r, columns i-1 .. i+2 clamped to [0, cw-1], packed little-endian: two aligned 32-bit
// loads and a funnel shift wherever no clamping applies and both words lie inside the row (rows start 8-byte
// aligned), the clamped byte path at the edges.
__device__ __forceinline__ uint32_t chroma4(const uint8_t* __restrict__ r, int i, int cw, int cstride) {
  const int a = (i - 1) & ~3;
  if (i >= 1 && i + 2 <= cw - 1 && a + 8 <= cstride) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(r + a);
    return __funnelshift_r(q[0], q[1], 8 * ((i - 1) & 3));
  }
  uint32_t v = 0;
#pragma unroll
  for (int d = 0; d < 4; d++) v |= (uint32_t)r[min(max(i - 1 + d, 0), cw - 1)] << (8 * d);
  return v;
}

// The triangle filter of jpeg/src/decode.rs:1806-1818 at columns x0 .. x0+3 (x0 even) of one output row, from its
// near chroma row rn and far chroma row rf (chroma4 words at i = x0/2).
__device__ __forceinline__ void chroma_up(uint32_t rn, uint32_t rf, int (&out)[4]) {
  int vert[4];
#pragma unroll
  for (int d = 0; d < 4; d++) vert[d] = 3 * (int)((rn >> (8 * d)) & 0xFF) + (int)((rf >> (8 * d)) & 0xFF);
  out[0] = (3 * vert[1] + vert[0] + 8) >> 4;
  out[1] = (3 * vert[1] + vert[2] + 7) >> 4;
  out[2] = (3 * vert[2] + vert[1] + 8) >> 4;
  out[3] = (3 * vert[2] + vert[3] + 7) >> 4;
}

// Fixed-point YCbCr -> RGB (jpeg/src/decode.rs:1438-1441) of 4 pixels (luma bytes in q) and the sRGB table.
__device__ __forceinline__ void ycc_linear(uint32_t q, const int (&cb4)[4], const int (&cr4)[4], const float* lut,
                                           float (&l)[3][4]) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int yv = (q >> (8 * k)) & 0xFF;
    const int cb = cb4[k] - 128, cr = cr4[k] - 128;
    l[0][k] = lut[min(max(yv + ((91881 * cr + 32768) >> 16), 0), 255)];
    l[1][k] = lut[min(max(yv - ((22554 * cb + 46802 * cr + 32768) >> 16), 0), 255)];
    l[2][k] = lut[min(max(yv + ((116130 * cb + 32768) >> 16), 0), 255)];
  }
}

// Linear-light values of four columns (x0 .. x0+3, x0 % 4 == 0) of output row y, for the layouts of an encoder's own
// candidates (layout_direct in capi.cu): Gray, 4:4:4, 4:2:2 and 4:2:0 with luma at full resolution
// (jpeg/src/decode.rs:1768-1828, :1438-1441).
__device__ __forceinline__ void planes_quad(const StepDesc* __restrict__ st, const uint8_t* __restrict__ planes, int w,
                                            int h, const float* lut, int x0, int y, float (&l)[3][4]) {
  const CompDesc& c0 = st->comp[0];
  const uint32_t q = *reinterpret_cast<const uint32_t*>(planes + c0.plane_off + (size_t)y * (c0.bw * 8) + x0);
  if (st->ncomp == 1) {
#pragma unroll
    for (int k = 0; k < 4; k++) l[0][k] = l[1][k] = l[2][k] = lut[(q >> (8 * k)) & 0xFF];
    return;
  }
  // Each chroma component has a stride of its own: a caller's block grids need only cover the MCU grid.
  int up[2][4];
  if (st->hmax == 1) {
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const CompDesc& cd = st->comp[1 + c];
      const uint32_t v = *reinterpret_cast<const uint32_t*>(planes + cd.plane_off + (size_t)y * (cd.bw * 8) + x0);
#pragma unroll
      for (int k = 0; k < 4; k++) up[c][k] = (v >> (8 * k)) & 0xFF;
    }
  } else if (st->vmax == 1) {
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int cstride = st->comp[1 + c].bw * 8;
      const uint32_t v = chroma4(planes + st->comp[1 + c].plane_off + (size_t)y * cstride, x0 / 2, (w + 1) / 2, cstride);
      const int b0 = v & 0xFF, b1 = (v >> 8) & 0xFF, b2 = (v >> 16) & 0xFF, b3 = v >> 24;
      up[c][0] = (3 * b1 + b0 + 1) >> 2;
      up[c][1] = (3 * b1 + b2 + 2) >> 2;
      up[c][2] = (3 * b2 + b1 + 1) >> 2;
      up[c][3] = (3 * b2 + b3 + 2) >> 2;
    }
  } else {
    const int j = y / 2, cw = (w + 1) / 2, ch = (h + 1) / 2;
    const int far = (y & 1) ? min(j + 1, ch - 1) : max(j - 1, 0);
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int cstride = st->comp[1 + c].bw * 8;
      const uint8_t* p = planes + st->comp[1 + c].plane_off;
      chroma_up(chroma4(p + (size_t)j * cstride, x0 / 2, cw, cstride),
                chroma4(p + (size_t)far * cstride, x0 / 2, cw, cstride), up[c]);
    }
  }
  ycc_linear(q, up[0], up[1], lut, l);
}

}  // namespace rcg
