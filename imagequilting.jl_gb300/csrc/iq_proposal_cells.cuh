// Cell inputs of the learned proposal's encoder (mask fraction, masked sum and masked sum of
// squares over the cell volume), for windows of the training image and for templates of the
// simulation grid.
#pragma once

#include "iq_internal.h"

namespace {

__device__ __forceinline__ void cell_of(const LpGeo& g, int cell, int& i, int& j, int& k) {
  i = cell % g.g[0];
  j = (cell / g.g[0]) % g.g[1];
  k = cell / (g.g[0] * g.g[1]);
}

// Voxels of cell `cell` (origin a, end b) and of its part inside the mask box (ia, ib); false
// when the box leaves the cell alone.
__device__ __forceinline__ bool cell_box(const LpGeo& g, const int* lo, const int* hi, int cell,
                                         int (&a)[3], int (&b)[3], int (&ia)[3], int (&ib)[3]) {
  int c3[3];
  cell_of(g, cell, c3[0], c3[1], c3[2]);
  bool inner = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    a[d] = c3[d] * g.c[d];
    b[d] = min(a[d] + g.c[d], g.t[d]);
    ia[d] = max(a[d], lo[d]);
    ib[d] = min(b[d], hi[d]);
    inner = inner && ia[d] < ib[d];
  }
  return inner;
}

// Sum over a box of an integral image kept modulo 2^32 (box sums of integer images below 2^31).
__device__ __forceinline__ int box_sum_i(const int* __restrict__ ii, int64_t sx, int64_t sxy,
                                         int64_t x0, int64_t y0, int64_t z0, int ex, int ey, int ez) {
  const int* p = ii + x0 + sx * y0 + sxy * z0;
  const int* q = p + sxy * ez;
  const int64_t dy = sx * ey;
  const unsigned lo = (unsigned)p[dy + ex] - (unsigned)p[dy] - (unsigned)p[ex] + (unsigned)p[0];
  const unsigned up = (unsigned)q[dy + ex] - (unsigned)q[dy] - (unsigned)q[ex] + (unsigned)q[0];
  return (int)(up - lo);
}

// Cell of a training-image window at image origin (x0, y0, z0) under the mask "tile minus box
// [lo, hi)", from the Float64 integral images ii1 (values) and ii2 (squares).
__device__ void window_cell(const LpGeo& g, const double* __restrict__ ii1,
                            const double* __restrict__ ii2, int64_t sx, int64_t sxy, int64_t x0,
                            int64_t y0, int64_t z0, const int* lo, const int* hi, int cell,
                            float* out) {
  int a[3], b[3], ia[3], ib[3];
  const bool inner = cell_box(g, lo, hi, cell, a, b, ia, ib);
  double s1 = 0.0, s2 = 0.0, cnt = 0.0;
  if (b[0] > a[0] && b[1] > a[1] && b[2] > a[2]) {
    s1 = iq_box_sum(ii1, sx, sxy, x0 + a[0], y0 + a[1], z0 + a[2], b[0] - a[0], b[1] - a[1],
                    b[2] - a[2]);
    s2 = iq_box_sum(ii2, sx, sxy, x0 + a[0], y0 + a[1], z0 + a[2], b[0] - a[0], b[1] - a[1],
                    b[2] - a[2]);
    cnt = (double)(b[0] - a[0]) * (b[1] - a[1]) * (b[2] - a[2]);
    if (inner) {
      s1 -= iq_box_sum(ii1, sx, sxy, x0 + ia[0], y0 + ia[1], z0 + ia[2], ib[0] - ia[0],
                       ib[1] - ia[1], ib[2] - ia[2]);
      s2 -= iq_box_sum(ii2, sx, sxy, x0 + ia[0], y0 + ia[1], z0 + ia[2], ib[0] - ia[0],
                       ib[1] - ia[1], ib[2] - ia[2]);
      cnt -= (double)(ib[0] - ia[0]) * (ib[1] - ia[1]) * (ib[2] - ia[2]);
    }
  }
  const double vol = (double)g.c[0] * g.c[1] * g.c[2];
  out[0] = (float)(cnt / vol);
  out[1] = (float)(s1 / vol);
  out[2] = (float)(s2 / vol);
}

// The same for integer-valued images whose tile sums stay below 2^24: 32-bit integral images, and
// FP32 quotients. Both operands are integers below 2^24, so the Float64 quotient rounded to FP32 is
// the FP32 quotient (a 53-bit intermediate holds more than twice 24 bits: rounding twice changes
// nothing), and the results equal window_cell's. The Float64 pipe of this part is 1/64 of its FP32
// pipe: the sums and divisions of a window cost more than its convolutions there.
__device__ void window_cell_int(const LpGeo& g, const int* __restrict__ ii1,
                                const int* __restrict__ ii2, int64_t sx, int64_t sxy, int64_t x0,
                                int64_t y0, int64_t z0, const int* lo, const int* hi, int cell,
                                float* out) {
  int a[3], b[3], ia[3], ib[3];
  const bool inner = cell_box(g, lo, hi, cell, a, b, ia, ib);
  int s1 = 0, s2 = 0, cnt = 0;
  if (b[0] > a[0] && b[1] > a[1] && b[2] > a[2]) {
    s1 = box_sum_i(ii1, sx, sxy, x0 + a[0], y0 + a[1], z0 + a[2], b[0] - a[0], b[1] - a[1], b[2] - a[2]);
    s2 = box_sum_i(ii2, sx, sxy, x0 + a[0], y0 + a[1], z0 + a[2], b[0] - a[0], b[1] - a[1], b[2] - a[2]);
    cnt = (b[0] - a[0]) * (b[1] - a[1]) * (b[2] - a[2]);
    if (inner) {
      s1 -= box_sum_i(ii1, sx, sxy, x0 + ia[0], y0 + ia[1], z0 + ia[2], ib[0] - ia[0], ib[1] - ia[1], ib[2] - ia[2]);
      s2 -= box_sum_i(ii2, sx, sxy, x0 + ia[0], y0 + ia[1], z0 + ia[2], ib[0] - ia[0], ib[1] - ia[1], ib[2] - ia[2]);
      cnt -= (ib[0] - ia[0]) * (ib[1] - ia[1]) * (ib[2] - ia[2]);
    }
  }
  const float vol = (float)(g.c[0] * g.c[1] * g.c[2]);
  out[0] = __fdiv_rn((float)cnt, vol);
  out[1] = __fdiv_rn((float)s1, vol);
  out[2] = __fdiv_rn((float)s2, vol);
}

// Cell of a template: the simulation grid at `src` (grid strides gx, gxy), summed directly over the
// cell's voxels outside the box. INT: integer values whose tile sums stay below 2^24, FP32 sums and
// quotients as in window_cell_int.
template <bool INT>
__device__ void template_cell(const LpGeo& g, const float* __restrict__ src, int64_t gx,
                              int64_t gxy, const int* lo, const int* hi, int cell, float* out) {
  int c3[3];
  cell_of(g, cell, c3[0], c3[1], c3[2]);
  // rows summed in FP32, rows added in Float64 (exact for integer codes; GB300's FP64 pipe is
  // narrow, so FP64 work per row rather than per voxel)
  double s1 = 0.0, s2 = 0.0;
  float f1 = 0.f, f2 = 0.f;
  int cnt = 0;
  const int a0 = c3[0] * g.c[0], a1 = c3[1] * g.c[1], a2 = c3[2] * g.c[2];
  const int b0 = min(a0 + g.c[0], g.t[0]), b1 = min(a1 + g.c[1], g.t[1]), b2 = min(a2 + g.c[2], g.t[2]);
  for (int z = a2; z < b2; ++z)
    for (int y = a1; y < b1; ++y) {
      const bool rin = y >= lo[1] && y < hi[1] && z >= lo[2] && z < hi[2];
      float r1 = 0.f, r2 = 0.f;
      for (int x = a0; x < b0; ++x) {
        if (rin && x >= lo[0] && x < hi[0]) continue;
        const float v = src[x + gx * y + gxy * z];
        r1 += v;
        r2 = fmaf(v, v, r2);
        ++cnt;
      }
      if (INT) {
        f1 += r1;
        f2 += r2;
      } else {
        s1 += (double)r1;
        s2 += (double)r2;
      }
    }
  if (INT) {
    const float vol = (float)(g.c[0] * g.c[1] * g.c[2]);
    out[0] = __fdiv_rn((float)cnt, vol);
    out[1] = __fdiv_rn(f1, vol);
    out[2] = __fdiv_rn(f2, vol);
    return;
  }
  const double vol = (double)g.c[0] * g.c[1] * g.c[2];
  out[0] = (float)((double)cnt / vol);
  out[1] = (float)(s1 / vol);
  out[2] = (float)(s2 / vol);
}

}  // namespace
