// The learned proposal's encoder: inference, training forward and backward, InfoNCE, Adam (layers
// as described in iq_proposal.cu). Every layer is computed by register-tiled kernels over batches of
// items with channel-contiguous activations ([cell][32], rows of 36 words in shared memory), the
// transposed weights resident in shared memory.
//
// What bounds them: shared-memory reads that two warps a scheduler do not cover (net_l2: the data pipe
// 0.58, FMA pipe 0.35, issue 0.48 of the cycles). Layer 2 is 0.75 of the 0.85 M multiply-adds of an item (8 x 8 x 4
// cells), layer 3 most of the rest. One CTA per item with one output per thread and two loads per
// multiply-add took 0.54 us a window (10.6 ms for 20,000) and 2.25 + 7.7 + 14.5 ms for the forward,
// backward and weight gradients of a training batch of 4,352 items, of about 0.25 ms each at the
// pipe's rate; a 4 x 4 tile per thread loads eight 16-byte words per 64 of them. Now (4,352 items):
// net_l2 0.26 ms, net_l3 0.08, net_b3 0.10, net_b2 0.23, net_wgrad 0.25 + 0.06; 20,000 windows 1.2 ms.
//
//   net_l2_kernel    cell inputs, layers 1 and 2 -> h2      (batch of 4 items, warp = output row)
//   net_l3_kernel    layer 3, linear -> embeddings          (batch of 16 items)
//   net_b3_kernel    d/dE -> gz3, gz2                       (batch of 8 items)
//   net_b2_kernel    gz2 -> d/dz1, reduced to W1's gradient (batch of 4 items)
//   net_wgrad_kernel gradients of W2 and W3                 (warp = (dy, dz) taps, 96 sums a thread)
//   net_w4_kernel    gradient of W4
//   net_reduce_kernel partial sums of the CTAs, in CTA order (no atomics: the same bits every time)
//
// Inference adds every output's terms in the order bias, taps 0..26, input channels 0..31, one fused
// multiply-add each, with BF16-rounded parameters.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "iq_proposal_cells.cuh"

namespace {

constexpr int CH = IQ_LP_CH;
constexpr int EMB = IQ_LP_EMB;
constexpr int NIN = 3;
constexpr int NT = 256;    // threads of the encoder kernels
constexpr int LD = 36;     // words per staged cell (32 channels and 4 of padding: conflict-free rows)

// prepared parameters (floats): small ones, then W2 and W3 as [tap][ci][co], W4 as [f][o], and for
// the backward pass W2 and W3 as [tap][co][ci]
constexpr int NW_W1 = 0, NW_B1 = 96, NW_B2 = 128, NW_B3 = 160, NW_B4 = 192, NW_SMALL = 256;
constexpr int NW_W2 = NW_SMALL, NW_W3 = NW_W2 + 27 * CH * CH, NW_W4 = NW_W3 + 27 * CH * CH;
constexpr int NW_W2B = NW_W4 + EMB * CH * IQ_LP_MAXG3, NW_W3B = NW_W2B + 27 * CH * CH;
constexpr int NW_END = NW_W3B + 27 * CH * CH;

__global__ void net_prep_kernel(LpGeo g, const float* __restrict__ w, int bf16, float* __restrict__ o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  auto rd = [&](int k) { return bf16 ? __bfloat162float(__float2bfloat16_rn(w[k])) : w[k]; };
  if (i < 27 * CH * CH) {
    const int t = i >> 10, a = (i >> 5) & 31, b = i & 31;
    o[NW_W2 + i] = rd(LP_OFF_W2 + (b * CH + a) * 27 + t);
    o[NW_W3 + i] = rd(LP_OFF_W3 + (b * CH + a) * 27 + t);
    o[NW_W2B + i] = rd(LP_OFF_W2 + (a * CH + b) * 27 + t);
    o[NW_W3B + i] = rd(LP_OFF_W3 + (a * CH + b) * 27 + t);
  }
  if (i < g.nf * EMB) o[NW_W4 + i] = rd(LP_OFF_W4 + (i & 63) * g.nf + (i >> 6));
  if (i < 96) o[NW_W1 + i] = rd(LP_OFF_W1 + i);
  if (i < 32) {
    o[NW_B1 + i] = rd(LP_OFF_B1 + i);
    o[NW_B2 + i] = rd(LP_OFF_B2 + i);
    o[NW_B3 + i] = rd(LP_OFF_B3 + i);
  }
  if (i < EMB) o[NW_B4 + i] = rd(g.off_b4 + i);
}

// One training item: the features of a template (feat >= 0: row of `feats`) or a window of the
// image at distance-map position `pos` under the mask box of anchor `box`.
struct TrainItem {
  int32_t feat;   // row of the anchor feature table, or -1
  int32_t pos;    // window position when feat < 0
  int32_t box;    // row of the box table
  int32_t pad_;
};

// Where the items' cell inputs come from.
struct NetSrc {
  // windows: of position pos[i], or base + i, of the distance map
  const double *ii1, *ii2;     // Float64 integral images
  const int *iq1, *iq2;        // 32-bit ones (integer data; nullptr: Float64)
  int64_t isx, isxy, dx, dxy;
  const int64_t* pos;
  int64_t base;
  int lo[3], hi[3];            // mask box
  // templates (tsrc set): item i reads grid + tsrc[i] under tbox[i] (nullable: lo, hi)
  const float* grid;
  const int64_t* tsrc;
  int64_t gx, gxy;
  const int* tbox;
  int tint;                    // integer templates (template_cell<true>)
  // training items (items set)
  const TrainItem* items;
  const float* feats;
  const int32_t* boxes;
};

__device__ void item_cell(const LpGeo& g, const NetSrc& s, int64_t i, int cell, float* f) {
  int lo[3], hi[3];
  int64_t q;
  if (s.items) {
    const TrainItem it = s.items[i];
    if (it.feat >= 0) {
#pragma unroll
      for (int c = 0; c < NIN; ++c) f[c] = s.feats[((int64_t)it.feat * NIN + c) * g.ng + cell];
      return;
    }
    for (int d = 0; d < 3; ++d) { lo[d] = s.boxes[6 * it.box + d]; hi[d] = s.boxes[6 * it.box + 3 + d]; }
    q = it.pos;
  } else {
    for (int d = 0; d < 3; ++d) {
      lo[d] = s.tbox ? s.tbox[6 * i + d] : s.lo[d];
      hi[d] = s.tbox ? s.tbox[6 * i + 3 + d] : s.hi[d];
    }
    if (s.tsrc) {
      if (s.tint) template_cell<true>(g, s.grid + s.tsrc[i], s.gx, s.gxy, lo, hi, cell, f);
      else template_cell<false>(g, s.grid + s.tsrc[i], s.gx, s.gxy, lo, hi, cell, f);
      return;
    }
    q = s.pos ? s.pos[i] : s.base + i;
  }
  const int64_t z = q / s.dxy, r = q - z * s.dxy, y = r / s.dx, x = r - y * s.dx;
  if (s.iq1) window_cell_int(g, s.iq1, s.iq2, s.isx, s.isxy, x, y, z, lo, hi, cell, f);
  else window_cell(g, s.ii1, s.ii2, s.isx, s.isxy, x, y, z, lo, hi, cell, f);
}

// layer 1 of channel c at one cell
__device__ __forceinline__ float layer1(const float* sP, int c, float x0, float x1, float x2) {
  float z = sP[NW_B1 + c];
  z = fmaf(sP[NW_W1 + 3 * c], x0, z);
  z = fmaf(sP[NW_W1 + 3 * c + 1], x1, z);
  return fmaf(sP[NW_W1 + 3 * c + 2], x2, z);
}

__device__ __forceinline__ void fma4(float (&acc)[4], const float4& w, float a) {
  acc[0] = fmaf(w.x, a, acc[0]);
  acc[1] = fmaf(w.y, a, acc[1]);
  acc[2] = fmaf(w.z, a, acc[2]);
  acc[3] = fmaf(w.w, a, acc[3]);
}

// acc[i][c] += sum over k of A[i][k] W[k][c] for NC rows of 32 staged values and a 32 x 4 block of
// weights (rows of 32), k ascending
template <int NC>
__device__ __forceinline__ void gemm32(float (&acc)[NC][4], const float* const (&p)[NC], const float* w) {
#pragma unroll 4
  for (int k = 0; k < 32; k += 4) {
    float4 a[NC], b[4];
#pragma unroll
    for (int i = 0; i < NC; ++i) a[i] = *reinterpret_cast<const float4*>(p[i] + k);
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = *reinterpret_cast<const float4*>(w + (k + q) * 32);
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      fma4(acc[i], b[0], a[i].x);
      fma4(acc[i], b[1], a[i].y);
      fma4(acc[i], b[2], a[i].z);
      fma4(acc[i], b[3], a[i].w);
    }
  }
}

// ---- cell inputs, layers 1 and 2 ------------------------------------------------------------------
// Warp = one (y, z) row of layer 2's output (up to 4 cells in x) of 4 items; lane = (item, 4
// channels). Layer 1 is staged one z tap at a time, the planes 2 z + dz - 1 that it reads.
struct L2Args {
  LpGeo g;
  NetSrc s;
  const float* nw;   // prepared parameters
  int64_t n;
  float* X;          // [n][3][cells] cell inputs (nullable)
  float* h2;         // [n][cells of layer 2][32]
};

constexpr int L2_X = 4 * NIN * IQ_LP_MAXG;                    // floats
constexpr int L2_H = 4 * (2 * 64 * LD + 4);
constexpr size_t L2_SMEM = sizeof(float) * (27 * CH * CH + NW_SMALL + L2_X + L2_H + LD + 256);  // (+4 words an item, up to 32 items)

__global__ void __launch_bounds__(NT, 1) net_l2_kernel(const L2Args a) {
  extern __shared__ __align__(16) float smf[];
  float* sW = smf;
  float* sP = sW + 27 * CH * CH;
  float* sZ = sP + NW_SMALL;       // a row of zeros (padding cells)
  float* sX = sZ + LD;
  float* sH = sX + L2_X + 28;      // (16-byte aligned)
  const LpGeo& g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < 27 * CH * CH / 4; i += NT)
    reinterpret_cast<float4*>(sW)[i] = reinterpret_cast<const float4*>(a.nw + NW_W2)[i];
  for (int i = tid; i < NW_SMALL; i += NT) sP[i] = a.nw[i];
  if (tid < LD) sZ[tid] = 0.f;
  const int gx = g.g[0], gy = g.g[1], gz = g.g[2], cxy = gx * gy;
  const int g2x = g.g2[0], g2y = g.g2[1], g2z = g.g2[2];
  const int nrows = g2y * g2z, ngrp = 8 / nrows, ipb = 4 * ngrp;
  const int istride = g2z * cxy * LD + 4;  // words per item (items on different banks)
  const int row = warp % nrows, oy = row % g2y, oz = row / g2y;
  const bool work = warp < nrows * ngrp;
  const int item = (warp / nrows) * 4 + (lane >> 3), co = 4 * (lane & 7);
  const int64_t nb = (a.n + ipb - 1) / ipb;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int64_t i0 = b * ipb;
    __syncthreads();  // the previous batch's readers are done
    for (int i = tid; i < ipb * g.ng; i += NT) {
      const int it = i / g.ng, cell = i - it * g.ng;
      float f[3] = {0.f, 0.f, 0.f};
      if (i0 + it < a.n) item_cell(g, a.s, i0 + it, cell, f);
#pragma unroll
      for (int c = 0; c < NIN; ++c) {
        sX[(it * NIN + c) * g.ng + cell] = f[c];
        if (a.X && i0 + it < a.n) a.X[((i0 + it) * NIN + c) * g.ng + cell] = f[c];
      }
    }
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][c] = sP[NW_B2 + co + c];
    for (int dz = 0; dz < 3; ++dz) {
      __syncthreads();
      for (int i = tid; i < ipb * g2z * cxy; i += NT) {
        const int it = i / (g2z * cxy), r = i - it * g2z * cxy, pz = r / cxy, c = r - pz * cxy;
        const int z = 2 * pz + dz - 1;
        if (z < 0 || z >= gz) continue;
        const float* x = sX + it * NIN * g.ng + z * cxy + c;
        const float x0 = x[0], x1 = x[g.ng], x2 = x[2 * g.ng];
        float* h = sH + it * istride + r * LD;
#pragma unroll
        for (int q = 0; q < CH; q += 4) {
          float4 v;
          v.x = fmaxf(layer1(sP, q, x0, x1, x2), 0.f);
          v.y = fmaxf(layer1(sP, q + 1, x0, x1, x2), 0.f);
          v.z = fmaxf(layer1(sP, q + 2, x0, x1, x2), 0.f);
          v.w = fmaxf(layer1(sP, q + 3, x0, x1, x2), 0.f);
          *reinterpret_cast<float4*>(h + q) = v;
        }
      }
      __syncthreads();
      const int z = 2 * oz + dz - 1;
      if (!work || z < 0 || z >= gz) continue;
      const float* plane = sH + item * istride + oz * cxy * LD;
      for (int dy = 0; dy < 3; ++dy) {
        const int y = 2 * oy + dy - 1;
        if (y < 0 || y >= gy) continue;
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
          const float* p[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int x = 2 * i + dx - 1;
            p[i] = (i < g2x && x >= 0 && x < gx) ? plane + (y * gx + x) * LD : sZ;
          }
          gemm32<4>(acc, p, sW + (dx + 3 * dy + 9 * dz) * CH * CH + co);
        }
      }
    }
    if (work && i0 + item < a.n) {
      float* o = a.h2 + ((i0 + item) * g.ng2 + g2x * (oy + g2y * oz)) * CH + co;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < g2x)
          *reinterpret_cast<float4*>(o + i * CH) =
              make_float4(fmaxf(acc[i][0], 0.f), fmaxf(acc[i][1], 0.f), fmaxf(acc[i][2], 0.f),
                          fmaxf(acc[i][3], 0.f));
    }
  }
}

// ---- layer 3 and the output layer -------------------------------------------------------------------
// Thread = (item, 2 channels) of layer 3 (all of its up to 4 cells), then (4 items, 1 output).
struct L3Args {
  LpGeo g;
  const float* nw;
  int64_t n;
  const float* h2;
  float* h3;              // [n][cells of layer 3][32] (nullable)
  float* E;               // [n][64] FP32 (nullable)
  __nv_bfloat16* out;     // [n][64] BF16 (nullable) and the squared norms of those
  float* norm;
};

constexpr int L3_IPB = 16;
constexpr int L3_H2 = L3_IPB * (IQ_LP_MAXG2 * LD + 4), L3_H3 = L3_IPB * CH * IQ_LP_MAXG3;
constexpr size_t L3_SMEM = sizeof(float) * (27 * CH * CH + L3_H2 + L3_H3 + L3_IPB * EMB + LD + 32);

__global__ void __launch_bounds__(NT, 1) net_l3_kernel(const L3Args a) {
  extern __shared__ __align__(16) float smf[];
  float* sW = smf;
  float* sH = sW + 27 * CH * CH;
  float* s3 = sH + L3_H2;
  float* sE = s3 + L3_H3;
  float* sZ = sE + L3_IPB * EMB;
  const LpGeo& g = a.g;
  const int tid = threadIdx.x;
  for (int i = tid; i < 27 * CH * CH / 4; i += NT)
    reinterpret_cast<float4*>(sW)[i] = reinterpret_cast<const float4*>(a.nw + NW_W3)[i];
  if (tid < LD) sZ[tid] = 0.f;
  const int G2 = g.ng2, G3 = g.ng3, nf = g.nf;
  const int istride = G2 * LD + 4;
  const int item = tid >> 4, co = 2 * (tid & 15);
  const float b3[2] = {a.nw[NW_B3 + co], a.nw[NW_B3 + co + 1]};
  const int64_t nb = (a.n + L3_IPB - 1) / L3_IPB;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int64_t i0 = b * L3_IPB;
    __syncthreads();
    for (int i = tid; i < L3_IPB * G2 * 8; i += NT) {
      const int it = i / (G2 * 8), r = i - it * G2 * 8, c = r >> 3, q = 4 * (r & 7);
      const float4 v = i0 + it < a.n
                           ? *reinterpret_cast<const float4*>(a.h2 + ((i0 + it) * G2 + c) * CH + q)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(sH + it * istride + c * LD + q) = v;
    }
    __syncthreads();
    float acc[4][2];
#pragma unroll
    for (int m = 0; m < 4; ++m) { acc[m][0] = b3[0]; acc[m][1] = b3[1]; }
    const float* hb = sH + item * istride;
    for (int t = 0; t < 27; ++t) {
      const float* p[4];
      bool any = false;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        p[m] = sZ;
        if (m < G3) {
          const int x = 2 * (m % g.g3[0]) + t % 3 - 1, y = 2 * ((m / g.g3[0]) % g.g3[1]) + (t / 3) % 3 - 1,
                    z = 2 * (m / (g.g3[0] * g.g3[1])) + t / 9 - 1;
          if (x >= 0 && y >= 0 && z >= 0 && x < g.g2[0] && y < g.g2[1] && z < g.g2[2]) {
            p[m] = hb + (x + g.g2[0] * (y + g.g2[1] * z)) * LD;
            any = true;
          }
        }
      }
      if (!any) continue;  // the same for every thread
      const float* w = sW + t * CH * CH + co;
#pragma unroll 4
      for (int k = 0; k < 32; k += 4) {
        float4 v[4];
        float2 c[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) v[m] = *reinterpret_cast<const float4*>(p[m] + k);
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] = *reinterpret_cast<const float2*>(w + (k + q) * 32);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          acc[m][0] = fmaf(c[0].x, v[m].x, acc[m][0]); acc[m][1] = fmaf(c[0].y, v[m].x, acc[m][1]);
          acc[m][0] = fmaf(c[1].x, v[m].y, acc[m][0]); acc[m][1] = fmaf(c[1].y, v[m].y, acc[m][1]);
          acc[m][0] = fmaf(c[2].x, v[m].z, acc[m][0]); acc[m][1] = fmaf(c[2].y, v[m].z, acc[m][1]);
          acc[m][0] = fmaf(c[3].x, v[m].w, acc[m][0]); acc[m][1] = fmaf(c[3].y, v[m].w, acc[m][1]);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if (m < G3) {
        const float2 v = make_float2(fmaxf(acc[m][0], 0.f), fmaxf(acc[m][1], 0.f));
        *reinterpret_cast<float2*>(s3 + item * nf + m * CH + co) = v;
        if (a.h3 && i0 + item < a.n) *reinterpret_cast<float2*>(a.h3 + (i0 + item) * nf + m * CH + co) = v;
      }
    __syncthreads();
    {  // linear: output o of items 4 q .. 4 q + 3
      const int o = tid & 63, it0 = 4 * (tid >> 6);
      float e[4];
      const float b4 = a.nw[NW_B4 + o];
#pragma unroll
      for (int i = 0; i < 4; ++i) e[i] = b4;
#pragma unroll 4
      for (int f = 0; f < nf; ++f) {
        const float w = __ldg(a.nw + NW_W4 + f * EMB + o);
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = fmaf(w, s3[(it0 + i) * nf + f], e[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) sE[(it0 + i) * EMB + o] = e[i];
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    for (int it = warp; it < L3_IPB && i0 + it < a.n; it += NT / 32) {
      const float e0 = sE[it * EMB + lane], e1 = sE[it * EMB + 32 + lane];
      if (a.E) {
        a.E[(i0 + it) * EMB + lane] = e0;
        a.E[(i0 + it) * EMB + 32 + lane] = e1;
      }
      if (a.out) {
        const __nv_bfloat16 v0 = __float2bfloat16_rn(e0), v1 = __float2bfloat16_rn(e1);
        a.out[(i0 + it) * EMB + lane] = v0;
        a.out[(i0 + it) * EMB + 32 + lane] = v1;
        const float f0 = __bfloat162float(v0), f1 = __bfloat162float(v1);
        float s = fmaf(f0, f0, 0.f);
        s = fmaf(f1, f1, s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) a.norm[i0 + it] = s;
      }
    }
  }
}

// ---- backward: transposed stride-2 convolution -----------------------------------------------------
// acc[i][c] (NC cells 2 i + px of input row (jy, jz), 4 input channels) = sum over the taps t that
// link them to output cells m, and over their channels, of gz[m][co] W[t][co][ci].
template <int NC>
__device__ __forceinline__ void tconv_row(float (&acc)[NC][4], const int* Go, const float* gz,
                                          const float* zero, const float* w, int px, int jy, int jz) {
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
  for (int dz = 0; dz < 3; ++dz) {
    const int az = jz + 1 - dz;
    if (az < 0 || (az & 1) || (az >> 1) >= Go[2]) continue;
    for (int dy = 0; dy < 3; ++dy) {
      const int ay = jy + 1 - dy;
      if (ay < 0 || (ay & 1) || (ay >> 1) >= Go[1]) continue;
      const float* r = gz + (Go[0] * ((ay >> 1) + Go[1] * (az >> 1))) * LD;
      for (int dx = px ? 0 : 1; dx < 3; dx += 2) {
        const int o = (px + 1 - dx) >> 1;  // output cell of cell i: i + o
        const float* p[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) p[i] = i + o < Go[0] ? r + (i + o) * LD : zero;
        gemm32<NC>(acc, p, w + (dx + 3 * dy + 9 * dz) * CH * CH);
      }
    }
  }
}

// d loss / dE -> gz3 (through the output layer and layer 3's ReLU) and gz2 (through layer 3 and
// layer 2's ReLU).
struct B3Args {
  LpGeo g;
  const float* w;        // FP32 parameters (W4)
  const float* nw;
  int64_t n;
  const float *gE, *h3, *h2;
  float *gz3, *gz2;
};

constexpr int B3_IPB = 8;
constexpr size_t B3_SMEM = sizeof(float) * (27 * CH * CH + B3_IPB * (IQ_LP_MAXG3 * LD + 4) + B3_IPB * EMB + LD + 32);

__global__ void __launch_bounds__(NT, 1) net_b3_kernel(const B3Args a) {
  extern __shared__ __align__(16) float smf[];
  float* sW = smf;
  float* sG = sW + 27 * CH * CH;
  float* sE = sG + B3_IPB * (IQ_LP_MAXG3 * LD + 4);
  float* sZ = sE + B3_IPB * EMB;
  const LpGeo& g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < 27 * CH * CH / 4; i += NT)
    reinterpret_cast<float4*>(sW)[i] = reinterpret_cast<const float4*>(a.nw + NW_W3B)[i];
  if (tid < LD) sZ[tid] = 0.f;
  const int G2 = g.ng2, nf = g.nf, istride = g.ng3 * LD + 4;
  const int64_t nb = (a.n + B3_IPB - 1) / B3_IPB;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int64_t i0 = b * B3_IPB;
    __syncthreads();
    for (int i = tid; i < B3_IPB * EMB; i += NT)
      sE[i] = i0 + i / EMB < a.n ? a.gE[i0 * EMB + i] : 0.f;
    __syncthreads();
    for (int f = lane; f < nf; f += 32) {  // warp = item
      float acc = 0.f;
#pragma unroll 8
      for (int o = 0; o < EMB; ++o) acc = fmaf(__ldg(a.w + LP_OFF_W4 + o * nf + f), sE[warp * EMB + o], acc);
      const int64_t it = i0 + warp;
      const float v = it < a.n && a.h3[it * nf + f] > 0.f ? acc : 0.f;
      sG[warp * istride + (f >> 5) * LD + (f & 31)] = v;
      if (it < a.n) a.gz3[it * nf + f] = v;
    }
    __syncthreads();
    // lane = (item of 4, 4 channels); rows (item group, x parity, y, z) over the warps
    const int ci = 4 * (lane & 7);
    const int rows = 2 * g.g2[1] * g.g2[2];
    for (int u = warp; u < 2 * rows; u += NT / 32) {
      const int item = 4 * (u / rows) + (lane >> 3), r = u % rows;
      const int px = r & 1, jy = (r >> 1) % g.g2[1], jz = (r >> 1) / g.g2[1];
      float acc[2][4];
      tconv_row<2>(acc, g.g3, sG + item * istride, sZ, sW + ci, px, jy, jz);
      if (i0 + item >= a.n) continue;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int jx = 2 * i + px;
        if (jx >= g.g2[0]) continue;
        const int64_t at = ((i0 + item) * G2 + jx + g.g2[0] * (jy + g.g2[1] * jz)) * CH + ci;
        const float4 h = *reinterpret_cast<const float4*>(a.h2 + at);
        *reinterpret_cast<float4*>(a.gz2 + at) =
            make_float4(h.x > 0.f ? acc[i][0] : 0.f, h.y > 0.f ? acc[i][1] : 0.f,
                        h.z > 0.f ? acc[i][2] : 0.f, h.w > 0.f ? acc[i][3] : 0.f);
      }
    }
  }
}

// gz2 -> d loss / dz1 through layer 2 and layer 1's ReLU, reduced at once to the gradient of W1 and
// b1 (partial sums of the CTA: part[cta][channel][3 weights, bias]).
struct B2Args {
  LpGeo g;
  const float* nw;
  int64_t n;
  const float *X, *gz2;
  float* part;
};

constexpr int B2_G = 4 * (IQ_LP_MAXG2 * LD + 4);
constexpr size_t B2_SMEM = sizeof(float) * (27 * CH * CH + NW_SMALL + B2_G + L2_X + LD + 32);

__global__ void __launch_bounds__(NT, 1) net_b2_kernel(const B2Args a) {
  extern __shared__ __align__(16) float smf[];
  float* sW = smf;
  float* sP = sW + 27 * CH * CH;
  float* sG = sP + NW_SMALL;
  float* sX = sG + B2_G;
  float* sZ = sX + L2_X;
  const LpGeo& g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < 27 * CH * CH / 4; i += NT)
    reinterpret_cast<float4*>(sW)[i] = reinterpret_cast<const float4*>(a.nw + NW_W2B)[i];
  for (int i = tid; i < NW_SMALL; i += NT) sP[i] = a.nw[i];
  if (tid < LD) sZ[tid] = 0.f;
  const int G2 = g.ng2, istride = G2 * LD + 4;
  const int ci = 4 * (lane & 7), item = lane >> 3;
  float gw[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int q = 0; q < 4; ++q) gw[c][q] = 0.f;
  const int64_t nb = (a.n + 3) / 4;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int64_t i0 = b * 4;
    __syncthreads();
    for (int i = tid; i < 4 * G2 * 8; i += NT) {
      const int it = i / (G2 * 8), r = i - it * G2 * 8, c = r >> 3, q = 4 * (r & 7);
      const float4 v = i0 + it < a.n
                           ? *reinterpret_cast<const float4*>(a.gz2 + ((i0 + it) * G2 + c) * CH + q)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(sG + it * istride + c * LD + q) = v;
    }
    for (int i = tid; i < 4 * NIN * g.ng; i += NT)
      sX[i] = i0 + i / (NIN * g.ng) < a.n ? a.X[i0 * NIN * g.ng + i] : 0.f;
    __syncthreads();
    const int ny = g.g[1], rows = 2 * ny * g.g[2];
    for (int u = warp; u < rows; u += NT / 32) {
      // rows of one warp take every y parity in turn (odd rows have twice the taps)
      const int k = u / ny, jy = (u + k) % ny, px = k & 1, jz = k >> 1;
      float acc[4][4];
      tconv_row<4>(acc, g.g2, sG + item * istride, sZ, sW + ci, px, jy, jz);
      const float* x = sX + item * NIN * g.ng + g.g[0] * (jy + ny * jz);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int jx = 2 * i + px;
        if (jx >= g.g[0]) continue;
        const float x0 = x[jx], x1 = x[g.ng + jx], x2 = x[2 * g.ng + jx];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float v = layer1(sP, ci + c, x0, x1, x2) > 0.f ? acc[i][c] : 0.f;
          gw[c][0] = fmaf(v, x0, gw[c][0]);
          gw[c][1] = fmaf(v, x1, gw[c][1]);
          gw[c][2] = fmaf(v, x2, gw[c][2]);
          gw[c][3] += v;
        }
      }
    }
  }
  // sums over the lanes of one channel group, then over the warps
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      gw[c][q] += __shfl_xor_sync(0xffffffffu, gw[c][q], 8);
      gw[c][q] += __shfl_xor_sync(0xffffffffu, gw[c][q], 16);
    }
  __syncthreads();
  float* red = sG;  // [8 warps][32 channels][4]
  if (lane < 8)
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int q = 0; q < 4; ++q) red[(warp * CH + ci + c) * 4 + q] = gw[c][q];
  __syncthreads();
  if (tid < CH * 4) {
    float s = 0.f;
    for (int w = 0; w < NT / 32; ++w) s += red[w * CH * 4 + tid];
    a.part[(int64_t)blockIdx.x * CH * 4 + tid] = s;
  }
}

// ---- weight gradients of the convolutions -----------------------------------------------------------
// grad W[co][ci][t] = sum over items and output cells m of gz[m][co] hin[cell(m, t)][ci]. Warp =
// (dy, dz); a thread holds the 3 dx taps of 8 input and 4 output channels. LAYER 2 stages layer 1's
// output from the cell inputs, LAYER 3 reads h2. part[cta][tap][ci][co], then the bias sums.
struct WgArgs {
  LpGeo g;
  const float* nw;
  int64_t n;
  const float* hin;   // LAYER 2: X; LAYER 3: h2
  const float* gz;
  float* part;
};

constexpr int WG_NT = 288;
constexpr int WG_PART = 27 * CH * CH + CH;
constexpr size_t wg_smem(int layer) {
  return sizeof(float) * (layer == 2 ? IQ_LP_MAXG * LD + IQ_LP_MAXG2 * LD + NIN * IQ_LP_MAXG + NW_SMALL
                                     : IQ_LP_MAXG2 * LD + IQ_LP_MAXG3 * LD);
}

template <int LAYER>
__global__ void __launch_bounds__(WG_NT, 1) net_wgrad_kernel(const WgArgs a) {
  extern __shared__ __align__(16) float smf[];
  const LpGeo& g = a.g;
  const int* Gi = LAYER == 2 ? g.g : g.g2;
  const int* Go = LAYER == 2 ? g.g2 : g.g3;
  const int nin = LAYER == 2 ? g.ng : g.ng2, nout = LAYER == 2 ? g.ng2 : g.ng3;
  float* sH = smf;
  float* sG = sH + (LAYER == 2 ? IQ_LP_MAXG : IQ_LP_MAXG2) * LD;
  float* sX = sG + (LAYER == 2 ? IQ_LP_MAXG2 : IQ_LP_MAXG3) * LD;
  float* sP = sX + NIN * IQ_LP_MAXG;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dy = warp % 3, dz = warp / 3;
  const int ci = 8 * (lane >> 3), co = 4 * (lane & 7);
  if (LAYER == 2)
    for (int i = tid; i < NW_SMALL; i += WG_NT) sP[i] = a.nw[i];
  float acc[3][8][4];
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[d][i][c] = 0.f;
  float bias = 0.f;
  for (int64_t item = blockIdx.x; item < a.n; item += gridDim.x) {
    __syncthreads();  // the previous item's readers are done
    for (int i = tid; i < nout * 8; i += WG_NT)
      *reinterpret_cast<float4*>(sG + (i >> 3) * LD + 4 * (i & 7)) =
          *reinterpret_cast<const float4*>(a.gz + (item * nout + (i >> 3)) * CH + 4 * (i & 7));
    if (LAYER == 3) {
      for (int i = tid; i < nin * 8; i += WG_NT)
        *reinterpret_cast<float4*>(sH + (i >> 3) * LD + 4 * (i & 7)) =
            *reinterpret_cast<const float4*>(a.hin + (item * nin + (i >> 3)) * CH + 4 * (i & 7));
    } else {
      for (int i = tid; i < NIN * nin; i += WG_NT) sX[i] = a.hin[item * NIN * nin + i];
      __syncthreads();
      for (int c = tid; c < nin; c += WG_NT) {
        const float x0 = sX[c], x1 = sX[nin + c], x2 = sX[2 * nin + c];
#pragma unroll
        for (int q = 0; q < CH; q += 4) {
          float4 v;
          v.x = fmaxf(layer1(sP, q, x0, x1, x2), 0.f);
          v.y = fmaxf(layer1(sP, q + 1, x0, x1, x2), 0.f);
          v.z = fmaxf(layer1(sP, q + 2, x0, x1, x2), 0.f);
          v.w = fmaxf(layer1(sP, q + 3, x0, x1, x2), 0.f);
          *reinterpret_cast<float4*>(sH + c * LD + q) = v;
        }
      }
    }
    __syncthreads();
    if (warp == 0)
      for (int m = 0; m < nout; ++m) bias += sG[m * LD + lane];
    for (int oz = 0; oz < Go[2]; ++oz) {
      const int z = 2 * oz + dz - 1;
      if (z < 0 || z >= Gi[2]) continue;
      for (int oy = 0; oy < Go[1]; ++oy) {
        const int y = 2 * oy + dy - 1;
        if (y < 0 || y >= Gi[1]) continue;
        const float* hr = sH + Gi[0] * (y + Gi[1] * z) * LD + ci;
        const float* gr = sG + Go[0] * (oy + Go[1] * oz) * LD + co;
        for (int ox = 0; ox < Go[0]; ++ox) {
          const float4 v = *reinterpret_cast<const float4*>(gr + ox * LD);
#pragma unroll
          for (int dx = 0; dx < 3; ++dx) {
            const int x = 2 * ox + dx - 1;
            if (x < 0 || x >= Gi[0]) continue;
            const float4 h0 = *reinterpret_cast<const float4*>(hr + x * LD);
            const float4 h1 = *reinterpret_cast<const float4*>(hr + x * LD + 4);
            fma4(acc[dx][0], v, h0.x);
            fma4(acc[dx][1], v, h0.y);
            fma4(acc[dx][2], v, h0.z);
            fma4(acc[dx][3], v, h0.w);
            fma4(acc[dx][4], v, h1.x);
            fma4(acc[dx][5], v, h1.y);
            fma4(acc[dx][6], v, h1.z);
            fma4(acc[dx][7], v, h1.w);
          }
        }
      }
    }
  }
  float* part = a.part + (int64_t)blockIdx.x * WG_PART;
#pragma unroll
  for (int dx = 0; dx < 3; ++dx)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<float4*>(part + ((dx + 3 * dy + 9 * dz) * CH + ci + i) * CH + co) =
          make_float4(acc[dx][i][0], acc[dx][i][1], acc[dx][i][2], acc[dx][i][3]);
  if (warp == 0) part[27 * CH * CH + lane] = bias;
}

// gradient of W4 and b4: part[cta][64][nf], then 64 bias sums
struct W4Args {
  LpGeo g;
  int64_t n;
  const float *gE, *h3;
  float* part;
};

constexpr int W4_IPB = 32;
constexpr int W4_PART = EMB * CH * IQ_LP_MAXG3 + EMB;

__global__ void __launch_bounds__(NT) net_w4_kernel(const W4Args a) {
  __shared__ __align__(16) float sE[W4_IPB * EMB];
  __shared__ __align__(16) float sF[W4_IPB * CH * IQ_LP_MAXG3];
  const int tid = threadIdx.x, nf = a.g.nf;
  const int f = 4 * (tid & 31), o = 8 * (tid >> 5);
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
  float bias = 0.f;
  const int64_t nb = (a.n + W4_IPB - 1) / W4_IPB;
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const int64_t i0 = b * W4_IPB;
    const int m = (int)min((int64_t)W4_IPB, a.n - i0);
    __syncthreads();
    for (int i = tid; i < m * EMB; i += NT) sE[i] = a.gE[i0 * EMB + i];
    for (int i = tid; i < m * nf; i += NT) sF[i] = a.h3[i0 * nf + i];
    __syncthreads();
    if (tid < EMB)
      for (int i = 0; i < m; ++i) bias += sE[i * EMB + tid];
    if (f < nf)
      for (int i = 0; i < m; ++i) {
        const float4 h = *reinterpret_cast<const float4*>(sF + i * nf + f);
        const float4 e0 = *reinterpret_cast<const float4*>(sE + i * EMB + o);
        const float4 e1 = *reinterpret_cast<const float4*>(sE + i * EMB + o + 4);
        fma4(acc[0], h, e0.x); fma4(acc[1], h, e0.y); fma4(acc[2], h, e0.z); fma4(acc[3], h, e0.w);
        fma4(acc[4], h, e1.x); fma4(acc[5], h, e1.y); fma4(acc[6], h, e1.z); fma4(acc[7], h, e1.w);
      }
  }
  float* part = a.part + (int64_t)blockIdx.x * W4_PART;
  if (f < nf)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<float4*>(part + (o + i) * nf + f) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  if (tid < EMB) part[EMB * CH * IQ_LP_MAXG3 + tid] = bias;
}

// grad[parameter] = its partial sums in CTA order
struct RedArgs {
  LpGeo g;
  const float *p1, *p2, *p3, *p4;  // W1, W2, W3, W4 partials
  int n1, n2, n3, n4;
  float* grad;
};

__global__ void net_reduce_kernel(const RedArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const float* p;
  int n, stride, dst;
  constexpr int C2 = WG_PART;
  int k = i;
  if (k < C2 || (k -= C2) < C2) {
    const bool l2 = i < C2;
    p = (l2 ? a.p2 : a.p3) + k;
    n = l2 ? a.n2 : a.n3;
    stride = WG_PART;
    if (k < 27 * CH * CH) {
      const int t = k >> 10, ci = (k >> 5) & 31, co = k & 31;
      dst = (l2 ? LP_OFF_W2 : LP_OFF_W3) + (co * CH + ci) * 27 + t;
    } else {
      dst = (l2 ? LP_OFF_B2 : LP_OFF_B3) + (k - 27 * CH * CH);
    }
  } else if ((k -= C2) < EMB * a.g.nf) {
    p = a.p4 + k; n = a.n4; stride = W4_PART; dst = LP_OFF_W4 + k;
  } else if ((k -= EMB * a.g.nf) < EMB) {
    p = a.p4 + EMB * CH * IQ_LP_MAXG3 + k; n = a.n4; stride = W4_PART; dst = a.g.off_b4 + k;
  } else if ((k -= EMB) < CH * 4) {
    const int c = k >> 2, q = k & 3;
    p = a.p1 + k; n = a.n1; stride = CH * 4;
    dst = q < NIN ? LP_OFF_W1 + c * NIN + q : LP_OFF_B1 + c;
  } else {
    return;
  }
  float s = 0.f;
#pragma unroll 8
  for (int b = 0; b < n; ++b) s += p[(int64_t)b * stride];
  a.grad[dst] = s;
}

__global__ void net_int_ii_kernel(const double* __restrict__ ii, int64_t n, int* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (int)(unsigned)(unsigned long long)(long long)ii[i];
}

// InfoNCE of anchor b (one warp): items b (anchor), nA + b (positive), 2 nA + b * nneg + n
// (negatives). Writes d loss / d embedding of those items (scaled by 1 / nA) and adds the loss.
__global__ void lp_loss_kernel(const float* __restrict__ E, int nA, int nneg, float temp,
                               float* gE, double* loss) {
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= nA) return;
  const int nj = 1 + nneg;
  auto item_of = [&](int j) -> int64_t {
    return j == 0 ? (int64_t)nA + b : 2 * (int64_t)nA + (int64_t)b * nneg + (j - 1);
  };
  const float a0 = E[(int64_t)b * EMB + lane], a1 = E[(int64_t)b * EMB + 32 + lane];
  // logits
  float zmax = -1e30f;
  for (int j = 0; j < nj; ++j) {
    const int64_t it = item_of(j);
    const float d0 = a0 - E[it * EMB + lane], d1 = a1 - E[it * EMB + 32 + lane];
    float s = d0 * d0 + d1 * d1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    zmax = fmaxf(zmax, -s / temp);
  }
  float den = 0.f, z0 = 0.f;
  for (int j = 0; j < nj; ++j) {
    const int64_t it = item_of(j);
    const float d0 = a0 - E[it * EMB + lane], d1 = a1 - E[it * EMB + 32 + lane];
    float s = d0 * d0 + d1 * d1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float z = -s / temp;
    if (j == 0) z0 = z;
    den += expf(z - zmax);
  }
  if (lane == 0) atomicAdd(loss, (double)(-z0 + zmax + logf(den)) / nA);
  float ga0 = 0.f, ga1 = 0.f;
  const float sc = 1.f / (float)nA;
  for (int j = 0; j < nj; ++j) {
    const int64_t it = item_of(j);
    const float d0 = a0 - E[it * EMB + lane], d1 = a1 - E[it * EMB + 32 + lane];
    float s = d0 * d0 + d1 * d1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    float gz = expf(-s / temp - zmax) / den - (j == 0 ? 1.f : 0.f);
    gz *= sc;
    // z_j = -|ea - ej|^2 / T: dz/dea = -2 d / T, dz/dej = 2 d / T
    ga0 += gz * (-2.f * d0 / temp);
    ga1 += gz * (-2.f * d1 / temp);
    gE[it * EMB + lane] = gz * (2.f * d0 / temp);
    gE[it * EMB + 32 + lane] = gz * (2.f * d1 / temp);
  }
  gE[(int64_t)b * EMB + lane] = ga0;
  gE[(int64_t)b * EMB + 32 + lane] = ga1;
}

__global__ void lp_adam_kernel(float* p, const float* g, float* m, float* v, int n, float lr,
                               float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace

// ---------------------------------------------------------------------------------------------
LpGeo iq_lp_geo(Dim3 tile) {
  LpGeo g{};
  const int64_t t[3] = {tile.x, tile.y, tile.z};
  const int gm[3] = {8, 8, 4};
  for (int d = 0; d < 3; ++d) {
    g.t[d] = (int)t[d];
    g.g[d] = (int)std::min<int64_t>(t[d], gm[d]);
    g.c[d] = (int)((t[d] + g.g[d] - 1) / g.g[d]);
    g.g2[d] = (g.g[d] + 1) / 2;
    g.g3[d] = (g.g2[d] + 1) / 2;
  }
  g.ng = g.g[0] * g.g[1] * g.g[2];
  g.ng2 = g.g2[0] * g.g2[1] * g.g2[2];
  g.ng3 = g.g3[0] * g.g3[1] * g.g3[2];
  g.nf = CH * g.ng3;
  g.off_b4 = LP_OFF_W4 + EMB * g.nf;
  g.npar = g.off_b4 + EMB;
  return g;
}

namespace {

// prepared parameters in scratch
int net_prep(iq_ctx* ctx, const LpGeo& g, const float* w, int bf16, float** out) {
  float* nw = (float*)iq_scratch(ctx, S_LP_W, sizeof(float) * NW_END);
  if (!nw) return IQ_ERR_ALLOC;
  net_prep_kernel<<<(27 * CH * CH + 255) / 256, 256, 0, ctx->stream>>>(g, w, bf16, nw);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  *out = nw;
  return IQ_OK;
}

int net_l2(iq_ctx* ctx, const LpGeo& g, const NetSrc& s, const float* nw, int64_t n, float* X, float* h2) {
  L2Args a{};
  a.g = g; a.s = s; a.nw = nw; a.n = n; a.X = X; a.h2 = h2;
  IQ_CUDA_OK(cudaFuncSetAttribute(net_l2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L2_SMEM));
  const int ipb = 4 * (8 / (g.g2[1] * g.g2[2]));
  net_l2_kernel<<<(unsigned)std::min<int64_t>((n + ipb - 1) / ipb, iq_sm_count()), NT, L2_SMEM, ctx->stream>>>(a);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int net_l3(iq_ctx* ctx, const L3Args& a) {
  IQ_CUDA_OK(cudaFuncSetAttribute(net_l3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L3_SMEM));
  net_l3_kernel<<<(unsigned)std::min<int64_t>((a.n + L3_IPB - 1) / L3_IPB, iq_sm_count()), NT, L3_SMEM, ctx->stream>>>(a);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

// Inference of n items: blocks of NET_BLOCK items through both kernels (their layer-2 outputs,
// 4 KB an item, stay in L2).
constexpr int64_t NET_BLOCK = 16384;

int net_encode(iq_ctx* ctx, const LpGeo& g, const float* w, NetSrc s, int64_t n, __nv_bfloat16* out,
               float* norm) {
  float* nw = nullptr;
  int rc = net_prep(ctx, g, w, 1, &nw);
  if (rc) return rc;
  float* h2 = (float*)iq_scratch(ctx, S_LP_BH2, sizeof(float) * std::min(n, NET_BLOCK) * g.ng2 * CH);
  if (!h2) return IQ_ERR_ALLOC;
  iq_timer_start(ctx, "lp.encode");
  for (int64_t i0 = 0; i0 < n; i0 += NET_BLOCK) {
    const int64_t m = std::min(NET_BLOCK, n - i0);
    NetSrc b = s;
    if (b.pos) b.pos += i0;
    else b.base += i0;
    if (b.tsrc) b.tsrc += i0;
    if (b.tbox) b.tbox += 6 * i0;
    if ((rc = net_l2(ctx, g, b, nw, m, nullptr, h2))) return rc;
    L3Args a{};
    a.g = g; a.nw = nw; a.n = m; a.h2 = h2; a.out = out + i0 * EMB; a.norm = norm + i0;
    if ((rc = net_l3(ctx, a))) return rc;
  }
  iq_timer_stop(ctx, "lp.encode");
  return IQ_OK;
}

}  // namespace

bool iq_lp_int_cells(const IqValueStats& s, Dim3 tile) {
  // integers whose squares summed over a tile stay below 2^24 (and the tile's voxels too)
  const double T = (double)tile.vol(), m = std::max(1.0, (double)s.amax);
  return s.narrow && s.lsbexp >= 0 && T * m * m < 16777216.0;
}

int iq_lp_int_integral(iq_ctx* ctx, const double* ii, int64_t n, int* out) {
  net_int_ii_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, ctx->stream>>>(ii, n, out);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int iq_lp_encode_windows(iq_ctx* ctx, const LpGeo& g, const float* w, const LpWindows& W,
                         const int* lo, const int* hi, __nv_bfloat16* out, float* norm,
                         const int64_t* pos, int64_t npos) {
  NetSrc s{};
  s.ii1 = W.ii1; s.ii2 = W.ii2; s.iq1 = W.iq1; s.iq2 = W.iq2;
  s.isx = W.img.x + 1; s.isxy = (W.img.x + 1) * (W.img.y + 1);
  s.dx = W.dist.x; s.dxy = W.dist.x * W.dist.y;
  s.pos = pos;
  for (int d = 0; d < 3; ++d) { s.lo[d] = lo[d]; s.hi[d] = hi[d]; }
  return net_encode(ctx, g, w, s, pos ? npos : W.dist.vol(), out, norm);
}

int iq_lp_encode_templates(iq_ctx* ctx, const LpGeo& g, const float* w, const float* grid,
                           Dim3 gdims, const int64_t* tsrc, const int* tbox, int64_t n, bool ints,
                           __nv_bfloat16* out, float* norm) {
  if (n <= 0) return IQ_OK;
  NetSrc s{};
  s.grid = grid; s.tsrc = tsrc; s.gx = gdims.x; s.gxy = gdims.x * gdims.y; s.tbox = tbox;
  s.tint = ints ? 1 : 0;
  return net_encode(ctx, g, w, s, n, out, norm);
}

int iq_lp_train_batch(iq_ctx* ctx, const LpGeo& g, const LpTrainBatch& B, double* loss_out) {
  const int64_t n = (int64_t)B.nA * (2 + B.nneg);
  const int nsm = iq_sm_count();
  cudaStream_t st = ctx->stream;
  float* nw = nullptr;
  int rc = net_prep(ctx, g, B.w, 0, &nw);
  if (rc) return rc;
  const int64_t G2 = g.ng2, nf = g.nf;
  float* h2 = (float*)iq_scratch(ctx, S_LP_BH2, sizeof(float) * n * (G2 * CH + nf) * 2);
  const int nw4 = (int)std::min<int64_t>((n + W4_IPB - 1) / W4_IPB, nsm), nwg = (int)std::min<int64_t>(n, nsm),
            nb2 = (int)std::min<int64_t>((n + 3) / 4, nsm);
  float* part = (float*)iq_scratch(ctx, S_LP_BH1, sizeof(float) * ((size_t)2 * nwg * WG_PART +
                                                                  (size_t)nw4 * W4_PART + (size_t)nb2 * CH * 4));
  if (!h2 || !part) return IQ_ERR_ALLOC;
  float* gz2 = h2 + n * G2 * CH;
  float* h3 = gz2 + n * G2 * CH;
  float* gz3 = h3 + n * nf;
  NetSrc s{};
  s.ii1 = B.win.ii1; s.ii2 = B.win.ii2; s.iq1 = B.win.iq1; s.iq2 = B.win.iq2;
  s.isx = B.win.img.x + 1; s.isxy = (B.win.img.x + 1) * (B.win.img.y + 1);
  s.dx = B.win.dist.x; s.dxy = B.win.dist.x * B.win.dist.y;
  s.items = static_cast<const TrainItem*>(B.items); s.feats = B.feats; s.boxes = B.boxes;
  if ((rc = net_l2(ctx, g, s, nw, n, B.X, h2))) return rc;
  L3Args a3{};
  a3.g = g; a3.nw = nw; a3.n = n; a3.h2 = h2; a3.h3 = h3; a3.E = B.E;
  if ((rc = net_l3(ctx, a3))) return rc;
  IQ_CUDA_OK(cudaMemsetAsync(B.loss, 0, sizeof(double), st));
  lp_loss_kernel<<<(unsigned)((B.nA + 7) / 8), 256, 0, st>>>(B.E, B.nA, B.nneg, B.temp, B.gE, B.loss);
  IQ_CUDA_OK(cudaGetLastError());
  B3Args b3{};
  b3.g = g; b3.w = B.w; b3.nw = nw; b3.n = n; b3.gE = B.gE; b3.h3 = h3; b3.h2 = h2; b3.gz3 = gz3; b3.gz2 = gz2;
  IQ_CUDA_OK(cudaFuncSetAttribute(net_b3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B3_SMEM));
  net_b3_kernel<<<(unsigned)std::min<int64_t>((n + B3_IPB - 1) / B3_IPB, nsm), NT, B3_SMEM, st>>>(b3);
  IQ_CUDA_OK(cudaGetLastError());
  float* p2 = part;
  float* p3 = p2 + (size_t)nwg * WG_PART;
  float* p4 = p3 + (size_t)nwg * WG_PART;
  float* p1 = p4 + (size_t)nw4 * W4_PART;
  B2Args b2{};
  b2.g = g; b2.nw = nw; b2.n = n; b2.X = B.X; b2.gz2 = gz2; b2.part = p1;
  IQ_CUDA_OK(cudaFuncSetAttribute(net_b2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B2_SMEM));
  net_b2_kernel<<<nb2, NT, B2_SMEM, st>>>(b2);
  IQ_CUDA_OK(cudaGetLastError());
  WgArgs wg{};
  wg.g = g; wg.nw = nw; wg.n = n; wg.hin = B.X; wg.gz = gz2; wg.part = p2;
  IQ_CUDA_OK(cudaFuncSetAttribute(net_wgrad_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wg_smem(2)));
  net_wgrad_kernel<2><<<nwg, WG_NT, wg_smem(2), st>>>(wg);
  wg.hin = h2; wg.gz = gz3; wg.part = p3;
  net_wgrad_kernel<3><<<nwg, WG_NT, wg_smem(3), st>>>(wg);
  IQ_CUDA_OK(cudaGetLastError());
  W4Args w4{};
  w4.g = g; w4.n = n; w4.gE = B.gE; w4.h3 = h3; w4.part = p4;
  net_w4_kernel<<<nw4, NT, 0, st>>>(w4);
  RedArgs r{};
  r.g = g; r.p1 = p1; r.p2 = p2; r.p3 = p3; r.p4 = p4; r.n1 = nb2; r.n2 = nwg; r.n3 = nwg; r.n4 = nw4;
  r.grad = B.grad;
  net_reduce_kernel<<<(2 * WG_PART + EMB * (int)nf + EMB + CH * 4 + 255) / 256, 256, 0, st>>>(r);
  IQ_CUDA_OK(cudaGetLastError());
  iq_count(ctx, 7);
  if (loss_out) {
    IQ_CUDA_OK(cudaMemcpyAsync(loss_out, B.loss, sizeof(double), cudaMemcpyDeviceToHost, st));
    IQ_CUDA_OK(cudaStreamSynchronize(st));
  }
  return IQ_OK;
}

int iq_lp_adam(iq_ctx* ctx, float* p, const float* g, float* m, float* v, int n, float lr, int step) {
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)step), c2 = 1.f - std::pow(b2, (float)step);
  lp_adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(p, g, m, v, n, lr, b1, b2, 1e-8f, c1, c2);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}
