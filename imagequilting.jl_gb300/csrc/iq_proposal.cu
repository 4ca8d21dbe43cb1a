// Learned proposal: a shortlist of training-image positions per (tile, realization) from a
// small 3-D convolutional encoder, so that the exact distance is evaluated only there instead
// of at every position. No counterpart in the reference, whose tile loop scans every position
// (src/iqsim.jl:206, src/utils.jl:5-13); the full scan stays the fallback and the judge of the
// shortlist's recall.
//
// Encoder (the same for a tile's masked overlap region and for a training-image window under
// the same mask; weights BF16 for inference, FP32 while training, FP32 accumulation):
//   cells    grid G = (min(tx, 8), min(ty, 8), min(tz, 4)) of cells of c = ceil(t / G) voxels;
//            per cell: mask fraction, masked sum of values / volume, masked sum of squares /
//            volume (windows: Float64 integral images of the image and of its squares;
//            templates: direct sums over the simulation grid)
//   layer 1  1x1x1 convolution 3 -> 32, bias, ReLU
//   layer 2  3x3x3 convolution 32 -> 32, stride 2, padding 1, bias, ReLU
//   layer 3  3x3x3 convolution 32 -> 32, stride 2, padding 1, bias, ReLU
//   output   linear (32 x cells of layer 3) -> 64, bias
// Training (InfoNCE on squared embedding distances, anchors = templates, positives = their exact
// candidates, negatives = random windows) runs in FP32 through hand-written forward and
// backward kernels and an Adam step.
//
// Shortlist of one column (template embedding e): every position's window embedding w_p
// (cached per training image and mask) is scored s_p = |e - w_p|^2 as a GEMM on the tensor
// cores (BF16 inputs, FP32 accumulation); a per-column threshold taken from a sample of the
// positions keeps about `k` of them. The exact distance is then summed directly at the
// shortlisted positions and the pick of src/iqsim.jl:236-246 runs on them.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "iq_proposal_cells.cuh"

namespace {

constexpr int EMB = IQ_LP_EMB;
constexpr int NIN = 3;
constexpr int LT = 256;  // threads of the template feature kernel

}  // namespace

// =============================================================================================
// Shortlist: sampled per-column threshold, then a tensor-core scan of every position
// =============================================================================================
namespace {

__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Scores of every position against every column with tensor-core MMAs (mma.sync m16n8k16, BF16
// in, FP32 accumulation): s = |w|^2 + |e|^2 - 2 w.e. The columns are staged in shared memory in chunks
// of LP_SCAN_COLS (rows padded to 36 words, conflict-free fragment loads); a warp keeps the A
// fragments of its 16 positions in registers and sweeps the chunk's columns, so the window embeddings
// are read once per chunk.
// Scan: the positions with s <= tau[col] leave as bits, four ballots per 16 positions x 8 columns;
// lp_list_kernel turns a column's bits into its list, ascending. (Appending each hit with a global
// atomic took 0.35 ms of a launch's 0.39 on a 0.46 M-position image with 55 columns: 16,384 adds to
// one address per column.)
// DENSE: every score is written to dense[col * P + row] instead (the sampled rows).
constexpr int LP_SCAN_COLS = 512;
constexpr int LP_SCAN_LD = 36;  // words per staged column (32 + 4 of padding)

constexpr int LP_SCAN_THREADS = 512;  // 16 warps: two CTAs fill half an SM's warp slots

template <bool DENSE>
__global__ void __launch_bounds__(LP_SCAN_THREADS) lp_scan_kernel(const __nv_bfloat16* __restrict__ W,
                                                      const float* __restrict__ nW, int64_t P,
                                                      const __nv_bfloat16* __restrict__ T,
                                                      const float* __restrict__ nT,
                                                      const float* __restrict__ tau, int N,
                                                      uint4* __restrict__ bits, float* dense) {
  extern __shared__ __align__(16) uint32_t sT[];
  float* sN = reinterpret_cast<float*>(sT + LP_SCAN_COLS * LP_SCAN_LD);
  float* sTau = sN + LP_SCAN_COLS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const uint32_t* T32 = reinterpret_cast<const uint32_t*>(T);
  const int64_t nblk = (P + 15) / 16;
  for (int c0 = 0; c0 < N; c0 += LP_SCAN_COLS) {
    const int nc = min(LP_SCAN_COLS, N - c0);
    __syncthreads();  // the previous chunk's readers are done
    for (int i = threadIdx.x; i < nc * 32; i += blockDim.x)
      sT[(i >> 5) * LP_SCAN_LD + (i & 31)] = T32[(int64_t)(c0 + (i >> 5)) * 32 + (i & 31)];
    // scan: |w|^2 - 2 w.e <= tau - |e|^2 (one FMA and a compare per pair)
    for (int i = threadIdx.x; i < nc; i += blockDim.x) {
      sN[i] = nT[c0 + i];
      sTau[i] = DENSE ? 0.f : tau[c0 + i] - nT[c0 + i];
    }
    __syncthreads();
    const int nw = blockDim.x >> 5;
    for (int64_t blk = (int64_t)blockIdx.x * nw + warp; blk < nblk; blk += (int64_t)gridDim.x * nw) {
      const int64_t p0 = blk * 16;
      const int64_t r0 = p0 + gid, r1 = p0 + gid + 8;
      const int64_t q0 = r0 < P ? r0 : P - 1, q1 = r1 < P ? r1 : P - 1;
      uint32_t af[4][4];
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const uint32_t* x0 = reinterpret_cast<const uint32_t*>(W + q0 * EMB + ks * 16 + 2 * tig);
        const uint32_t* x1 = reinterpret_cast<const uint32_t*>(W + q1 * EMB + ks * 16 + 2 * tig);
        af[ks][0] = x0[0];
        af[ks][1] = x1[0];
        af[ks][2] = x0[4];
        af[ks][3] = x1[4];
      }
      const float w0 = nW[q0], w1 = nW[q1];
      for (int cb = 0; cb < nc; cb += 64) {
#pragma unroll 2
        for (int nt = 0; nt < 8; ++nt) {
          const int cl = cb + nt * 8 + gid;
          // word ks * 8 + tig holds dims ks * 16 + 2 tig, +1 (b0); +4 words: dims + 8 (b1)
          const uint32_t* src = sT + (cl < nc ? cl : 0) * LP_SCAN_LD + tig;
          float acc[4] = {0.f, 0.f, 0.f, 0.f};
          unsigned hit[4];
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint32_t b0 = cl < nc ? src[ks * 8] : 0u, b1 = cl < nc ? src[ks * 8 + 4] : 0u;
            mma_bf16(acc, af[ks], b0, b1);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int cc = cb + nt * 8 + 2 * tig + (e & 1);  // column within the chunk
            const int64_t row = e < 2 ? r0 : r1;
            const bool in = cc < nc && row < P;
            if (DENSE) {
              if (in) dense[(int64_t)(c0 + cc) * P + row] = (e < 2 ? w0 : w1) + sN[cc] - 2.f * acc[e];
            } else {
              hit[e] = __ballot_sync(0xffffffffu, in && fmaf(-2.f, acc[e], e < 2 ? w0 : w1) <= sTau[cc]);
            }
          }
          // word e: bit 4 g + t is row g (e < 2) or g + 8, column 2 t + (e & 1) of the tile
          if (!DENSE && lane == 0 && cb + nt * 8 < nc)
            bits[(int64_t)((c0 + cb) / 8 + nt) * nblk + blk] = make_uint4(hit[0], hit[1], hit[2], hit[3]);
        }
      }
    }
  }
}

// The lists from the scan's bits: a column's positions in ascending order (the first `cap`), and
// their count. A CTA takes the eight columns that share a word over one slice of the blocks of 16
// positions, a thread four blocks at a time (four loads in flight). COUNT: the slice's counts only,
// which the slices after it start from. A chain of scans and barriers bounds a CTA, so the blocks are
// cut into as many slices as fill the chip (one slice, without the counting pass, where one pass of
// a CTA covers the image). One CTA per column over all blocks, each reading its eight columns' words:
// scan and lists 1.23 ms a launch over 5.7 M positions (185 columns), with slices 0.98; calls on
// 0.46 M positions 89.5 -> 87.7 ms.
constexpr int LL_NT = 512, LL_BLK = 4;

template <bool COUNT>
__global__ void __launch_bounds__(LL_NT) lp_list_kernel(const uint4* __restrict__ bits, int64_t nblk,
                                                        int64_t per, int N, int* counts, int32_t* list,
                                                        int32_t* cnt, int cap) {
  __shared__ unsigned long long wsum[2][LL_NT / 32];
  const int grp = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint4* src = bits + (int64_t)grp * nblk;
  const int64_t lo = blockIdx.y * per, hi = min(lo + per, nblk);
  int base[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (!COUNT)
    for (unsigned s = 0; s < blockIdx.y; ++s) {
      const int4* q = reinterpret_cast<const int4*>(counts + ((int64_t)s * gridDim.x + grp) * 8);
      const int4 x = q[0], y = q[1];
      base[0] += x.x; base[1] += x.y; base[2] += x.z; base[3] += x.w;
      base[4] += y.x; base[5] += y.y; base[6] += y.z; base[7] += y.w;
    }
  for (int64_t b0 = lo; b0 < hi; b0 += LL_NT * LL_BLK) {
    const int64_t b = b0 + (int64_t)threadIdx.x * LL_BLK;
    uint4 w[LL_BLK];
#pragma unroll
    for (int k = 0; k < LL_BLK; ++k) w[k] = b + k < hi ? src[b + k] : make_uint4(0u, 0u, 0u, 0u);
    // column j's rows are bits 4 g + j / 2 of words x, z (j even) or y, w (j odd); its count is the
    // 16-bit field j % 4 of c[j / 4] (a CTA's 2,048 blocks hold 32,768 positions)
    unsigned long long c[2] = {0ull, 0ull}, inc[2], tot[2];
#pragma unroll
    for (int k = 0; k < LL_BLK; ++k) {
      if (!(w[k].x | w[k].y | w[k].z | w[k].w)) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const unsigned m0 = ((j & 1 ? w[k].y : w[k].x) >> (j >> 1)) & 0x11111111u;
        const unsigned m1 = ((j & 1 ? w[k].w : w[k].z) >> (j >> 1)) & 0x11111111u;
        c[j >> 2] += (unsigned long long)(__popc(m0) + __popc(m1)) << (16 * (j & 3));
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      inc[q] = c[q];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, inc[q], o);
        if (lane >= o) inc[q] += y;
      }
      if (lane == 31) wsum[q][warp] = inc[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const unsigned long long ws = lane < LL_NT / 32 ? wsum[q][lane] : 0ull;
      unsigned long long wi = ws;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += y;
      }
      inc[q] += __shfl_sync(0xffffffffu, wi - ws, warp) - c[q];
      tot[q] = __shfl_sync(0xffffffffu, wi, 31);
    }
    if (!COUNT && (c[0] | c[1])) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (!(c[j >> 2] >> (16 * (j & 3)) & 0xFFFFu)) continue;  // (columns >= N have no bits)
        int at = base[j] + (int)(inc[j >> 2] >> (16 * (j & 3)) & 0xFFFFu);
        int32_t* out = list + (int64_t)(grp * 8 + j) * cap;
#pragma unroll
        for (int k = 0; k < 2 * LL_BLK; ++k) {
          const uint4 v = w[k >> 1];
          const unsigned word = k & 1 ? (j & 1 ? v.w : v.z) : (j & 1 ? v.y : v.x);
          for (unsigned m = (word >> (j >> 1)) & 0x11111111u; m; m &= m - 1, ++at)
            if (at < cap) out[at] = (int32_t)(b * 16 + 8 * k + ((__ffs(m) - 1) >> 2));
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) base[j] += (int)(tot[j >> 2] >> (16 * (j & 3)) & 0xFFFFu);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (COUNT) counts[((int64_t)blockIdx.y * gridDim.x + grp) * 8 + j] = base[j];
      else if (blockIdx.y == gridDim.y - 1 && grp * 8 + j < N) cnt[grp * 8 + j] = base[j];
    }
  }
}

// Rows i * stride of the window embeddings (the positions the per-column thresholds sample).
__global__ void lp_sample_rows_kernel(const __nv_bfloat16* __restrict__ W, const float* __restrict__ nW,
                                      int64_t P, int64_t stride, int S, __nv_bfloat16* Ws,
                                      float* nWs) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)S * EMB) return;
  const int64_t row = i / EMB, d = i - row * EMB;
  const int64_t p = row * stride;
  Ws[i] = p < P ? W[p * EMB + d] : __float2bfloat16_rn(0.f);
  if (d == 0) nWs[row] = p < P ? nW[p] : 3.0e38f;
}

// The m-th smallest of each column's S = IQ_LP_SAMPLES sampled scores, one CTA per column: the scores
// stay in registers as order-preserving keys, and the largest v with fewer than m keys below it is
// found a bit at a time (32 counts over the CTA; a radix select's histogram had all keys in a few of
// its bins).
constexpr int SEL_NT = 256;

__global__ void __launch_bounds__(SEL_NT) lp_select_kernel(const float* __restrict__ dense, int m,
                                                           float* tau) {
  __shared__ int wcnt[2][SEL_NT / 32];
  const float* x = dense + (int64_t)blockIdx.x * IQ_LP_SAMPLES;
  unsigned key[IQ_LP_SAMPLES / SEL_NT];
#pragma unroll
  for (int i = 0; i < IQ_LP_SAMPLES / SEL_NT; ++i) {
    const unsigned b = __float_as_uint(x[i * SEL_NT + threadIdx.x]);
    key[i] = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  }
  unsigned v = 0;
  for (int bit = 31; bit >= 0; --bit) {
    const unsigned t = v | (1u << bit);
    int c = 0;
#pragma unroll
    for (int i = 0; i < IQ_LP_SAMPLES / SEL_NT; ++i) c += key[i] < t ? 1 : 0;
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) wcnt[bit & 1][threadIdx.x >> 5] = c;
    __syncthreads();
    c = 0;
#pragma unroll
    for (int w = 0; w < SEL_NT / 32; ++w) c += wcnt[bit & 1][w];
    if (c < m) v = t;
  }
  if (threadIdx.x == 0) tau[blockIdx.x] = __uint_as_float((v & 0x80000000u) ? (v & 0x7FFFFFFFu) : ~v);
}

__global__ void lp_template_features_kernel(LpGeo g, const float* grid, const int64_t* tsrc,
                                            const int* tbox, int64_t gx, int64_t gxy, int64_t n,
                                            float* out) {
  for (int64_t item = blockIdx.x; item < n; item += gridDim.x) {
    int lo[3], hi[3];
    for (int d = 0; d < 3; ++d) { lo[d] = tbox[6 * item + d]; hi[d] = tbox[6 * item + 3 + d]; }
    for (int cell = threadIdx.x; cell < g.ng; cell += blockDim.x) {
      float f[3];
      template_cell<false>(g, grid + tsrc[item], gx, gxy, lo, hi, cell, f);
      for (int c = 0; c < NIN; ++c) out[item * NIN * g.ng + c * g.ng + cell] = f[c];
    }
  }
}

// Exact distance (byte-valued image, integer sums) of one column at every position, and its
// minimum (the monitor). A column whose template values are not bytes leaves dmin at +Inf.
__global__ void __launch_bounds__(256) lp_full_kernel(const LpImg im, int64_t dx, int64_t dxy,
                                                      int64_t P, LpColumn col, float* D,
                                                      unsigned* dmin) {
  extern __shared__ __align__(16) unsigned char dyn[];
  uint4* qd = reinterpret_cast<uint4*>(dyn);
  const int nst = iq_stage(im, col, qd);
  if (nst < 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned mn = 0x7F800000u;
  for (int64_t p0 = ((int64_t)blockIdx.x * 8 + warp) * 32; p0 < P; p0 += (int64_t)gridDim.x * 8 * 32) {
    const uint2 o = iq_lp_origin(im, (uint32_t)min(p0 + lane, P - 1), (uint32_t)dx, (uint32_t)dxy);
    const int m = (int)min((int64_t)32, P - p0);
    float mine = 0.f;
    for (int e = 0; e < m; ++e) {
      const uint2 oe = make_uint2(__shfl_sync(0xffffffffu, o.x, e), __shfl_sync(0xffffffffu, o.y, e));
      const float acc = (float)iq_lp_ssd(im, qd, nst, oe, [] { return INFINITY; });
      if (lane == e) mine = acc;
      mn = min(mn, __float_as_uint(acc));
    }
    if (lane < m) D[p0 + lane] = mine;
  }
  if (lane == 0) atomicMin(dmin, mn);
}

__global__ void lp_mark_kernel(const int32_t* list, const int32_t* cnt, int cap, uint32_t* bits) {
  const int n = min(*cnt, cap);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    atomicOr(bits + (list[i] >> 5), 1u << (list[i] & 31));
}

// counters[0] += |{D <= (1 + tol) min D}|, counters[1] += those in the shortlist
__global__ void lp_recall_kernel(const float* D, const unsigned* dmin, int64_t P, double tol,
                                 const uint32_t* bits, unsigned long long* counters) {
  if (*dmin >= 0x7F800000u) return;  // the column was not evaluated
  const float thr = f_dn(__dmul_rn(__dadd_rn(1.0, tol), (double)__uint_as_float(*dmin)));
  unsigned long long t = 0, h = 0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < P;
       p += (int64_t)gridDim.x * blockDim.x) {
    if (D[p] <= thr) {
      t++;
      if (bits[p >> 5] >> (p & 31) & 1u) h++;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    t += __shfl_xor_sync(0xffffffffu, t, o);
    h += __shfl_xor_sync(0xffffffffu, h, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counters, t);
    atomicAdd(counters + 1, h);
  }
}

}  // namespace

namespace {
// The image as bytes; *bad = 1 when a value is not an integer in [0, 255].
__global__ void lp_to_u8_kernel(const float* __restrict__ src, int64_t n, uint8_t* dst, int* bad) {
  int b = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float v = src[i];
    const bool ok = v >= 0.f && v <= 255.f && v == floorf(v);
    dst[i] = ok ? (uint8_t)v : 0;
    b |= !ok;
  }
  if (__syncthreads_or(b) && threadIdx.x == 0) atomicOr(bad, 1);
}
}  // namespace

namespace {
// Plane form of an image of codes 0..3 (see LpImg); *bad = 1 for any other value.
__global__ void lp_to_planes_kernel(const float* __restrict__ src, Dim3 d, int64_t ntx, uint4* dst,
                                    int* bad) {
  const int64_t nw = d.z * ntx * d.y;
  int b = 0;
  for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < nw;
       w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t y = w % d.y, t = w / d.y, tx = t % ntx, z = t / ntx;
    uint32_t p0[2] = {0, 0}, p1[2] = {0, 0};
#pragma unroll
    for (int k = 0; k < 2; ++k)
      for (int i = 0; i < 32; ++i) {
        const int64_t x = (tx + k) * 32 + i;
        if (x >= d.x) break;
        const float v = src[x + d.x * y + d.x * d.y * z];
        if (!(v == 0.f || v == 1.f || v == 2.f || v == 3.f)) b = 1;
        const uint32_t c = (uint32_t)v & 3u;
        p0[k] |= (c & 1u) << i;
        p1[k] |= (c >> 1) << i;
      }
    dst[w] = make_uint4(p0[0], p0[1], p1[0], p1[1]);
  }
  if (__syncthreads_or(b) && threadIdx.x == 0) atomicOr(bad, 1);
}
}  // namespace

int iq_lp_to_planes(iq_ctx* ctx, const float* src, Dim3 d, int64_t ntx, uint4* dst, int* bad) {
  IQ_CUDA_OK(cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
  const int64_t nw = d.z * ntx * d.y;
  lp_to_planes_kernel<<<(unsigned)std::min<int64_t>((nw + 255) / 256, 4096), 256, 0, ctx->stream>>>(
      src, d, ntx, dst, bad);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int iq_lp_to_u8(iq_ctx* ctx, const float* src, int64_t n, uint8_t* dst, int* bad) {
  IQ_CUDA_OK(cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
  IQ_CUDA_OK(cudaMemsetAsync(dst + n, 0, 16, ctx->stream));
  lp_to_u8_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, ctx->stream>>>(
      src, n, dst, bad);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int iq_lp_sample_rows(iq_ctx* ctx, const __nv_bfloat16* W, const float* nW, int64_t P,
                      __nv_bfloat16* Ws, float* nWs) {
  const int64_t stride = (P + IQ_LP_SAMPLES - 1) / IQ_LP_SAMPLES;
  const int64_t n = (int64_t)IQ_LP_SAMPLES * EMB;
  lp_sample_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(W, nW, P, stride,
                                                                            IQ_LP_SAMPLES, Ws, nWs);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int iq_lp_shortlist(iq_ctx* ctx, const __nv_bfloat16* W, const float* nW, int64_t P,
                    const __nv_bfloat16* Ws, const float* nWs, const __nv_bfloat16* T,
                    const float* nT, int N, int64_t k, float* tau, float* dense, int32_t* list,
                    int32_t* cnt, int cap) {
  if (N <= 0) return IQ_OK;
  const int64_t nblk = (P + 15) / 16;
  // slices of the lists: four CTAs per SM, each at least one pass of its threads
  const int nsm = iq_sm_count();
  const int64_t grps = (N + 7) / 8, npass = (nblk + LL_NT * LL_BLK - 1) / (LL_NT * LL_BLK);
  const int64_t want = std::max<int64_t>(1, std::min<int64_t>(npass, 4 * nsm / grps));
  const int64_t per = (npass + want - 1) / want * (LL_NT * LL_BLK), slices = (nblk + per - 1) / per;
  uint4* bits = (uint4*)iq_scratch(ctx, S_LP_BITS2, sizeof(uint4) * (size_t)grps * nblk +
                                                        sizeof(int) * 8 * (size_t)(grps * slices));
  if (!bits) return IQ_ERR_ALLOC;
  int* counts = (int*)(bits + grps * nblk);
  const int S = IQ_LP_SAMPLES;
  const int64_t stride = (P + S - 1) / S;
  // the m-th smallest sampled score stands for about m * stride positions
  const int m = (int)std::max<int64_t>(4, std::min<int64_t>(S, (k + stride - 1) / stride));
  cudaStream_t st = ctx->stream;
  iq_timer_start(ctx, "lp.scan");
  // per-column thresholds: the sampled rows' scores as one GEMM, then a select per column
  const size_t sm = sizeof(uint32_t) * LP_SCAN_COLS * LP_SCAN_LD + 2 * sizeof(float) * LP_SCAN_COLS;
  IQ_CUDA_OK(cudaFuncSetAttribute(lp_scan_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  IQ_CUDA_OK(cudaFuncSetAttribute(lp_scan_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  lp_scan_kernel<true><<<(unsigned)((S / 16 + 15) / 16), LP_SCAN_THREADS, sm, st>>>(
      Ws, nWs, S, T, nT, nullptr, N, nullptr, dense);
  lp_select_kernel<<<(unsigned)N, SEL_NT, 0, st>>>(dense, m, tau);
  IQ_CUDA_OK(cudaGetLastError());
  const int64_t gx = std::max<int64_t>(1, std::min<int64_t>((nblk + 15) / 16, (int64_t)nsm * 2));
  lp_scan_kernel<false><<<(unsigned)gx, LP_SCAN_THREADS, sm, st>>>(W, nW, P, T, nT, tau, N, bits,
                                                                   nullptr);
  const dim3 lgrid((unsigned)grps, (unsigned)slices);
  if (slices > 1)
    lp_list_kernel<true><<<lgrid, LL_NT, 0, st>>>(bits, nblk, per, N, counts, list, cnt, cap);
  lp_list_kernel<false><<<lgrid, LL_NT, 0, st>>>(bits, nblk, per, N, counts, list, cnt, cap);
  iq_timer_stop(ctx, "lp.scan", 2.0 * (double)(P + S) * N * EMB);
  iq_count(ctx, slices > 1 ? 5 : 4);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int iq_lp_template_features(iq_ctx* ctx, const LpGeo& g, const float* grid, Dim3 gdims,
                            const int64_t* tsrc, const int* tbox, int64_t n, float* out) {
  if (n <= 0) return IQ_OK;
  lp_template_features_kernel<<<(unsigned)std::min<int64_t>(n, 4096), LT, 0, ctx->stream>>>(
      g, grid, tsrc, tbox, gdims.x, gdims.x * gdims.y, n, out);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int iq_lp_recall(iq_ctx* ctx, const LpImg& im, Dim3 dist, const LpColumn& col,
                 const int32_t* list, const int32_t* cnt, int cap, double tol, float* Dbuf,
                 unsigned* dmin, uint32_t* bits, unsigned long long* counters) {
  const int64_t P = dist.vol();
  const size_t sm = (size_t)16 * (im.p2 ? (size_t)col.tdim[1] * col.tdim[2] : (size_t)col.nq) + 16;
  if (sm > 227 * 1024) return iq_set_error(IQ_ERR_LIMIT, "recall check: mask too large");
  IQ_CUDA_OK(cudaFuncSetAttribute(lp_full_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  const unsigned inf = 0x7F800000u;
  IQ_CUDA_OK(cudaMemcpyAsync(dmin, &inf, sizeof(unsigned), cudaMemcpyHostToDevice, ctx->stream));
  IQ_CUDA_OK(cudaMemsetAsync(bits, 0, sizeof(uint32_t) * ((P + 31) / 32), ctx->stream));
  iq_timer_start(ctx, "lp.monitor");
  lp_full_kernel<<<(unsigned)std::min<int64_t>((P + 255) / 256, 8 * iq_sm_count()), 256, sm, ctx->stream>>>(
      im, dist.x, dist.x * dist.y, P, col, Dbuf, dmin);
  lp_mark_kernel<<<64, 256, 0, ctx->stream>>>(list, cnt, cap, bits);
  lp_recall_kernel<<<(unsigned)std::min<int64_t>((P + 255) / 256, 1024), 256, 0, ctx->stream>>>(
      Dbuf, dmin, P, tol, bits, counters);
  iq_timer_stop(ctx, "lp.monitor");
  iq_count(ctx, 3);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}
