// Tensor-core distance maps of many templates with the Toeplitz structure on the template side
// (tcgen05, sm_103a): the same maps as iq_corr_tc.cu,
//   D[n][p] = |A2(p) - 2 AB[n][p] + B2[n]|     (src/utils.jl:5-13, src/imfilter.jl:5-28),
// for masks "tile minus a box" and operands that FP16 halves represent.
//
// What bounds a masked correlation on this part is not the MMA itself but feeding it: as a GEMM
// over positions the image operand is a Hankel matrix, eight 16-byte rows per eight values, and
// with the few dozen templates of a dependency level each MMA reads 4 KB of it for little work
// (iq_corr_tc.cu: 119 TFLOP/s issued at 16-64 columns, its one issuing thread and its image
// builders busy throughout). Here eight consecutive positions p = base + 8 i + s (s = 0..7) are
// one GEMM row i, and the shift s moves to the template:
//   AB[n][base + 8 i + s] = sum_k' A[i][k'] B[8 n + s][k'],
//   A[i][k'] = TI[base + 8 i + k' + row],  B[8 n + s][k'] = tmpl_n[k' - s] (0 outside the mask).
// A is then the plain FP16 image: the core matrix of rows 8 q.. and offsets 8 j.. is the 128
// contiguous bytes at 16 (8 q + j), so a descriptor with leading offset 16 * (chunk distance)
// and stride offset 128 reads it, and one bulk copy per (ky, kz) row of the mask stages it with
// no conversion and no redundancy. B is the template packed once per launch with its eight
// shifts (tz_pack_kernel); its columns fill N = 8 x templates. The price is 7 extra offsets per
// row: a row of w offsets takes ceil((w + 7) / 8) chunks of 8.
// Measured, correlation time of whole simulations before (iq_corr_tc.cu) and after: image
// 256 x 256 x 128 of 4 codes, tile 32 x 32 x 16, 752 columns: 751 -> 98 ms (1330 TFLOP/s of issued
// FP16 MMA work, the measured cuBLAS peak is 1901); 128 x 128 x 64, 1720 columns: 184 -> 30 ms;
// continuous (SPLIT) 91 x 83 x 47, tile 21 x 19 x 11, 1257 columns: 33.7 -> 13.2 ms.
//
//   M   128 rows = 1024 consecutive linear positions per accumulator, MB accumulators per CTA;
//       x rows of the image are padded to a multiple of 8 values, so that every row offset is a
//       16-byte one; positions past the valid extents are computed and dropped
//   N   8 x the columns of a group (at most 32 templates, even)
//   K   the 8-offset chunks of the union of the group's masks, two per K-step of 16
//
// EXACT (values of at most 11 significant bits): one MMA per K-step, the sums exact. SPLIT:
// v = hi + lo in FP16 halves; hi * hi accumulates in one set of TMEM columns, hi * lo + lo * hi in
// another, added once at the end, so the FP32 accumulator of the large terms takes one rounding
// per K-step instead of three.
//
// Pipeline: warp 0 (one lane) waits for a free stage and issues its bulk copies (image rows,
// packed templates, the stage's 64-byte step table), warp 1 (one lane) waits for them, issues the
// stage's MMAs and commits them to the stage's "done" barrier. All 8 warps run the epilogue:
// TMEM -> a 1 KB transpose per warp and column -> coalesced stores of |A2 + B2 - 2 AB| with the
// column's minimum and largest finite value. A2 comes from maps made once per call
// (iq_tz_a2_maps; +Inf at disabled windows). Every wait is bounded (iq_tcgen05.cuh); on expiry the
// kernel records IQ_ERR_TIMEOUT, stops issuing, waits for its copies, frees its TMEM, returns.
#include <float.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "iq_tcgen05.cuh"

namespace {

constexpr int TZ_THREADS = 256;
constexpr int TZ_MAXST = 4;    // most pipeline stages
constexpr int TZ_MAXCH = 8;    // chunks a row entry spans

struct TzArgs {
  const __half* hi;          // padded image, high halves (pitch ixp, planes of ixp * iy)
  const __half* lo;          // low halves (SPLIT)
  int64_t ixp, plane;        // padded row pitch, padded plane
  int64_t dx, dy, dz;        // valid extents
  int64_t run, nrun;         // positions of one run (a plane, or the volume), number of runs
  int tiles;                 // CTAs per run
  int slot;                  // 16-byte units of one staged image row
  int nst;                   // pipeline stages
  uint32_t stage_bytes, b_off, t_off;  // stage layout: rows (hi, lo), packed templates, table
  int Nmax;
  uint32_t tmem_cols;
  const TzGroup* groups;
  const TzStage* stages;
  const char* B;
  const TcCol* cols;
  const float* a2;           // A2 maps, box b at a2 + b * P
  int64_t P;
  float ab2;
  int* status;
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&r)[16]) {
  uint32_t u[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]),
        "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]),
        "=r"(u[14]), "=r"(u[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) r[i] = __uint_as_float(u[i]);
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

// MB: accumulators (1024 positions each) per CTA.
template <bool SPLIT, int MB>
__global__ void __launch_bounds__(TZ_THREADS, 1) corr_tz_kernel(const TzArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t bars[2 * TZ_MAXST + 1];
  __shared__ float* s_out[IQ_TZ_COLS];
  __shared__ unsigned* s_mmp[IQ_TZ_COLS];
  __shared__ const float* s_a2[IQ_TZ_COLS];
  __shared__ float s_b2[IQ_TZ_COLS];
  __shared__ unsigned s_mn[IQ_TZ_COLS], s_mx[IQ_TZ_COLS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const TzGroup g = a.groups[blockIdx.y];
  const uint32_t bar_full = smem_u32(bars), bar_done = bar_full + 8 * TZ_MAXST,
                 bar_fin = bar_full + 16 * TZ_MAXST;
  if (tid < g.ncol) {
    const TcCol c = a.cols[g.col0 + tid];
    const bool live = c.src >= 0;
    s_out[tid] = live ? c.out : nullptr;
    s_mmp[tid] = live ? c.mm : nullptr;
    s_b2[tid] = (live && c.b2) ? (float)*c.b2 : 0.f;
    s_a2[tid] = a.a2 + (live ? (int64_t)c.box : 0) * a.P;
    s_mn[tid] = 0x7F800000u;
    s_mx[tid] = 0u;
  }
  if (tid == 0) {
    for (int i = 0; i < 2 * TZ_MAXST + 1; ++i) mbar_init(bar_full + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem)),
                 "r"(a.tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  const int N = g.N;
  const int64_t runi = blockIdx.x / a.tiles;
  const int64_t rel0 = (int64_t)(blockIdx.x - runi * a.tiles) * (1024 * MB);
  const int64_t p0 = runi * a.plane + rel0;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t rowlo = (uint32_t)(IQ_TZ_ROWS * a.slot) * 16u;  // low images of a stage (SPLIT)

  int fail = 0;
  if (warp == 0) {
    if (lane == 0) {
      // ---- copies ----
      int issued = 0;
      TzStage nx = g.nstage > 0 ? a.stages[g.stage0] : TzStage{};
      for (int e = 0; e < g.nstage; ++e) {
        const TzStage st = nx;
        if (e + 1 < g.nstage) nx = a.stages[g.stage0 + e + 1];
        const int b = e % a.nst, use = e / a.nst;
        if (use > 0 && !mbar_wait(bar_done + 8 * b, (uint32_t)(use - 1) & 1u)) { fail = 1; break; }
        const uint32_t sS = sbase + b * a.stage_bytes, bar = bar_full + 8 * b;
        const int nent = (int)(st.w[0] & 15u), nks = (int)((st.w[0] >> 8) & 15u);
        const uint32_t bbytes = (uint32_t)nks * 32u * (uint32_t)N;
        uint32_t total = 64u + bbytes * (SPLIT ? 2u : 1u);
        for (int i = 0; i < nent; ++i)
          total += (uint32_t)(128 * MB + ((st.w[7] >> (4 * i)) & 15u) - 1) * (SPLIT ? 32u : 16u);
        mbar_expect(bar, total);
        bulk_copy(sS + a.t_off, a.stages + g.stage0 + e, 64u, bar);
        for (int i = 0; i < nent; ++i) {
          const uint32_t bytes = (uint32_t)(128 * MB + ((st.w[7] >> (4 * i)) & 15u) - 1) * 16u;
          const int64_t src = p0 + 8 * (int64_t)st.w[2 + i];
          bulk_copy(sS + (uint32_t)(i * a.slot) * 16u, a.hi + src, bytes, bar);
          if (SPLIT) bulk_copy(sS + rowlo + (uint32_t)(i * a.slot) * 16u, a.lo + src, bytes, bar);
        }
        const char* B = a.B + g.boff + (int64_t)st.w[1] * 32 * N;
        bulk_copy(sS + a.b_off, B, bbytes, bar);
        if (SPLIT) bulk_copy(sS + a.b_off + bbytes, B + (int64_t)g.nstep * 32 * N, bbytes, bar);
        issued = e + 1;
      }
      // the last copies have landed (bounded waits) before the buffers go away
      for (int e = issued - 1; e >= 0 && e >= issued - a.nst; --e)
        mbar_wait(bar_full + 8 * (e % a.nst), (uint32_t)(e / a.nst) & 1u);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMAs ----
      const uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
      uint32_t acc = 0;
      for (int e = 0; e < g.nstage; ++e) {
        const int b = e % a.nst;
        if (!mbar_wait(bar_full + 8 * b, (uint32_t)(e / a.nst) & 1u)) { fail = 1; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sS = sbase + b * a.stage_bytes;
        const uint32_t* tab = reinterpret_cast<const uint32_t*>(smem + b * a.stage_bytes + a.t_off);
        const int nks = (int)((tab[0] >> 8) & 15u);
        const uint64_t dB = make_desc(sS + a.b_off, 16u * N, 128u);
#pragma unroll 1
        for (int t = 0; t < nks; ++t) {
          const uint32_t w = tab[8 + t];
          const uint32_t u0 = (w & 15u) * a.slot + ((w >> 4) & 15u);
          const uint32_t u1 = ((w >> 8) & 15u) * a.slot + ((w >> 12) & 15u);
          const uint64_t dA = make_desc(sS + 16u * u0, 16u * (u1 - u0), 128u);
          const uint64_t bh = dB + (uint64_t)(2u * N * t);
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) {
            mma_f16(tmem + (uint32_t)(mb * N * (SPLIT ? 2 : 1)), dA + 128u * mb, bh, idesc, acc);
            if (SPLIT) {
              const uint32_t d2 = tmem + (uint32_t)(mb * N * 2 + N);
              mma_f16(d2, dA + 128u * mb, bh + 2u * N * nks, idesc, acc);
              mma_f16(d2, dA + (rowlo >> 4) + 128u * mb, bh, idesc, 1u);
            }
          }
          acc = 1u;
        }
        mma_commit(bar_done + 8 * b);
      }
      if (g.nstage > 0) mma_commit(bar_fin);  // every MMA issued has completed
      else mbar_arrive(bar_fin);
    }
    __syncwarp();
  }
  if (!mbar_wait(bar_fin, 0)) fail = 1;
  const int aborted = __syncthreads_or(fail);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  if (!aborted) {
    // warp = (lane quadrant lq: 32 rows = 256 positions, half: even or odd pairs of columns)
    const int lq = warp & 3, half = warp >> 2;
    float* tr = reinterpret_cast<float*>(smem) + warp * 256;
#pragma unroll 1
    for (int mb = 0; mb < MB; ++mb) {
      // this lane's positions: j-th store instruction covers 32 consecutive ones
      int64_t po[8];
      const int64_t r0 = rel0 + 1024 * mb + 256 * lq + lane;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t r = (uint32_t)(r0 + 32 * j);  // a run has fewer than 2^31 positions
        const uint32_t zr = r / (uint32_t)a.plane, q = r - zr * (uint32_t)a.plane;
        const uint32_t y = q / (uint32_t)a.ixp, x = q - y * (uint32_t)a.ixp;
        const int64_t z = runi + zr;
        po[j] = ((int64_t)r < a.run && x < a.dx && y < a.dy && z < a.dz)
                    ? (int64_t)x + a.dx * ((int64_t)y + a.dy * z) : -1;
      }
      const float* pa2 = nullptr;
      float a2v[8];
#pragma unroll 1
      for (int c0 = 2 * half; c0 < g.ncol; c0 += 4) {
        float r[16];
        if (g.nstage > 0) {
          const uint32_t ta = tmem + ((uint32_t)(32 * lq) << 16) +
                              (uint32_t)(mb * N * (SPLIT ? 2 : 1) + 8 * c0);
          tmem_ld16(ta, r);
          if (SPLIT) {
            float r2[16];
            tmem_ld16(ta + N, r2);
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i] = __fadd_rn(r[i], r2[i]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = 0.f;  // no offsets: AB = 0
        }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const int n = c0 + cc;
          float* o = s_out[n];
          if (!o) continue;  // the same for the whole warp
          float4* tw = reinterpret_cast<float4*>(tr + 8 * lane);
          __syncwarp();
          tw[0] = make_float4(r[8 * cc], r[8 * cc + 1], r[8 * cc + 2], r[8 * cc + 3]);
          tw[1] = make_float4(r[8 * cc + 4], r[8 * cc + 5], r[8 * cc + 6], r[8 * cc + 7]);
          __syncwarp();
          const float* ca2 = s_a2[n];
          if (ca2 != pa2) {  // columns are grouped by mask
            pa2 = ca2;
#pragma unroll
            for (int j = 0; j < 8; ++j) a2v[j] = po[j] >= 0 ? __ldg(ca2 + po[j]) : 0.f;
          }
          const float b2 = s_b2[n];
          unsigned mn = 0x7F800000u, mx = 0u;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (po[j] < 0) continue;
            // A2 is +Inf at disabled windows, and so is D
            const float df = fabsf(__fmaf_rn(-a.ab2, tr[32 * j + lane], __fadd_rn(a2v[j], b2)));
            o[po[j]] = df;
            const unsigned u = __float_as_uint(df);
            mn = min(mn, u);
            if (u < 0x7F800000u) mx = max(mx, u);
          }
          mn = __reduce_min_sync(0xffffffffu, mn);
          mx = __reduce_max_sync(0xffffffffu, mx);
          if (lane == 0) {
            if (mn != 0x7F800000u) atomicMin(s_mn + n, mn);
            if (mx != 0u) atomicMax(s_mx + n, mx);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(a.tmem_cols));
  if (aborted) {
    if (tid == 0 && a.status) atomicCAS(a.status, 0, IQ_ERR_TIMEOUT);
    return;
  }
  if (tid < g.ncol) {
    unsigned* mm = s_mmp[tid];
    if (mm && s_mn[tid] != 0x7F800000u) atomicMin(mm, s_mn[tid]);
    if (mm && s_mx[tid] != 0u) atomicMax(mm + 1, s_mx[tid]);
  }
}

// ---- packing of the templates: thread per (chunk, column, shift), 16 bytes each ----
struct TzPackArgs {
  const float* grid;
  int64_t gx, gxy, tx;
  const TcCol* cols;
  const TcBox* boxes;
  const TzGroup* groups;
  const uint32_t* chunks;
  float scale;
  int split;
  char* B;
};

__global__ void __launch_bounds__(256) tz_pack_kernel(const TzPackArgs p) {
  const TzGroup g = p.groups[blockIdx.y];
  const int64_t units = (int64_t)g.nstep * 2 * g.N;
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < units;
       u += (int64_t)gridDim.x * blockDim.x) {
    const int ch = (int)(u / g.N), rem = (int)(u - (int64_t)ch * g.N);
    const int n = rem >> 3, s = rem & 7;
    const uint32_t w = p.chunks[g.chunk0 + ch];
    const TcCol col = p.cols[g.col0 + n];
    uint32_t h[4] = {0, 0, 0, 0}, l[4] = {0, 0, 0, 0};
    if (w != 0xFFFFFFFFu && col.src >= 0) {
      const int ky = (int)(w & 1023u), kz = (int)((w >> 10) & 1023u);
      const int k0 = 8 * (int)(w >> 20) - s;
      const TcBox bx = p.boxes[col.box];
      const float* row = p.grid + col.src + p.gx * ky + p.gxy * kz;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int kx = k0 + q;
        const float v = (kx >= 0 && kx < p.tx && !in_box(bx, kx, ky, kz)) ? row[kx] : 0.f;
        uint16_t hh, ll;
        f16_split(v, p.scale, hh, ll);
        h[q >> 1] |= (uint32_t)hh << (16 * (q & 1));
        l[q >> 1] |= (uint32_t)ll << (16 * (q & 1));
      }
    }
    char* dst = p.B + g.boff + u * 16;
    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
    if (p.split)
      *reinterpret_cast<uint4*>(dst + (int64_t)g.nstep * 32 * g.N) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

// ---- the FP16 image, x rows padded to a multiple of 8, zeros past the end ----
__global__ void tz_image_kernel(const float* __restrict__ img, int64_t ix, int64_t rows, int64_t ixp,
                                int64_t total, float scale, __half* hi, __half* lo) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / ixp, x = i - r * ixp;
    const float v = (r < rows && x < ix) ? img[x + ix * r] : 0.f;
    uint16_t h, l;
    f16_split(v, scale, h, l);
    hi[i] = __ushort_as_half(h);
    if (lo) lo[i] = __ushort_as_half(l);
  }
}

// A2 of every box at every position: Float64 sums of the integral image, stored as FP32 (+Inf at
// disabled windows).
__global__ void tz_a2_kernel(const double* __restrict__ ii, Dim3 img, Dim3 od, Dim3 tile,
                             const TcBox* boxes, int nbox, const uint8_t* disabled, float* out) {
  const int64_t P = od.vol(), sx = img.x + 1, sxy = (img.x + 1) * (img.y + 1);
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < P;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t z = p / (od.x * od.y), q = p - z * od.x * od.y, y = q / od.x, x = q - y * od.x;
    const bool dis = disabled && disabled[p];
    const double full = iq_box_sum(ii, sx, sxy, x, y, z, tile.x, tile.y, tile.z);
    for (int b = 0; b < nbox; ++b) {
      const TcBox bx = boxes[b];
      double A2 = full;
      if (bx.hi[0] > bx.lo[0] && bx.hi[1] > bx.lo[1] && bx.hi[2] > bx.lo[2])
        A2 -= iq_box_sum(ii, sx, sxy, x + bx.lo[0], y + bx.lo[1], z + bx.lo[2],
                         bx.hi[0] - bx.lo[0], bx.hi[1] - bx.lo[1], bx.hi[2] - bx.lo[2]);
      out[(int64_t)b * P + p] = dis ? __int_as_float(0x7F800000) : (float)A2;
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// Plans
// ---------------------------------------------------------------------------------------------
void iq_tz_list(Dim3 img, Dim3 tile, const TcBox* boxes, int nbox, TzList& out) {
  out = TzList();
  out.touched.assign(nbox, 0);
  const int64_t ixp = (img.x + 7) / 8 * 8, plane = ixp * img.y;
  const int nj = (int)((tile.x + 7 + 7) / 8);  // chunks of a whole row
  struct Entry { uint32_t off; int j0, span; std::vector<int> ch; uint32_t row; };
  std::vector<Entry> ent;
  std::vector<uint8_t> act(nj);
  auto has = [&](const TcBox& bx, int64_t ky, int64_t kz, int j) {
    // any offset kx of [8 j - 7, 8 j + 7] in the mask
    const int64_t a = std::max<int64_t>(8 * j - 7, 0), b = std::min<int64_t>(8 * j + 7, tile.x - 1);
    if (a > b) return false;
    const bool rowin = ky >= bx.lo[1] && ky < bx.hi[1] && kz >= bx.lo[2] && kz < bx.hi[2];
    return !rowin || a < bx.lo[0] || b >= bx.hi[0] || bx.hi[0] <= bx.lo[0];
  };
  for (int64_t kz = 0; kz < tile.z; ++kz)
    for (int64_t ky = 0; ky < tile.y; ++ky) {
      for (int j = 0; j < nj; ++j) {
        act[j] = 0;
        for (int b = 0; b < nbox && !act[j]; ++b) act[j] = has(boxes[b], ky, kz, j);
      }
      for (int j0 = 0; j0 < nj;) {
        if (!act[j0]) { ++j0; continue; }
        Entry e;
        e.j0 = j0;
        e.off = (uint32_t)((8 * j0 + ixp * ky + plane * kz) / 8);
        e.row = (uint32_t)ky | (uint32_t)kz << 10;
        for (int j = j0; j < std::min(nj, j0 + TZ_MAXCH); ++j)
          if (act[j]) { e.ch.push_back(j - j0); e.span = j - j0 + 1; }
        j0 += e.span;
        ent.push_back(e);
      }
    }
  // stages of at most IQ_TZ_ROWS entries and 2 IQ_TZ_STEPS chunks
  for (size_t i = 0; i < ent.size();) {
    size_t k = i;
    int nch = 0;
    while (k < ent.size() && (int)(k - i) < IQ_TZ_ROWS &&
           nch + (int)ent[k].ch.size() <= 2 * IQ_TZ_STEPS)
      nch += (int)ent[k++].ch.size();
    TzStage st{};
    const int nks = (nch + 1) / 2;
    st.w[0] = (uint32_t)(k - i) | (uint32_t)nks << 8;
    st.w[1] = (uint32_t)out.nstep;
    uint32_t prev = 0;
    int c = 0;
    for (size_t q = i; q < k; ++q) {
      const Entry& e = ent[q];
      st.w[2 + (q - i)] = e.off;
      st.w[7] |= (uint32_t)(e.span + 1) << (4 * (q - i));  // one chunk more for an odd end
      for (int lc : e.ch) {
        const uint32_t pos = (uint32_t)(q - i) | (uint32_t)lc << 4;
        st.w[8 + c / 2] |= pos << (8 * (c & 1));
        out.chunk.push_back(e.row | (uint32_t)(e.j0 + lc) << 20);
        prev = pos;
        ++c;
      }
    }
    if (c & 1) {  // the last step's second chunk: the next image block against zero templates
      st.w[8 + c / 2] |= (prev + 16u) << 8;
      out.chunk.push_back(0xFFFFFFFFu);
    }
    out.stage.push_back(st);
    out.nstep += nks;
    i = k;
  }
  // K-steps that hold an offset of each mask (its roundings in the FP32 accumulator)
  for (int b = 0; b < nbox; ++b)
    for (size_t s = 0; s + 1 < out.chunk.size(); s += 2) {
      bool any = false;
      for (int h = 0; h < 2; ++h) {
        const uint32_t w = out.chunk[s + h];
        if (w != 0xFFFFFFFFu)
          any = any || has(boxes[b], w & 1023u, (w >> 10) & 1023u, (int)(w >> 20));
      }
      out.touched[b] += any;
    }
}

double iq_map_kappa_tz(const IqValueStats& A, const IqValueStats& B, int64_t K, int64_t nsteps) {
  if (!(iq_map_kappa(A, B, K, 1) > 0.0)) return 0.0;  // exact sums
  // the hi * hi accumulator rounds once per K-step (4u of sum |a||b| each, as in iq_map_kappa);
  // the hi * lo + lo * hi accumulator holds terms 2^-11 as large and rounds twice per K-step;
  // adding the two rounds once; split (12u), epilogue (4u) and slack as in iq_map_kappa
  const double u = std::ldexp(1.0, -24);
  const double acc = 4.0 * (double)nsteps * (1.0 + 2.0 * 2.0 / 1024.0);
  return (acc + 2.0 + 12.0 + 4.0 + 8.0) * u * 1.01;
}

bool iq_tz_fits(Dim3 img, Dim3 tile, Dim3 out) {
  // row offsets in units of 8 values in 32 bits; chunk numbers in 12 bits; one run's positions in
  // 31 bits (rows padded to 8); the staged slots hold any tile extent below 1024
  const int64_t ixp = (img.x + 7) / 8 * 8;
  return tile.x < 1024 && tile.y < 1024 && tile.z < 1024 && ixp * img.y * img.z < ((int64_t)1 << 31) - (1 << 16) &&
         out.vol() > 0;
}

int64_t iq_tz_image_halves(Dim3 img) {
  // slack: a CTA's last accumulators and row spans read past the last run's end
  return (img.x + 7) / 8 * 8 * img.y * img.z + 4096 + 1024 + 128;
}

int iq_tz_image(iq_ctx* ctx, const float* img, Dim3 d, const IqValueStats& st, bool split, void* dst) {
  const int64_t ixp = (d.x + 7) / 8 * 8, total = iq_tz_image_halves(d);
  __half* hi = (__half*)dst;
  const int64_t pitch = (total + 63) / 64 * 64;
  const int ka = st.amax > 0.f ? st.maxexp() - 14 : 0;
  tz_image_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256, 4096), 256, 0, ctx->stream>>>(
      img, d.x, d.y * d.z, ixp, total, std::ldexp(1.f, -ka), hi, split ? hi + pitch : nullptr);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

int iq_tz_a2_maps(iq_ctx* ctx, const double* ii, Dim3 img, Dim3 out, Dim3 tile, const TcBox* boxes,
                  int nbox, const uint8_t* disabled, float* maps) {
  if (nbox <= 0 || out.vol() <= 0) return IQ_OK;
  tz_a2_kernel<<<(unsigned)std::min<int64_t>((out.vol() + 255) / 256, 8192), 256, 0, ctx->stream>>>(
      ii, img, out, tile, boxes, nbox, disabled, maps);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}

namespace {

struct TzShape {
  int MB, nst, slot;
  int64_t run, nrun, tiles, ctas;
  size_t smem;
  uint32_t stage_bytes, b_off, t_off;
};

TzShape tz_shape(const TzLaunch& L, int MB, bool split, int smem_lim) {
  TzShape s{};
  const int64_t ixp = (L.img_dims.x + 7) / 8 * 8, plane = ixp * L.img_dims.y;
  const Dim3 od = L.out_dims;
  const int64_t M = 1024 * MB;
  // runs: one per z plane, or the whole volume when that takes fewer CTAs
  const int64_t r1 = (od.y - 1) * ixp + od.x, rv = (od.z - 1) * plane + r1;
  const int64_t t1 = (r1 + M - 1) / M, tv = (rv + M - 1) / M;
  s.MB = MB;
  if (tv < t1 * od.z) { s.run = rv; s.nrun = 1; s.tiles = tv; }
  else { s.run = r1; s.nrun = od.z; s.tiles = t1; }
  s.ctas = s.tiles * s.nrun * L.ngroup;
  s.slot = 128 * MB + TZ_MAXCH + 1;
  const uint32_t rows = (uint32_t)(IQ_TZ_ROWS * s.slot) * 16u * (split ? 2u : 1u);
  const uint32_t bb = (uint32_t)IQ_TZ_STEPS * 32u * (uint32_t)L.Nmax * (split ? 2u : 1u);
  s.b_off = (rows + 127u) & ~127u;
  s.t_off = (s.b_off + bb + 127u) & ~127u;
  s.stage_bytes = s.t_off + 128u;
  s.nst = (int)std::min<int64_t>(TZ_MAXST, smem_lim / s.stage_bytes);
  s.smem = std::max<size_t>((size_t)s.nst * s.stage_bytes, (size_t)(TZ_THREADS / 32) * 1024);
  return s;
}

template <bool SPLIT>
cudaError_t tz_launch(const TzArgs& a, const TzShape& s, dim3 grid, cudaStream_t st) {
  void (*k)(TzArgs) = s.MB == 4 ? corr_tz_kernel<SPLIT, 4> : s.MB == 2 ? corr_tz_kernel<SPLIT, 2>
                                                                       : corr_tz_kernel<SPLIT, 1>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
  if (e != cudaSuccess) return e;
  k<<<grid, TZ_THREADS, s.smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace

int iq_launch_corr_tz(iq_ctx* ctx, const TzLaunch& L) {
  if (L.ngroup <= 0) return IQ_OK;
  const bool split = !(L.img_stats.narrow && L.tmpl_stats.narrow);
  if (L.Nmax < 16 || L.Nmax % 16 || L.Nmax > 8 * IQ_TZ_COLS || (split && 2 * L.Nmax > 512) ||
      !L.groups || !L.stages || !L.cols || !L.boxes || !L.img || !L.a2)
    return iq_set_error(IQ_ERR_ARG, "tensor-core correlation: bad launch");
  const Dim3 od = L.out_dims;
  const int64_t ixp = (L.img_dims.x + 7) / 8 * 8;
  int dev = 0, lim = 0;
  const int nsm = iq_sm_count();
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  lim -= 4096;  // the kernel's static shared memory
  // Accumulators per CTA: more of them reuse a staged template chunk for more positions, fewer
  // spread a small map over more SMs. Cycles of one K-step: the MMAs (N / 2 each, three when
  // split) or its bytes from L2 at ~32 per cycle and SM; times the waves of CTAs.
  TzShape best{};
  double best_cost = 0.0;
  for (int MB : {4, 2, 1}) {
    if (MB * L.Nmax * (split ? 2 : 1) > 512) continue;
    const TzShape s = tz_shape(L, MB, split, lim);
    if (s.nst < 2) continue;
    const double mma = MB * L.Nmax * 0.5 * (split ? 3.0 : 1.0);
    const double mem = (32.0 * L.Nmax + 1024.0 * MB) * (split ? 2.0 : 1.0) / 32.0;
    const double cost = std::ceil((double)s.ctas / nsm) * (std::max(mma, mem) + 24.0);
    if (best.MB == 0 || cost < best_cost) { best = s; best_cost = cost; }
  }
  if (best.MB == 0) return iq_set_error(IQ_ERR_LIMIT, "tensor-core correlation: no launch shape fits");
  TzArgs a{};
  const int ka = L.img_stats.amax > 0.f ? L.img_stats.maxexp() - 14 : 0;
  const int kb = L.tmpl_stats.amax > 0.f ? L.tmpl_stats.maxexp() - 14 : 0;
  a.hi = (const __half*)L.img;
  a.lo = a.hi + (iq_tz_image_halves(L.img_dims) + 63) / 64 * 64;
  a.ixp = ixp; a.plane = ixp * L.img_dims.y;
  a.dx = od.x; a.dy = od.y; a.dz = od.z;
  a.run = best.run; a.nrun = best.nrun; a.tiles = (int)best.tiles;
  a.slot = best.slot; a.nst = best.nst;
  a.stage_bytes = best.stage_bytes; a.b_off = best.b_off; a.t_off = best.t_off;
  a.Nmax = L.Nmax;
  uint32_t tc = 32;
  while (tc < (uint32_t)(best.MB * L.Nmax * (split ? 2 : 1))) tc <<= 1;
  a.tmem_cols = tc;
  a.groups = L.groups; a.stages = L.stages; a.B = (const char*)L.B; a.cols = L.cols;
  a.a2 = L.a2; a.P = od.vol();
  a.ab2 = std::ldexp(1.f, ka + kb + 1);
  a.status = ctx->d_status;
  iq_timer_start(ctx, "corr");
  if (L.max_units > 0) {
    TzPackArgs p{};
    p.grid = L.grid; p.gx = L.grid_dims.x; p.gxy = L.grid_dims.x * L.grid_dims.y; p.tx = L.tile.x;
    p.cols = L.cols; p.boxes = L.boxes; p.groups = L.groups; p.chunks = L.chunks;
    p.scale = std::ldexp(1.f, -kb); p.split = split ? 1 : 0; p.B = (char*)L.B;
    const dim3 pg((unsigned)std::min<int64_t>((L.max_units + 255) / 256, 2048), (unsigned)L.ngroup);
    tz_pack_kernel<<<pg, 256, 0, ctx->stream>>>(p);
    iq_count(ctx);
    IQ_CUDA_OK(cudaGetLastError());
  }
  const dim3 grid((unsigned)(best.tiles * best.nrun), (unsigned)L.ngroup);
  const cudaError_t e = split ? tz_launch<true>(a, best, grid, ctx->stream)
                              : tz_launch<false>(a, best, grid, ctx->stream);
  iq_count(ctx);
  iq_timer_stop(ctx, "corr", L.flops);
  if (e != cudaSuccess)
    return iq_set_error(IQ_ERR_CUDA, "tensor-core correlation: %s", cudaGetErrorString(e));
  if (ctx->prof) {
    ctx->prof_mma_flops += L.mma_flops * (split ? 3 : 1) * (double)(best.tiles * best.nrun) * best.MB;
    ctx->prof_mma_flops16 += L.mma_flops * (split ? 3 : 1) * (double)(best.tiles * best.nrun) * best.MB;
    ctx->prof_mma_launches += 1;
    ctx->prof_tc_cols += L.ncols;
  }
  return IQ_OK;
}
