// Minimum-error boundary cut of the overlap slabs (src/graphcut.jl:5-84).
//
// One CTA per (realization, slab). The lattice graph, the capacities
//   c(u, v) = (|A-B|_u + |A-B|_v) / (|A_v-A_u| + |A_w-A_v| + |B_v-B_u| + |B_w-B_v| + eps())
// (Float32 differences and sums, Float64 division, as Julia does for Float32 arrays) and the
// infinite source/sink slices follow the reference. The max-flow is a synchronous
// push-relabel instead of Boykov-Kolmogorov:
//   * the first slice along the cut dimension is contracted into s, the last into t;
//   * capacities are rounded to multiples of q = 2^(ilogb(cmax) - 47), cmax the largest of
//     the slab, so that every residual (<= 2 cmax) and excess (<= 12 cmax) is a multiple of q
//     below 2^53 q and all flow arithmetic is exact (zero gradient sums give eps-denominator
//     capacities ~2^52 times the others, which unquantized Float64 flows cannot resolve);
//   * so residuals and excesses are kept as int64 counts of q (the same values as the exact
//     Float64 arithmetic, without GB300's narrow FP64 pipe); an arc is open when its residual
//     is positive (the oracle quantizes and tests the same way);
//   * each round: every node on the active list pushes its excess along its arcs to lower
//     neighbours and, if some is left, relabels to 1 + its lowest open neighbour; the receivers
//     and the nodes still active form the next list (a few percent of the slab per round). The
//     flow found depends on the order of the atomics, the cut does not: integer sums are exact,
//     and the set of nodes that can reach t is the same for every maximum preflow;
//   * a global relabel (BFS from t over open arcs) runs at the start, every GR rounds and at
//     the end; nodes that cannot reach t get height NH and stop being active. The cut is done
//     when it finds no node with excess that reaches t.
// Only the interior nodes (the slab without its s and t slices) are kept: arcs to s never carry
// flow here (heights stay below NH) and arcs from t are never used, so a node's state is its six
// outgoing residuals, its excess and its height: 3,072 of a slab of 4,096 voxels fit shared memory
// whole. What bounds the cut is latency: the rounds (some 50 active nodes of 3,072, 35-80 rounds a
// slab) and the searches are chains of dependent shared-memory steps, and a launch ends with its
// slowest slab. Eight lanes serve a node, a direction each, one phase and one barrier make a round, and
// excesses, flags and lists go through native 32-bit shared-memory atomics. Cut time of whole
// simulations, before (a thread per node, two phases, 64-bit adds and 16-bit compare-and-swaps, the
// 4,096-node slabs' excesses in global memory) and after: 128 x 128 x 64 facies 28.6 -> 10.1 ms,
// proposal 55 -> 18.9, 3-D conditioned 46 -> 26.8, 3-D continuous 31.5 -> 15.9, 2-D continuous
// 3.7 -> 2.1.
// At the end the nodes that can reach t are the sink side of the canonical minimum cut (the
// same set for every maximum flow, which is what BK's sink tree holds at termination), and
// mask = not sink side (graphcut.jl:75-81).
#include <algorithm>

#include "iq_internal.h"

namespace {

constexpr int CUT_MAX_THREADS = 1024;

struct CutArgs {
  StepTask t0;                 // used when tasks is null
  const StepTask* tasks;
  int nreal;                   // CTA (s, y): slab s of realization y % nreal of task y / nreal
  const float* sim; int64_t sx, sy; int64_t sim_rs;
  const float* ti; int64_t tix, tiy; int64_t dx, dy;
  const int64_t* rind;
  const float* A; const float* B;
  uint8_t* out; int64_t slabmax;
  char* scratch; int64_t scratch_per_cta;
  int* status;
  int round_cap;
  unsigned long long* stats;
  int gr_period;
};

__device__ __forceinline__ long long dbits(double x) { return __double_as_longlong(x); }

// *p += d. In shared memory as two 32-bit adds, the low one's carry joined to the high one: the sum
// is right once every add is done, whatever their order. A round reads a node's excess while others may
// push into the node (one_round): every such add is positive and its high word follows its low one, so a
// read between the two is at most the excess after the round. The node then pushes no more than it has,
// does not relabel, and whoever pushed into it has put it on the next list.
template <bool SHARED>
__device__ __forceinline__ void add64(long long* p, long long d) {
  if (SHARED) {
    unsigned* w = reinterpret_cast<unsigned*>(p);
    const unsigned lo = (unsigned)d;
    unsigned hi = (unsigned)((unsigned long long)d >> 32);
    if (lo) {
      const unsigned old = atomicAdd(w, lo);
      hi += old + lo < old ? 1u : 0u;
    }
    if (hi) atomicAdd(w + 1, hi);
  } else {
    atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)d);
  }
}

template <bool SHARED, typename T>
__device__ __forceinline__ T ldv(const T* p) {
  if (SHARED) return *p;
  return __ldcg(p);  // written by other threads' atomics: past the L1
}

// Most active nodes of a round on one warp (two passes of four). Cut time at 0, 4, 8 and 16: 2-D
// continuous 2.07, 2.11, 2.19, 2.23 ms; 3-D conditioned 26.5, 26.7, 27.0, 28.6; 128 x 128 x 64 facies
// 10.06, 9.92, 10.13, 10.72: little is at stake up to 8, and more is worse.
constexpr int CUT_WARP = 8;
// Past this many rounds a search follows every round: with exact heights at each start a round only
// pushes along shortest paths, distances to t never fall, and the rounds are bounded whatever labels
// came out too high before (the most seen in any workload is 391).
constexpr int CUT_SAFE = 1 << 12;
constexpr int CUT_CODES = 8;  // categorical codes 0..7 take their capacities from a table
constexpr int CUT_TAB = (2 * (CUT_CODES - 1) + 1) * (4 * (CUT_CODES - 1) + 1);

// capacity of one edge u -> v (w: the voxel after v along the edge, or v's difference again)
__device__ __forceinline__ void edge_terms(const float* A, const float* B, int u, int v, int w,
                                           bool ok, float& num, float& den) {
  const float Au = A[u], Av = A[v], Bu = B[u], Bv = B[v];
  const float Du = fabsf(__fsub_rn(Au, Bu));
  const float Dv = fabsf(__fsub_rn(Av, Bv));
  const float gAu = fabsf(__fsub_rn(Av, Au));
  const float gBu = fabsf(__fsub_rn(Bv, Bu));
  const float gAv = ok ? fabsf(__fsub_rn(A[w], Av)) : gAu;
  const float gBv = ok ? fabsf(__fsub_rn(B[w], Bv)) : gBu;
  num = __fadd_rn(Du, Dv);
  den = __fadd_rn(gAu, gAv);
  den = __fadd_rn(den, gBu);
  den = __fadd_rn(den, gBv);
}

__device__ __forceinline__ double edge_cap(float num, float den) {
  const double EPS = 2.220446049250313e-16;  // eps(Float64) = 2^-52
  return __ddiv_rn((double)num, __dadd_rn((double)den, EPS));
}

// capacity in units of q = 2^sh, rounded half to even
__device__ __forceinline__ long long edge_units(double cap, int sh) {
  return (long long)rint(ldexp(cap, -sh));
}

// Bytes of the arrays over n interior nodes of a slab of nf voxels; heights and list entries are HT:
// 16-bit for slabs below 32768 nodes, else 32-bit.
struct CutLayout {
  size_t ab, ex, h, l, nl, info, flag, end;  // offsets behind the residuals (ab aliases ex..nl)
};
__host__ __device__ inline CutLayout cut_layout(int64_t n, int64_t nf, int hb) {
  CutLayout c;
  auto up = [](size_t b) { return (b + 15) & ~(size_t)15; };
  c.ab = up((size_t)n * 48);
  c.ex = c.ab;
  c.h = up(c.ex + (size_t)n * 8);
  c.l = up(c.h + (size_t)n * hb);
  c.nl = up(c.l + (size_t)n * hb);
  const size_t e1 = up(c.nl + (size_t)n * hb), e2 = up(c.ab + (size_t)nf * 8);
  c.info = e1 > e2 ? e1 : e2;
  c.flag = up(c.info + (size_t)n);
  c.end = (c.flag + (size_t)(n + 31) / 32 * 8 + 255) & ~(size_t)255;
  return c;
}
// MODE 2: the residuals, heights, node info and flags in shared memory
struct CutLayout2 {
  size_t h, info, flag, end;     // shared
  size_t ex, l, nl, gend;        // global (A and B alias ex..nl and what follows)
};
__host__ __device__ inline CutLayout2 cut_layout2(int64_t n, int64_t nf, int hb) {
  CutLayout2 c;
  auto up = [](size_t b) { return (b + 15) & ~(size_t)15; };
  c.h = up((size_t)n * 48);
  c.info = up(c.h + (size_t)n * hb);
  c.flag = up(c.info + (size_t)n);
  c.end = (c.flag + (size_t)(n + 31) / 32 * 8 + 255) & ~(size_t)255;
  c.ex = 0;
  c.l = up((size_t)n * 8);
  c.nl = up(c.l + (size_t)n * hb);
  const size_t e1 = up(c.nl + (size_t)n * hb), e2 = up((size_t)nf * 8);
  c.gend = ((e1 > e2 ? e1 : e2) + 255) & ~(size_t)255;
  return c;
}

// MODE 0: the slab lives in shared memory. MODE 2: the residuals, heights and node info (what every
// push and relabel reads) in shared memory, the excesses and lists in global scratch. MODE 1:
// everything in global scratch.
template <typename HT, int MODE, int NTHR>
__global__ void __launch_bounds__(NTHR, NTHR == 256 ? 3 : 1) cut_kernel(const CutArgs a) {
  extern __shared__ __align__(16) char smem[];
  constexpr bool SX = MODE == 0;   // excesses and lists in shared memory
  constexpr bool SR = MODE != 1;   // residuals and heights in shared memory
  const int s_id = blockIdx.x;
  const int y = blockIdx.y;
  const int r = y % a.nreal;
  const StepTask& tk = a.tasks ? a.tasks[y / a.nreal] : a.t0;
  if (s_id >= tk.nslab) return;
  const CutSlab sl = tk.slab[s_id];
  const int64_t tile_start = tk.start;
  const bool prof = a.stats != nullptr && threadIdx.x == 0;
  const long long t_start = prof ? clock64() : 0;
  long long t_gr = 0;
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31;
  // slab extents and strides; interior extents, strides and count
  const int e0 = (int)sl.ext[0], e1 = (int)sl.ext[1], e2 = (int)sl.ext[2];
  const int d = sl.dim;
  const int Ld = d == 0 ? e0 : (d == 1 ? e1 : e2);
  const int f1 = e0, f2 = e0 * e1, nf = f2 * e2, fd = d == 0 ? 1 : (d == 1 ? f1 : f2);
  const int in = Ld > 2 ? Ld - 2 : 0;
  const int m0 = d == 0 ? in : e0, m1 = d == 1 ? in : e1, m2 = d == 2 ? in : e2;
  const int s1 = m0, s2 = m0 * m1, n = s2 * m2;
  const int NH = n + 2;            // height of s
  const int fw = (n + 31) / 32;    // words of one flag mask

  char* gbase = a.scratch + (int64_t)(blockIdx.y * gridDim.x + blockIdx.x) * a.scratch_per_cta;
  char* base = MODE == 1 ? gbase : smem;
  long long* const R = reinterpret_cast<long long*>(base);  // R[dir n + u]: residual of u's arc
  long long* ex;
  HT *hc, *L, *Nl;
  uint8_t* info;                   // bits 0-5: interior neighbour in direction 0..5; 6: next to t
  unsigned* flag;                  // two bit masks: listed, by round parity (rounds); reached (search)
  float* Av;
  if (MODE == 2) {
    const CutLayout2 c = cut_layout2(n, nf, sizeof(HT));
    hc = reinterpret_cast<HT*>(smem + c.h);
    info = reinterpret_cast<uint8_t*>(smem + c.info);
    flag = reinterpret_cast<unsigned*>(smem + c.flag);
    ex = reinterpret_cast<long long*>(gbase + c.ex);
    L = reinterpret_cast<HT*>(gbase + c.l);
    Nl = reinterpret_cast<HT*>(gbase + c.nl);
    Av = reinterpret_cast<float*>(gbase);
  } else {
    const CutLayout c = cut_layout(n, nf, sizeof(HT));
    ex = reinterpret_cast<long long*>(base + c.ex);
    hc = reinterpret_cast<HT*>(base + c.h);
    L = reinterpret_cast<HT*>(base + c.l);
    Nl = reinterpret_cast<HT*>(base + c.nl);
    info = reinterpret_cast<uint8_t*>(base + c.info);
    flag = reinterpret_cast<unsigned*>(base + c.flag);
    Av = reinterpret_cast<float*>(base + c.ab);
  }
  float* Bv = Av + nf;  // A and B alias the excesses, heights and lists, written after the capacities
  __shared__ unsigned long long s_cmax;  // bits of the largest capacity
  __shared__ unsigned s_code;            // largest categorical code (all ones: not categorical)
  __shared__ double s_tab[CUT_TAB];      // categorical capacities, then their units
  __shared__ uint8_t s_has[CUT_TAB];
  __shared__ int s_cnt[2];
  if (tid == 0) { s_cmax = 0ull; s_code = 0u; }

  // ---- load A (simulation grid) and B (training image at the drawn pattern) ----
  int64_t bstart = 0;
  if (!a.A) {
    const int64_t ri = a.rind[y];
    if (ri < 0) {  // pick failed: no cut (status already set)
      for (int u = tid; u < nf; u += nthr) a.out[((int64_t)y * 6 + s_id) * a.slabmax + u] = 0;
      return;
    }
    const int64_t rx = ri % a.dx, rr = ri / a.dx, ry = rr % a.dy, rz = rr / a.dy;
    bstart = rx + a.tix * (ry + a.tiy * rz);
  }
  __syncthreads();
  unsigned code = 0;
  if (n > 0) {
    for (int u = tid; u < nf; u += nthr) {
      float va, vb;
      if (a.A) {
        va = a.A[u];
        vb = a.B[u];
      } else {
        const int x = u % e0, yy = (u / e0) % e1, z = u / f2;
        const int64_t lx = sl.off[0] + x, ly = sl.off[1] + yy, lz = sl.off[2] + z;
        va = a.sim[(int64_t)r * a.sim_rs + tile_start + lx + a.sx * (ly + a.sy * lz)];
        vb = a.ti[bstart + lx + a.tix * (ly + a.tiy * lz)];
      }
      Av[u] = va;
      Bv[u] = vb;
      const float top = (float)(CUT_CODES - 1);
      const bool cat = va >= 0.f && va <= top && va == floorf(va) && vb >= 0.f && vb <= top && vb == floorf(vb);
      code = max(code, cat ? (unsigned)fmaxf(va, vb) : 0xFFFFFFFFu);
    }
    code = __reduce_max_sync(0xffffffffu, code);
    if (lane == 0) atomicMax(&s_code, code);
  }
  for (int i = tid; i < CUT_TAB; i += nthr) s_has[i] = 0;
  __syncthreads();
  code = s_code;
  const bool cat = code < (unsigned)CUT_CODES;
  const int tw = 4 * (int)code + 1;  // table row length: denominators 0 .. 4 code

  // ---- capacities (graphcut.jl:22-50) ----
  // Every edge counts for the largest capacity; edges with an interior end are kept, in R of their
  // lower end (of the upper end's opposite direction for the s slice). Integer codes take their few
  // distinct quotients from a table (one Float64 division each instead of one per edge: the FP64 pipe
  // made the set-up a third of the categorical cuts). Otherwise edges inside the s and t slices only
  // divide in Float64 when a float quotient comes near the largest capacity of the others.
  const int wd0 = d == 0 ? 1 : 0, wd1 = d == 1 ? 1 : 0, wd2 = d == 2 ? 1 : 0;
  auto each_edge = [&](auto&& fn) {
    for (int u = tid; u < nf; u += nthr) {
      const int x = u % e0, yy = (u / e0) % e1, z = u / f2;
      const int cd = d == 0 ? x : (d == 1 ? yy : z);
      // interior index of u (meaningful for cd in [1, Ld - 2]) and of the voxel after it along d
      const int ui = (x - wd0) + s1 * (yy - wd1) + s2 * (z - wd2);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const int c = e == 0 ? x : (e == 1 ? yy : z), ne = e == 0 ? e0 : (e == 1 ? e1 : e2);
        if (c + 1 >= ne) continue;
        const int st = e == 0 ? 1 : (e == 1 ? f1 : f2), sti = e == 0 ? 1 : (e == 1 ? s1 : s2);
        const int v = u + st;
        const bool ok = c + 2 < ne;
        float num, den;
        edge_terms(Av, Bv, u, v, ok ? v + st : v, ok, num, den);
        // where the edge's value is kept: direction slot and node; -1: inside the s or t slice
        int slot = -1;
        if (e == d) {
          if (cd >= 1) slot = (2 * e + 1) * n + ui;        // interior or t end
          else slot = (2 * e) * n + ui + sti;              // from s to interior node ui + sti
        } else if (cd >= 1 && cd < Ld - 1) {
          slot = (2 * e + 1) * n + ui;
        }
        fn(slot, e, ui, sti, cd, num, den);
      }
    }
  };
  int sh = 0;
  if (n > 0) {
    if (cat) {
      each_edge([&](int, int, int, int, int, float num, float den) { s_has[(int)num * tw + (int)den] = 1; });
      __syncthreads();
      for (int i = tid; i < (2 * (int)code + 1) * tw; i += nthr) {
        const double c = edge_cap((float)(i / tw), (float)(i % tw));
        s_tab[i] = c;
        if (s_has[i]) atomicMax(&s_cmax, (unsigned long long)dbits(c));
      }
    } else {
      unsigned long long mx = 0ull;
      each_edge([&](int slot, int, int, int, int, float num, float den) {
        if (slot < 0) return;
        const double c = edge_cap(num, den);
        R[slot] = dbits(c);  // the double's bits until the quantization below
        const unsigned long long b = (unsigned long long)dbits(c);
        mx = b > mx ? b : mx;
      });
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = w > mx ? w : mx;
      }
      if (lane == 0) atomicMax(&s_cmax, mx);
      __syncthreads();
      const float lim = fminf((float)__longlong_as_double((long long)s_cmax) * 0.9999f, 1e38f);
      each_edge([&](int slot, int, int, int, int, float num, float den) {
        if (slot >= 0) return;
        if (!(__fdiv_rn(num, den + 2.2204460e-16f) < lim))
          atomicMax(&s_cmax, (unsigned long long)dbits(edge_cap(num, den)));
      });
    }
    __syncthreads();
    // ---- capacities in units of q = 2^(ilogb(cmax) - 47), rounded half to even: the flows are then
    // exact integers (<= 2^49 per arc), the same numbers the oracle's quantized Float64 arithmetic
    // produces ----
    sh = s_cmax != 0ull ? ilogb(__longlong_as_double((long long)s_cmax)) - 47 : 0;
    if (sh < -1074) sh = -1074;
    if (cat) {
      for (int i = tid; i < (2 * (int)code + 1) * tw; i += nthr)
        s_tab[i] = __longlong_as_double(s_cmax != 0ull && s_has[i] ? edge_units(s_tab[i], sh) : 0ll);
      __syncthreads();
    }
    // both arcs of every kept edge; an edge from s only becomes its node's first excess, in the slot
    // of the node's (unused) arc to s until the excesses' memory is free
    each_edge([&](int slot, int e, int ui, int sti, int cd, float num, float den) {
      if (slot < 0) return;
      long long k;
      if (cat) k = dbits(s_tab[(int)num * tw + (int)den]);
      else k = s_cmax != 0ull ? edge_units(__longlong_as_double(R[slot]), sh) : 0ll;
      R[slot] = k;
      if (e != d || (cd >= 1 && cd < Ld - 2)) R[(2 * e) * n + ui + sti] = k;  // the opposite arc
    });
    __syncthreads();
  }
  // ---- node info, first excesses (the source slice saturated) ----
  const int dsink = 2 * d + 1, dsrc = 2 * d;
  for (int u = tid; u < n; u += nthr) {
    const int x = u % m0, yy = (u / m0) % m1, z = u / s2;
    const int cd = d == 0 ? x : (d == 1 ? yy : z);
    uint8_t f = 0;
    if (x > 0) f |= 1u;
    if (x + 1 < m0) f |= 2u;
    if (yy > 0) f |= 4u;
    if (yy + 1 < m1) f |= 8u;
    if (z > 0) f |= 16u;
    if (z + 1 < m2) f |= 32u;
    if (cd == in - 1) f |= 64u;
    info[u] = f;
    long long c = 0;
    if (cd == 0) {
      c = R[dsrc * n + u];
      R[dsrc * n + u] = 0;
    }
    ex[u] = c;
  }
  __syncthreads();

  // Lists of active nodes (excess and height below NH), double-buffered by round parity; their lengths
  // rotate through three counters (this round's, the next round's, one zeroed for the round after), so
  // a round needs one barrier.
  __shared__ int s_cl[3];
  int k6 = 0;  // rounds since the list was rebuilt, modulo 6
  int round = 0, levels = 0;
  long long nactive = 0;
  const long long t_setup = prof ? clock64() : 0;
  constexpr int FAR = 0x3FFFFFFF;
  // Exact heights: breadth-first search from t over open arcs; each level examines the neighbours of
  // the previous level's frontier (in L and Nl).
  auto relabel_all = [&]() {
    const long long t = prof ? clock64() : 0;
    if (tid == 0) { s_cnt[0] = 0; s_cnt[1] = 0; }
    __syncthreads();
    const int nw = (n + 31) / 32 * 32;
    for (int u = tid; u < nw; u += nthr) {
      bool one = false;
      if (u < n) {
        one = (info[u] & 64) && R[dsink * n + u] > 0;
        hc[u] = (HT)(one ? 1 : NH);
      }
      const unsigned b = __ballot_sync(0xffffffffu, one);
      int at = 0;
      if (lane == 0) {
        flag[u >> 5] = b;
        if (b) at = atomicAdd(&s_cnt[0], __popc(b));
      }
      at = __shfl_sync(0xffffffffu, at, 0);
      if (one) L[at + __popc(b & ((1u << lane) - 1u))] = (HT)u;
    }
    __syncthreads();
    int level = 1, cur = 0;
    for (;;) {
      const int nfr = s_cnt[cur];
      if (nfr == 0) break;
      HT* front = cur ? Nl : L;
      HT* next = cur ? L : Nl;
      __syncthreads();  // every thread has read the count
      if (tid == 0) s_cnt[cur] = 0;  // (next read two levels on)
      for (int i0 = 4 * (tid >> 5); i0 < nfr; i0 += 4 * (nthr >> 5)) {
        // eight lanes per frontier node, one per direction
        const int sb = lane & 7;
        const bool in = i0 + (lane >> 3) < nfr;
        const int v = in ? (int)ldv<SX>(front + i0 + (lane >> 3)) : 0;
        const int st = (sb >> 1) == 0 ? 1 : ((sb >> 1) == 1 ? s1 : s2);
        const bool ok = in && sb < 6 && (info[v] >> sb & 1);
        const int u = ok ? ((sb & 1) ? v + st : v - st) : v;
        bool add = false;
        if (ok && (int)ldv<SR>(hc + u) == NH && ldv<SR>(R + (sb ^ 1) * n + u) > 0) {  // arc u -> v
          add = !(atomicOr(&flag[u >> 5], 1u << (u & 31)) >> (u & 31) & 1u);
          if (add) hc[u] = (HT)(level + 1);
        }
        const unsigned b = __ballot_sync(0xffffffffu, add);
        if (b) {
          int at = 0;
          if (lane == 0) at = atomicAdd(&s_cnt[cur ^ 1], __popc(b));
          at = __shfl_sync(0xffffffffu, at, 0);
          if (add) next[at + __popc(b & ((1u << lane) - 1u))] = (HT)u;
        }
      }
      __syncthreads();
      cur ^= 1;
      ++level;
    }
    levels += level;
    __syncthreads();
    if (prof) t_gr += clock64() - t;
  };
  // the active list from scratch (after a search, which used the lists as frontiers)
  auto rebuild = [&]() {
    k6 = 0;
    if (tid == 0) { s_cl[0] = 0; s_cl[1] = 0; s_cl[2] = 0; }
    __syncthreads();
    const int nw = (n + 31) / 32 * 32;
    for (int u = tid; u < nw; u += nthr) {
      const bool act = u < n && ldv<SX>(ex + u) > 0 && (int)hc[u] < NH;
      const unsigned b = __ballot_sync(0xffffffffu, act);
      int at = 0;
      if (lane == 0) {
        flag[u >> 5] = 0;
        flag[fw + (u >> 5)] = 0;
        if (b) at = atomicAdd(&s_cl[0], __popc(b));
      }
      at = __shfl_sync(0xffffffffu, at, 0);
      if (act) L[at + __popc(b & ((1u << lane) - 1u))] = (HT)u;
    }
    __syncthreads();
  };
  // One round over the list cur[0, A): every listed node pushes along its admissible arcs (to lower
  // neighbours) while it has excess, then, if some is left, moves to 1 + the lowest neighbour it still
  // has residual capacity to. Two ends of one edge never push on it in the same round: each uses its
  // own height from before the round, and a neighbour's height read later can only be larger. A node
  // that relabels may miss an arc opened in the same round by a push into it, so its label may come
  // out too high; it then pushes back along the steep arc. Labels only steer: the search at the end
  // checks that no excess can still reach t, and goes on where it can.
  // Eight lanes per node, one per direction (two spare): one thread going through a node's six
  // directions took some 3,400 cycles a round, a chain of ~500 dependent instructions, whatever the
  // number of nodes.
  const int sub = lane & 7, grp = lane >> 3;
  const int dst = (sub >> 1) == 0 ? 1 : ((sub >> 1) == 1 ? s1 : s2);
  const int doff = (sub & 1) ? dst : -dst;       // this lane's neighbour
  const int rown = (sub < 6 ? sub : 0) * n, rrev = ((sub ^ 1) < 6 ? sub ^ 1 : 0) * n;
  const unsigned lt = (1u << lane) - 1u;
  auto one_round = [&](int A, int w0, int nw) {
    const int bit = k6 & 1;
    HT* cur = bit ? Nl : L;
    HT* nxt = bit ? L : Nl;
    unsigned* fc = flag + (bit ? fw : 0);
    unsigned* fn = flag + (bit ? 0 : fw);
    int* cn = &s_cl[(k6 + 1) % 3];
    for (int i0 = 4 * w0; i0 < A; i0 += 4 * nw) {
      const bool in = i0 + grp < A;
      const int u = in ? (int)ldv<SX>(cur + i0 + grp) : 0;
      const int f = in ? info[u] : 0;
      const int hu = (int)hc[u];
      const long long x0 = in ? ldv<SX>(ex + u) : 0ll;
      const bool ok = sub < 6 && (f >> sub & 1);
      const int v = ok ? u + doff : u;
      const int hv = ok ? (int)hc[v] : ((f & 64) && sub == dsink ? 0 : FAR);
      const long long rr = (in && sub < 6) ? R[rown + u] : 0ll;
      const bool open = rr > 0, adm = open && hu > hv;
      if (in && sub == 0) fc[u >> 5] = 0;  // every node of the word leaves this list
      // the excess goes to the admissible arcs in order of direction
      long long inc = adm ? rr : 0ll;
      int mh = open && !adm ? hv : FAR;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, inc, o, 8);
        if (sub >= o) inc += t;
        mh = min(mh, __shfl_xor_sync(0xffffffffu, mh, o));
      }
      const long long room = x0 - (inc - (adm ? rr : 0ll));
      const long long delta = adm ? (room <= 0 ? 0ll : (room < rr ? room : rr)) : 0ll;
      const long long all = __shfl_sync(0xffffffffu, inc, 7, 8);
      const bool left = x0 > all;          // every arc to a lower neighbour is saturated
      bool add = false;
      int at_v = v;
      if (delta > 0) {
        R[rown + u] = rr - delta;
        if (ok) {  // (flow into t leaves the graph)
          R[rrev + v] += delta;
          add64<SX>(ex + v, delta);
          add = !(atomicOr(&fn[v >> 5], 1u << (v & 31)) >> (v & 31) & 1u);
        }
      }
      if (sub == 7 && in) {
        const long long pushed = left ? all : x0;
        if (pushed > 0) add64<SX>(ex + u, -pushed);
        if (left) {
          const int h = mh >= NH - 1 ? NH : mh + 1;
          hc[u] = (HT)h;
          if (h < NH) {
            add = !(atomicOr(&fn[u >> 5], 1u << (u & 31)) >> (u & 31) & 1u);
            at_v = u;
          }
        }
      }
      const unsigned b = __ballot_sync(0xffffffffu, add);
      if (b) {
        int at = 0;
        if (lane == 0) at = atomicAdd(cn, __popc(b));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (add) nxt[at + __popc(b & lt)] = (HT)at_v;
      }
    }
  };
  __shared__ int s_round, s_k6;
  if (n > 0) {
    bool capped = false;
    relabel_all();
    rebuild();
    while (s_cl[0] > 0 && !capped) {
      for (;;) {
        const int A = s_cl[k6 % 3];
        if (A == 0) break;
        if (A <= CUT_WARP) {
          // Rounds with few active nodes run on warp 0 alone, synchronised by __syncwarp,
          // until the list grows past CUT_WARP or empties, or the round cap or a global relabel is due
          // (the same rounds as the block form, without its barriers).
          __syncthreads();  // every thread has read A before warp 0 moves the counters on
          if (tid < 32) {
            int Aw = A;
            for (;;) {
              nactive += Aw;
              if (lane == 0) s_cl[(k6 + 2) % 3] = 0;
              one_round(Aw, 0, 1);
              __syncwarp();
              ++round;
              k6 = k6 == 5 ? 0 : k6 + 1;
              Aw = s_cl[k6 % 3];
              __syncwarp();
              if (Aw == 0 || Aw > CUT_WARP || round >= a.round_cap || round % a.gr_period == 0 ||
                  round > CUT_SAFE)
                break;
            }
            if (lane == 0) { s_round = round; s_k6 = k6; }
          }
          __syncthreads();
          round = s_round;
          k6 = s_k6;
        } else {
          nactive += A;
          if (tid == 0) s_cl[(k6 + 2) % 3] = 0;
          one_round(A, tid >> 5, nthr >> 5);
          __syncthreads();
          ++round;
          k6 = k6 == 5 ? 0 : k6 + 1;
        }
        if (round >= a.round_cap && s_cl[k6 % 3] > 0) { capped = true; break; }
        if (round % a.gr_period == 0 || round > CUT_SAFE) break;
      }
      __syncthreads();
      relabel_all();
      rebuild();
    }
    if (capped && tid == 0) iq_dev_fail(a.status, IQ_ERR_CUTCAP);
  }

  if (a.stats && tid == 0) {
    const long long t_end = clock64();
    atomicAdd(a.stats + ST_CUT_TSETUP, (unsigned long long)(t_setup - t_start));
    atomicAdd(a.stats + ST_CUT_TGR, (unsigned long long)t_gr);
    atomicAdd(a.stats + ST_CUT_TROUNDS, (unsigned long long)(t_end - t_setup - t_gr));
    atomicAdd(a.stats + ST_CUT_ROUNDS, (unsigned long long)round);
    atomicAdd(a.stats + ST_CUT_NODES, (unsigned long long)nf);
    atomicAdd(a.stats + ST_CUT_ACTIVE, (unsigned long long)nactive);
    atomicAdd(a.stats + ST_CUT_LEVELS, (unsigned long long)levels);
    atomicAdd(a.stats + ST_CUT_CTAS, 1ull);
    atomicMax(a.stats + ST_CUT_MAXROUNDS, (unsigned long long)round);
    atomicMax(a.stats + ST_CUT_MAXLEVELS, (unsigned long long)levels);
  }
  // ---- mask: not sink side ----
  uint8_t* out = a.out + ((int64_t)y * 6 + s_id) * a.slabmax;
  for (int u = tid; u < nf; u += nthr) {
    const int x = u % e0, yy = (u / e0) % e1, z = u / f2;
    const int cd = d == 0 ? x : (d == 1 ? yy : z);
    int M;
    if (cd == 0) M = 1;
    else if (cd == Ld - 1) M = 0;
    else M = (int)hc[(x - wd0) + s1 * (yy - wd1) + s2 * (z - wd2)] >= NH ? 1 : 0;
    out[u] = (uint8_t)(sl.next ? !M : M);
  }
}

}  // namespace

namespace {
constexpr int64_t CUT_SHORT_MAX = 32767;  // largest slab with 16-bit heights and indices
}  // namespace

size_t iq_cut_scratch_bytes(int64_t nodes) {
  // either form of scratch, for a slab of that many voxels whatever its cut dimension
  const int hb = nodes <= CUT_SHORT_MAX ? 2 : 4;
  return std::max(cut_layout(nodes, nodes, hb).end, cut_layout2(nodes, nodes, hb).gend);
}

int iq_launch_cut(iq_ctx* ctx, const CutLaunch& L) {
  const int nslab_max = L.tasks ? L.nslab_max : L.t0.nslab;
  if (nslab_max <= 0 || L.nreal <= 0 || L.ntask <= 0) return IQ_OK;
  CutArgs a;
  a.t0 = L.t0;
  a.tasks = L.tasks;
  a.nreal = L.nreal;
  a.sim = L.sim; a.sx = L.sim_dims.x; a.sy = L.sim_dims.y; a.sim_rs = L.sim_rstride;
  a.ti = L.ti; a.tix = L.ti_dims.x; a.tiy = L.ti_dims.y;
  a.dx = L.dist_dims.x; a.dy = L.dist_dims.y;
  a.rind = L.rind;
  a.A = L.A; a.B = L.B;
  a.out = L.out; a.slabmax = L.slabmax;
  a.status = L.status;
  a.round_cap = L.round_cap;
  a.stats = L.stats;
  a.gr_period = L.gr_period > 0 ? L.gr_period : 16;
  const int64_t nmax = L.slabmax, nint = L.intmax >= 0 ? std::min(L.intmax, nmax) : nmax;
  const bool narrow = nmax <= CUT_SHORT_MAX;
  const int hb = narrow ? 2 : 4;
  const size_t need = cut_layout(nint, nmax, hb).end;
  // dynamic shared memory may use the opt-in maximum minus the kernel's static part
  auto limit_of = [&](void (*k)(CutArgs), int& lim) -> int {
    int dev = 0, v = 0;
    IQ_CUDA_OK(cudaGetDevice(&dev));
    IQ_CUDA_OK(cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa;
    IQ_CUDA_OK(cudaFuncGetAttributes(&fa, k));
    lim = v - (int)fa.sharedSizeBytes;
    IQ_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
    return IQ_OK;
  };
  // (a slab of 32-bit heights has more interior nodes than shared memory holds residuals for)
  const int threads = (L.threads == 256 || L.threads == 1024) ? L.threads : 512;
  void (*kern)(CutArgs) = threads == 256   ? cut_kernel<short, 0, 256>
                          : threads == 512 ? cut_kernel<short, 0, 512>
                                           : cut_kernel<short, 0, 1024>;
  int smem_limit = 0;
  if (int rc = limit_of(kern, smem_limit)) return rc;
  size_t dyn = 0;
  a.scratch = nullptr;
  a.scratch_per_cta = 0;
  if (narrow && (int64_t)need <= smem_limit) {
    dyn = need;
  } else {
    if (!L.scratch || L.scratch_per_cta < (int64_t)iq_cut_scratch_bytes(nmax))
      return iq_set_error(IQ_ERR_LIMIT, "graph cut slab of %lld nodes needs global scratch",
                          (long long)nmax);
    a.scratch = (char*)L.scratch;
    a.scratch_per_cta = L.scratch_per_cta;
    void (*k2)(CutArgs) = cut_kernel<short, 2, CUT_MAX_THREADS>;
    int lim2 = 0;
    if (int rc = limit_of(k2, lim2)) return rc;
    if (narrow && (int64_t)cut_layout2(nint, nmax, hb).end <= lim2) {
      kern = k2;
      dyn = cut_layout2(nint, nmax, hb).end;
    } else {
      kern = narrow ? cut_kernel<short, 1, CUT_MAX_THREADS> : cut_kernel<int, 1, CUT_MAX_THREADS>;
    }
  }
  dim3 grid((unsigned)nslab_max, (unsigned)(L.ntask * L.nreal));
  iq_timer_start(ctx, "graphcut");
  kern<<<grid, threads, dyn, ctx->stream>>>(a);
  iq_timer_stop(ctx, "graphcut", 0);
  iq_count(ctx);
  IQ_CUDA_OK(cudaGetLastError());
  return IQ_OK;
}
