// Host-side plan of the Toeplitz tensor-core correlation (iq_corr_tz.cu), used by iq_simulate and
// iq_fastdistance.
#pragma once

#include <string.h>

#include <algorithm>
#include <map>
#include <vector>

#include "iq_internal.h"

namespace {

// Groups of columns for the Toeplitz tensor-core correlation (iq_corr_tz.cu): host arrays filled
// launch by launch, uploaded once.
struct TzPlan {
  Dim3 img, tile;
  std::vector<TcBox> boxes;     // the masks the columns' box indexes
  bool split = false;
  std::vector<TzGroup> groups;
  std::vector<TzStage> stages;
  std::vector<uint32_t> chunks;
  std::vector<TcCol> cols;
  std::vector<int64_t> touched; // per mask: most K-steps of a list that hold one of its offsets
  struct Ref { int stage0, nstage, nstep, chunk0; };
  std::map<std::vector<int>, Ref> lists;
  struct Launch { int group0, ngroup, Nmax, ncols; int64_t units, bytes; double flops, mma; };
  std::vector<Launch> launches;
  // What upload() copies from: a copy of pageable memory may still be reading it when the call returns,
  // so the plan outlives the stream's next synchronization.
  std::vector<char> host;
  // device copies
  const TzGroup* d_groups = nullptr;
  const TzStage* d_stages = nullptr;
  const uint32_t* d_chunks = nullptr;
  const TcBox* d_boxes = nullptr;
  const TcCol* d_cols = nullptr;

  Ref list_of(const std::vector<int>& set) {
    auto it = lists.find(set);
    if (it != lists.end()) return it->second;
    std::vector<TcBox> bx;
    for (int b : set) bx.push_back(boxes[b]);
    TzList l;
    iq_tz_list(img, tile, bx.data(), (int)bx.size(), l);
    touched.resize(boxes.size(), 0);
    for (size_t i = 0; i < set.size(); ++i)
      touched[set[i]] = std::max(touched[set[i]], l.touched[i]);
    Ref r{(int)stages.size(), (int)l.stage.size(), (int)l.nstep, (int)chunks.size()};
    stages.insert(stages.end(), l.stage.begin(), l.stage.end());
    chunks.insert(chunks.end(), l.chunk.begin(), l.chunk.end());
    lists[set] = r;
    return r;
  }
  // Launches over `c` (columns grouped by mask): groups of balanced, even width, as many to a launch
  // as `cap` bytes of packed templates hold (one at least; the launches follow one another in the same
  // buffer). Split data take groups of at most 16 columns, so that the two accumulators of two
  // 1024-position blocks fill TMEM (the templates of a K-step then serve 2048 positions).
  void add_launches(const std::vector<TcCol>& c, double flops, int64_t cap) {
    const int64_t most = split ? IQ_TZ_COLS / 2 : IQ_TZ_COLS, n = (int64_t)c.size();
    const int64_t ng = (n + most - 1) / most;
    const int64_t per = ng > 0 ? ((n + ng - 1) / ng + 1) / 2 * 2 : 0;
    Launch L{};
    for (int64_t q = 0; q < n; q += per) {
      const int64_t m = std::min(per, n - q);
      std::vector<int> set;
      for (int64_t i = q; i < q + m; ++i)
        if (set.empty() || set.back() != c[i].box) set.push_back(c[i].box);
      std::sort(set.begin(), set.end());
      set.erase(std::unique(set.begin(), set.end()), set.end());
      const Ref r = list_of(set);
      TzGroup g{};
      g.ncol = (int32_t)(m + (m & 1));
      g.N = 8 * g.ncol;
      g.stage0 = r.stage0; g.nstage = r.nstage; g.nstep = r.nstep; g.chunk0 = r.chunk0;
      const int64_t bytes = ((int64_t)g.nstep * 32 * g.N * (split ? 2 : 1) + 255) / 256 * 256;
      if (L.ngroup > 0 && L.bytes + bytes > cap) {
        launches.push_back(L);
        L = Launch{};
      }
      if (L.ngroup == 0) L.group0 = (int)groups.size();
      g.col0 = (int32_t)cols.size();
      cols.insert(cols.end(), c.begin() + q, c.begin() + q + m);
      if (m & 1) cols.push_back(TcCol{-1, nullptr, nullptr, nullptr, 0, 0});
      g.boff = L.bytes;
      L.bytes += bytes;
      L.units = std::max<int64_t>(L.units, (int64_t)g.nstep * 2 * g.N);
      L.Nmax = std::max(L.Nmax, (int)g.N);
      L.mma += 2.0 * 128 * 16 * (double)g.nstep * g.N;
      L.flops += flops * (double)m / (double)n;
      L.ncols += (int)m;
      L.ngroup++;
      groups.push_back(g);
    }
    if (L.ngroup > 0) launches.push_back(L);
  }
  // K-steps of mask b (0: no column has it)
  int64_t steps_of(size_t b) const { return b < touched.size() ? touched[b] : 0; }
  int64_t max_bytes() const {
    int64_t b = 1;
    for (const Launch& l : launches) b = std::max(b, l.bytes);
    return (b + 255) / 256 * 256;
  }
  int upload(iq_ctx* ctx, int slot, cudaStream_t st) {
    auto pad = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t sz[5] = {sizeof(TzGroup) * groups.size(), sizeof(TzStage) * stages.size(),
                          4 * chunks.size(), sizeof(TcBox) * boxes.size(), sizeof(TcCol) * cols.size()};
    const void* src[5] = {groups.data(), stages.data(), chunks.data(), boxes.data(), cols.data()};
    size_t total = 0;
    for (size_t b : sz) total += pad(b);
    host.assign(total + 1, 0);
    char* d = (char*)iq_scratch(ctx, slot, total + 256);
    if (!d) return IQ_ERR_ALLOC;
    size_t at[5], off = 0;
    for (int i = 0; i < 5; ++i) {
      at[i] = off;
      if (sz[i]) memcpy(host.data() + off, src[i], sz[i]);
      off += pad(sz[i]);
    }
    IQ_CUDA_OK(cudaMemcpyAsync(d, host.data(), total, cudaMemcpyHostToDevice, st));
    d_groups = (const TzGroup*)(d + at[0]);
    d_stages = (const TzStage*)(d + at[1]);
    d_chunks = (const uint32_t*)(d + at[2]);
    d_boxes = (const TcBox*)(d + at[3]);
    d_cols = (const TcCol*)(d + at[4]);
    return IQ_OK;
  }
  // launch l of the plan
  int launch(iq_ctx* ctx, const Launch& l, const void* image, Dim3 out, const float* a2,
             const float* grid, Dim3 gdims, void* B, const IqValueStats& is, const IqValueStats& ts) const {
    TzLaunch T;
    T.img = image; T.img_dims = img; T.out_dims = out; T.tile = tile;
    T.groups = d_groups + l.group0; T.ngroup = l.ngroup; T.Nmax = l.Nmax;
    T.stages = d_stages; T.chunks = d_chunks; T.boxes = d_boxes; T.a2 = a2;
    T.grid = grid; T.grid_dims = gdims; T.cols = d_cols; T.B = B; T.max_units = l.units;
    T.img_stats = is; T.tmpl_stats = ts; T.flops = l.flops; T.mma_flops = l.mma; T.ncols = l.ncols;
    return iq_launch_corr_tz(ctx, T);
  }
};

}  // namespace
