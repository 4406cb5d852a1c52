// batch.cu — the batched campaign engine: many independent cells (Hamming,
// Lee, torus, grid; any sizes) resident at once, and their count, gain and
// loss transforms run as one graph of persistent launches.
//
// The reference runs a campaign as one process per cell, each with its own
// singleton plugin context (coldcore src/coldcore/campaign.py:186-221,
// src/include/coldcore/plugin.h:8-10), so every cell pays its own context,
// allocations and per-axis launches.  Here a batch owns one device arena;
// each cell's transforms are split into passes (one per axis group) and
// passes into tiles, and the whole step — for every cell: recount from its
// code, the uncovered/deficit count, gain map + maximum, loss map + maximum
// — is one CUDA graph: a persistent launch per register kernel over a
// level-ordered work table (batch_groups.cu), one of batch_kernel
// (transform_group.cu) for the cells without such a kernel, and the big
// cells' own launches, on forked streams.  Handles, not the v1 singleton:
// batches never touch the dct_* cell.
//
// Tile size is the one schedule knob (shared memory per tile); the
// autotuner times a few and keeps the fastest.
#include <algorithm>
#include <climits>
#include <cstring>
#include <map>
#include <unordered_map>
#include <vector>

#include "../../include/coldcore_b200/plugin.h"
#include "engine.h"

using namespace cc;

namespace {

struct Cell {
  Geometry g;
  int R1 = 1;
  long long plane = 0;
  std::vector<long long> code;       // sorted
  // device pointers into the arena
  int32_t *layers = nullptr, *gain = nullptr, *loss = nullptr;
  uint16_t *cnt = nullptr;
  long long *dcode = nullptr, *bounds = nullptr;
  long long nbounds = 0;
  int first_pass = 0, npass = 0;     // global pass range (small cells)
  int kid = -1;                      // register kernel of a small cell's passes
  int gain_pass = 0, ngain = 0;      // its gain transform alone (greedy)
  double gain_us = 0;                // estimate of that transform's time
  bool regs = false;                 // one axis size, with a register kernel
  bool big = false;                  // own register-blocked launches
  int side = 0;                      // its side stream (big cells)
  bool tuned = false;                // fast[] tuned (big cells)
  std::vector<GroupPlan> fast[3];    // recount, gain, loss (big cells)
  // codes may be replaced between launches (dct_batch_set_code): the
  // device buffer holds code_cap words, its length lives on the device
  long long code_cap = 0;
  long long *dncode = nullptr;
  // support table for the cell's walks (dct_batch_set_table), SoA slots
  int32_t *dtbl_base = nullptr, *dtbl = nullptr;
  uint32_t *dpk = nullptr;           // its packed form (pack_walk)
  int4 *dent = nullptr;
  int noff = 0;
  int slots = 0;
  long long tlen = 0;
  bool ball_ok = false;              // the table is exactly the metric ball
  bool moved = false;                // cnt or gain changed since the last step
};

// one cell's code slices per first-group tile, computed on the device from
// the code length on the device (so a replaced code needs no re-capture)
struct BoundsJob {
  const long long *code;
  const long long *ncode;
  long long tile_words, ntiles;
  long long *bounds;
};

__global__ void k_batch_bounds(const BoundsJob *jobs) {
  const BoundsJob j = jobs[blockIdx.x];
  const long long n = *j.ncode;
  for (long long t = threadIdx.x; t <= j.ntiles; t += blockDim.x) {
    const long long x = t * j.tile_words;
    long long lo = 0, hi = n;
    while (lo < hi) {
      const long long md = (lo + hi) >> 1;
      if (j.code[md] < x) lo = md + 1; else hi = md;
    }
    j.bounds[t] = lo;
  }
}

// Cells of at least 2^16 words whose axes all have one size with a
// register-blocked kernel run as their own launches (captured on forked
// streams of the same graph); smaller cells share the persistent kernel.
// (CC_BATCH_BIG: log2 of that threshold; CC_BATCH_ITEM: the words of one
// work item of the persistent kernels, at least)
long long big_cell_words() {
  const char *e = getenv("CC_BATCH_BIG");
  const int lg = e ? atoi(e) : 16;
  return 1LL << (lg < 8 ? 8 : lg > 40 ? 40 : lg);
}
// (register kernels: a step of 256 cells of 10^3..10^5 words took 0.95 ms
// with items of 2,048 words, 0.99 with 4,096, 1.33 with 8,192, 1.89 with
// 16,384: one tile an item keeps the most CTAs busy)
long long item_words(bool regs) {
  const char *e = getenv("CC_BATCH_ITEM");
  const long long w = e ? atoll(e) : regs ? 2048 : 32768;
  return w < 256 ? 256 : w;
}
// side streams the big cells are spread over (CC_BATCH_STREAMS, 1..16,
// default 4: 4, 8 and 16 timed within 3% of each other on the 256-cell
// campaign), largest cells first onto the least loaded stream
constexpr int kSideStreams = 16;
int side_streams() {
  const char *e = getenv("CC_BATCH_STREAMS");
  const int n = e ? atoi(e) : 4;
  return n < 1 ? 1 : n > kSideStreams ? kSideStreams : n;
}

// one persistent launch: the small cells one kernel serves (kid -1: the
// runtime-size tiles)
struct Group {
  int kid = -1;
  long long item0 = 0, nitems = 0;   // its range of the item table
  size_t smem = 0;
  int grid = 1;
  int side = -1;                     // side stream, -1 the main stream
  int next = 0;                      // its claim counter
};

struct Batch {
  std::vector<Cell> cells;
  bool built = false;
  char *arena = nullptr;
  size_t arena_bytes = 0;
  std::vector<GroupPlan> passes;     // the step's nstep, then gain alone
  int nstep = 0;
  std::vector<int> dep;
  std::vector<unsigned> need;
  std::vector<int> pass_cell;
  std::vector<Group> groups;         // persistent launches, one a kernel
  // the gain transforms alone, without reductions: the greedy's rebuilds
  std::vector<Group> gain_groups;
  GroupArgs *d_passes = nullptr;
  int *d_dep = nullptr;
  unsigned *d_need = nullptr;
  int *d_pass_cell = nullptr;
  int4 *d_items = nullptr;
  long long nitems = 0;
  unsigned *d_done = nullptr;
  unsigned long long *d_next = nullptr;
  int *d_err = nullptr;
  long long *d_scal = nullptr;       // per cell: deficit, gain max, loss max
  long long *d_bounds = nullptr;     // per-tile code slices of every cell
  long long bounds_cap = 0;
  long long *d_ncode = nullptr;      // per cell: its code length
  BoundsJob *d_jobs = nullptr;       // per cell: its bounds job
  // staging of the per-cell calls (updates, gathers, extraction)
  long long *d_words = nullptr;
  int32_t *d_out = nullptr;
  void *d_ext = nullptr;
  int32_t *d_extv = nullptr;
  long long ext_cap = 0;
  long long *d_count = nullptr;
  // the greedy's workspace, grown to the largest call, and its state ring
  char *d_greedy = nullptr;
  size_t greedy_cap = 0;
  char *h_greedy = nullptr;
  size_t h_greedy_cap = 0;
  cudaEvent_t ev_greedy[2] = {nullptr};
  size_t tile_budget = 48 * 1024;
  int grid = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t side[kSideStreams] = {nullptr};
  cudaEvent_t fork = nullptr, join[kSideStreams] = {nullptr};
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  float tuned_ms = 0;
  int nside = 4;                     // side streams of the big cells
  int nnext = 0;                     // claim counters of d_next
};

std::unordered_map<long long, Batch *> g_batches;
long long g_next_handle = 1;

Batch *get(long long h) {
  auto it = g_batches.find(h);
  return it == g_batches.end() ? nullptr : it->second;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Groups of consecutive axes whose tile fits `budget` bytes of shared
// memory (runtime-size tile kernel: any axis size up to 16).
std::vector<GroupArgs> plan_cell(const Cell &c, size_t budget) {
  std::vector<GroupArgs> out;
  const Geometry &g = c.g;
  long long reach = 0;
  int j = 0;
  while (j < g.n) {
    GroupArgs a{};
    a.layers = c.layers;
    a.plane = c.plane;
    a.cnt = c.cnt;
    a.inner = g.pw[j];
    a.W = a.inner >= 32 ? 32 : (int)a.inner;
    a.prob = g.prob;
    a.R = g.R;
    a.mu = g.mu;
    long long mid = 1;
    while (j + a.k < g.n && a.k < kMaxRounds) {
      GroupArgs t = a;
      const long long mid2 = mid * g.ax[j + a.k];
      const long long outer = g.space / (a.inner * mid2);
      t.k = a.k + 1;
      t.mid = (int)mid2;
      t.Bo = a.W >= 32 ? 1
             : (int)std::max<long long>(1, std::min<long long>(
                   outer, 1024 / (a.W * mid2)));
      if (a.k > 0 && group_smem_bytes(t, c.R1) > budget) break;
      a = t;
      mid = mid2;
    }
    for (int t = 0; t < a.k; t++) a.qax[t] = g.ax[j + t];
    a.outer = g.space / (a.inner * (long long)a.mid);
    a.nchunk = (a.inner + a.W - 1) / a.W;
    a.ntiles = (a.outer + a.Bo - 1) / a.Bo * a.nchunk;
    long long reach2 = reach;
    for (int t = 0; t < a.k; t++)
      reach2 += g.prob == kLee ? g.ax[j + t] / 2 : 1;
    const bool layered = c.R1 > 1;
    a.lin = layered ? (int)std::min<long long>(reach, g.R) + 1 : 1;
    a.lout = layered ? (int)std::min<long long>(reach2, g.R) + 1 : 1;
    out.push_back(a);
    reach = reach2;
    j += a.k;
  }
  return out;
}

// |B| of the metric ball (the most words one codeword covers): the
// coefficient sum up to R of prod_j (per-axis weight enumerator) for the
// sum metrics, prod_j min(2R+1, a_j) for the L-infinity families
long long ball_cardinality(const Geometry &g) {
  if (g.prob == kTorus || g.prob == kGrid) {
    long long b = 1;
    for (int j = 0; j < g.n; j++) b *= std::min(2 * g.R + 1, g.ax[j]);
    return b;
  }
  std::vector<long long> poly(g.R + 1, 0);
  poly[0] = 1;
  for (int j = 0; j < g.n; j++) {
    std::vector<long long> nx(g.R + 1, 0);
    const int a = g.ax[j];
    for (int w = 0; w <= g.R; w++) {
      if (!poly[w]) continue;
      for (int d = 0; d < a; d++) {
        const int c = d < a - d ? d : a - d;       // circular weight
        const int e = g.prob == kHamming ? (d ? 1 : 0) : c;
        if (w + e <= g.R) nx[w + e] += poly[w];
      }
    }
    poly = nx;
  }
  long long t = 0;
  for (long long v : poly) t += v;
  return t;
}

void release(Batch *b) {
  if (b->stream) cudaStreamSynchronize(b->stream);
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->exec = nullptr;
  b->graph = nullptr;
  auto F = [](void *p) { if (p) cudaFree(p); };
  F(b->arena); F(b->d_passes); F(b->d_dep); F(b->d_need); F(b->d_items);
  F(b->d_pass_cell);
  F(b->d_done); F(b->d_next); F(b->d_err); F(b->d_scal); F(b->d_bounds);
  F(b->d_ncode); F(b->d_jobs); F(b->d_words); F(b->d_out); F(b->d_ext);
  F(b->d_extv); F(b->d_count); F(b->d_greedy);
  if (b->h_greedy) cudaFreeHost(b->h_greedy);
  for (auto &ev : b->ev_greedy) {
    if (ev) cudaEventDestroy(ev);
    ev = nullptr;
  }
  b->d_greedy = b->h_greedy = nullptr;
  b->greedy_cap = b->h_greedy_cap = 0;
  for (Cell &c : b->cells) {
    F(c.dtbl_base);
    c.dtbl_base = c.dtbl = nullptr; c.dpk = nullptr; c.dent = nullptr;
  }
  b->d_ncode = nullptr; b->d_jobs = nullptr; b->d_words = nullptr;
  b->d_out = nullptr; b->d_ext = nullptr; b->d_extv = nullptr;
  b->d_count = nullptr; b->ext_cap = 0;
  b->d_bounds = nullptr;
  b->bounds_cap = 0;
  b->d_pass_cell = nullptr;
  b->arena = nullptr; b->d_passes = nullptr; b->d_dep = nullptr;
  b->d_need = nullptr; b->d_items = nullptr; b->d_done = nullptr;
  b->d_next = nullptr; b->d_err = nullptr; b->d_scal = nullptr;
  b->built = false;
}

// Per-launch tuning of the cells with their own launches, as the singleton
// tunes its plan: every variant group_variants offers for a launch (register
// block, row width, prefetching, streamed form, CTA width) is timed on the
// batch stream (three launches after a warm one) and the fastest is kept.
// Cells of at least 2^CC_BATCH_TUNE words (default 16: every such cell; 0
// turns it off, as does CC_TUNE=0), once per batch.  On the 256-cell
// campaign it took the step from 22.7 ms to 17.9 ms for under a second of
// build time.  A variant run again works in place on
// the cell's planes, which only scrambles values; every step recomputes
// from the code.
int tune_big_cells(Batch *b) {
  const char *te = getenv("CC_TUNE");
  if (te && atoi(te) == 0) return 0;
  const char *be = getenv("CC_BATCH_TUNE");
  const int lg = be ? atoi(be) : 16;
  if (lg <= 0) return 0;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  CC_CK(cudaEventCreate(&e0));
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    cudaGetLastError();
    return -1;
  }
  int rc = 0;
  for (Cell &c : b->cells) {
    if (rc) break;
    if (!c.big || c.tuned || c.g.space < (1LL << lg) || c.fast[0].empty())
      continue;
    // the recount's first group reads its code slices: bounds for its tiles
    const GroupArgs &a0 = c.fast[0][0].a;
    rc = launch_code_bounds(c.dcode, (long long)c.code.size(),
                            (long long)a0.Bo * a0.mid * a0.inner, a0.ntiles,
                            c.bounds, b->stream);
    for (int t = 0; t < 3 && !rc; t++)
      for (size_t gi = 0; gi < c.fast[t].size() && !rc; gi++) {
        const std::vector<GroupPlan> vars =
            group_variants(c.fast[t][gi], c.R1, 220 << 10);
        if (vars.size() < 2) continue;
        float bv = 1e30f;
        size_t bi = 0;
        for (size_t vi = 0; vi < vars.size() && !rc; vi++) {
          const GroupPlan &v = vars[vi];
          if ((rc = prepare_group(v))) break;
          rc = launch_group(v, b->stream);
          if (rc == -9) { rc = 0; continue; }   // a form the launcher refused
          if (rc) break;
          if (cudaEventRecord(e0, b->stream) != cudaSuccess) { rc = -1; break; }
          for (int r = 0; r < 3 && !rc; r++) rc = launch_group(v, b->stream);
          if (rc) break;
          float ms = 0;
          if (cudaEventRecord(e1, b->stream) != cudaSuccess ||
              cudaEventSynchronize(e1) != cudaSuccess ||
              cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
            rc = -1;
            break;
          }
          if (ms < bv) { bv = ms; bi = vi; }
        }
        if (!rc) c.fast[t][gi] = vars[bi];
      }
    c.tuned = !rc;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc == -1) cudaGetLastError();
  return rc;
}

// passes + level-ordered work table for the current tile budget
int make_schedule(Batch *b) {
  b->passes.clear();
  b->dep.clear();
  b->need.clear();
  b->pass_cell.clear();
  b->groups.clear();
  b->gain_groups.clear();
  // per kernel (-1 first): its passes by level
  typedef std::map<int, std::vector<std::vector<int>>> ByKid;
  ByKid by_kid, gain_by_kid;
  const char *tma_env = getenv("CC_TMA");
  const bool streams_off = tma_env && atoi(tma_env) == 0;
  for (size_t i = 0; i < b->cells.size(); i++) {
    Cell &c = b->cells[i];
    c.first_pass = (int)b->passes.size();
    c.npass = 0;
    if (c.big && c.tuned) continue;     // its tuned launches stand
    if (c.big) {
      // 16-bit planes between launches (and packed pairs where the
      // planner can) when every layer value stays below 2^16: always for
      // the recount (the occurrence bound checked at add), for the
      // predicate transforms when the ball has at most 65,535 words
      const long long ball = ball_cardinality(c.g);
      for (int t = 0; t < 3; t++) {
        Knobs kn{100 * 1024, 1};
        kn.half = c.R1 >= 2 && (t == 0 || ball <= 65535) ? 1 : 0;
        PlanPtrs ptr{c.layers, c.plane, c.cnt, c.dcode,
                     (long long)c.code.size(), t == 1 ? c.gain : c.loss};
        ptr.layers16 = reinterpret_cast<uint16_t *>(c.layers + c.plane);
        const int src = t == 0 ? kSrcCode : kSrcCnt;
        const int dst = t == 0 ? kDstCnt : kDstMap;
        const Geometry tg = transform_geometry(c.g);
        c.fast[t] = plan_groups(tg, c.R1, ptr, src, dst, kn);
        // the streamed forms where they apply (CC_TMA=0 keeps the
        // register kernels): a ternary cell's padded plan, else every
        // group a streamed form serves
        if (!streams_off && kn.half &&
            !pad_plan(c.fast[t], tg, ptr, dst, c.R1,
                      (long long)(c.R1 - 1) * c.plane * 2)) {
          stream_groups(c.fast[t], c.R1);
          u8_plan(c.fast[t], c.R1, (long long)(c.R1 - 1) * c.plane * 2);
        }
        for (auto &gp : c.fast[t]) {
          if (prepare_group(gp)) return -1;
          if (gp.a.tma && gp.grid < 1) {
            // sized here: the graph capture records launches only
            const int per_sm = std::max(1, tma_blocks_per_sm(gp));
            gp.grid = (int)std::max<long long>(1, std::min<long long>(
                gp.a.ntiles, (long long)sm_count() * per_sm));
          }
          gp.a.pmode = kPredEq;
          gp.a.ptarget = t == 1 ? 0 : 1;
          if (c.g.mu > 1) gp.a.pmode = t == 1 ? kPredDef : kPredCrit;
        }
      }
      continue;
    }
    // a small cell: three transforms of the same groups on one kernel
    std::vector<std::vector<GroupPlan>> plans(3);
    c.kid = -1;
    if (c.regs) {
      const long long ball = ball_cardinality(c.g);
      for (int t = 0; t < 3; t++) {
        Knobs kn{b->tile_budget, 0};
        kn.half = c.R1 >= 2 && (t == 0 || ball <= 65535) ? 1 : 0;
        PlanPtrs ptr{c.layers, c.plane, c.cnt, c.dcode,
                     (long long)c.code.size(), t == 1 ? c.gain : c.loss};
        ptr.layers16 = reinterpret_cast<uint16_t *>(c.layers + c.plane);
        plans[t] = plan_groups(transform_geometry(c.g), c.R1, ptr,
                               t == 0 ? kSrcCode : kSrcCnt,
                               t == 0 ? kDstCnt : kDstMap, kn);
        if (plans[t].empty()) return -1;
      }
      c.kid = plans[0][0].kernel;
    } else {
      for (const GroupArgs &ga : plan_cell(c, b->tile_budget)) {
        GroupPlan p;
        p.a = ga;
        p.kernel = -1;
        p.threads = 256;
        p.smem = group_smem_bytes(ga, c.R1);
        p.grid = (int)std::min<long long>(ga.ntiles,
                                          (long long)sm_count() * 4);
        for (auto &v : plans) v.push_back(p);
      }
    }
    auto &by_level = by_kid[c.kid];
    for (int t = 0; t < 3; t++) {            // recount, gain, loss
      const int G = (int)plans[t].size();
      for (int k = 0; k < G; k++) {
        GroupPlan p = plans[t][k];
        GroupArgs &a = p.a;
        const bool first = k == 0, last = k == G - 1;
        a.src = !first ? kSrcLayers : t == 0 ? kSrcCode : kSrcCnt;
        a.dst = !last ? kDstLayers : t == 0 ? kDstCnt : kDstMap;
        a.code = c.dcode;
        a.ncode = (long long)c.code.size();
        a.code_bounds = c.bounds;
        a.pmode = kPredEq;
        a.ptarget = t == 1 ? 0 : 1;
        if (c.g.mu > 1) a.pmode = t == 1 ? kPredDef : kPredCrit;
        a.map = t == 1 ? c.gain : c.loss;
        a.red = b->d_scal + 3 * i + t;
        a.red_mode = last ? (t == 0 ? 1 : 2) : 0;
        if (prepare_group(p)) return -1;
        const int pid = (int)b->passes.size();
        b->passes.push_back(p);
        b->pass_cell.push_back((int)i);
        b->dep.push_back(pid == c.first_pass ? -1 : pid - 1);
        b->need.push_back((unsigned)a.ntiles);
        const int level = pid - c.first_pass;
        if ((int)by_level.size() <= level) by_level.resize(level + 1);
        by_level[level].push_back(pid);
      }
    }
    c.npass = (int)b->passes.size() - c.first_pass;
  }
  b->nstep = (int)b->passes.size();
  // the gain transforms again, on their own
  for (size_t i = 0; i < b->cells.size(); i++) {
    Cell &c = b->cells[i];
    double bytes = 0;
    if (c.big)
      for (const auto &gp : c.fast[1]) bytes += group_bytes(gp.a);
    const int G = c.npass / 3;
    c.gain_pass = (int)b->passes.size();
    c.ngain = G;
    for (int k = 0; k < G; k++) {
      GroupPlan p = b->passes[c.first_pass + G + k];
      p.a.red_mode = 0;
      bytes += group_bytes(p.a);
      const int pid = (int)b->passes.size();
      b->passes.push_back(p);
      b->pass_cell.push_back((int)i);
      b->dep.push_back(k == 0 ? -1 : pid - 1);
      b->need.push_back((unsigned)p.a.ntiles);
      auto &by_level = gain_by_kid[c.kid];
      if ((int)by_level.size() <= k) by_level.resize(k + 1);
      by_level[k].push_back(pid);
    }
    c.gain_us = 1.0 + bytes / 1.8e6;
  }
  // big cells onto the side streams: largest (algorithmic bytes) first,
  // each onto the least loaded stream
  {
    b->nside = side_streams();
    std::vector<std::pair<long long, size_t>> order;
    for (size_t i = 0; i < b->cells.size(); i++) {
      const Cell &c = b->cells[i];
      if (!c.big) continue;
      long long by = 0;
      for (int t = 0; t < 3; t++)
        for (const auto &gp : c.fast[t]) by += group_bytes(gp.a);
      order.push_back({by, i});
    }
    std::sort(order.begin(), order.end(),
              [](const std::pair<long long, size_t> &x,
                 const std::pair<long long, size_t> &y) {
                return x.first != y.first ? x.first > y.first
                                          : x.second < y.second;
              });
    std::vector<long long> load(b->nside, 0);
    for (const auto &o : order) {
      int k = 0;
      for (int j = 1; j < b->nside; j++)
        if (load[j] < load[k]) k = j;
      b->cells[o.second].side = k;
      load[k] += o.first;
    }
  }
  // tile slices of each cell's code for this schedule's first groups
  auto first_tiles = [&](const Cell &c) {
    return c.big ? c.fast[0][0].a.ntiles
                 : b->passes[c.first_pass].a.ntiles;
  };
  long long nb = 0;
  for (const Cell &c : b->cells) nb += first_tiles(c) + 1;
  if (nb > b->bounds_cap) {
    if (b->d_bounds) cudaFree(b->d_bounds);
    b->d_bounds = nullptr;
    CC_CK(cudaMalloc(&b->d_bounds, (size_t)nb * 8));
    b->bounds_cap = nb;
  }
  nb = 0;
  for (Cell &c : b->cells) {
    c.bounds = b->d_bounds + nb;
    c.nbounds = first_tiles(c) + 1;
    nb += c.nbounds;
    for (int p = c.first_pass; p < c.first_pass + c.npass; p++)
      b->passes[p].a.code_bounds = c.bounds;
    if (c.big)
      for (int t = 0; t < 3; t++)
        for (auto &gp : c.fast[t]) gp.a.code_bounds = c.bounds;
  }
  {
    const int rc = tune_big_cells(b);
    if (rc) return rc;
  }
  // the bounds job of every cell (its first group's tiles)
  std::vector<BoundsJob> jobs;
  for (const Cell &c : b->cells) {
    BoundsJob j{};
    j.code = c.dcode;
    j.ncode = c.dncode;
    j.bounds = c.bounds;
    if (c.big) {
      const GroupArgs &a0 = c.fast[0][0].a;
      j.tile_words = (long long)a0.Bo * a0.mid * a0.inner;
      j.ntiles = a0.ntiles;
    } else {
      const GroupArgs &a0 = b->passes[c.first_pass].a;
      j.tile_words = (long long)a0.Bo * a0.mid * a0.inner;
      j.ntiles = a0.ntiles;
    }
    jobs.push_back(j);
  }
  if (b->d_jobs) cudaFree(b->d_jobs);
  b->d_jobs = nullptr;
  CC_CK(cudaMalloc(&b->d_jobs, std::max<size_t>(1, jobs.size()) *
                                   sizeof(BoundsJob)));
  if (!jobs.empty())
    CC_CK(cudaMemcpyAsync(b->d_jobs, jobs.data(),
                          jobs.size() * sizeof(BoundsJob),
                          cudaMemcpyHostToDevice, b->stream));
  // the work items: per kernel, level by level; largest passes first inside
  // a level (long tails start early).  A cell all of whose passes are single
  // tiles is one chained item of its first level (register kernels).
  std::vector<int4> items;
  auto add_items = [&](ByKid &kids, std::vector<Group> &out, bool gain) {
    for (auto &kv : kids) {
      Group gr;
      gr.kid = kv.first;
      gr.item0 = (long long)items.size();
      long long most = 1;                 // items of the widest level
      for (auto &lv : kv.second) {
        std::stable_sort(lv.begin(), lv.end(), [&](int x, int y) {
          return b->passes[x].a.ntiles > b->passes[y].a.ntiles;
        });
        const long long before = (long long)items.size();
        for (int pid : lv) {
          const GroupArgs &a = b->passes[pid].a;
          const Cell &c = b->cells[b->pass_cell[pid]];
          gr.smem = std::max(gr.smem, b->passes[pid].smem);
          if (gr.kid >= 0) {
            const int p0 = gain ? c.gain_pass : c.first_pass;
            const int np = gain ? c.ngain : c.npass;
            bool single = true;
            for (int p = p0; p < p0 + np; p++)
              single = single && b->passes[p].a.ntiles == 1;
            if (single) {
              if (pid == p0) items.push_back(make_int4(pid, 0, 1, np));
              continue;
            }
          }
          const long long tw = (long long)a.Bo * a.mid * a.W;
          const long long per = std::max<long long>(
              1, item_words(gr.kid >= 0) / tw);
          for (long long t = 0; t < a.ntiles; t += per)
            items.push_back(make_int4(
                pid, (int)t, (int)std::min<long long>(per, a.ntiles - t), 1));
        }
        most = std::max(most, (long long)items.size() - before);
      }
      gr.nitems = (long long)items.size() - gr.item0;
      gr.grid = gr.kid < 0 ? batch_grid(gr.smem)
                           : (int)std::min<long long>(
                                 batch_groups_grid(gr.kid, gr.smem), most);
      gr.next = (int)(b->groups.size() + b->gain_groups.size());
      out.push_back(gr);
    }
    // the register kernels' launches onto the streams the big cells leave,
    // most items first
    std::vector<size_t> order;
    for (size_t k = 0; k < out.size(); k++)
      if (out[k].kid >= 0) order.push_back(k);
    std::sort(order.begin(), order.end(), [&](size_t x, size_t y) {
      return out[x].nitems > out[y].nitems;
    });
    const int first = b->nside < kSideStreams ? b->nside : 0;
    for (size_t k = 0; k < order.size(); k++)
      out[order[k]].side =
          first + (int)(k % (size_t)(kSideStreams - first));
  };
  add_items(by_kid, b->groups, false);
  b->nitems = (long long)items.size();
  add_items(gain_by_kid, b->gain_groups, true);
  b->grid = 0;
  for (const Group &gr : b->groups) b->grid += gr.grid;
  auto F = [](void *p) { if (p) cudaFree(p); };
  F(b->d_passes); F(b->d_dep); F(b->d_need); F(b->d_items); F(b->d_done);
  F(b->d_pass_cell); F(b->d_next);
  const size_t np = b->passes.size();
  const size_t npa = std::max<size_t>(1, np);
  CC_CK(cudaMalloc(&b->d_passes, npa * sizeof(GroupArgs)));
  CC_CK(cudaMalloc(&b->d_dep, npa * sizeof(int)));
  CC_CK(cudaMalloc(&b->d_need, npa * sizeof(unsigned)));
  CC_CK(cudaMalloc(&b->d_done, npa * sizeof(unsigned)));
  CC_CK(cudaMalloc(&b->d_pass_cell, npa * sizeof(int)));
  b->nnext = (int)(b->groups.size() + b->gain_groups.size());
  CC_CK(cudaMalloc(&b->d_next, std::max<size_t>(1, b->nnext) * 8));
  CC_CK(cudaMalloc(&b->d_items, std::max<size_t>(1, items.size()) *
                                    sizeof(int4)));
  std::vector<GroupArgs> args;
  for (const GroupPlan &p : b->passes) args.push_back(p.a);
  if (np) {
    CC_CK(cudaMemcpyAsync(b->d_passes, args.data(),
                          np * sizeof(GroupArgs), cudaMemcpyHostToDevice,
                          b->stream));
    CC_CK(cudaMemcpyAsync(b->d_pass_cell, b->pass_cell.data(),
                          np * sizeof(int), cudaMemcpyHostToDevice,
                          b->stream));
    CC_CK(cudaMemcpyAsync(b->d_dep, b->dep.data(), np * sizeof(int),
                          cudaMemcpyHostToDevice, b->stream));
    CC_CK(cudaMemcpyAsync(b->d_need, b->need.data(), np * sizeof(unsigned),
                          cudaMemcpyHostToDevice, b->stream));
  }
  if (!items.empty())
    CC_CK(cudaMemcpyAsync(b->d_items, items.data(), items.size() * sizeof(int4),
                          cudaMemcpyHostToDevice, b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return 0;
}

// one big cell's step on stream s (its code bounds computed before):
// recount, deficit, gain, gain max, loss, loss max (register-blocked group
// kernels)
int run_big_cell(Batch *b, size_t i, cudaStream_t s) {
  Cell &c = b->cells[i];
  int rc = 0;
  for (int t = 0; t < 3; t++) {
    long long *slot = b->d_scal + 3 * i + t;
    // the deficit count (recount) or the map maximum folded into the last
    // launch where its kernel reduces what it writes (a register kernel or
    // a streamed strided group); else a separate reduction pass
    bool folded = false;
    for (size_t k = 0; k < c.fast[t].size(); k++) {
      GroupPlan gp = c.fast[t][k];
      if (k + 1 == c.fast[t].size() && gp.a.dst != kDstLayers &&
          (gp.a.tma == 1 || (gp.a.tma == 0 && gp.kernel >= 0))) {
        gp.a.red = slot;
        gp.a.red_mode = t == 0 ? 1 : 2;
        folded = true;
      }
      if ((rc = launch_group(gp, s))) return rc;
    }
    if (folded) continue;
    rc = t == 0 ? launch_cnt_reduce(c.cnt, c.g.space, kPredDef, 0, c.g.mu,
                                    slot, s)
                : launch_max(t == 1 ? c.gain : c.loss, c.g.space, slot, s);
    if (rc) return rc;
  }
  return 0;
}

// one persistent launch of the batch on its stream (nullptr active: every
// cell's items run)
int launch_items(Batch *b, const Group &gr, const int *active) {
  if (!gr.nitems) return 0;
  BatchLaunch L{b->d_passes, b->d_dep, b->d_need, b->d_items + gr.item0,
                gr.nitems, b->d_done, b->d_next + gr.next, b->d_err, gr.smem,
                gr.grid, gr.kid, b->d_pass_cell, active};
  cudaStream_t s = gr.side < 0 ? b->stream : b->side[gr.side];
  return gr.kid < 0 ? launch_batch(L, s) : launch_batch_groups(L, s);
}

// the gain map of every cell with active[i] again (d_active: the same flags
// on the device), on the streams the step uses; `beside` puts on the main
// stream what runs at the same time
template <class Beside>
int rebuild_gains(Batch *b, const std::vector<int> &active,
                  const int *d_active, Beside beside) {
  const size_t np = std::max<size_t>(1, b->passes.size());
  CC_CK(cudaMemsetAsync(b->d_next, 0, std::max<size_t>(1, b->nnext) * 8,
                        b->stream));
  CC_CK(cudaMemsetAsync(b->d_done, 0, np * sizeof(unsigned), b->stream));
  CC_CK(cudaEventRecord(b->fork, b->stream));
  int rc = beside();
  bool used[kSideStreams] = {false};
  auto fork = [&](int k) -> int {
    if (used[k]) return 0;
    used[k] = true;
    CC_CK(cudaStreamWaitEvent(b->side[k], b->fork, 0));
    return 0;
  };
  for (size_t i = 0; i < b->cells.size() && !rc; i++) {
    const Cell &c = b->cells[i];
    if (!c.big || !active[i]) continue;
    rc = fork(c.side);
    for (size_t k = 0; k < c.fast[1].size() && !rc; k++)
      rc = launch_group(c.fast[1][k], b->side[c.side]);
  }
  for (size_t k = 0; k < b->gain_groups.size() && !rc; k++) {
    const Group &gr = b->gain_groups[k];
    bool any = false;
    for (size_t i = 0; i < b->cells.size(); i++)
      any = any || (active[i] && !b->cells[i].big && b->cells[i].kid == gr.kid);
    if (!any) continue;
    if (gr.side >= 0) rc = fork(gr.side);
    if (!rc) rc = launch_items(b, gr, d_active);
  }
  for (int k = 0; k < kSideStreams; k++) {
    if (!used[k]) continue;
    CC_CK(cudaEventRecord(b->join[k], b->side[k]));
    CC_CK(cudaStreamWaitEvent(b->stream, b->join[k], 0));
  }
  return rc;
}

int capture_graph(Batch *b) {
  if (b->exec) { cudaGraphExecDestroy(b->exec); b->exec = nullptr; }
  if (b->graph) { cudaGraphDestroy(b->graph); b->graph = nullptr; }
  const size_t np = std::max<size_t>(1, b->passes.size());
  CC_CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  int rc = 0;
  auto ck = [&](cudaError_t e, const char *what) {
    if (e != cudaSuccess && !rc) {
      fprintf(stderr, "coldcore_b200: batch capture: %s: %s\n", what,
              cudaGetErrorString(e));
      rc = -(100 + (int)e);
    }
  };
  ck(cudaMemsetAsync(b->d_next, 0, std::max<size_t>(1, b->nnext) * 8,
                     b->stream), "memset next");
  ck(cudaMemsetAsync(b->d_err, 0, 4, b->stream), "memset err");
  ck(cudaMemsetAsync(b->d_done, 0, np * sizeof(unsigned), b->stream),
     "memset done");
  ck(cudaMemsetAsync(b->d_scal, 0, b->cells.size() * 3 * 8, b->stream),
     "memset scalars");
  // every cell's code slices, from the code lengths on the device
  k_batch_bounds<<<(unsigned)b->cells.size(), 256, 0, b->stream>>>(
      b->d_jobs);
  ck(cudaGetLastError(), "bounds launch");
  // big cells and the register kernels' small cells fork onto side streams,
  // the runtime-size tiles run on the main stream, and everything joins
  // before the end
  ck(cudaEventRecord(b->fork, b->stream), "fork record");
  bool used[kSideStreams] = {false};
  for (const Cell &c : b->cells) if (c.big) used[c.side] = true;
  for (const Group &gr : b->groups) if (gr.side >= 0) used[gr.side] = true;
  for (int k = 0; k < kSideStreams; k++)
    if (used[k]) ck(cudaStreamWaitEvent(b->side[k], b->fork, 0), "fork wait");
  for (size_t k = 0; k < b->groups.size() && !rc; k++)
    rc = launch_items(b, b->groups[k], nullptr);
  for (size_t i = 0; i < b->cells.size() && !rc; i++)
    if (b->cells[i].big)
      rc = run_big_cell(b, i, b->side[b->cells[i].side]);
  for (int k = 0; k < kSideStreams; k++) {
    if (!used[k]) continue;
    ck(cudaEventRecord(b->join[k], b->side[k]), "join record");
    ck(cudaStreamWaitEvent(b->stream, b->join[k], 0), "join wait");
  }
  cudaGraph_t graph = nullptr;
  const cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
  if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
  CC_CK(e);
  b->graph = graph;
  CC_CK(cudaGraphInstantiate(&b->exec, graph, 0));
  return 0;
}

int run_persistent(Batch *b) {
  CC_CK(cudaGraphLaunch(b->exec, b->stream));
  int err = 0;
  CC_CK(cudaMemcpyAsync(&err, b->d_err, 4, cudaMemcpyDeviceToHost,
                        b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return err ? -7 : 0;
}

// The same step as one launch per pass: every big cell's own launches on
// the same side streams as the graph, every small cell's passes as
// one launch each of the same tile code on the main stream, no host wait
// until the end.  Only the launch structure differs from the persistent
// graph launch, which is what the comparison measures.
int run_per_pass(Batch *b) {
  CC_CK(cudaMemsetAsync(b->d_scal, 0, b->cells.size() * 3 * 8, b->stream));
  k_batch_bounds<<<(unsigned)b->cells.size(), 256, 0, b->stream>>>(
      b->d_jobs);
  CC_CK(cudaGetLastError());
  CC_CK(cudaEventRecord(b->fork, b->stream));
  for (int k = 0; k < b->nside; k++)
    CC_CK(cudaStreamWaitEvent(b->side[k], b->fork, 0));
  for (size_t i = 0; i < b->cells.size(); i++) {
    const Cell &c = b->cells[i];
    if (c.big) {
      const int rc = run_big_cell(b, i, b->side[c.side]);
      if (rc) return rc;
      continue;
    }
    for (int p = c.first_pass; p < c.first_pass + c.npass; p++) {
      const int rc = launch_group(b->passes[p], b->stream);
      if (rc) return rc;
    }
  }
  for (int k = 0; k < b->nside; k++) {
    CC_CK(cudaEventRecord(b->join[k], b->side[k]));
    CC_CK(cudaStreamWaitEvent(b->stream, b->join[k], 0));
  }
  CC_CK(cudaStreamSynchronize(b->stream));
  return 0;
}

}  // namespace

extern "C" {

long long dct_batch_create(void) {
  Batch *b = new Batch();
  bool ok = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) ==
                cudaSuccess &&
            cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming) ==
                cudaSuccess;
  for (int k = 0; k < kSideStreams && ok; k++)
    ok = cudaStreamCreateWithFlags(&b->side[k], cudaStreamNonBlocking) ==
             cudaSuccess &&
         cudaEventCreateWithFlags(&b->join[k], cudaEventDisableTiming) ==
             cudaSuccess;
  if (!ok) {
    delete b;
    return -1;
  }
  const long long h = g_next_handle++;
  g_batches[h] = b;
  return h;
}

int dct_batch_add(long long h, int problem, int n, const int *ax, int R,
                  int mu, const long long *code, int M) {
  Batch *b = get(h);
  if (!b || b->built || problem < 0 || problem > 3 || n < 1 ||
      n > kMaxAxes || !ax || R < 1 || mu < 1 || mu > 65535 || M < 0 ||
      (M && !code))
    return -1;
  const bool layered = problem == kHamming || problem == kLee;
  if (layered && R + 1 > kMaxLayers) return -1;
  Cell c;
  c.g.prob = problem; c.g.n = n; c.g.R = R; c.g.mu = mu;
  c.g.pw[0] = 1;
  for (int i = 0; i < n; i++) {
    if (ax[i] < 2 || ax[i] > 16) return -1;          // tile kernel fibres
    if (problem == kTorus && 2 * R + 1 > ax[i]) return -1;
    if (c.g.pw[i] > (1LL << 40) / ax[i]) return -2;
    c.g.ax[i] = ax[i];
    c.g.pw[i + 1] = c.g.pw[i] * ax[i];
  }
  c.g.space = c.g.pw[n];
  c.R1 = layered ? R + 1 : 1;
  c.plane = (c.g.space + kPlaneAlign - 1) / kPlaneAlign * kPlaneAlign;
  c.code.assign(code, code + M);
  for (long long w : c.code)
    if (w < 0 || w >= c.g.space) return -1;
  std::sort(c.code.begin(), c.code.end());
  // the exact uint16 bound of the singleton engine: no counter exceeds
  // min(total occurrences, max multiplicity x |B|)
  long long maxmult = 0, run = 0;
  for (size_t i = 0; i < c.code.size(); i++) {
    run = (i && c.code[i] == c.code[i - 1]) ? run + 1 : 1;
    if (run > maxmult) maxmult = run;
  }
  if (std::min<long long>(M, maxmult * ball_cardinality(c.g)) > 65535)
    return -1;
  bool homog = true;
  for (int i = 1; i < n; i++) homog &= ax[i] == ax[0];
  int bm = 0;
  c.regs = homog && pick_group_kernel(transform_geometry(c.g).prob, ax[0],
                                      c.R1, &bm) >= 0;
  c.big = c.g.space >= big_cell_words() && homog &&
          pick_group_kernel(problem, ax[0], c.R1, &bm) >= 0;
  b->cells.push_back(std::move(c));
  return (int)b->cells.size() - 1;
}

int dct_batch_build(long long h, int tile_kb) {
  Batch *b = get(h);
  if (!b || b->built || b->cells.empty()) return -1;
  if (tile_kb > 0) b->tile_budget = (size_t)std::max(16, tile_kb) * 1024;
  // arena: per cell layers, cnt, gain, loss, code (room for a code of
  // four times its first size, at least 4096 words)
  for (Cell &c : b->cells)
    c.code_cap = std::max<long long>(
        4 * (long long)c.code.size(),
        std::min<long long>(c.g.space, 1LL << 18));
  size_t total = 0;
  std::vector<size_t> off(b->cells.size());
  for (size_t i = 0; i < b->cells.size(); i++) {
    const Cell &c = b->cells[i];
    off[i] = total;
    total += align256((size_t)c.plane * c.R1 * 4) + align256(c.plane * 2) +
             2 * align256((size_t)c.plane * 4) +
             align256((size_t)b->cells[i].code_cap * 8);
  }
  CC_CK(cudaMalloc(&b->arena, total));
  b->arena_bytes = total;
  CC_CK(cudaMalloc(&b->d_err, 4));
  CC_CK(cudaMalloc(&b->d_scal, b->cells.size() * 3 * 8));
  CC_CK(cudaMalloc(&b->d_ncode, b->cells.size() * 8));
  {
    std::vector<long long> nc;
    for (const Cell &c : b->cells) nc.push_back((long long)c.code.size());
    CC_CK(cudaMemcpy(b->d_ncode, nc.data(), nc.size() * 8,
                     cudaMemcpyHostToDevice));
  }
  for (size_t i = 0; i < b->cells.size(); i++) {
    Cell &c = b->cells[i];
    char *p = b->arena + off[i];
    c.layers = reinterpret_cast<int32_t *>(p);
    p += align256((size_t)c.plane * c.R1 * 4);
    c.cnt = reinterpret_cast<uint16_t *>(p);
    p += align256(c.plane * 2);
    c.gain = reinterpret_cast<int32_t *>(p);
    p += align256((size_t)c.plane * 4);
    c.loss = reinterpret_cast<int32_t *>(p);
    p += align256((size_t)c.plane * 4);
    c.dcode = reinterpret_cast<long long *>(p);
    c.dncode = b->d_ncode + i;
    if (!c.code.empty())
      CC_CK(cudaMemcpyAsync(c.dcode, c.code.data(), c.code.size() * 8,
                            cudaMemcpyHostToDevice, b->stream));
  }
  b->built = true;
  // tile bounds depend on the tile size: computed per schedule
  auto schedule = [&]() -> int {
    int rc = make_schedule(b);
    if (rc) return rc;
    return capture_graph(b);          // code bounds inside the graph
  };
  int rc;
  if (tile_kb > 0) return schedule();
  // autotune the tile budget: time one graph launch per candidate
  static const int cand_kb[] = {24, 48, 96};
  EventPair ev;
  if ((rc = ev.create())) return rc;
  cudaEvent_t e0 = ev.e0, e1 = ev.e1;
  float best = 1e30f;
  int best_kb = 48;
  for (int kb : cand_kb) {
    b->tile_budget = (size_t)kb * 1024;
    if ((rc = schedule())) return rc;
    if ((rc = run_persistent(b))) return rc;               // warm
    CC_CK(cudaEventRecord(e0, b->stream));
    if ((rc = run_persistent(b))) return rc;
    CC_CK(cudaEventRecord(e1, b->stream));
    CC_CK(cudaEventSynchronize(e1));
    float ms = 0;
    CC_CK(cudaEventElapsedTime(&ms, e0, e1));
    if (ms < best) { best = ms; best_kb = kb; }
  }
  b->tile_budget = (size_t)best_kb * 1024;
  b->tuned_ms = best;
  return schedule();
}

int dct_batch_run(long long h, int mode) {
  Batch *b = get(h);
  if (!b || !b->built) return -1;
  if (mode == 0 || mode == 1) {
    for (Cell &c : b->cells) c.moved = false;
    const int rc = mode == 0 ? run_persistent(b) : run_per_pass(b);
    const int late = tma_fault_take();   // the launches have drained
    return rc ? rc : late;
  }
  if (mode == 2) {
    // self-test of the bounded dependency wait: one launch in which the
    // first pass needs one more tile than it has, so its dependents time
    // out; the launch must end with an error status, not hang
    if (b->nstep < 2) return -1;
    std::vector<unsigned> poisoned = b->need;
    poisoned[0] += 1;
    CC_CK(cudaMemcpyAsync(b->d_need, poisoned.data(),
                          poisoned.size() * sizeof(unsigned),
                          cudaMemcpyHostToDevice, b->stream));
    const int rc = run_persistent(b);
    CC_CK(cudaMemcpyAsync(b->d_need, b->need.data(),
                          b->need.size() * sizeof(unsigned),
                          cudaMemcpyHostToDevice, b->stream));
    CC_CK(cudaStreamSynchronize(b->stream));
    return rc;
  }
  return -1;
}

int dct_batch_read(long long h, int cell, int field, long long off,
                   long long len, void *out) {
  Batch *b = get(h);
  if (!b || !b->built || cell < 0 || cell >= (int)b->cells.size() ||
      field < 0 || field > 2 || off < 0 || len < 0 || (len && !out))
    return -1;
  const Cell &c = b->cells[cell];
  if (off + len > c.g.space) return -1;
  const void *src = field == 0 ? (const void *)(c.cnt + off)
                    : field == 1 ? (const void *)(c.gain + off)
                                 : (const void *)(c.loss + off);
  if (len)
    CC_CK(cudaMemcpyAsync(out, src, (size_t)len * (field == 0 ? 2 : 4),
                          cudaMemcpyDeviceToHost, b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return 0;
}

int dct_batch_scalars(long long h, long long *out, int cap) {
  Batch *b = get(h);
  if (!b || !b->built || !out) return -1;
  const int n = (int)std::min<long long>(cap, (long long)b->cells.size() * 3);
  CC_CK(cudaMemcpyAsync(out, b->d_scal, (size_t)n * 8, cudaMemcpyDeviceToHost,
                        b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return n;
}

int dct_batch_info(long long h, long long *out, int cap) {
  Batch *b = get(h);
  if (!b || !out || cap < 6) return -1;
  out[0] = (long long)b->cells.size();
  out[1] = b->nstep;
  out[2] = b->nitems;
  out[3] = (long long)(b->tile_budget / 1024);
  out[4] = b->grid;
  out[5] = (long long)(b->tuned_ms * 1000.0f);
  if (cap < 8) return 6;
  // the step's algorithmic HBM bytes (every launch's source read once and
  // destination written once, the deficit count and the two maxima), and
  // those of the big cells alone
  long long all = 0, big = 0;
  for (const Cell &c : b->cells) {
    long long cb = 0;
    if (c.big) {
      for (int t = 0; t < 3; t++)
        for (const auto &gp : c.fast[t]) {
          GroupArgs a = gp.a;
          a.ncode = (long long)c.code.size();
          cb += group_bytes(a);
        }
    } else {
      for (int p = c.first_pass; p < c.first_pass + c.npass; p++) {
        GroupArgs a = b->passes[p].a;
        a.ncode = (long long)c.code.size();
        cb += group_bytes(a);
      }
    }
    cb += c.g.space * (2 + 4 + 4);         // deficit count, gain / loss max
    all += cb;
    if (c.big) big += cb;
  }
  out[6] = all;
  out[7] = big;
  return 8;
}

// ------------------------------------------------------------ per cell
// The calls a search on one cell of a batch makes between graph launches.
// They run on the batch's stream and return after it drains.

int dct_batch_set_code(long long h, int cell, const long long *code, int M) {
  Batch *b = get(h);
  if (!b || !b->built || cell < 0 || cell >= (int)b->cells.size() || M < 0 ||
      (M && !code))
    return -1;
  Cell &c = b->cells[cell];
  if (M > c.code_cap) return -3;                   // beyond the room kept
  std::vector<long long> v(code, code + M);
  for (long long w : v)
    if (w < 0 || w >= c.g.space) return -1;
  std::sort(v.begin(), v.end());
  long long maxmult = 0, run = 0;
  for (size_t i = 0; i < v.size(); i++) {
    run = (i && v[i] == v[i - 1]) ? run + 1 : 1;
    if (run > maxmult) maxmult = run;
  }
  if (std::min<long long>(M, maxmult * ball_cardinality(c.g)) > 65535)
    return -1;                                     // the uint16 bound
  c.code.swap(v);
  const long long n = (long long)c.code.size();
  if (n)
    CC_CK(cudaMemcpyAsync(c.dcode, c.code.data(), (size_t)n * 8,
                          cudaMemcpyHostToDevice, b->stream));
  CC_CK(cudaMemcpyAsync(c.dncode, &n, 8, cudaMemcpyHostToDevice, b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return 0;
}

// the cell's support table: `len` patterns of `slots` int32 slots
// (pos << 24) | shift, row-major as dct_init3w takes it; entry 0 the centre
int dct_batch_set_table(long long h, int cell, const int32_t *tbl, int slots,
                        long long len) {
  Batch *b = get(h);
  if (!b || !b->built || cell < 0 || cell >= (int)b->cells.size() ||
      !tbl || slots < 1 || slots > kMaxSlots || len < 1)
    return -1;
  Cell &c = b->cells[cell];
  std::vector<int32_t> soa((size_t)slots * len);
  for (long long t = 0; t < len; t++)
    for (int k = 0; k < slots; k++) {
      const int32_t v = tbl[t * slots + k];
      if (v) {
        const int pos = v >> 24, dl = v & 0xFFFFFF;
        if (pos < 0 || pos >= c.g.n || dl < 1 || dl >= c.g.ax[pos]) return -1;
      }
      soa[(size_t)k * len + t] = v;
    }
  // one allocation and one copy: the entries, the table, its packed form
  std::vector<uint32_t> pk;
  std::vector<int4> ent;
  if (!pack_walk(c.g, soa, slots, len, pk, ent)) { pk.clear(); ent.clear(); }
  std::vector<int32_t> all(4 * ent.size() + soa.size() + pk.size());
  memcpy(all.data(), ent.data(), ent.size() * sizeof(int4));
  memcpy(all.data() + 4 * ent.size(), soa.data(), soa.size() * 4);
  memcpy(all.data() + 4 * ent.size() + soa.size(), pk.data(), pk.size() * 4);
  if (c.dtbl_base) cudaFree(c.dtbl_base);
  c.dtbl_base = nullptr;
  c.dtbl = nullptr;
  CC_CK(cudaMalloc(&c.dtbl_base, all.size() * 4));
  CC_CK(cudaMemcpy(c.dtbl_base, all.data(), all.size() * 4,
                   cudaMemcpyHostToDevice));
  c.dent = reinterpret_cast<int4 *>(c.dtbl_base);
  c.dtbl = c.dtbl_base + 4 * ent.size();
  c.dpk = pk.empty() ? nullptr
                     : reinterpret_cast<uint32_t *>(c.dtbl + soa.size());
  c.noff = (int)ent.size();
  c.slots = slots;
  c.tlen = len;
  c.ball_ok = metric_ball_table(c.g, soa, slots, len);
  return 0;
}

namespace {

int stage_cell_words(Batch *b, const Cell &c, const long long *words,
                     int nw) {
  if (nw < 0 || nw > (1 << 16) || (nw && !words)) return -1;
  for (int i = 0; i < nw; i++)
    if (words[i] < 0 || words[i] >= c.g.space) return -1;
  if (!b->d_words) {
    CC_CK(cudaMalloc(&b->d_words, (size_t)(1 << 16) * 8));
    CC_CK(cudaMalloc(&b->d_out, (size_t)(1 << 16) * 4));
    CC_CK(cudaMalloc(&b->d_count, 16));
  }
  if (nw)
    CC_CK(cudaMemcpyAsync(b->d_words, words, (size_t)nw * 8,
                          cudaMemcpyHostToDevice, b->stream));
  return 0;
}

WalkArgs cell_walk(const Cell &c) {
  WalkArgs w{};
  w.g = c.g;
  w.tbl = c.dtbl;
  w.slots = c.slots;
  w.len = c.tlen;
  w.cnt = c.cnt;
  w.pk = c.dpk;
  w.ent = c.dent;
  w.noff = c.noff;
  return w;
}

Cell *live_cell(long long h, int cell, Batch **pb) {
  Batch *b = get(h);
  if (!b || !b->built || cell < 0 || cell >= (int)b->cells.size())
    return nullptr;
  *pb = b;
  return &b->cells[cell];
}

}  // namespace

// cnt += delta over the balls of nw words (delta +1 or -1; the caller keeps
// the multiset valid, as the search core does)
int dct_batch_update(long long h, int cell, const long long *words, int nw,
                     int delta) {
  Batch *b = nullptr;
  Cell *c = live_cell(h, cell, &b);
  if (!c || !c->dtbl || (delta != 1 && delta != -1)) return -1;
  int rc = stage_cell_words(b, *c, words, nw);
  if (rc || !nw) return rc;
  c->moved = true;
  rc = launch_update(cell_walk(*c), b->d_words, nullptr, nw, delta, nullptr,
                     b->stream);
  if (rc) return rc;
  CC_CK(cudaStreamSynchronize(b->stream));
  return 0;
}

// out[i] = #{x in B(w_i) : role(cnt[x])}: role 0 deficient (cnt < mu),
// 1 critical (1 <= cnt <= mu), else the literal cnt == role
int dct_batch_gather(long long h, int cell, const long long *words, int nw,
                     int role, int32_t *out) {
  Batch *b = nullptr;
  Cell *c = live_cell(h, cell, &b);
  if (!c || !c->dtbl || role < 0 || (nw && !out)) return -1;
  int rc = stage_cell_words(b, *c, words, nw);
  if (rc || !nw) return rc;
  const int mode = role == 0 ? (c->g.mu > 1 ? kPredDef : kPredEq)
                   : role == 1 ? (c->g.mu > 1 ? kPredCrit : kPredEq)
                               : kPredEq;
  rc = launch_gather(cell_walk(*c), b->d_words, nw, mode, role, b->d_out,
                     false, b->stream);
  if (rc) return rc;
  CC_CK(cudaMemcpyAsync(out, b->d_out, (size_t)nw * 4,
                        cudaMemcpyDeviceToHost, b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return 0;
}

// entries of the gain (field 1) or loss (field 2) map at or above thr:
// up to cap (index, value) pairs, unordered; returns how many there are
long long dct_batch_extract(long long h, int cell, int field, int32_t thr,
                            long long *idx, int32_t *val, int cap) {
  Batch *b = nullptr;
  Cell *c = live_cell(h, cell, &b);
  if (!c || (field != 1 && field != 2) || cap < 0 || (cap && (!idx || !val)))
    return -1;
  if (cap > b->ext_cap) {
    if (b->d_ext) cudaFree(b->d_ext);
    if (b->d_extv) cudaFree(b->d_extv);
    b->d_ext = nullptr;
    b->d_extv = nullptr;
    CC_CK(cudaMalloc(&b->d_ext, (size_t)cap * 8));
    CC_CK(cudaMalloc(&b->d_extv, (size_t)cap * 4));
    b->ext_cap = cap;
  }
  if (!b->d_count) CC_CK(cudaMalloc(&b->d_count, 16));
  CC_CK(cudaMemsetAsync(b->d_count, 0, 8, b->stream));
  const int32_t *A = field == 1 ? c->gain : c->loss;
  int rc = launch_extract(A, c->g.space, thr, b->d_ext, true, b->d_extv, cap,
                          b->d_count, b->stream);
  if (rc) return rc;
  long long found = 0;
  CC_CK(cudaMemcpyAsync(&found, b->d_count, 8, cudaMemcpyDeviceToHost,
                        b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  const long long n = std::min<long long>(found, cap);
  if (n) {
    CC_CK(cudaMemcpyAsync(idx, b->d_ext, (size_t)n * 8,
                          cudaMemcpyDeviceToHost, b->stream));
    CC_CK(cudaMemcpyAsync(val, b->d_extv, (size_t)n * 4,
                          cudaMemcpyDeviceToHost, b->stream));
    CC_CK(cudaStreamSynchronize(b->stream));
  }
  return found;
}

// Exact greedy on the listed cells at once (the device repair of a
// campaign's searches): from each cell's gain map as the last launch left
// it — the caller runs the step after its last update — with the cell's
// code words excluded, each step places, in every cell still placing, the
// word of largest gain (ties: smallest index) until the cell's deficit is 0,
// no word gains, or max_add[k] words are placed.  placed_out holds cap words
// per listed cell; nplaced_out and deficit_out one value per listed cell.
int dct_batch_greedy(long long h, const int *cells, int n, const int *max_add,
                     long long *placed_out, int cap, int *nplaced_out,
                     long long *deficit_out) {
  Batch *b = get(h);
  if (!b || !b->built || n < 0 || (n && (!cells || !max_add || !placed_out ||
                                         !nplaced_out || !deficit_out)) ||
      cap < 0)
    return -1;
  if (n == 0) return 0;
  std::vector<long long> sc(b->cells.size() * 3);
  CC_CK(cudaMemcpyAsync(sc.data(), b->d_scal, sc.size() * 8,
                        cudaMemcpyDeviceToHost, b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  long long steps = 0;
  for (int k = 0; k < n; k++) {
    if (cells[k] < 0 || cells[k] >= (int)b->cells.size() || max_add[k] < 0 ||
        max_add[k] > cap)
      return -1;
    const Cell &c = b->cells[cells[k]];
    if (!c.dtbl || c.g.space >= (1LL << 32)) return -1;
    // placed words are new (multiplicity 1): the counters stay within
    // min(occurrences, max multiplicity x |B|) <= 65,535
    long long maxmult = 1, run = 0;
    for (size_t i = 0; i < c.code.size(); i++) {
      run = (i && c.code[i] == c.code[i - 1]) ? run + 1 : 1;
      if (run > maxmult) maxmult = run;
    }
    if (std::min<long long>((long long)c.code.size() + max_add[k],
                            maxmult * ball_cardinality(c.g)) > 65535)
      return -1;
    steps = std::max<long long>(steps, std::min<long long>(
        max_add[k], sc[3 * cells[k]]));
  }
  // workspace: per cell its table entry, state, placed words and chunk keys;
  // the rebuild flags of the listed cells and of the batch's
  // cells; the jobs of the two launches of a step
  auto pad = [](size_t x) { return (x + 63) / 64 * 64; };
  const size_t st_b = (size_t)n * kGreedyStateBytes;
  const size_t pl_b = (size_t)n * std::max(cap, 1) * 8;
  std::vector<int2> jam, jpl;
  std::vector<int> pats(n);
  // blocks of a cell's ball: enough for all cells together to fill the GPU
  const int ball_blocks = std::max(8, sm_count() * 16 / n);
  size_t chunks = 0, fresh_words = 0;
  for (int k = 0; k < n; k++) {
    const Cell &c = b->cells[cells[k]];
    chunks += (size_t)greedy_chunks(c.g.space);
    fresh_words += (size_t)c.tlen;
    for (int j = 0; j < greedy_argmax_blocks(c.g.space); j++)
      jam.push_back(make_int2(k, j));
    pats[k] = greedy_pats(c.tlen, ball_blocks);
    for (long long j = 0; j * pats[k] < c.tlen; j++)
      jpl.push_back(make_int2(k, (int)j));
  }
  size_t off = 0;
  auto take = [&](size_t bytes) { const size_t o = off; off += pad(bytes);
                                  return o; };
  const size_t o_tab = take((size_t)n * sizeof(BatchGreedyCell));
  const size_t o_st = take(st_b), o_pl = take(pl_b);
  const size_t o_key = take(chunks * 8);
  const size_t o_fresh = take(fresh_words * 8);
  const size_t o_flag = take((size_t)n * 4);
  const size_t o_act = take(b->cells.size() * 4);
  const size_t o_jam = take(jam.size() * 8), o_jpl = take(jpl.size() * 8);
  if (off > b->greedy_cap) {
    if (b->d_greedy) CC_CK(cudaFree(b->d_greedy));
    b->d_greedy = nullptr;
    b->greedy_cap = 0;
    CC_CK(cudaMalloc(&b->d_greedy, off));
    b->greedy_cap = off;
  }
  if (2 * st_b > b->h_greedy_cap) {
    if (b->h_greedy) CC_CK(cudaFreeHost(b->h_greedy));
    b->h_greedy = nullptr;
    b->h_greedy_cap = 0;
    CC_CK(cudaHostAlloc((void **)&b->h_greedy, 2 * st_b,
                        cudaHostAllocDefault));
    b->h_greedy_cap = 2 * st_b;
  }
  for (auto &ev : b->ev_greedy)
    if (!ev) CC_CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  char *ws = b->d_greedy;
  int rc = 0;
  std::vector<BatchGreedyCell> tab(n);
  std::vector<GreedyHost> st0(n);
  std::vector<int> flag(n, 0), act(b->cells.size(), 0);
  {
    size_t co = 0, fo = 0;
    for (int k = 0; k < n; k++) {
      Cell &c = b->cells[cells[k]];
      BatchGreedyCell &g = tab[k];
      g.w = cell_walk(c);
      g.map = c.gain;
      g.st = ws + o_st + (size_t)k * kGreedyStateBytes;
      g.placed = reinterpret_cast<long long *>(ws + o_pl) +
                 (size_t)k * std::max(cap, 1);
      g.ckey = reinterpret_cast<unsigned long long *>(ws + o_key) + co;
      g.code = c.dcode;
      g.ncode = (long long)c.code.size();
      g.max_add = max_add[k];
      g.pats = pats[k];
      g.fresh = reinterpret_cast<long long *>(ws + o_fresh) + fo;
      co += (size_t)greedy_chunks(c.g.space);
      fo += (size_t)c.tlen;
      // done from the start when there is nothing to do
      st0[k] = GreedyHost{};
      st0[k].deficit = sc[3 * cells[k]];
      st0[k].done = (max_add[k] == 0 || sc[3 * cells[k]] == 0) ? 1 : 0;
      deficit_out[k] = sc[3 * cells[k]];
      nplaced_out[k] = 0;
    }
  }
  const BatchGreedyCell *dtab =
      reinterpret_cast<const BatchGreedyCell *>(ws + o_tab);
  int *d_flag = reinterpret_cast<int *>(ws + o_flag);
  int *d_act = reinterpret_cast<int *>(ws + o_act);
  const int2 *d_jam = reinterpret_cast<const int2 *>(ws + o_jam);
  const int2 *d_jpl = reinterpret_cast<const int2 *>(ws + o_jpl);
  constexpr int32_t kExcluded = INT_MIN / 2;
  auto ck = [&](cudaError_t e) {
    if (e != cudaSuccess && !rc) rc = -(100 + (int)e);
  };
  auto up = [&](size_t o, const void *src, size_t bytes) {
    if (bytes) ck(cudaMemcpyAsync(ws + o, src, bytes, cudaMemcpyHostToDevice,
                                  b->stream));
  };
  up(o_tab, tab.data(), (size_t)n * sizeof(BatchGreedyCell));
  up(o_st, st0.data(), st_b);
  up(o_jam, jam.data(), jam.size() * 8);
  up(o_jpl, jpl.data(), jpl.size() * 8);
  up(o_flag, flag.data(), (size_t)n * 4);
  // the rebuilds' error word: an earlier step's is not this call's
  ck(cudaMemsetAsync(b->d_err, 0, 4, b->stream));
  // incumbents never re-enter
  if (!rc) rc = launch_greedy_exclude(dtab, n, nullptr, kExcluded, b->stream);
  GreedyHost *ring[2] = {
      reinterpret_cast<GreedyHost *>(b->h_greedy),
      reinterpret_cast<GreedyHost *>(b->h_greedy + st_b)};
  auto read_states = [&](int slot) {
    ck(cudaMemcpyAsync(ring[slot], ws + o_st, st_b, cudaMemcpyDeviceToHost,
                       b->stream));
    ck(cudaEventRecord(b->ev_greedy[slot], b->stream));
  };
  // A map that updates or an earlier greedy have left behind or ahead of cnt
  // is never rebuilt: a transform would raise gains that the keys kept of its
  // chunks bound, and bring back words that an earlier greedy took out.
  // While a placement of some cell may be worth a rebuild of its map, the
  // host follows the gains one step behind (the first step knows them from
  // the last launch) and the device stays busy; gains never grow, so after
  // that the steps go out in chunks with one look between them.
  long long issued = 0, chunk = 32;
  bool follow = true;
  while (!rc && issued < steps) {
    const int par = (int)(issued & 1);
    if (follow) {
      rc = launch_greedy_argmax(dtab, d_jam, (int)jam.size(), par,
                                issued == 0, b->stream);
      read_states(par);
      const GreedyHost *h = ring[par ^ 1];
      if (issued) ck(cudaEventSynchronize(b->ev_greedy[par ^ 1]));
      if (rc) break;
      bool live = issued == 0, any = false, changed = false;
      for (int k = 0; k < n; k++) {
        const Cell &c = b->cells[cells[k]];
        const bool done = issued ? h[k].done != 0 : st0[k].done != 0;
        const long long gain = issued ? h[k].gain(par ^ 1)
                                      : sc[3 * cells[k] + 1];
        const int want = !done && c.ball_ok && !c.moved &&
                         greedy_rebuild_pays(gain, c.tlen, c.gain_us);
        live = live || !done;
        any = any || want;
        changed = changed || want != flag[k];
        flag[k] = act[cells[k]] = want;
      }
      if (!live) break;
      if (changed) {
        up(o_flag, flag.data(), (size_t)n * 4);
        up(o_act, act.data(), act.size() * 4);
      }
      if (!rc)
        rc = launch_greedy_place(dtab, d_jpl, (int)jpl.size(), par, kExcluded,
                                 b->stream);
      // the other cells' refresh runs while the side streams rebuild
      auto refresh = [&] {
        return launch_greedy_refresh(dtab, n, ball_blocks, d_flag, b->stream);
      };
      if (!rc) rc = any ? rebuild_gains(b, act, d_act, refresh) : refresh();
      if (any && !rc)
        rc = launch_greedy_exclude(dtab, n, d_flag, kExcluded, b->stream);
      follow = any;
      issued++;
      continue;
    }
    const long long m = std::min(chunk, steps - issued);
    for (long long i = 0; i < m && !rc; i++, issued++) {
      const int p2 = (int)(issued & 1);
      rc = launch_greedy_argmax(dtab, d_jam, (int)jam.size(), p2, 0,
                                b->stream);
      if (!rc) rc = launch_greedy_place(dtab, d_jpl, (int)jpl.size(), p2,
                                        kExcluded, b->stream);
      if (!rc) rc = launch_greedy_refresh(dtab, n, ball_blocks, d_flag,
                                          b->stream);
    }
    read_states(0);
    ck(cudaEventSynchronize(b->ev_greedy[0]));
    bool all = true;
    for (int k = 0; k < n; k++) all = all && ring[0][k].done;
    if (all) break;
    chunk = std::min<long long>(chunk * 2, 512);
  }
  for (int k = 0; k < n; k++) b->cells[cells[k]].moved = true;
  if (!rc) {
    read_states(0);
    ck(cudaStreamSynchronize(b->stream));
    int err = 0;
    ck(cudaMemcpyAsync(&err, b->d_err, 4, cudaMemcpyDeviceToHost, b->stream));
    // the placed words: one copy while that is small, else cell by cell
    std::vector<long long> words;
    const bool once = pl_b <= (8u << 20);
    if (once && !rc) {
      words.resize(pl_b / 8);
      ck(cudaMemcpyAsync(words.data(), ws + o_pl, pl_b, cudaMemcpyDeviceToHost,
                         b->stream));
      ck(cudaStreamSynchronize(b->stream));
    }
    for (int k = 0; k < n && !rc; k++) {
      const GreedyHost &h = ring[0][k];
      const int got = h.placed_now();
      deficit_out[k] = h.deficit_now();
      nplaced_out[k] = got;
      if (!got) continue;
      if (once)
        memcpy(placed_out + (size_t)k * cap, words.data() + (size_t)k * cap,
               (size_t)got * 8);
      else
        ck(cudaMemcpyAsync(placed_out + (size_t)k * cap, tab[k].placed,
                           (size_t)got * 8, cudaMemcpyDeviceToHost,
                           b->stream));
    }
    ck(cudaStreamSynchronize(b->stream));
    if (!rc && err) rc = -7;
  }
  cudaStreamSynchronize(b->stream);
  const int late = tma_fault_take();     // a rebuild's streamed launch
  return rc ? rc : late;
}

// mode 0: #{x : cnt[x] == target}; 1: the deficit sum max(0, mu - cnt)
long long dct_batch_count(long long h, int cell, int mode, int target) {
  Batch *b = nullptr;
  Cell *c = live_cell(h, cell, &b);
  if (!c || mode < 0 || mode > 1) return -1;
  if (!b->d_count) CC_CK(cudaMalloc(&b->d_count, 16));
  CC_CK(cudaMemsetAsync(b->d_count, 0, 8, b->stream));
  const int rc = launch_cnt_reduce(c->cnt, c->g.space,
                                   mode == 1 ? kPredDef : kPredEq, target,
                                   c->g.mu, b->d_count, b->stream);
  if (rc) return rc;
  long long v = 0;
  CC_CK(cudaMemcpyAsync(&v, b->d_count, 8, cudaMemcpyDeviceToHost,
                        b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return v;
}

// the gain (field 1) or loss (field 2) map at k words
int dct_batch_read_at(long long h, int cell, int field, const long long *idx,
                      int k, int32_t *out) {
  Batch *b = nullptr;
  Cell *c = live_cell(h, cell, &b);
  if (!c || (field != 1 && field != 2) || (k && !out)) return -1;
  int rc = stage_cell_words(b, *c, idx, k);
  if (rc || !k) return rc;
  rc = launch_read_at(field == 1 ? c->gain : c->loss, b->d_words, k,
                      b->d_out, b->stream);
  if (rc) return rc;
  CC_CK(cudaMemcpyAsync(out, b->d_out, (size_t)k * 4, cudaMemcpyDeviceToHost,
                        b->stream));
  CC_CK(cudaStreamSynchronize(b->stream));
  return 0;
}

int dct_batch_free(long long h) {
  Batch *b = get(h);
  if (!b) return -1;
  release(b);
  if (b->stream) cudaStreamDestroy(b->stream);
  for (int k = 0; k < kSideStreams; k++) {
    if (b->side[k]) cudaStreamDestroy(b->side[k]);
    if (b->join[k]) cudaEventDestroy(b->join[k]);
  }
  if (b->fork) cudaEventDestroy(b->fork);
  g_batches.erase(h);
  delete b;
  return 0;
}

}  // extern "C"
