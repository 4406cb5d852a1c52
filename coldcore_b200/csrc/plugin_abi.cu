// plugin_abi.cu — the extern "C" plugin ABI v1 of the B200 covering engine.
//
// Host side of every entry point declared in include/coldcore_b200/plugin.h:
// validation before any mutation, the represented multisets (uploaded /
// active, coldcore src/plugins/covering/dct_hc.cu:46-56), staging through
// pinned buffers, the transform planner, and the result copies.  Semantics
// follow the reference entry points cited per function; the device work is
// this engine's own (transform_group.cu, transform_window.cu, walks.cu,
// reduce.cu) and runs in call order on one engine-owned stream.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <map>
#include <unordered_map>
#include <vector>

#include "../../include/coldcore_b200/plugin.h"
#include "engine.h"

namespace cc {

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

int g_dct_blocks = 0;

}  // namespace cc

using namespace cc;

namespace {

constexpr long long kCounterMax = 65535;    // uint16 cnt
constexpr long long kStageCap = 1 << 16;    // words per staged chunk
// Extracted entries that come back with their count, through pinned memory;
// the rest take a second wait and a copy into the caller's pageable arrays.
// On K_3(14,3)'s map (4.8 M words), us a call with room for 2^12 / 2^15 /
// 2^16 entries: one found 47 / 51 / 55, 10,097 found 98 / 68 / 74, 30,290
// found 153 / 96 / 101, 60,076 found 282 / 241 / 178.  A doubling from 2^15
// costs every small answer as much again as all the room up to there.
constexpr long long kExtFirst = 1 << 15;
constexpr int kGreedyRing = 2;              // steps whose states are in flight

struct Plan {
  std::vector<GroupPlan> groups;   // layered / small-axis path
  std::vector<WindowArgs> passes;  // wide window path
  bool window = false;
  int scatter_plane = -1;          // window recount: plane of the code counts
};

// sorted words in pinned host memory
struct WordBuf {
  long long *p = nullptr;
  long long cap = 0, n = 0;
  // room for m words; a refusal leaves the words that are there
  int reserve(long long m) {
    if (m <= cap) return 0;
    const long long want = std::max<long long>(m + m / 2, 1024);
    if (fault_due(kFaultPinned))
      return -(100 + (int)cudaErrorMemoryAllocation);
    void *q = nullptr;
    CC_CK(cudaHostAlloc(&q, (size_t)want * 8, cudaHostAllocDefault));
    if (p) cudaFreeHost(p);
    p = static_cast<long long *>(q);
    cap = want;
    n = 0;
    return 0;
  }
  long long count(long long w) const {
    const auto r = std::equal_range(p, p + n, w);
    return r.second - r.first;
  }
};
// multiplicity -> distinct words that have it
typedef std::map<int, long long> MultHist;
inline int max_mult(const MultHist &h) {
  return h.empty() ? 0 : h.rbegin()->first;
}

// a greedy's state and its launches' barrier state as they lie on the device
struct GreedySlot {
  GreedyHost st;
  char pad[64 - kGreedyStateBytes];
  int run[kGreedyRunBytes / 4];    // [1]: a barrier timed out
};
static_assert(sizeof(GreedySlot) == 64 + kGreedyRunBytes, "greedy slot");

struct State {
  bool live = false;
  Geometry g{};
  int R1 = 1;                      // planes the transform math uses
  int nplanes = 0;                 // planes allocated
  long long plane = 0;
  int32_t *layers = nullptr;
  uint16_t *cnt = nullptr;
  long long cnt_len = 0;
  uint32_t *owner = nullptr;
  int use_owner = 0;
  int layers_mode = 0, cnt_mode = 0;
  // layers_mode 1: the R+1 layer planes in pinned host memory (plane d at
  // h_layers + d*|X|), streamed by every transform (outofcore.cu); the
  // device keeps plane 0 alone, the map
  bool streamed = false;
  int32_t *h_layers = nullptr;
  long long h_layers_bytes = 0;
  // support tables, SoA slots
  int32_t *tbl = nullptr, *tbl2 = nullptr;
  uint32_t *pk = nullptr, *pk2 = nullptr;    // packed forms (pack_walk)
  int4 *ent = nullptr;
  int noff = 0;
  int slots = 0, slots2 = 0;
  long long len = 0;
  int fmt = 0;
  // code
  long long *d_code = nullptr;
  long long code_cap = 0, codeM = 0;
  long long *d_bounds = nullptr;   // per-tile code slices of a recount
  long long bounds_cap = 0;
  // staging
  long long *h_words = nullptr, *d_words = nullptr;
  int32_t *h_out = nullptr, *d_out = nullptr;
  cudaEvent_t ev_stage[2] = {nullptr};
  long long *h_scalar = nullptr, *d_scalar = nullptr;
  // one bit per word, the predicate of a large gather call (walks.cu)
  uint8_t *d_bits = nullptr;
  int32_t *d_hist = nullptr;
  char *h_ext = nullptr;           // pinned: the first extracted entries
  uint32_t *d_ext32 = nullptr;
  int64_t *d_ext64 = nullptr;
  int32_t *d_extv = nullptr;
  long long extract_cap = 0;
  // multisets (coldcore dct_hc.cu:46-56).  uploaded: the staged code, sorted
  // in pinned memory (buffer `up`).  active: the represented multiset, the
  // code of the last recount (buffer `act`) plus `delta`, what updates
  // added and removed since.  A recount is act = up: nothing is built.
  WordBuf code_buf[2];
  int up = 0, act = 0;
  bool code_in_flight = false;     // a copy from code_buf[up] may be running
  std::unordered_map<long long, int> delta;
  long long active_size = 0;
  MultHist up_hist, act_hist;      // distinct words per multiplicity
  long long stats[9] = {0};
  long long bytes_dev = 0, bytes_host = 0;
  unsigned long long dd_last = 0;
  bool torn = false;               // a call failed while it changed cnt
  bool layered_out = false;        // last transform left N_0..N_R
  // set side (setside.cu): the listed predicate set Z, cached per cnt state
  bool metric_table = false;       // support table proven == metric ball
  bool ball_ok = false;            // ... on a cell the set side takes
  bool set_ok = false;             // ... and the set side is on
  bool metric_tbl2 = false;        // dct_set_tbl2's table is the ball too
  int set_policy = 1;              // DCT_SET_GATHER: 0 off, 1 auto, 2 force
  long long set_min = -1;          // DCT_SET_MIN: walk size that tries it
  long long set_ratio = 2;         // DCT_SET_RATIO: set side while |Z| <= r|B|
  unsigned long long *zbuf = nullptr, *d_found = nullptr;
  long long zcap = 0, zcap_max = 0;
  unsigned long long cnt_ver = 1;  // bumped by every cnt mutation
  int z_mode = -1, z_target = 0, z_mu = 0;
  unsigned long long z_ver = 0;
  bool z_valid = false;
  long long z_n = 0;
  // swap_eval fast path: packed host/device staging and the drop lists
  char *h_swap = nullptr, *d_swap = nullptr;
  long long *d_list = nullptr;
  long long lcap = 0;
  // device greedy: state, placed words, words satisfied per placement
  // [the cell's BatchGreedyCell][its state][chunk keys][fresh words]
  char *d_greedy = nullptr;
  GreedySlot *h_greedy = nullptr;  // pinned ring of kGreedyRing states
  cudaEvent_t ev_greedy[kGreedyRing] = {nullptr};
  long long *d_placed = nullptr, *h_placed = nullptr;
  long long placed_cap = 0;
  long long *d_active = nullptr;   // active words (mu > 1: excluded again)
  long long active_cap = 0;
  Plan gather_plan;                // a predicate's counts, untuned
  bool gather_plan_ok = false;
  Plan plans[3][4];                // [init_mode][out_mode]
  bool plan_ok[3][4] = {{false}};
  bool tuned[3][4] = {{false}};
  float tune_ms[3][4] = {{0}};
};

State S;
cudaStream_t g_stream = nullptr;
int g_mu = 1;

// per-launch device timing of the last transform (DCT_TIMING=1 in the
// environment at load, or dct_b200_set_timing(1)): events around every
// launch, read after the transform's final synchronisation
constexpr int kMaxTimed = 64;
int g_timing = -1;
cudaEvent_t g_ev[kMaxTimed + 1];
float g_last_ms[kMaxTimed];
int g_last_n = 0;

bool timing_on() {
  if (g_timing < 0) g_timing = getenv("DCT_TIMING") ? 1 : 0;
  return g_timing == 1;
}

int timing_mark(int i) {
  if (!timing_on() || i > kMaxTimed) return 0;
  if (!g_ev[i]) CC_CK(cudaEventCreate(&g_ev[i]));
  CC_CK(cudaEventRecord(g_ev[i], g_stream));
  return 0;
}

long long round_up(long long x, long long a) { return (x + a - 1) / a * a; }

int dev_alloc(void **p, size_t bytes, int mode) {
  cudaError_t e;
  if (mode == 0) {
    e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) S.bytes_dev += bytes;
  } else {
    // the reference's LPDDR / managed placements (dct_hc.cu alloc_buf):
    // a B200 host has no coherent C2C memory, so both map to managed
    // memory that the driver pages in on demand
    e = cudaMallocManaged(p, bytes);
    if (e == cudaSuccess) S.bytes_host += bytes;
  }
  if (e != cudaSuccess) {
    fprintf(stderr, "coldcore_b200: allocation of %zu bytes failed: %s\n",
            bytes, cudaGetErrorString(e));
    *p = nullptr;
    return -1;
  }
  return 0;
}

bool valid_words(const long long *w, long long n) {
  if (n < 0 || (n && !w)) return false;
  for (long long i = 0; i < n; i++)
    if (w[i] < 0 || w[i] >= S.g.space) return false;
  return true;
}

// exact uint16 bound: no counter can exceed min(total, maxmult * |B|)
bool within_counter(long long total, long long maxmult) {
  long long b = maxmult * S.len;
  if (b > total) b = total;
  return b <= kCounterMax;
}

void hist_move(MultHist &h, int from, int to) {
  if (from > 0) {
    auto it = h.find(from);
    if (--it->second == 0) h.erase(it);
  }
  if (to > 0) ++h[to];
}

// the multiplicity of w in the active multiset
int active_count(long long w) {
  const auto it = S.delta.find(w);
  return (int)S.code_buf[S.act].count(w) +
         (it == S.delta.end() ? 0 : it->second);
}

// f(word, multiplicity) for every active word
template <typename F>
void each_active(F f) {
  const WordBuf &b = S.code_buf[S.act];
  for (long long i = 0; i < b.n;) {
    long long j = i + 1;
    while (j < b.n && b.p[j] == b.p[i]) j++;
    const auto it = S.delta.empty() ? S.delta.end() : S.delta.find(b.p[i]);
    const int c = (int)(j - i) + (it == S.delta.end() ? 0 : it->second);
    if (c > 0) f(b.p[i], c);
    i = j;
  }
  for (const auto &e : S.delta)
    if (e.second > 0 && !b.count(e.first)) f(e.first, e.second);
}

// an update's distinct words and their occurrences
typedef std::vector<std::pair<long long, int>> Batch1;
void count_words(const long long *words, int nw, Batch1 &batch) {
  std::vector<long long> v(words, words + nw);
  if (!std::is_sorted(v.begin(), v.end())) std::sort(v.begin(), v.end());
  for (size_t i = 0; i < v.size();) {
    size_t j = i + 1;
    while (j < v.size() && v[j] == v[i]) j++;
    batch.push_back({v[i], (int)(j - i)});
    i = j;
  }
}

void apply_active(const Batch1 &batch, int delta, long long nw) {
  for (const auto &e : batch) {
    const int before = active_count(e.first), d = delta * e.second;
    int &c = S.delta[e.first];
    c += d;
    if (c == 0) S.delta.erase(e.first);
    hist_move(S.act_hist, before, before + d);
  }
  S.active_size += delta * nw;
}

// validate an update batch against `active`; fills `batch`
int check_update(const long long *words, int nw, int delta, Batch1 &batch) {
  if (!valid_words(words, nw) || (delta != 1 && delta != -1)) return -1;
  count_words(words, nw, batch);
  if (delta == -1) {
    for (const auto &e : batch)
      if (active_count(e.first) < e.second) return -1;
  } else {
    long long mx = max_mult(S.act_hist);
    for (const auto &e : batch)
      mx = std::max(mx, (long long)active_count(e.first) + e.second);
    if (!within_counter(S.active_size + nw, mx)) return -1;
  }
  return 0;
}

// 0 where cnt is the counters of the active multiset; -1 without a cell, -8
// after a call that failed while it changed cnt, until a recount
int cnt_ready() {
  if (!S.live) return -1;
  if (!S.torn) return 0;
  fprintf(stderr, "coldcore_b200: an earlier call failed while it changed "
          "the counters; recount first\n");
  return -8;
}

int fetch_scalar(long long *r, int slot = 0) {
  CC_CK(cudaMemcpyAsync(S.h_scalar + slot, S.d_scalar + slot, 8,
                        cudaMemcpyDeviceToHost, g_stream));
  CC_CK(cudaStreamSynchronize(g_stream));
  *r = S.h_scalar[slot];
  return 0;
}

// a query's accumulator (d_scalar), and its result's way to the host
constexpr int kQuerySlot = 40, kTicketSlot = 44;
RedOut red_out(void *host = nullptr) {
  RedOut r;
  r.ticket = reinterpret_cast<unsigned *>(S.d_scalar + kTicketSlot);
  r.host = host ? static_cast<long long *>(host) : S.h_scalar + kQuerySlot;
  return r;
}
int query_result(long long *r) {
  CC_CK(cudaStreamSynchronize(g_stream));
  *r = *(volatile long long *)(S.h_scalar + kQuerySlot);
  return 0;
}

int stage_words(const long long *words, long long nb) {
  memcpy(S.h_words, words, (size_t)nb * 8);
  CC_CK(cudaMemcpyAsync(S.d_words, S.h_words, (size_t)nb * 8,
                        cudaMemcpyHostToDevice, g_stream));
  return 0;
}

// out[i] = f(words[i]) for many words: half the staging buffers at a time,
// so the host stages one half while the device works on the other.
// launch(dwords, nb, dout) queues one half's work.
template <typename F>
int staged_words(const long long *words, long long n, int32_t *out,
                 F launch) {
  const long long half = kStageCap / 2;
  const long long steps = (n + half - 1) / half;
  auto take = [&](long long i) -> int {      // step i's answers
    const int k = (int)(i & 1);
    CC_CK(cudaEventSynchronize(S.ev_stage[k]));
    memcpy(out + i * half, S.h_out + k * half,
           (size_t)std::min(half, n - i * half) * 4);
    return 0;
  };
  for (auto &ev : S.ev_stage)
    if (!ev) CC_CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  int rc = 0;
  for (long long i = 0; i < steps; i++) {
    const int k = (int)(i & 1);
    const long long nb = std::min(half, n - i * half);
    if (i >= 2 && (rc = take(i - 2))) return rc;
    memcpy(S.h_words + k * half, words + i * half, (size_t)nb * 8);
    CC_CK(cudaMemcpyAsync(S.d_words + k * half, S.h_words + k * half,
                          (size_t)nb * 8, cudaMemcpyHostToDevice, g_stream));
    if ((rc = launch(S.d_words + k * half, (int)nb, S.d_out + k * half)))
      return rc;
    CC_CK(cudaMemcpyAsync(S.h_out + k * half, S.d_out + k * half,
                          (size_t)nb * 4, cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaEventRecord(S.ev_stage[k], g_stream));
  }
  for (long long i = std::max(0LL, steps - 2); i < steps; i++)
    if ((rc = take(i))) return rc;
  return 0;
}

WalkArgs walk_args() {
  WalkArgs w;
  w.g = S.g;
  w.g.mu = g_mu;
  const bool ox = S.fmt == 1 && S.tbl2;
  w.tbl = ox ? S.tbl2 : S.tbl;
  w.slots = ox ? S.slots2 : S.slots;
  w.len = S.len;
  w.cnt = S.cnt;
  w.pk = ox ? S.pk2 : S.pk;
  w.ent = S.ent;
  w.noff = S.noff;
  return w;
}

void free_all() {
  if (g_stream) cudaStreamSynchronize(g_stream);
  auto F = [](void *p) { if (p) cudaFree(p); };
  auto FH = [](void *p) { if (p) cudaFreeHost(p); };
  F(S.layers); F(S.cnt); F(S.owner); F(S.tbl); F(S.tbl2); F(S.d_code);
  F(S.pk); F(S.pk2); F(S.ent);
  F(S.d_bounds);
  F(S.d_words); F(S.d_out); F(S.d_scalar); F(S.d_hist); F(S.d_ext32);
  F(S.d_ext64); F(S.d_extv); F(S.zbuf); F(S.d_found);
  F(S.d_swap); F(S.d_list); FH(S.h_swap);
  for (WordBuf &b : S.code_buf) FH(b.p);
  F(S.d_greedy); F(S.d_placed); F(S.d_active); FH(S.h_placed);
  FH(S.h_greedy);
  for (cudaEvent_t e : S.ev_greedy) if (e) cudaEventDestroy(e);
  for (cudaEvent_t e : S.ev_stage) if (e) cudaEventDestroy(e);
  F(S.d_bits);
  FH(S.h_layers);
  FH(S.h_words); FH(S.h_out); FH(S.h_scalar); FH(S.h_ext);
  S.~State();
  new (&S) State();
}

// ------------------------------------------------------------ planner
// shared-memory budget of one tile (CC_SMEM_BUDGET_KB overrides; read
// whenever a plan is built, i.e. once per cell and transform kind)
size_t smem_budget() {
  const char *e = getenv("CC_SMEM_BUDGET_KB");
  long long b = e ? atoll(e) * 1024 : 100 * 1024;
  if (b < 16 * 1024) b = 16 * 1024;
  if (b > 220 * 1024) b = 220 * 1024;
  return (size_t)b;
}

// Schedule knobs of a group plan (planner.cu): CC_SMEM_BUDGET_KB /
// CC_PIPE override the defaults; the autotuner tries several.
Knobs default_knobs() {
  const char *pe = getenv("CC_PIPE");
  return {smem_budget(), pe ? atoi(pe) : 1};
}

// 16-bit planes between the launches of one transform are exact when no
// intermediate layer value can pass 65535: a layer counts words within a
// distance, so it is at most the occurrences (<= 65535 by the rule that
// set_code enforces) for a code, and at most |B| for a predicate.  They sit
// from int32 plane 1 on, clear of the int32 map in plane 0; a transform
// that outputs every layer keeps int32 planes throughout.  CC_HALF=0 turns
// them off.
bool half_planes_ok(int src, int dst) {
  const char *e = getenv("CC_HALF");
  if (e && atoi(e) == 0) return false;
  if (S.R1 < 2 || dst == kDstLayers) return false;
  return src == kSrcCode || S.len <= 65535;
}

Plan build_group_plan(int src, int dst, Knobs kn) {
  Plan P;
  PlanPtrs ptr{S.layers, S.plane, S.cnt, S.d_code, S.codeM, nullptr};
  kn.half = half_planes_ok(src, dst) ? 1 : 0;
  ptr.layers16 = reinterpret_cast<uint16_t *>(S.layers + S.plane);
  Geometry g = transform_geometry(S.g);
  g.mu = g_mu;
  P.groups = plan_groups(g, S.R1, ptr, src, dst, kn);
  if (kn.pad) {
    // a padded plan or none (the tuner then skips this knob setting)
    if (!kn.half || !pad_plan(P.groups, g, ptr, dst, S.R1,
                              (long long)(S.nplanes - 1) * S.plane * 2))
      P.groups.clear();
    return P;
  }
  // CC_TMA=1: every group the streamed form serves takes it (64-word rows
  // first, three stages where they fit); the autotuner otherwise times it
  // beside the other forms
  const char *ue = getenv("CC_U8");
  const bool u8_off = ue && atoi(ue) == 0;
  if (kn.u8) {
    // 8-bit planes after the streamed first group, or no plan
    stream_groups(P.groups, S.R1);
    if (u8_off || !u8_plan(P.groups, S.R1,
                         (long long)(S.nplanes - 1) * S.plane * 2)) P.groups.clear();
    return P;
  }
  const char *te = getenv("CC_TMA");
  if (te && atoi(te) == 1) {
    stream_groups(P.groups, S.R1);
    if (!u8_off) u8_plan(P.groups, S.R1,
                         (long long)(S.nplanes - 1) * S.plane * 2);
  }
  return P;
}

bool any_wide_axis() {
  for (int j = 0; j < S.g.n; j++)
    if (S.g.ax[j] > 16) return true;
  return false;
}

// window path: pass j reads buf[j] and writes buf[j+1]; buffers are planes
// 0..2, kSrc from cnt (-1) or a plane, the last one the map / cnt (-2)
Plan build_window_plan(int init_mode, int out_mode) {
  Plan P;
  P.window = true;
  const Geometry &g = S.g;
  // passes: two axes at a time where the pair form applies
  std::vector<std::pair<int, int>> axes;        // (first, how many)
  for (int j = 0; j < g.n;) {
    const int k = j + 1 < g.n && window_pair_ok(g.pw[j], g.ax[j], g.R) ? 2 : 1;
    axes.push_back({j, k});
    j += k;
  }
  const int n = (int)axes.size();
  std::vector<int> buf(n + 1);
  buf[0] = init_mode == 0 ? 2 : -1;
  P.scatter_plane = init_mode == 0 ? 2 : -1;
  buf[n] = out_mode == 2 ? -2 : 0;
  for (int j = n - 1; j >= 1; j--) {
    const int nxt = buf[j + 1];
    int pick = 0;
    while (pick == nxt || (j == 1 && pick == buf[0])) pick++;
    buf[j] = pick;
  }
  for (int j = 0; j < n; j++) {
    WindowArgs w{};
    const int s = buf[j], d = buf[j + 1];
    if (s == -1) w.src16 = S.cnt; else w.src32 = S.layers + s * S.plane;
    if (d == -2) w.dst16 = S.cnt; else w.dst32 = S.layers + d * S.plane;
    w.pmode = kPredEq;
    w.mu = g_mu;
    w.space = g.space;
    w.stride = g.pw[axes[j].first];
    w.q = g.ax[axes[j].first];
    w.R = g.R;
    w.grid = g.prob == kGrid;
    w.q2 = axes[j].second == 2 ? g.ax[axes[j].first + 1] : 0;
    P.passes.push_back(w);
  }
  return P;
}

Plan make_plan(int init_mode, int out_mode, Knobs kn) {
  const int src = init_mode == 0 ? kSrcCode : kSrcCnt;
  const int dst = out_mode == 1 ? kDstMap
                  : out_mode == 2 ? kDstCnt : kDstLayers;
  if ((S.g.prob == kTorus || S.g.prob == kGrid) && any_wide_axis())
    return build_window_plan(init_mode, out_mode);
  return build_group_plan(src, dst, kn);
}

Plan &plan_for(int init_mode, int out_mode) {
  if (!S.plan_ok[init_mode][out_mode]) {
    Plan P;
    // CC_TMA=1 also asks for the padded plan where a cell has one
    const char *te = getenv("CC_TMA");
    if (te && atoi(te) == 1) {
      Knobs kn = default_knobs();
      kn.pad = 1;
      P = make_plan(init_mode, out_mode, kn);
    }
    if (P.groups.empty() && !P.window)
      P = make_plan(init_mode, out_mode, default_knobs());
    S.plans[init_mode][out_mode] = P;
    S.plan_ok[init_mode][out_mode] = true;
  }
  return S.plans[init_mode][out_mode];
}

void set_predicate(int init_mode, int *pm, int *pt) {
  *pm = kPredEq;
  *pt = 0;
  if (init_mode == 1) {
    if (g_mu == 1) *pt = 0; else *pm = kPredDef;
  } else if (init_mode == 2) {
    if (g_mu == 1) *pt = 1; else *pm = kPredCrit;
  }
}

// Device bytes a streamed transform may allocate: CC_OOC_BUDGET_KB, else
// 80% of the free device memory less 256 MiB.
long long ooc_budget() {
  if (const char *e = getenv("CC_OOC_BUDGET_KB")) return atoll(e) << 10;
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return std::max(0LL, (long long)(fr / 10 * 8) - (256LL << 20));
}

// A transform of a layers_mode-1 cell: the code (uploaded, sorted) or cnt
// in, the map (plane 0) or cnt out on the device, or every layer out into
// the host planes.
int run_streamed(int init_mode, int out_mode) {
  CC_CK(cudaStreamSynchronize(g_stream));
  void *out = out_mode == 1 ? static_cast<void *>(S.layers)
              : out_mode == 2 ? static_cast<void *>(S.cnt) : nullptr;
  float ms[2] = {0, 0};
  const long long M = init_mode == 0 ? S.codeM : 0;
  const int rc = dct_b200_ooc_transform(
      S.g.prob, S.g.n, S.g.ax, S.g.R, init_mode, out_mode, g_mu,
      M ? S.code_buf[S.up].p : nullptr, M, S.cnt, out, S.h_layers,
      S.h_layers_bytes, ooc_budget(), 0, ms);
  if (rc) return rc;
  g_last_n = 0;
  if (timing_on()) {
    g_last_ms[0] = ms[0];
    g_last_ms[1] = ms[1];
    g_last_n = 2;
  }
  return 0;
}

int run_transform(int init_mode, int out_mode) {
  if (const int rc = tma_fault_take()) return rc;   // a tuning launch's
  if (S.streamed) {
    const int rc = run_streamed(init_mode, out_mode);
    // begun: neither refused (arguments, no split, host planes too few) nor
    // out of device memory for its pieces
    S.torn = S.torn || (out_mode == 2 && rc < -5 &&
                        rc != -(100 + (int)cudaErrorMemoryAllocation));
    return rc;
  }
  Plan &P = plan_for(init_mode, out_mode);
  int pm, pt;
  set_predicate(init_mode, &pm, &pt);
  int nt = 0, rc = 0;
  if (!P.window && P.groups.empty()) return -1;   // the planner found no tile
  if (P.window) {
    if (init_mode == 0) {
      int32_t *pl = S.layers + P.scatter_plane * S.plane;
      CC_CK(cudaMemsetAsync(pl, 0, (size_t)S.g.space * 4, g_stream));
      rc = launch_scatter(pl, S.d_code, S.codeM, g_stream);
      if (rc) return rc;
    }
    S.torn = S.torn || out_mode == 2;    // until the recount has drained
    if ((rc = timing_mark(nt))) return rc;
    for (auto &w : P.passes) {
      WindowArgs x = w;
      x.pmode = pm;
      x.ptarget = pt;
      x.mu = g_mu;
      if ((rc = launch_window(x, g_stream))) return rc;
      if ((rc = timing_mark(++nt))) return rc;
    }
  } else {
    if (init_mode == 0) {
      const GroupArgs &a0 = P.groups[0].a;
      const long long need = a0.ntiles + 1;
      if (need > S.bounds_cap) {
        if (S.d_bounds) cudaFree(S.d_bounds);
        S.d_bounds = nullptr;
        CC_CK(cudaMalloc(&S.d_bounds, (size_t)need * 8));
        S.bounds_cap = need;
      }
      rc = launch_code_bounds(S.d_code, S.codeM,
                              (long long)a0.Bo * a0.mid * a0.inner,
                              a0.ntiles,
                              S.d_bounds, g_stream);
      if (rc) return rc;
    }
    S.torn = S.torn || out_mode == 2;
    if ((rc = timing_mark(nt))) return rc;
    for (auto &gp : P.groups) {
      GroupPlan p = gp;
      p.a.pmode = pm;
      p.a.ptarget = pt;
      p.a.mu = g_mu;
      p.a.code = S.d_code;
      p.a.ncode = S.codeM;
      p.a.code_bounds = S.d_bounds;
      if ((rc = launch_group(p, g_stream))) return rc;
      if ((rc = timing_mark(++nt))) return rc;
    }
  }
  g_last_n = 0;
  if (timing_on()) {
    CC_CK(cudaStreamSynchronize(g_stream));
    const int m = nt < kMaxTimed ? nt : kMaxTimed;
    for (int i = 0; i < m; i++)
      CC_CK(cudaEventElapsedTime(&g_last_ms[i], g_ev[i], g_ev[i + 1]));
    g_last_n = m;
    if (getenv("DCT_TIMING"))
      for (int i = 0; i < m; i++)
        fprintf(stderr, "DCT_TIMING transform(%d,%d) launch %d: %.4f ms\n",
                init_mode, out_mode, i, g_last_ms[i]);
  }
  return 0;
}

// CC_TUNE_LOG=1: every timed variant of the per-launch tuning on stderr
bool tune_log() {
  static const bool on = [] {
    const char *e = getenv("CC_TUNE_LOG");
    return e && atoi(e) == 1;
  }();
  return on;
}

// Per-launch tuning of plan P with its grouping fixed: every register block
// size, row width, prefetching form and CTA width of each launch, each
// timed alone (three launches after a warm one).  A launch run again works
// in place on its own planes, which only scrambles values; the real
// transform runs from scratch afterwards.
int tune_launches(Plan &P, int init_mode, int out_mode, cudaEvent_t e0,
                  cudaEvent_t e1) {
  // one transform with P: its code bounds (a recount's first group) and
  // planes are then the ones every variant below reads; the variants keep
  // the first group's tiles, so the bounds stay valid for all of them
  S.plans[init_mode][out_mode] = P;
  S.plan_ok[init_mode][out_mode] = true;
  int rc = run_transform(init_mode, out_mode);
  if (rc) return rc;
  int pm, pt;
  set_predicate(init_mode, &pm, &pt);
  for (size_t gi = 0; gi < P.groups.size(); gi++) {
    std::vector<GroupPlan> vars = group_variants(P.groups[gi], S.R1,
                                                 220 << 10);
    if (vars.size() < 2) continue;
    float bv = 1e30f;
    size_t bi = 0;
    for (size_t vi = 0; vi < vars.size(); vi++) {
      GroupPlan p = vars[vi];
      p.a.pmode = pm;
      p.a.ptarget = pt;
      p.a.mu = g_mu;
      p.a.code = S.d_code;
      p.a.ncode = S.codeM;
      p.a.code_bounds = S.d_bounds;
      if ((rc = prepare_group(p))) return rc;
      rc = launch_group(p, g_stream);
      if (rc == -9) { rc = 0; continue; }     // a form the launcher refused
      if (rc) return rc;
      CC_CK(cudaEventRecord(e0, g_stream));
      for (int r = 0; r < 3; r++)
        if ((rc = launch_group(p, g_stream))) return rc;
      CC_CK(cudaEventRecord(e1, g_stream));
      CC_CK(cudaEventSynchronize(e1));
      float ms = 0;
      CC_CK(cudaEventElapsedTime(&ms, e0, e1));
      if (ms < bv) { bv = ms; bi = vi; }
      if (tune_log())
        fprintf(stderr, "CC_TUNE_LOG transform(%d,%d) group %zu variant %zu: "
                "kernel %d tma %d stages %d W %d threads %d grid %d smem %zu "
                "pipe %d in8 %d out8 %d: %.4f ms\n", init_mode, out_mode, gi,
                vi, p.kernel, p.a.tma, p.a.stages, p.a.W, p.threads, p.grid,
                p.smem, p.a.pipe, p.a.in8, p.a.out8, ms / 3);
    }
    P.groups[gi] = vars[bi];
  }
  return 0;
}

// the axes, rows and prefetching of each launch: two knob settings that
// give the same grouping are tuned once
std::vector<long long> grouping_key(const Plan &P) {
  std::vector<long long> k;
  for (const auto &g : P.groups)
    k.push_back(((long long)g.a.k << 32) | (g.a.W << 8) | (g.a.pipe << 1) |
                g.a.pair_axis | ((g.a.pitch ? 1LL : 0LL) << 24) |
                ((long long)(g.a.in8 | g.a.out8) << 25));
  return k;
}

// Autotuner: on the first transform of a kind on a large cell, every
// distinct grouping the knob settings give (shared-memory budget x
// prefetching mode) gets its per-launch tuning, and then the whole tuned
// transform is timed (CUDA events on the engine stream, two runs after a
// warm one); the fastest is kept.  Every schedule computes the same
// integers, so tuning runs are ordinary transforms.  CC_TUNE=0 turns it
// off; explicit CC_PIPE / CC_SMEM_BUDGET_KB settings also pin the schedule.
int autotune(int init_mode, int out_mode) {
  if (S.streamed || S.tuned[init_mode][out_mode]) return 0;
  S.tuned[init_mode][out_mode] = true;
  const char *te = getenv("CC_TUNE");
  if ((te && atoi(te) == 0) || getenv("CC_PIPE") ||
      getenv("CC_SMEM_BUDGET_KB") || S.g.space < (1LL << 22) ||
      ((S.g.prob == kTorus || S.g.prob == kGrid) && any_wide_axis()))
    return 0;
  static const Knobs cands[] = {{100 << 10, 1}, {160 << 10, 1},
                                {64 << 10, 1}, {200 << 10, 1},
                                {100 << 10, 2}, {100 << 10, 3},
                                {200 << 10, 3}, {160 << 10, 2},
                                {200 << 10, 2},
                                // padded plans (ternary cells)
                                {64 << 10, 1, 0, 1, 1},
                                {100 << 10, 1, 0, 1, 1},
                                {160 << 10, 1, 0, 1, 1},
                                {200 << 10, 1, 0, 1, 1},
                                // 8-bit planes after the first group
                                {64 << 10, 1, 0, 1, 0, 1},
                                {100 << 10, 1, 0, 1, 0, 1},
                                {160 << 10, 1, 0, 1, 0, 1}};
  EventPair ev;
  int rc = ev.create();
  if (rc) return rc;
  cudaEvent_t e0 = ev.e0, e1 = ev.e1;
  float best = 1e30f;
  Plan keep;
  std::vector<std::vector<long long>> seen;
  for (const Knobs &kn : cands) {
    Plan P = make_plan(init_mode, out_mode, kn);
    if (P.window || P.groups.empty()) continue;
    const std::vector<long long> key = grouping_key(P);
    bool dup = false;
    for (const auto &k : seen) dup = dup || k == key;
    if (dup) continue;
    seen.push_back(key);
    if ((rc = tune_launches(P, init_mode, out_mode, e0, e1))) break;
    S.plans[init_mode][out_mode] = P;
    S.plan_ok[init_mode][out_mode] = true;
    if ((rc = run_transform(init_mode, out_mode))) break;      // warm
    CC_CK(cudaEventRecord(e0, g_stream));
    for (int r = 0; r < 2 && !rc; r++) rc = run_transform(init_mode, out_mode);
    if (rc) break;
    CC_CK(cudaEventRecord(e1, g_stream));
    CC_CK(cudaEventSynchronize(e1));
    float ms = 0;
    CC_CK(cudaEventElapsedTime(&ms, e0, e1));
    if (tune_log()) {
      fprintf(stderr, "CC_TUNE_LOG transform(%d,%d) plan budget %zu KB pipe "
              "%d pad %d u8 %d axes", init_mode, out_mode, kn.budget >> 10,
              kn.pipe, kn.pad, kn.u8);
      for (const auto &gp : P.groups)
        fprintf(stderr, " %d", gp.a.k + gp.a.pair_axis);
      fprintf(stderr, ": %.4f ms\n", ms / 2);
    }
    if (ms < best) { best = ms; keep = P; }
  }
  if (rc) return rc;
  if (!keep.groups.empty()) S.plans[init_mode][out_mode] = keep;
  else S.plans[init_mode][out_mode] = make_plan(init_mode, out_mode,
                                                default_knobs());
  S.plan_ok[init_mode][out_mode] = true;
  S.tune_ms[init_mode][out_mode] = best < 1e29f ? best / 2 : 0.f;
  return 0;
}

int ensure_stream() {
  if (!g_stream)
    CC_CK(cudaStreamCreateWithFlags(&g_stream, cudaStreamNonBlocking));
  return 0;
}

// v1 packed table -> SoA slots; -1 on malformed entries
int unpack_v1(const uint64_t *pat, long long len, std::vector<int32_t> &out,
              int *slots) {
  int w = 1;
  for (long long t = 0; t < len; t++) {
    int k = 0;
    while (k < 8 && ((pat[t] >> (8 * k)) & 255u)) k++;
    if (k > w) w = k;
  }
  out.assign((size_t)w * len, 0);
  for (long long t = 0; t < len; t++) {
    for (int k = 0; k < 8; k++) {
      const unsigned b = (unsigned)(pat[t] >> (8 * k)) & 255u;
      if (!b) break;
      const int pos = (int)(b >> 4), dl = (int)(b & 15u);
      if (pos >= S.g.n || dl < 1 || dl >= S.g.ax[pos]) return -1;
      out[(size_t)k * len + t] = (pos << 24) | dl;
    }
  }
  *slots = w;
  return 0;
}

int init_common(int problem, int n, const int *ax, int R, long long len,
                int extract_cap, int layers_mode, int cnt_mode,
                int use_owner) {
  if (n < 1 || n > kMaxAxes || R < 1 || !ax || len < 1 || len > INT_MAX ||
      extract_cap < 1)
    return -1;
  const bool layered = problem == kHamming || problem == kLee;
  if (problem < 0 || problem > 3) return -1;
  if (layered && R + 1 > kMaxLayers) return -1;
  for (int i = 0; i < n; i++) {
    if (ax[i] < 2 || ax[i] >= (1 << 24)) return -1;
    if (layered && ax[i] > 16) return -1;        // register / tile kernels
    if (problem == kTorus && (ax[i] < 3 || 2 * R + 1 > ax[i])) return -1;
  }
  long long space = 1;
  for (int i = 0; i < n; i++) {
    if (space > (1LL << 40) / ax[i]) return -2;
    space *= ax[i];
  }
  free_all();
  int rc = ensure_stream();
  if (rc) return rc;
  // coldcore's launch-size knob: 256 CTAs at least (dct_hc.cu:274-276)
  const char *bl = getenv("DCT_BLOCKS");
  g_dct_blocks = bl ? std::max(256, atoi(bl)) : 0;
  S.g.prob = problem; S.g.n = n; S.g.R = R; S.g.mu = g_mu;
  S.g.space = space;
  S.g.pw[0] = 1;
  for (int i = 0; i < n; i++) {
    S.g.ax[i] = ax[i];
    S.g.pw[i + 1] = S.g.pw[i] * ax[i];
  }
  S.R1 = layered ? R + 1 : 1;
  S.nplanes = layered ? R + 1 : 3;
  S.plane = round_up(space, kPlaneAlign);
  S.layers_mode = layers_mode;
  S.cnt_mode = cnt_mode;
  S.use_owner = use_owner;
  S.len = len;
  // layers_mode 1, the reference's host placement of the layer planes
  // (dctcore_core.cuh:86-119): pinned host planes streamed through the
  // device (cells with a two-phase split, i.e. group-transform cells of
  // two or more axes); otherwise, and for mode 2, managed planes
  bool wide = false;
  for (int i = 0; i < n; i++) wide = wide || ax[i] > 16;
  S.streamed = layers_mode == 1 && n >= 2 && !wide;
  if (S.streamed) {
    if (dev_alloc((void **)&S.layers, (size_t)S.plane * 4, 0)) {
      free_all(); return -3;
    }
    S.h_layers_bytes = (long long)S.R1 * space * 4;
    if (cudaHostAlloc((void **)&S.h_layers, (size_t)S.h_layers_bytes,
                      cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      S.h_layers = nullptr;
      fprintf(stderr, "coldcore_b200: pinned host planes of %lld bytes "
              "failed\n", S.h_layers_bytes);
      free_all(); return -3;
    }
    S.bytes_host += S.h_layers_bytes;
  } else if (dev_alloc((void **)&S.layers, (size_t)S.plane * S.nplanes * 4,
                       layers_mode)) { free_all(); return -3; }
  S.cnt_len = round_up(space, kPlaneAlign);
  if (dev_alloc((void **)&S.cnt, (size_t)S.cnt_len * 2, cnt_mode)) {
    free_all(); return -4;
  }
  CC_CK(cudaMemsetAsync(S.cnt, 0, (size_t)S.cnt_len * 2, g_stream));
  if (use_owner) {
    if (dev_alloc((void **)&S.owner, (size_t)space * 4, cnt_mode)) {
      free_all(); return -5;
    }
  }
  CC_CK(cudaMalloc(&S.d_words, kStageCap * 8));
  CC_CK(cudaMalloc(&S.d_out, kStageCap * 4));
  CC_CK(cudaMalloc(&S.d_scalar, 64 * 8));
  CC_CK(cudaMalloc(&S.d_hist, 4096 * 4));
  CC_CK(cudaHostAlloc((void **)&S.h_words, kStageCap * 8,
                      cudaHostAllocDefault));
  CC_CK(cudaHostAlloc((void **)&S.h_out, kStageCap * 4,
                      cudaHostAllocDefault));
  CC_CK(cudaHostAlloc((void **)&S.h_scalar, 64 * 8, cudaHostAllocDefault));
  CC_CK(cudaMemsetAsync(S.d_scalar, 0, 64 * 8, g_stream));
  CC_CK(cudaMemsetAsync(S.d_hist, 0, 4096 * 4, g_stream));
  S.bytes_dev += kStageCap * 12 + 64 * 8 + 4096 * 4;
  S.extract_cap = extract_cap;
  CC_CK(cudaMalloc(&S.d_ext32, (size_t)extract_cap * 4));
  CC_CK(cudaMalloc(&S.d_ext64, (size_t)extract_cap * 8));
  CC_CK(cudaMalloc(&S.d_extv, (size_t)extract_cap * 4));
  S.bytes_dev += (long long)extract_cap * 16;
  S.live = true;
  return 0;
}

int upload_table(const std::vector<int32_t> &soa, int slots, int32_t **dst,
                 int *dslots, uint32_t **dpk) {
  CC_CK(cudaMalloc(dst, soa.size() * 4));
  CC_CK(cudaMemcpyAsync(*dst, soa.data(), soa.size() * 4,
                        cudaMemcpyHostToDevice, g_stream));
  S.bytes_dev += (long long)soa.size() * 4;
  *dslots = slots;
  std::vector<uint32_t> pk;
  std::vector<int4> ent;
  if (pack_walk(S.g, soa, slots, S.len, pk, ent)) {
    CC_CK(cudaMalloc(dpk, pk.size() * 4));
    CC_CK(cudaMemcpyAsync(*dpk, pk.data(), pk.size() * 4,
                          cudaMemcpyHostToDevice, g_stream));
    S.bytes_dev += (long long)pk.size() * 4;
    if (!S.ent) {                        // the cell's, whatever the table
      CC_CK(cudaMalloc(&S.ent, ent.size() * sizeof(int4)));
      CC_CK(cudaMemcpyAsync(S.ent, ent.data(), ent.size() * sizeof(int4),
                            cudaMemcpyHostToDevice, g_stream));
      S.noff = (int)ent.size();
    }
  }
  CC_CK(cudaStreamSynchronize(g_stream));
  return 0;
}

int finish_init(long long *bytes) {
  CC_CK(cudaStreamSynchronize(g_stream));
  if (bytes) *bytes = S.bytes_dev + S.bytes_host;
  return 0;
}

// May a gather count listed words by distance instead of walking the table?
// Only where the table is exactly the metric ball (coldcore dct_hc.cu:158-204
// states the same test), on at most 16 axes of at most 16 values.
bool table_is_ball() {
  if (S.g.n > 16) return false;
  for (int i = 0; i < S.g.n; i++)
    if (S.g.ax[i] > 16) return false;
  return S.metric_table;
}

void set_side_init(const std::vector<int32_t> &soa, int slots) {
  const char *sp = getenv("DCT_SET_GATHER");
  const char *sm = getenv("DCT_SET_MIN");
  const char *sr = getenv("DCT_SET_RATIO");
  S.set_policy = sp ? atoi(sp) : 1;
  S.set_min = sm ? atoll(sm) : -1;
  S.set_ratio = sr ? std::max(1LL, atoll(sr)) : 2;
  S.metric_table = metric_ball_table(S.g, soa, slots, S.len);
  S.ball_ok = table_is_ball();
  S.set_ok = S.set_policy != 0 && S.ball_ok;
  S.zcap_max = std::min<long long>(S.g.space, 1LL << 27);
  S.z_mode = -1;
}

// the walk of nb candidates reads nb*|B| counters: worth trying the list?
bool want_set(int mode, int target, int nb) {
  if (!S.set_ok || !(mode == kPredDef || (mode == kPredEq && target == 0)))
    return false;
  if (S.set_policy == 2) return true;
  const long long walk = (long long)nb * S.len;
  const long long lim = S.set_min >= 0 ? S.set_min
                        : std::max<long long>(S.g.space / 8, 1LL << 21);
  return walk >= lim;
}

// List Z = {x : pred(cnt[x])} for the current cnt, unless it is listed
// already.  Returns 1 when the list is usable (|Z| <= ratio*|B|), 0 when
// the caller must walk, negative on error.
int ensure_zlist(int mode, int target) {
  if (S.z_mode == mode && S.z_target == target && S.z_mu == g_mu &&
      S.z_ver == S.cnt_ver)
    return S.z_valid ? 1 : 0;
  const long long lim = std::min(S.len * S.set_ratio, S.zcap_max);
  if (!S.d_found) CC_CK(cudaMalloc(&S.d_found, 8));
  long long want = std::min<long long>(std::max<long long>(S.len / 4, 4096),
                                       1LL << 22);
  want = std::min(want, lim);
  for (;;) {
    if (S.zcap < want) {
      if (S.zbuf) CC_CK(cudaFree(S.zbuf));
      S.zbuf = nullptr;
      S.zcap = 0;
      CC_CK(cudaMalloc(&S.zbuf, (size_t)want * 8));
      S.zcap = want;
    }
    Geometry g = S.g;
    g.mu = g_mu;
    int rc = launch_list_pred(g, S.cnt, mode, target, S.zbuf, S.zcap,
                              S.d_found, g_stream);
    if (rc) return rc;
    CC_CK(cudaMemcpyAsync(S.h_scalar + 8, S.d_found, 8,
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaStreamSynchronize(g_stream));
    const long long found = S.h_scalar[8];
    S.stats[2]++;
    if (found > S.zcap && found <= lim) { want = found; continue; }
    S.z_mode = mode; S.z_target = target; S.z_mu = g_mu;
    S.z_ver = S.cnt_ver;
    S.z_n = found;
    S.z_valid = found <= lim;
    if (!S.z_valid) S.stats[3]++;
    return S.z_valid ? 1 : 0;
  }
}

// launch the gather of nb staged words into dout (set side or walk)
int gather_launch(int mode, int target, int nb, const long long *dw,
                  int32_t *dout, bool zeroed) {
  const int zs = want_set(mode, target, nb) ? ensure_zlist(mode, target) : 0;
  if (zs < 0) return zs;
  if (zs == 1) {
    S.stats[0]++;
    if (S.z_n > 32768) S.stats[7]++;
    Geometry g = S.g;
    g.mu = g_mu;
    return launch_gather_set(g, dw, nb, S.zbuf, S.z_n, dout, zeroed,
                             g_stream);
  }
  S.stats[1]++;
  const WalkArgs wa = walk_args();
  uint8_t *bits = nullptr;
  if (gather_bits_pay(wa, nb)) {
    if (!S.d_bits)
      CC_CK(cudaMalloc(&S.d_bits, (size_t)((S.g.space + 7) / 8 + 16)));
    bits = S.d_bits;
  }
  return launch_gather(wa, dw, nb, mode, target, dout, zeroed, g_stream,
                       bits);
}

// A transform of the predicate counts EVERY word's ball at once, so a call
// that would walk enough of them (candidates x |B|) is a transform and a
// read: 10^5 candidates of ternary n = 16, R = 4 walk 3.4e9 patterns in
// 5.5 ms, the transform takes 0.48 ms.
//
// The counts go to the last layer plane and nothing else that a caller can
// see changes: the launches pass 16-bit planes, which start at plane 1 and
// leave plane 0, the map, alone, and by the last launch they end before the
// last plane.  So: a layered cell in device memory with R >= 3, a table that
// is the metric ball (the walk's answer), 16-bit exactness, and no exact
// layers of an earlier call in the planes.  (The table in use: dct_use_fmt's
// second one may hold other patterns.)  Returns the plan, or nullptr.
// An untuned cell takes the streamed forms without tuning (a tuning run
// costs hundreds of such calls, and would write the map).
Plan *gather_transform_plan() {
  if (S.streamed || S.layers_mode != 0 || S.cnt_mode != 0 || !S.ball_ok ||
      (S.fmt == 1 && !S.metric_tbl2) || S.layered_out || S.R1 < 4 ||
      !half_planes_ok(kSrcCnt, kDstMap))
    return nullptr;
  Plan *P = nullptr;
  if (S.tuned[1][1] && S.plan_ok[1][1]) {
    P = &S.plans[1][1];
  } else {
    if (!S.gather_plan_ok) {
      S.gather_plan_ok = true;
      Knobs kn = default_knobs();
      kn.pad = 1;
      S.gather_plan = make_plan(1, 1, kn);
      if (S.gather_plan.groups.empty()) {
        S.gather_plan = make_plan(1, 1, default_knobs());
        const char *te = getenv("CC_TMA");
        if (!(te && atoi(te) == 0)) stream_groups(S.gather_plan.groups, S.R1);
      }
    }
    P = &S.gather_plan;
  }
  if (P->window || P->groups.size() < 2) return nullptr;
  for (size_t i = 0; i + 1 < P->groups.size(); i++)
    if (!P->groups[i].a.out16 && !P->groups[i].a.out8) return nullptr;
  const GroupArgs &last = P->groups.back().a;
  // the last launch's source planes end before the last plane
  if (!last.in16 || last.in8 ||
      (long long)S.R1 * last.plane * 2 > (long long)(S.R1 - 2) * S.plane * 4)
    return nullptr;
  return P;
}

// Microseconds of a walk of nw candidates (k_gather_tiled over a bit plane:
// 620,000 patterns a microsecond) against the transform: launches, and its
// bytes at 3 TB/s.  CC_GATHER_TRANSFORM = 0 / 1 pins the choice.
bool gather_transform_pays(const Plan &P, long long nw) {
  const char *e = getenv("CC_GATHER_TRANSFORM");
  if (e) return atoi(e) != 0;
  double us = 20.0 + 5.0 * P.groups.size();
  for (const auto &gp : P.groups) us += group_bytes(gp.a) / 3.0e6;
  return (double)nw * (double)S.len / 6.2e5 > us;
}

int run_gather_transform(const Plan &P, int mode, int target) {
  for (const auto &gp : P.groups) {
    GroupPlan p = gp;
    p.a.pmode = mode;
    p.a.ptarget = target;
    p.a.mu = g_mu;
    p.a.map = S.layers + (long long)(S.R1 - 1) * S.plane;
    const int rc = launch_group(p, g_stream);
    if (rc) return rc;
  }
  return 0;
}

int gather_impl(const long long *words, int nwords, int mode, int target,
                int32_t *out) {
  if (nwords <= 0) return 0;
  if (!out || !valid_words(words, nwords)) return -1;
  // one route for the whole call: the set side where it serves, else the
  // transform where that is cheaper than the walk
  const int32_t *counts = nullptr;
  Plan *P = (long long)nwords * S.len > (1 << 24) ? gather_transform_plan()
                                                  : nullptr;
  if (P && gather_transform_pays(*P, nwords)) {
    const int nb = (int)std::min<long long>(kStageCap, nwords);
    const int zs = want_set(mode, target, nb) ? ensure_zlist(mode, target) : 0;
    if (zs < 0) return zs;
    if (zs == 0) {
      const int rc = run_gather_transform(*P, mode, target);
      if (rc) return rc;
      counts = S.layers + (long long)(S.R1 - 1) * S.plane;
    }
  }
  if (counts) {
    S.stats[1] += (nwords + kStageCap - 1) / kStageCap;
    S.stats[8]++;
    const int rc = staged_words(
        words, nwords, out, [&](const long long *w, int nb, int32_t *o) {
          return launch_read_at(counts, w, nb, o, g_stream);
        });
    // the streams have drained: a launch that timed out is this call's
    return rc ? rc : tma_fault_take();
  }
  for (long long off = 0; off < nwords; off += kStageCap) {
    const int nb = (int)std::min<long long>(kStageCap, nwords - off);
    int rc = stage_words(words + off, nb);
    if (rc) return rc;
    rc = gather_launch(mode, target, nb, S.d_words, S.d_out, false);
    if (rc) return rc;
    CC_CK(cudaMemcpyAsync(S.h_out, S.d_out, (size_t)nb * 4,
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaStreamSynchronize(g_stream));
    memcpy(out + off, S.h_out, (size_t)nb * 4);
  }
  return 0;
}

// cnt += delta over the balls of `words`; trans: running transition counter
int update_impl(const long long *words, int nwords, int delta,
                unsigned long long *trans) {
  const WalkArgs w = walk_args();
  S.cnt_ver++;
  for (long long off = 0; off < nwords; off += kStageCap) {
    const int nb = (int)std::min<long long>(kStageCap, nwords - off);
    int rc;
    if (nb <= kParamWords) {
      WordsParam p;
      memcpy(p.w, words + off, (size_t)nb * 8);
      rc = launch_update(w, nullptr, &p, nb, delta, trans, g_stream);
      if (rc) return rc;
    } else {
      rc = stage_words(words + off, nb);
      if (rc) return rc;
      rc = launch_update(w, S.d_words, nullptr, nb, delta, trans, g_stream);
      if (rc) return rc;
      CC_CK(cudaStreamSynchronize(g_stream));   // staging buffer reused
    }
  }
  return 0;
}

int mode_role(int role, int *mode, int *target) {
  if (role == 0) { *mode = g_mu == 1 ? kPredEq : kPredDef; *target = 0; }
  else { *mode = g_mu == 1 ? kPredEq : kPredCrit; *target = 1; }
  return 0;
}

}  // namespace

extern "C" {

long long dct_host_bytes(void) { return S.bytes_host; }

int dct_set_mu(int mu) {
  if (mu < 1 || mu > 65535) return -1;
  g_mu = mu;
  S.g.mu = mu;
  return 0;
}

int dct_get_mu(void) { return g_mu; }

int dct_init3(int problem, int n, const int *ax, int R,
              const uint64_t *ballpat, long long balllen, int extract_cap,
              long long *bytes, int layers_mode, int cnt_mode,
              int use_owner) {
  // the v1 table packs position and delta in one nibble each: n <= 16,
  // axes <= 16 (wider cells use dct_init3w)
  if (!ballpat || !ax || n < 1 || n > 16) return -1;
  for (int i = 0; i < n; i++)
    if (ax[i] < 2 || ax[i] > 16) return -1;
  if (layers_mode < 0 || layers_mode > 2 || cnt_mode < 0 || cnt_mode > 2)
    return -1;
  int rc = init_common(problem, n, ax, R, balllen, extract_cap, layers_mode,
                       cnt_mode, use_owner);
  if (rc) return rc;
  std::vector<int32_t> soa;
  int slots = 0;
  if (unpack_v1(ballpat, balllen, soa, &slots)) { free_all(); return -1; }
  rc = upload_table(soa, slots, &S.tbl, &S.slots, &S.pk);
  if (rc) return rc;
  set_side_init(soa, slots);
  return finish_init(bytes);
}

int dct_init3w(int problem, int n, const int *ax, int R, const int32_t *tbl,
               int slots, long long len, int extract_cap, long long *bytes) {
  return dct_b200_init3wm(problem, n, ax, R, tbl, slots, len, extract_cap,
                          bytes, 0, 0);
}

int dct_b200_init3wm(int problem, int n, const int *ax, int R,
                     const int32_t *tbl, int slots, long long len,
                     int extract_cap, long long *bytes, int layers_mode,
                     int cnt_mode) {
  if (!tbl || slots < 1 || slots > kMaxSlots) return -1;
  if (layers_mode < 0 || layers_mode > 2 || cnt_mode < 0 || cnt_mode > 2)
    return -1;
  int rc = init_common(problem, n, ax, R, len, extract_cap, layers_mode,
                       cnt_mode, 0);
  if (rc) return rc;
  std::vector<int32_t> soa((size_t)slots * len, 0);
  for (long long t = 0; t < len; t++)
    for (int k = 0; k < slots; k++) {
      const int32_t c = tbl[t * slots + k];
      if (!c) continue;
      const int pos = c >> 24, dl = c & 0xFFFFFF;
      if (pos < 0 || pos >= n || dl < 1 || dl >= ax[pos]) {
        free_all();
        return -1;
      }
      soa[(size_t)k * len + t] = c;
    }
  rc = upload_table(soa, slots, &S.tbl, &S.slots, &S.pk);
  if (rc) return rc;
  set_side_init(soa, slots);
  return finish_init(bytes);
}

int dct_init2(int q, int n, int R, const uint64_t *ballpat, long long balllen,
              int extract_cap, long long *bytes, int layers_mode,
              int cnt_mode, int use_owner) {
  int ax[kMaxAxes];
  if (n < 1 || n > kMaxAxes) return -1;
  for (int i = 0; i < n; i++) ax[i] = q;
  return dct_init3(kHamming, n, ax, R, ballpat, balllen, extract_cap, bytes,
                   layers_mode, cnt_mode, use_owner);
}

int dct_init(int q, int n, int R, const uint64_t *ballpat, long long balllen,
             int extract_cap, long long *bytes) {
  return dct_init2(q, n, R, ballpat, balllen, extract_cap, bytes, 0, 0, 0);
}

int dct_free(void) {
  free_all();
  g_mu = 1;                       // singleton: mu never leaks into a new cell
  return 0;
}

int dct_set_tbl2(const uint16_t *mask, const uint64_t *offs, long long len) {
  if (!S.live || len != S.len || !mask || !offs) return -1;
  int w = 1;
  for (long long t = 0; t < len; t++) w = std::max(w, __builtin_popcount(mask[t]));
  std::vector<int32_t> soa((size_t)w * len, 0);
  for (long long t = 0; t < len; t++) {
    unsigned m = mask[t];
    int k = 0;
    while (m) {
      const int p = __builtin_ctz(m);
      m &= m - 1;
      const int dl = (int)((offs[t] >> (4 * p)) & 15u);
      if (p >= S.g.n || dl < 1 || dl >= S.g.ax[p]) return -1;
      soa[(size_t)k * len + t] = (p << 24) | dl;
      k++;
    }
  }
  if (S.tbl2) { cudaFree(S.tbl2); S.tbl2 = nullptr; }
  if (S.pk2) { cudaFree(S.pk2); S.pk2 = nullptr; }
  S.metric_tbl2 = metric_ball_table(S.g, soa, w, S.len);
  return upload_table(soa, w, &S.tbl2, &S.slots2, &S.pk2);
}

int dct_use_fmt(int fmt) {
  if (fmt < 0 || fmt > 1) return -1;
  if (fmt == 1 && !S.tbl2) return -1;
  if (fmt == 1 && S.g.prob == kGrid) return -1;   // the ox walk is circulant
  S.fmt = fmt;
  return 0;
}

int dct_set_code(const long long *idx, int M) {
  if (!S.live || M < 0 || (M && !idx)) return -1;
  // one pass: in range, ascending, free of repeats
  unsigned outside = 0, down = 0, same = 0;
  const unsigned long long space = (unsigned long long)S.g.space;
  for (int i = 0; i < M; i++) {
    outside |= (unsigned long long)idx[i] >= space;
    if (i) {
      down |= idx[i] < idx[i - 1];
      same |= idx[i] == idx[i - 1];
    }
  }
  if (outside) return -1;
  MultHist hist;
  std::vector<long long> sorted;
  const long long *src = idx;
  if (down || same) {
    sorted.assign(idx, idx + M);
    if (down) std::sort(sorted.begin(), sorted.end());
    for (int i = 0; i < M;) {
      int j = i + 1;
      while (j < M && sorted[j] == sorted[i]) j++;
      ++hist[j - i];
      i = j;
    }
    src = sorted.data();
  } else if (M) {
    hist[1] = M;
  }
  if (!within_counter(M, max_mult(hist))) return -1;
  // all the room first: a call that is refused leaves the staged code, on the
  // device and here, as it was
  long long *room = nullptr;
  const long long cap = std::max<long long>(M, 1024);
  if (M > S.code_cap) CC_CK(cudaMalloc(&room, (size_t)cap * 8));
  // the buffer that does not hold the active multiset; a copy out of it may
  // still be on its way when the last call staged a code that no transform
  // has used since
  const int to = S.act == S.up ? 1 - S.up : S.up;
  WordBuf &b = S.code_buf[to];
  int rc = 0;
  if (S.code_in_flight) {
    const cudaError_t e = cudaStreamSynchronize(g_stream);
    if (e != cudaSuccess) rc = -(100 + (int)e);
  }
  if (!rc) rc = b.reserve(M);
  if (rc) {
    if (room) cudaFree(room);
    return rc;
  }
  S.code_in_flight = false;
  if (room) {
    if (S.d_code) cudaFree(S.d_code);
    S.d_code = room;
    S.code_cap = cap;
  }
  if (M) {
    memcpy(b.p, src, (size_t)M * 8);
    CC_CK(cudaMemcpyAsync(S.d_code, b.p, (size_t)M * 8,
                          cudaMemcpyHostToDevice, g_stream));
    S.code_in_flight = true;
  }
  b.n = M;
  S.up = to;
  S.codeM = M;
  S.up_hist.swap(hist);
  return 0;
}

int dct_transform(int init_mode, int out_mode) {
  if (!S.live) return -1;
  if (init_mode < 0 || init_mode > 2 || out_mode < 1 || out_mode > 3 ||
      (out_mode == 2 && init_mode != 0))
    return -1;
  if (out_mode == 3 && S.R1 == 1) return -1;
  int rc = init_mode ? cnt_ready() : 0;
  if (rc) return rc;
  rc = autotune(init_mode, out_mode);
  if (rc) return rc;
  rc = run_transform(init_mode, out_mode);
  if (rc) return rc;
  CC_CK(cudaStreamSynchronize(g_stream));
  if ((rc = tma_fault_take())) {
    S.torn = S.torn || out_mode == 2;
    return rc;
  }
  S.code_in_flight = false;
  S.layered_out = out_mode == 3;
  if (out_mode == 2) {
    // active = uploaded
    S.act = S.up;
    S.delta.clear();
    S.active_size = S.codeM;
    S.act_hist = S.up_hist;
    S.cnt_ver++;
    S.torn = false;
  }
  return 0;
}

int dct_ball_update(const long long *words, int nwords, int delta) {
  int rc = cnt_ready();
  if (rc) return rc;
  Batch1 batch;
  if (check_update(words, nwords, delta, batch)) return -1;
  if (nwords == 0) return 0;
  rc = update_impl(words, nwords, delta, nullptr);
  if (rc) return rc;
  apply_active(batch, delta, nwords);
  return 0;
}

int dct_ball_update_delta(const long long *words, int nwords, int delta,
                          long long *dd) {
  if (!dd) return -1;
  *dd = 0;
  int rc = cnt_ready();
  if (rc) return rc;
  Batch1 batch;
  if (check_update(words, nwords, delta, batch)) return -1;
  if (nwords == 0) return 0;
  auto *trans = reinterpret_cast<unsigned long long *>(S.d_scalar + 2);
  rc = update_impl(words, nwords, delta, trans);
  if (rc) return rc;
  long long now;
  rc = fetch_scalar(&now, 2);
  if (rc) return rc;
  const long long tr = (long long)((unsigned long long)now - S.dd_last);
  S.dd_last = (unsigned long long)now;
  *dd = delta > 0 ? -tr : tr;
  apply_active(batch, delta, nwords);
  return 0;
}

int dct_ball_gather(const long long *words, int nwords, int target,
                    int32_t *out) {
  if (const int rc = cnt_ready()) return rc;
  return gather_impl(words, nwords, kPredEq, target, out);
}

int dct_ball_gather_mu(const long long *words, int nwords, int role,
                       int32_t *out) {
  if (const int rc = cnt_ready()) return rc;
  if (nwords <= 0) return 0;
  if (role < 0 || role > 1) return -1;
  return gather_impl(words, nwords, role == 0 ? kPredDef : kPredCrit, 0, out);
}

// Read-only swap evaluation with one synchronisation (coldcore
// dct_hc.cu:882-963): loss[i] and the list of drop i's ball words at exactly
// mu come from two walks of its ball; gain[j] is the role-0 gather of cand j
// on the current cnt (set side or walk) plus the listed words of its drop
// within distance R, the words that removing the drop makes deficient.
// Returns 1 when the list overflowed (the caller falls back), else 0 or an
// error code.
int swap_eval_fast(const long long *drops, int k, const long long *cand,
                   const long long *off, int32_t *gain, int32_t *loss) {
  // one staging block of what this call needs, inputs then results:
  // [cand nc x 8][drops k x 8][coff (k + 1) x 4]
  // [gain nc x 4][loss k x 4][nmu k x 4][offs (k + 1) x 4][cursor k x 4]
  const long long nc = off[k];
  const size_t in_drop = (size_t)nc * 8, in_coff = in_drop + (size_t)k * 8;
  const size_t in_bytes = in_coff + (size_t)(k + 1) * 4;
  const size_t r0 = (in_bytes + 15) / 16 * 16;
  const size_t r_loss = r0 + (size_t)nc * 4, r_nmu = r_loss + (size_t)k * 4;
  const size_t r_offs = r_nmu + (size_t)k * 4;
  const size_t r_cur = r_offs + (size_t)(k + 1) * 4;
  if (!S.d_swap) {
    constexpr size_t kMaxN = 65536;
    const size_t total_bytes = kMaxN * 40 + 256;
    CC_CK(cudaMalloc(&S.d_swap, total_bytes));
    CC_CK(cudaHostAlloc((void **)&S.h_swap, total_bytes,
                        cudaHostAllocDefault));
    S.lcap = std::min<long long>(std::max<long long>(4 * S.len, 1 << 16),
                                 1LL << 22);
    CC_CK(cudaMalloc(&S.d_list, (size_t)S.lcap * 8));
  }
  char *h = S.h_swap, *d = S.d_swap;
  if (nc) memcpy(h, cand, (size_t)nc * 8);
  memcpy(h + in_drop, drops, (size_t)k * 8);
  int32_t *hc = reinterpret_cast<int32_t *>(h + in_coff);
  for (int i = 0; i <= k; i++) hc[i] = (int32_t)off[i];
  const long long *d_cand = reinterpret_cast<const long long *>(d);
  const long long *d_drop = reinterpret_cast<const long long *>(d + in_drop);
  const int32_t *d_coff = reinterpret_cast<const int32_t *>(d + in_coff);
  int32_t *d_gain = reinterpret_cast<int32_t *>(d + r0);
  int32_t *d_loss = reinterpret_cast<int32_t *>(d + r_loss);
  int32_t *d_nmu = reinterpret_cast<int32_t *>(d + r_nmu);
  int32_t *d_offs = reinterpret_cast<int32_t *>(d + r_offs);
  int32_t *d_cur = reinterpret_cast<int32_t *>(d + r_cur);
  CC_CK(cudaMemcpyAsync(d, h, in_bytes, cudaMemcpyHostToDevice, g_stream));
  CC_CK(cudaMemsetAsync(d + r0, 0, r_offs - r0, g_stream));
  WalkArgs w = walk_args();
  int rc = launch_drop_walks(w, d_drop, k, d_loss, d_nmu, d_offs, d_cur,
                             S.lcap, S.d_list, g_stream);
  if (rc) return rc;
  if (nc) {
    int gm, gt;
    mode_role(0, &gm, &gt);
    rc = gather_launch(gm, gt, (int)nc, d_cand, d_gain, true);
    if (rc) return rc;
    Geometry g = S.g;
    g.mu = g_mu;
    rc = launch_swap_corr(g, k, d_cand, d_coff, d_offs, S.d_list, S.lcap,
                          d_gain, g_stream);
    if (rc) return rc;
  }
  // gain, loss and the list total (offs[k]) in one copy
  CC_CK(cudaMemcpyAsync(h + r0, d + r0, r_offs - r0 + (size_t)(k + 1) * 4,
                        cudaMemcpyDeviceToHost, g_stream));
  CC_CK(cudaStreamSynchronize(g_stream));
  const int32_t listed = reinterpret_cast<int32_t *>(h + r_offs)[k];
  if (listed > S.lcap) return 1;
  memcpy(loss, h + r_loss, (size_t)k * 4);
  if (nc) memcpy(gain, h + r0, (size_t)nc * 4);
  S.stats[4]++;
  return 0;
}

// Exact greedy repair on the device (no counterpart in the reference; its
// greedy_fill is the Python lazy greedy of search.py:260-360).  From the
// gain map of the current cnt, with the active words excluded, each
// step places the word of largest exact gain (ties: smallest index),
// updates cnt over its ball and lowers the gain of every candidate whose
// ball holds a word the placement satisfied, all without leaving the GPU;
// it stops at zero deficit, at no positive gain, or after max_add words.
// The placed words are added to the active multiset.  placed (capacity
// max_add) receives them in placement order; *deficit the deficit left.
// Returns the number placed, or a negative error.  The map is clobbered.
int greedy_fill_impl(int max_add, long long *placed, long long *deficit) {
  if (!S.live || max_add < 0 || (max_add && !placed) || !deficit) return -1;
  if (const int rc = cnt_ready()) return rc;
  if (S.g.space >= (1LL << 32)) return -1;    // 32-bit index in the key
  // placed words are new (multiplicity 1): the counters stay within uint16
  if (!within_counter(S.active_size + max_add, std::max(max_mult(S.act_hist), 1)))
    return -1;
  const int mu = g_mu;
  const long long nch = greedy_chunks(S.g.space);
  const size_t o_st = (sizeof(BatchGreedyCell) + 63) / 64 * 64;
  const size_t o_run = o_st + 64;
  const size_t o_key = o_run + kGreedyRunBytes;
  static_assert(kGreedyStateBytes <= 64, "greedy state");
  const size_t o_fresh = o_key + (size_t)nch * 8;
  if (!S.d_greedy) {
    CC_CK(cudaMalloc(&S.d_greedy, o_fresh + (size_t)S.len * 8));
    CC_CK(cudaHostAlloc((void **)&S.h_greedy, kGreedyRing * sizeof(GreedySlot),
                        cudaHostAllocDefault));
    for (auto &ev : S.ev_greedy)
      CC_CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  }
  if (max_add > S.placed_cap) {
    if (S.d_placed) CC_CK(cudaFree(S.d_placed));
    if (S.h_placed) CC_CK(cudaFreeHost(S.h_placed));
    S.d_placed = S.h_placed = nullptr;
    S.placed_cap = 0;
    const long long cap = std::max<long long>(max_add, 1024);
    CC_CK(cudaMalloc(&S.d_placed, (size_t)cap * 8));
    CC_CK(cudaHostAlloc((void **)&S.h_placed, (size_t)cap * 8,
                        cudaHostAllocDefault));
    S.placed_cap = cap;
  }
  // the deficit to start from, and the gain map of the current cnt
  int rc = launch_cnt_reduce(S.cnt, S.g.space, kPredDef, 0, mu,
                             S.d_scalar + kQuerySlot, g_stream, red_out());
  if (rc) return rc;
  long long d0;
  rc = query_result(&d0);
  if (rc) return rc;
  *deficit = d0;
  if (max_add == 0 || d0 == 0) return 0;
  rc = autotune(1, 1);
  if (rc) return rc;
  constexpr int32_t kExcluded = INT_MIN / 2;
  // At mu = 1, with a table that is the metric ball, an active word's whole
  // ball is covered: its gain is 0 and it is never placed.  Otherwise the
  // active words are taken out of the map, after every transform of it.  (A
  // second table that is not the ball may have placed some of them.)
  const bool exclude = mu > 1 || !S.set_ok || S.fmt != 0 ||
                       (S.tbl2 && !S.metric_tbl2);
  std::vector<long long> code;
  if (exclude) {
    each_active([&](long long w, int) { code.push_back(w); });
    if ((long long)code.size() > S.active_cap) {
      if (S.d_active) CC_CK(cudaFree(S.d_active));
      S.d_active = nullptr;
      S.active_cap = 0;
      const long long cap = std::max<long long>(2 * code.size(), 1024);
      CC_CK(cudaMalloc(&S.d_active, (size_t)cap * 8));
      S.active_cap = cap;
    }
    if (!code.empty())
      CC_CK(cudaMemcpyAsync(S.d_active, code.data(), code.size() * 8,
                            cudaMemcpyHostToDevice, g_stream));
  }
  BatchGreedyCell gc{};
  gc.w = walk_args();
  gc.map = S.layers;
  gc.st = S.d_greedy + o_st;
  gc.placed = S.d_placed;
  gc.fresh = reinterpret_cast<long long *>(S.d_greedy + o_fresh);
  gc.ckey = reinterpret_cast<unsigned long long *>(S.d_greedy + o_key);
  gc.code = S.d_active;
  gc.ncode = (long long)code.size();
  gc.max_add = max_add;
  gc.pats = greedy_pats(S.len, sm_count() * 4);
  GreedyHost st{};
  st.deficit = d0;
  BatchGreedyCell *dcell = reinterpret_cast<BatchGreedyCell *>(S.d_greedy);
  CC_CK(cudaMemcpyAsync(dcell, &gc, sizeof(gc), cudaMemcpyHostToDevice,
                        g_stream));
  CC_CK(cudaMemcpyAsync(gc.st, &st, sizeof(st), cudaMemcpyHostToDevice,
                        g_stream));
  GreedyRun *run = reinterpret_cast<GreedyRun *>(S.d_greedy + o_run);
  CC_CK(cudaMemsetAsync(run, 0, kGreedyRunBytes, g_stream));
  auto build_map = [&]() -> int {
    const int r = run_transform(1, 1);
    if (r || !exclude) return r;
    return launch_greedy_exclude(dcell, 1, nullptr, kExcluded, g_stream);
  };
  if ((rc = build_map())) return rc;
  S.layered_out = false;
  const int nam = greedy_argmax_blocks(S.g.space);
  const int npl = (int)((S.len + gc.pats - 1) / gc.pats);
  const int nrf = sm_count() * 4;
  // the time of a gain transform: measured by the autotuner, else launches
  // and bytes at a small cell's rate; a streamed cell is never rebuilt, nor
  // one whose table is not the ball that the transform sums over
  double rebuild_us = S.tune_ms[1][1] * 1e3;
  if (rebuild_us <= 0) {
    const Plan &P = plan_for(1, 1);
    rebuild_us = 4.0 * (P.groups.size() + P.passes.size());
    for (const auto &gp : P.groups) rebuild_us += group_bytes(gp.a) / 2.0e6;
    for (size_t i = 0; i < P.passes.size(); i++)
      rebuild_us += 6.0 * S.g.space / 1.0e6;
  }
  if (S.streamed || !S.metric_table || S.fmt != 0) rebuild_us = 1e30;
  auto read_state = [&](int slot) -> int {
    CC_CK(cudaMemcpyAsync(S.h_greedy + slot, gc.st, sizeof(GreedySlot),
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaEventRecord(S.ev_greedy[slot], g_stream));
    return 0;
  };
  // Every placement serves at least one deficient word: at most d0 steps;
  // those after the stop return at once.  While a placement may still be
  // worth a rebuild the host follows the gains one step behind (the first
  // step waits for its own), and the device stays busy; after that steps go
  // out in chunks with one look at the state between them.
  const long long steps = std::min<long long>(max_add, d0);
  long long issued = 0, chunk = 32;
  bool follow = true;
  S.cnt_ver++;
  S.torn = true;                   // until every step has been accounted for
  while (issued < steps) {
    if (follow) {
      const int par = (int)(issued & 1);
      rc = launch_greedy_argmax(dcell, nullptr, nam, par, issued == 0,
                                g_stream);
      if (rc || (rc = read_state(par))) return rc;
      const int look = issued ? par ^ 1 : par;
      CC_CK(cudaEventSynchronize(S.ev_greedy[look]));
      const GreedyHost &h = S.h_greedy[look].st;
      if (h.done) break;
      const bool rebuild = greedy_rebuild_pays(h.gain(look), S.len,
                                               rebuild_us);
      rc = launch_greedy_place(dcell, nullptr, npl, par, kExcluded, g_stream);
      if (rc) return rc;
      rc = rebuild ? build_map()
                   : launch_greedy_refresh(dcell, 1, nrf, nullptr, g_stream);
      if (rc) return rc;
      follow = rebuild;
      issued++;
      continue;
    }
    const long long n = std::min(chunk, steps - issued);
    rc = launch_greedy_run(gc, (int)(issued & 1), (int)n, kExcluded, run,
                           g_stream);
    if (rc) return rc;
    issued += n;
    if (fault_due(kFaultBarrier))
      CC_CK(cudaMemsetAsync(reinterpret_cast<int *>(run) + 1, 1, 1, g_stream));
    if ((rc = read_state(0))) return rc;
    CC_CK(cudaEventSynchronize(S.ev_greedy[0]));
    if (S.h_greedy[0].run[1]) {    // no further launch on a half-done step
      fprintf(stderr, "coldcore_b200: a greedy launch timed out at its grid "
              "barrier\n");
      return -8;
    }
    if (S.h_greedy[0].st.done) break;
    chunk = std::min<long long>(chunk * 2, 512);
  }
  if ((rc = read_state(0))) return rc;
  CC_CK(cudaStreamSynchronize(g_stream));
  if ((rc = tma_fault_take())) return rc;      // a rebuild's streamed launch
  st = S.h_greedy[0].st;
  const int n = st.placed_now();
  if (n) {
    CC_CK(cudaMemcpyAsync(S.h_placed, S.d_placed, (size_t)n * 8,
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaStreamSynchronize(g_stream));
    memcpy(placed, S.h_placed, (size_t)n * 8);
    Batch1 batch;
    count_words(placed, n, batch);
    apply_active(batch, +1, n);
  }
  S.torn = false;
  *deficit = st.deficit_now();
  return n;
}

int dct_b200_greedy_fill(int max_add, long long *placed, long long *deficit) {
  return greedy_fill_impl(max_add, placed, deficit);
}

int dct_swap_eval(const long long *drops, int k, const long long *cand,
                  const long long *off, int32_t *gain, int32_t *loss) {
  if (const int rc = cnt_ready()) return rc;
  if (k <= 0) return 0;
  if (k > 65535 || !off || off[0] != 0 || !drops || !loss) return -1;
  for (int i = 0; i < k; i++)
    if (off[i + 1] < off[i]) return -1;
  const long long nc = off[k];
  if (nc > 65535 || (nc && (!cand || !gain))) return -1;
  if (!valid_words(drops, k) || !valid_words(cand, nc)) return -1;
  for (int i = 0; i < k; i++)
    if (active_count(drops[i]) <= 0) return -1;
  if (S.set_ok) {
    const int rc = swap_eval_fast(drops, k, cand, off, gain, loss);
    if (rc <= 0) return rc;                  // done (0) or an error
  }
  // drop / gather / undo per drop word; cnt ends where it started
  S.stats[5]++;
  int lm, lt, gm, gt;
  mode_role(1, &lm, &lt);
  mode_role(0, &gm, &gt);
  for (int i = 0; i < k; i++) {
    int rc = gather_impl(drops + i, 1, lm, lt, loss + i);
    if (rc) return rc;
    const long long ni = off[i + 1] - off[i];
    if (!ni) continue;
    rc = update_impl(drops + i, 1, -1, nullptr);
    if (rc) return rc;
    rc = gather_impl(cand + off[i], (int)ni, gm, gt, gain + off[i]);
    const int rc2 = update_impl(drops + i, 1, +1, nullptr);
    if (rc) return rc;
    if (rc2) return rc2;
  }
  return 0;
}

int dct_loss_owner(const long long *words, int M, int32_t *out) {
  if (!S.live || !S.owner) return -1;
  if (!valid_words(words, M) || (M && !out)) return -2;
  Batch1 batch;
  count_words(words, M, batch);
  MultHist hist;
  for (const auto &e : batch) ++hist[e.second];
  if (!within_counter(M, max_mult(hist))) return -2;
  // the words become the active multiset: into the buffer that does not
  // hold the staged code
  const int to = S.act == S.up ? 1 - S.up : S.act;
  if (S.code_buf[to].reserve(M)) return -2;
  S.torn = true;
  CC_CK(cudaMemsetAsync(S.cnt, 0, (size_t)S.cnt_len * 2, g_stream));
  int rc = update_impl(words, M, +1, nullptr);
  if (rc) return rc;
  long long *p = S.code_buf[to].p;
  for (const auto &e : batch)
    for (int i = 0; i < e.second; i++) *p++ = e.first;
  S.code_buf[to].n = M;
  S.act = to;
  S.delta.clear();
  S.active_size = M;
  S.act_hist.swap(hist);
  S.torn = false;
  if (M == 0) return 0;
  int lm, lt;
  mode_role(1, &lm, &lt);
  return gather_impl(words, M, lm, lt, out);
}

int dct_stats(long long *out, int n) {
  if (n > 9) n = 9;
  for (int i = 0; i < n; i++) out[i] = S.stats[i];
  return n < 0 ? 0 : n;
}

long long dct_count_eq(int target) {
  if (const int rc = cnt_ready()) return rc;
  // the zero-word list of a set-side gather already counted them
  if (target == 0 && S.z_valid && S.z_ver == S.cnt_ver &&
      (S.z_mode == kPredEq ? S.z_target == 0
                           : (S.z_mode == kPredDef && S.z_mu == 1))) {
    S.stats[6]++;
    return S.z_n;
  }
  int rc = launch_cnt_reduce(S.cnt, S.g.space, kPredEq, target, g_mu,
                             S.d_scalar + kQuerySlot, g_stream, red_out());
  if (rc) return rc;
  long long r;
  rc = query_result(&r);
  return rc ? rc : r;
}

long long dct_count_deficit(void) {
  int rc = cnt_ready();
  if (rc) return rc;
  rc = launch_cnt_reduce(S.cnt, S.g.space, kPredDef, 0, g_mu,
                             S.d_scalar + kQuerySlot, g_stream, red_out());
  if (rc) return rc;
  long long r;
  rc = query_result(&r);
  return rc ? rc : r;
}

int dct_map_max(int32_t *out) {
  if (!S.live || !out) return -1;
  int rc = launch_max(S.layers, S.g.space, S.d_scalar + kQuerySlot, g_stream,
                      red_out());
  if (rc) return rc;
  long long r;
  rc = query_result(&r);
  if (rc) return rc;
  *out = (int32_t)r;
  return 0;
}

int dct_map_hist(int nbins, int32_t vmax, int32_t *out) {
  if (!S.live || nbins < 1 || nbins > 4096 || vmax < 1 || !out) return -1;
  const int rc = launch_hist(S.layers, S.g.space, nbins, vmax, S.d_hist,
                             g_stream, red_out(S.h_out));
  if (rc) return rc;
  CC_CK(cudaStreamSynchronize(g_stream));
  memcpy(out, S.h_out, (size_t)nbins * 4);
  return 0;
}

static long long extract_impl(int32_t thr, void *out_idx, bool wide,
                              int32_t *out_val, int cap) {
  if (!S.live) return -1;
  if (cap > S.extract_cap) cap = (int)S.extract_cap;
  if (cap < 0) cap = 0;
  void *didx = wide ? (void *)S.d_ext64 : (void *)S.d_ext32;
  int rc = launch_extract(S.layers, S.g.space, thr, didx, wide, S.d_extv, cap,
                          S.d_scalar + kQuerySlot, g_stream, red_out());
  if (rc) return rc;
  // the first entries come back with the count, through pinned memory; a
  // larger answer's rest is copied once the count is known
  const size_t isz = wide ? 8 : 4;
  const long long first = std::min<long long>(cap, kExtFirst);
  if (first && !S.h_ext)
    CC_CK(cudaHostAlloc((void **)&S.h_ext, (size_t)kExtFirst * 12,
                        cudaHostAllocDefault));
  char *hv = S.h_ext + (size_t)kExtFirst * 8;
  if (first) {
    CC_CK(cudaMemcpyAsync(S.h_ext, didx, (size_t)first * isz,
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaMemcpyAsync(hv, S.d_extv, (size_t)first * 4,
                          cudaMemcpyDeviceToHost, g_stream));
  }
  long long found;
  rc = query_result(&found);
  if (rc) return rc;
  const long long m = found < cap ? found : cap;
  const long long m0 = std::min(m, first);
  if (m0 > 0) {
    memcpy(out_idx, S.h_ext, (size_t)m0 * isz);
    memcpy(out_val, hv, (size_t)m0 * 4);
  }
  if (m > m0) {
    CC_CK(cudaMemcpyAsync(static_cast<char *>(out_idx) + m0 * isz,
                          static_cast<char *>(didx) + m0 * isz,
                          (size_t)(m - m0) * isz, cudaMemcpyDeviceToHost,
                          g_stream));
    CC_CK(cudaMemcpyAsync(out_val + m0, S.d_extv + m0, (size_t)(m - m0) * 4,
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaStreamSynchronize(g_stream));
  }
  return found;
}

long long dct_map_extract(int32_t thr, uint32_t *idx, int32_t *val, int cap) {
  return extract_impl(thr, idx, false, val, cap);
}

long long dct_map_extract64(int32_t thr, int64_t *idx, int32_t *val,
                            int cap) {
  return extract_impl(thr, idx, true, val, cap);
}

int dct_map_read_at(const long long *idx, int k, int32_t *out) {
  if (!S.live) return -1;
  if (k <= 0) return 0;
  if (!out || !valid_words(idx, k)) return -1;
  return staged_words(idx, k, out,
                      [](const long long *w, int nb, int32_t *o) {
                        return launch_read_at(S.layers, w, nb, o, g_stream);
                      });
}

int dct_read_cnt(long long off, long long len, uint16_t *out) {
  if (!S.live || off < 0 || len < 0 || off + len > S.g.space ||
      (len && !out))
    return -1;
  if (const int rc = cnt_ready()) return rc;
  if (len)
    CC_CK(cudaMemcpyAsync(out, S.cnt + off, (size_t)len * 2,
                          cudaMemcpyDefault, g_stream));
  CC_CK(cudaStreamSynchronize(g_stream));   // async updates were in flight
  return 0;
}

long long dct_b200_stream(void) {
  if (ensure_stream()) return 0;
  return (long long)(uintptr_t)g_stream;
}

int dct_b200_plan(int init_mode, int out_mode, long long *info, int cap) {
  // a streamed cell runs the out-of-core schedule (dct_b200_ooc_plan)
  if (!S.live || S.streamed || init_mode < 0 || init_mode > 2 ||
      out_mode < 1 || out_mode > 3)
    return -1;
  Plan &P = plan_for(init_mode, out_mode);
  const long long X = S.g.space;
  int n = 0;
  if (P.window) {
    int axis = 0;
    for (size_t i = 0; i < P.passes.size(); i++, n++) {
      const WindowArgs &w = P.passes[i];
      const long long by = X * ((w.src16 ? 2 : 4) + (w.dst16 ? 2 : 4));
      const int first = axis, many = w.q2 ? 2 : 1;
      axis += many;
      if (info && 4 * n + 3 < cap) {
        info[4 * n] = first; info[4 * n + 1] = many;
        info[4 * n + 2] = by; info[4 * n + 3] = -2;
      }
    }
    return n;
  }
  int j = 0;
  for (const auto &p : P.groups) {
    long long rd = 0, wr = 0;
    if (p.a.src == kSrcCnt) rd = 2;
    else if (p.a.src == kSrcLayers)
      rd = (p.a.in8 ? 1LL : p.a.in16 ? 2LL : 4LL) * p.a.lin;
    if (p.a.dst == kDstLayers)
      wr = (p.a.out8 ? 1LL : p.a.out16 ? 2LL : 4LL) * p.a.lout;
    else if (p.a.dst == kDstMap) wr = 4;
    else wr = 2;
    long long by = X * (rd + wr);
    if (p.a.src == kSrcCode) by += 8 * S.codeM;
    if (info && 4 * n + 3 < cap) {
      info[4 * n] = j; info[4 * n + 1] = p.a.k + p.a.pair_axis;
      info[4 * n + 2] = by; info[4 * n + 3] = p.kernel;
    }
    j += p.a.k + p.a.pair_axis;
    n++;
  }
  return n;
}

int dct_b200_plan_probe(int problem, int n, const int *ax, int R,
                        int init_mode, int out_mode, int budget_kb, int pipe,
                        int half, long long *rows, int cap) {
  if (n < 1 || n > kMaxAxes || R < 1 || !ax || problem < 0 || problem > 3 ||
      init_mode < 0 || init_mode > 2 || out_mode < 1 || out_mode > 3 ||
      (out_mode == 2 && init_mode != 0) || budget_kb < 16 ||
      budget_kb > 220 || pipe < 0 || pipe > 3 || cap < 0)
    return -1;
  const bool layered = problem == kHamming || problem == kLee;
  if (layered && R + 1 > kMaxLayers) return -1;
  if (!layered && out_mode == 3) return -1;
  Geometry g{};
  g.prob = problem; g.n = n; g.R = R; g.mu = 1;
  g.pw[0] = 1;
  for (int i = 0; i < n; i++) {
    if (ax[i] < 2 || ax[i] >= (1 << 24)) return -1;
    if (layered && ax[i] > 16) return -1;
    if (problem == kTorus && (ax[i] < 3 || 2 * R + 1 > ax[i])) return -1;
    if (g.pw[i] > (1LL << 40) / ax[i]) return -2;
    g.ax[i] = ax[i];
    g.pw[i + 1] = g.pw[i] * ax[i];
  }
  g.space = g.pw[n];
  g = transform_geometry(g);                  // as a cell would plan it
  bool wide = false;
  for (int i = 0; i < n; i++) wide = wide || ax[i] > 16;
  if (!layered && wide) return 0;             // window passes, not groups
  const int R1 = layered ? R + 1 : 1;
  const int src = init_mode == 0 ? kSrcCode : kSrcCnt;
  const int dst = out_mode == 1 ? kDstMap
                  : out_mode == 2 ? kDstCnt : kDstLayers;
  // never dereferenced: aligned stand-ins for the planes
  int32_t *const fake = reinterpret_cast<int32_t *>(uintptr_t(1) << 12);
  const long long plane = round_up(g.space, kPlaneAlign);
  PlanPtrs ptr{fake, plane, reinterpret_cast<uint16_t *>(fake),
               reinterpret_cast<long long *>(fake), 0, nullptr};
  ptr.layers16 = reinterpret_cast<uint16_t *>(fake + plane);
  Knobs kn{(size_t)budget_kb << 10, pipe};
  kn.half = half && R1 >= 2 && dst != kDstLayers;
  const std::vector<GroupPlan> P = plan_groups(g, R1, ptr, src, dst, kn);
  int m = 0, j = 0;
  for (const auto &p : P) {
    const GroupArgs &a = p.a;
    int rbsum = 0;
    for (int r = 0; r < a.nrounds; r++) rbsum += a.rb[r];
    const long long row[24] = {
        j, a.k + a.pair_axis, a.pair_axis, a.W, a.mid, a.Bo, a.inner,
        a.outer, a.ntiles, p.kernel, a.pipe, a.pack, a.in16, a.out16,
        (long long)p.smem, p.threads, a.lin, a.lout, a.skew, p.grid, a.src,
        a.dst, a.nrounds, rbsum};
    if (rows && 24 * (m + 1) <= cap)
      for (int t = 0; t < 24; t++) rows[24 * m + t] = row[t];
    j += a.k + a.pair_axis;
    m++;
  }
  return m;
}

int dct_b200_plan_forms(int init_mode, int out_mode, int *forms, int cap) {
  if (!S.live || S.streamed || init_mode < 0 || init_mode > 2 || out_mode < 1 ||
      out_mode > 3 || cap < 0)
    return -1;
  Plan &P = plan_for(init_mode, out_mode);
  if (P.window) return 0;
  int n = 0;
  for (const auto &p : P.groups) {
    if (forms && n < cap)
      forms[n] = (p.a.pipe ? 1 : 0) | (p.a.pack ? 2 : 0) |
                 (p.a.in16 ? 4 : 0) | (p.a.out16 ? 8 : 0) |
                 (p.a.pair_axis ? 16 : 0) | (p.a.tma ? 32 : 0) |
                 (p.a.in8 || p.a.out8 ? 64 : 0);
    n++;
  }
  return n;
}

int dct_b200_ball_hist(const long long *words, int nw, int src, int nbins,
                       int32_t *out) {
  if (!S.live || nbins < 1 || nbins > 32 || !out || (src != 0 && src != 1))
    return -1;
  if (nw <= 0) return 0;
  if (!valid_words(words, nw)) return -1;
  if (const int rc = src == 1 ? cnt_ready() : 0) return rc;
  const WalkArgs w = walk_args();
  const long long cap = kStageCap / nbins;   // nb * nbins fits d_out
  for (long long off = 0; off < nw; off += cap) {
    const int nb = (int)std::min<long long>(cap, nw - off);
    int rc = stage_words(words + off, nb);
    if (rc) return rc;
    rc = launch_ball_hist(w, S.d_words, nb, S.layers, src, nbins, S.d_out,
                          g_stream);
    if (rc) return rc;
    CC_CK(cudaMemcpyAsync(S.h_out, S.d_out, (size_t)nb * nbins * 4,
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaStreamSynchronize(g_stream));
    memcpy(out + off * nbins, S.h_out, (size_t)nb * nbins * 4);
  }
  return 0;
}

int dct_b200_layers_at(const long long *idx, int k, int32_t *out) {
  if (!S.live || !S.layered_out || (k && !out)) return -1;
  if (k <= 0) return 0;
  if (!valid_words(idx, k)) return -1;
  if (S.streamed) {
    const long long X = S.g.space;
    for (int i = 0; i < k; i++)
      for (int d = 0; d < S.R1; d++)
        out[(long long)i * S.R1 + d] = S.h_layers[d * X + idx[i]];
    return 0;
  }
  const long long cap = kStageCap / S.R1;
  for (long long off = 0; off < k; off += cap) {
    const int nb = (int)std::min<long long>(cap, k - off);
    int rc = stage_words(idx + off, nb);
    if (rc) return rc;
    rc = launch_layers_at(S.layers, S.plane, S.R1, S.d_words, nb, S.d_out,
                          g_stream);
    if (rc) return rc;
    CC_CK(cudaMemcpyAsync(S.h_out, S.d_out, (size_t)nb * S.R1 * 4,
                          cudaMemcpyDeviceToHost, g_stream));
    CC_CK(cudaStreamSynchronize(g_stream));
    memcpy(out + off * S.R1, S.h_out, (size_t)nb * S.R1 * 4);
  }
  return 0;
}

int dct_b200_set_timing(int on) {
  g_timing = on ? 1 : 0;
  return 0;
}

int dct_b200_last_timings(float *ms, int cap) {
  const int n = g_last_n < cap ? g_last_n : cap;
  for (int i = 0; i < n && ms; i++) ms[i] = g_last_ms[i];
  return g_last_n;
}

int dct_b200_read_map(long long off, long long len, int32_t *out) {
  if (!S.live || off < 0 || len < 0 || off + len > S.g.space ||
      (len && !out))
    return -1;
  if (len)
    CC_CK(cudaMemcpyAsync(out, S.layers + off, (size_t)len * 4,
                          cudaMemcpyDeviceToHost, g_stream));
  CC_CK(cudaStreamSynchronize(g_stream));
  return 0;
}

int dct_b200_read_layer(int d, long long off, long long len, int32_t *out) {
  if (!S.live || !S.layered_out || d < 0 || d >= S.R1 || off < 0 ||
      len < 0 || off + len > S.g.space || (len && !out))
    return -1;
  if (len && S.streamed) {
    memcpy(out, S.h_layers + d * S.g.space + off, (size_t)len * 4);
    return 0;
  }
  if (len)
    CC_CK(cudaMemcpyAsync(out, S.layers + d * S.plane + off,
                          (size_t)len * 4, cudaMemcpyDeviceToHost, g_stream));
  CC_CK(cudaStreamSynchronize(g_stream));
  return 0;
}

}  // extern "C"
