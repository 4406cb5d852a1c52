// engine.h — internal state and launch interfaces of the B200 covering engine.
//
// One process-wide cell (the plugin ABI v1 singleton model, coldcore
// src/include/coldcore/plugin.h:8-10).  Every kernel takes its geometry by
// value (no __constant__ state shared between translation units), and every
// launch goes to the engine's own stream, so device work runs in call order.
#pragma once
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>
#include <vector>

#include "query_out.h"

namespace cc {

constexpr int kMaxAxes = 40;      // |X| <= 2^40 with every axis >= 2
constexpr int kMaxLayers = 8;     // R + 1 distance layers (R <= 7)
constexpr int kMaxSlots = 8;      // changed positions per support pattern
constexpr int kPlaneAlign = 64;   // plane stride rounded to 64 elements

// problem ids: coldcore src/include/coldcore/plugin.h:45-53
enum Problem { kHamming = 0, kTorus = 1, kLee = 2, kGrid = 3 };

// cnt predicates (coldcore src/plugins/covering/dctcore_mu.cuh:28-40)
enum Pred { kPredEq = 0, kPredDef = 1, kPredCrit = 2, kPredIdent = 3 };

struct Geometry {
  int prob, n, R, mu;
  long long space;
  int ax[kMaxAxes];
  long long pw[kMaxAxes + 1];
};

__host__ __device__ inline bool cnt_pred(int mode, int c, int target, int mu) {
  if (mode == kPredDef) return c < mu;
  if (mode == kPredCrit) return c >= 1 && c <= mu;
  return c == target;
}

// ------------------------------------------------------------ transform plan
// One kernel launch covers a GROUP of consecutive axes [j0, j0+k).  The
// group's words factor as x = o*(inner*mid) + m*inner + i with
// inner = pw[j0], mid = prod of the group's axes; a tile is W consecutive
// inner positions x mid x Bo consecutive outer slabs, staged in shared
// memory.  Rounds process `rb` axes each in registers (local stride rs in m).
constexpr int kMaxRounds = 24;
constexpr int kGroupThreads = 512;   // CTA size cap: 128 registers per thread

enum Src { kSrcLayers = 0, kSrcCnt = 1, kSrcCode = 2 };
enum Dst { kDstLayers = 0, kDstMap = 1, kDstCnt = 2 };

struct GroupArgs {
  int32_t *layers;        // plane 0 base; plane d at layers + d*plane
  long long plane;        // plane stride (elements)
  uint16_t *cnt;
  const long long *code;  // sorted code (kSrcCode)
  long long ncode;
  const long long *code_bounds;  // per-tile slice of the code (kSrcCode)
  long long inner, outer, ntiles, nchunk;
  int mid, W, Bo, k;
  int nrounds;
  int rb[kMaxRounds];     // axes per round
  int rs[kMaxRounds];     // local stride (in m) of the round's first axis
  int rq[kMaxRounds];     // axis size of the round (all axes of a round equal)
  int qax[kMaxRounds];    // per-axis size inside the group (generic kernel)
  int src, dst, lin, lout;
  int pmode, ptarget, mu, R;
  int skew;               // log2 of the shared-memory skew period (0 = none)
  int prob;
  int pipe;               // prefetch the next tile while computing (cp.async)
  int32_t *map;           // kDstMap target (nullptr: plane 0 of layers)
  // 16-bit intermediate planes: plane d at layers16 + d*plane (u16 words),
  // read when in16, written when out16 (values provably <= 65535)
  uint16_t *layers16;
  int in16, out16;
  // 8-bit planes between a streamed binary first group (out8) and the
  // streamed launch after it (in8), where every layer value after the
  // first group's k axes stays below 256: a 0/1 predicate source and
  // C(k, d) <= 255 for every d <= R.  Plane d at byte off8 + d*plane of
  // the 16-bit plane region, past the 16-bit planes that the launch
  // reading them writes (so no tile overwrites bytes another has yet to
  // read).
  int in8, out8;
  long long off8;
  // streamed group: axes per register round (0: RoundAxes, the default)
  int tbm;
  int pack;               // two inner words per 32-bit lane (group_kernel)
  // first group of a binary Hamming cell: axis 0 is the word pair itself
  // (inner = 2), applied once as a swap-add inside each packed lane
  int pair_axis;
  long long *red;         // epilogue reduction target (generic tiles, the
                          // register kernels and the streamed groups)
  int red_mode;           // 0 none, 1 deficit of the cnt written, 2 map max
  // streamed form (transform_tma.cu): tensor loads into `stages` shared
  // memory stages, W = 2 x lanes inner words a tile (tma 1); the first
  // group staged from cnt by bulk copies (tma 2); a ternary first group
  // over row pairs packed in 32-bit lanes (tma 3, Bo = 2)
  int tma;
  int stages;
  // padded layout of the 16-bit planes (ternary cells): every run of t0
  // words (the first group's mid) is stored at a pitch of `pitch` words
  // (a multiple of 64), so rows of the later groups start on 128-byte
  // boundaries.  The first group writes its layers padded; the later
  // groups' `inner` is then the padded one, and the last group's map or
  // cnt goes back to the canonical index.  0 = the canonical layout.
  long long pitch;
  long long t0;
};

// arguments of a streamed group launch (transform_tma.cu)
constexpr int kTmaMaxStages = 4;
struct TmaArgs {
  uint16_t *layers16;
  long long plane;
  int32_t *map;
  uint16_t *cnt;
  long long inner, nchunk, ntiles;
  int lin, lout, stages;
  int *fault;             // mapped host word, set when a wait runs out
  // first group (tma_first): the cnt source and its predicate
  const uint16_t *cnt_in;
  int pmode, ptarget, mu;
  // first group of a recount (code_first): the sorted code, per-tile slices
  const long long *code;
  const long long *code_bounds;
  // padded planes (GroupArgs::pitch): the canonical inner stride, the
  // pitch and the valid words of each padded run
  long long inner_c, pitch, t0;
  // first group over row pairs (rows_first): the rows of the cell
  long long rows;
  // 8-bit layer planes (tma_first OUT 5): their byte offset from layers16
  long long off8;
  // epilogue reduction of a map or cnt written (GroupArgs::red_mode)
  long long *red;
  int red_mode;
};

struct GroupPlan {
  GroupArgs a;
  int kernel;             // index into the launcher table
  int threads;
  size_t smem;
  int grid;
};

// planner.cu: schedule knobs and the group plan of one transform
// pipe: see plan_groups; half: 16-bit planes between the launches
// pair: allow the pair first group (binary Hamming, 16-bit planes)
// pad: the padded 16-bit layout for a ternary cell (streamed later groups)
// u8: 8-bit planes after a streamed binary first group (gain / loss)
struct Knobs { size_t budget; int pipe; int half = 0; int pair = 1;
               int pad = 0; int u8 = 0; };
struct PlanPtrs {
  int32_t *layers; long long plane; uint16_t *cnt;
  const long long *code; long long ncode; int32_t *map;
  uint16_t *layers16 = nullptr;   // u16 plane region (Knobs::half)
};
// An axis range of one transform: the launches cover axes [begin, end) of
// g (end < 0: through the last axis).  reach0 is the distance reach of axes
// applied by an earlier range (so the live layers at axis j are
// min(reach0 + reach of axes [begin, j), R) + 1); `final` is false when
// the range's layers feed a later range, which keeps the last launch's
// plane width (16-bit planes) and writes only its live layers.
struct AxisRange {
  int begin = 0;
  int end = -1;
  long long reach0 = 0;
  bool final = true;
};
std::vector<GroupPlan> plan_groups(const Geometry &g, int R1,
                                   const PlanPtrs &ptr, int src, int dst,
                                   Knobs kn, AxisRange range = AxisRange());
// distance reach of one axis: 1 for Hamming, floor(a/2) for Lee
inline long long axis_reach(int prob, int a) { return prob == kLee ? a / 2 : 1; }
// The transform geometry of a cell: Lee distance on axes of size 2 or 3 is
// the Hamming distance (every nonzero digit difference has weight
// min(d, q - d) = 1), so such a cell plans and runs as Hamming, with the
// Hamming kernels' streamed forms.
inline Geometry transform_geometry(Geometry g) {
  if (g.prob != kLee) return g;
  for (int j = 0; j < g.n; j++)
    if (g.ax[j] > 3) return g;
  g.prob = kHamming;
  return g;
}

// launchers (transform_*.cu)
int launch_group(const GroupPlan &p, cudaStream_t s);
int prepare_group(const GroupPlan &p);
int group_blocks_per_sm(const GroupPlan &p);
size_t group_smem_bytes(const GroupArgs &a, int R1);
// the prefetching kernel has a packed form for 16-bit layer sources
bool pipe_pairs_ok(const GroupArgs &a);
int pick_group_kernel(int prob, int q, int R1, int *bm);
int group_kernel_variants(int prob, int q, int R1, int *kids, int *bms,
                          int cap);
// the same group with every other register-blocked kernel and CTA width
// (rounds, skew and grid recomputed; tiles unchanged), the plan itself first
// the padded plan of a ternary cell (planner.cu), in place; false leaves
// `groups` unchanged
bool pad_plan(std::vector<GroupPlan> &groups, const Geometry &g,
              const PlanPtrs &ptr, int dst, int R1, long long room16);
// every group a streamed form serves takes it (planner.cu)
void stream_groups(std::vector<GroupPlan> &groups, int R1);
// 8-bit planes between the streamed first group and the launch after it
// (planner.cu), in place; false leaves `groups` unchanged
bool u8_plan(std::vector<GroupPlan> &groups, int R1, long long room16);
// algorithmic HBM bytes of one group launch (planner.cu)
long long group_bytes(const GroupArgs &a);
std::vector<GroupPlan> group_variants(const GroupPlan &p, int R1,
                                      size_t smem_cap);
// streamed form of a strided group (transform_tma.cu)
size_t tma_smem_bytes(int q, int k, int r1, int lanes, int stages,
                      int in8 = 0);
bool tma_group_ok(const GroupArgs &a, int q, int r1, int lanes, int stages);
GroupPlan tma_variant(const GroupPlan &p, int lanes, int stages, int threads);
// the first group read from cnt (axis 0 in the pair), a.tma == 2
size_t tma_first_smem_bytes(int kk, int r1, int stages);
bool tma_first_ok(const GroupArgs &a, int r1, int stages);
GroupPlan tma_first_variant(const GroupPlan &p, int stages, int threads);
// the first group of a ternary Hamming cell over row pairs, a.tma == 3
bool rows_first_ok(const GroupArgs &a, int r1);
GroupPlan rows_first_variant(const GroupPlan &p, int threads);
int launch_tma_group(const GroupPlan &p, cudaStream_t s);
int tma_prepare(const GroupPlan &p);
int tma_blocks_per_sm(const GroupPlan &p);
// A streamed launch that gave up waiting for its loads leaves its output
// unfinished: -8 (and a message) when one has since the last look, else 0.
// To be asked once the launches in question have drained.
int tma_fault_take();
// Failures made on the host, for tests of the paths behind them
// (dct_b200_fault_inject): true when this event of `kind` is the armed one.
enum FaultKind { kFaultStreamed = 0, kFaultBarrier = 1, kFaultPinned = 2,
                 kFaultKinds = 3 };
bool fault_due(int kind);
int launch_code_bounds(const long long *code, long long ncode,
                       long long tile_words, long long ntiles,
                       long long *bounds, cudaStream_t s);

// batched engine: persistent launches over (pass, tile) work items
struct BatchLaunch {
  const GroupArgs *passes;
  const int *dep;
  const unsigned *need;
  // (pass, first tile, tiles, chain): chain > 1 runs the item's pass and the
  // chain - 1 after it (single-tile passes of one cell) in the same CTA
  const int4 *items;
  long long nitems;
  unsigned *done;
  unsigned long long *next;
  int *err;
  size_t smem;
  int grid;
  int kernel;                   // -1 the runtime-size tiles, else a kernel id
  const int *pass_cell;         // cell of each pass
  const int *active;            // per cell: its items run (nullptr: all do)
};
int launch_batch(const BatchLaunch &b, cudaStream_t s);
int batch_grid(size_t smem);
// the register-blocked kernel `kernel` over work items (batch_groups.cu)
int launch_batch_groups(const BatchLaunch &b, cudaStream_t s);
// resident CTAs of that kernel over the whole GPU, opted in to `smem` bytes
int batch_groups_grid(int kernel, size_t smem);

// window pass (torus / grid) over one axis, or (q2) that axis and the next,
// any width, out of place
constexpr int kWindowPairMaxR = 3;
bool window_pair_ok(long long stride, int q, int R);
struct WindowArgs {
  const int32_t *src32; const uint16_t *src16; int pmode, ptarget, mu;
  int32_t *dst32; uint16_t *dst16;
  long long space, stride; int q, R, grid;
  int q2;                   // size of the next axis (0: one axis)
};
int launch_window(const WindowArgs &w, cudaStream_t s);

// ------------------------------------------------------------ walks
// Support table in structure-of-arrays form: slot s of pattern t is
// tbl[s*len + t] = (pos << 24) | delta, delta a circular shift in
// 1..ax_pos-1; 0 = unused slot.  Entry 0 is the centre.
struct WalkArgs {
  Geometry g;
  const int32_t *tbl;
  int slots;
  long long len;
  uint16_t *cnt;
  // the packed form of the table (pack_walk), nullptr where it has none:
  // pattern t is four 8-bit indices into the noff + 1 offsets that a word's
  // (position, shift) entries give, entry noff the 0 of an unused slot
  const uint32_t *pk = nullptr;
  const int4 *ent = nullptr;            // (stride, axis size, shift, -)
  int noff = 0;
};
constexpr int kMaxPackOff = 255;
// Is the table exactly the metric ball: distinct patterns, each moving
// distinct axes by admissible shifts within radius R, as many as the ball
// has?  Only then do a transform and walks over the table agree.
bool metric_ball_table(const Geometry &g, const std::vector<int32_t> &soa,
                       int slots, long long len);
// Packs a validated SoA table; false when the cell does not qualify: the
// open grid (it rejects patterns), 2^31 words or more, more than four slots
// or more than 255 (position, shift) entries.
bool pack_walk(const Geometry &g, const std::vector<int32_t> &soa, int slots,
               long long len, std::vector<uint32_t> &pk,
               std::vector<int4> &ent);
constexpr int kParamWords = 1024;       // words passed by value per launch
struct WordsParam { long long w[kParamWords]; };

// nb words from `dwords` (device) or, when dwords == nullptr, from `pw`
int launch_update(const WalkArgs &w, const long long *dwords,
                  const WordsParam *pw, int nb, int delta,
                  unsigned long long *trans, cudaStream_t s);
// bits: (|X|+7)/8 bytes of scratch for the predicate bit plane of a large
// call (gather_bits_pay), or nullptr
int launch_gather(const WalkArgs &w, const long long *dwords, int nb,
                  int mode, int target, int32_t *out, bool zeroed,
                  cudaStream_t s, uint8_t *bits = nullptr);
bool gather_bits_pay(const WalkArgs &w, int nb);
int pick_split(long long len, int nb);
// set side (setside.cu): list {x : pred(cnt[x])} as packed digit words, then
// count, per candidate, the listed words within distance R
int launch_list_pred(const Geometry &g, const uint16_t *cnt, int mode,
                     int target, unsigned long long *out, long long cap,
                     unsigned long long *found, cudaStream_t s);
int launch_gather_set(const Geometry &g, const long long *dcand, int nc,
                      const unsigned long long *Z, long long zn, int32_t *out,
                      bool zeroed, cudaStream_t s);
// device-side exact greedy (walks.cu) over one cell or many: a step is an
// argmax over chunk keys and a placement that lowers the gains it changes
constexpr int kGreedyStateBytes = 48;
constexpr int kGreedyChunk = 1024;        // map words per kept key
constexpr int kGreedyBlockChunks = 32;    // chunks per argmax block
constexpr int kGreedyMaxPat = 1024;       // ball patterns per place block
// host view of one cell's state (GreedyState)
struct GreedyHost {
  unsigned long long best[2];
  long long deficit;
  unsigned long long served;
  int done, placed, pend, nnew;
  long long deficit_now() const { return deficit - (pend ? (long long)served : 0); }
  int placed_now() const { return placed + (pend ? 1 : 0); }
  int gain(int par) const {
    return best[par] ? (int)((uint32_t)(best[par] >> 32) ^ 0x80000000u) : 0;
  }
};
static_assert(sizeof(GreedyHost) == kGreedyStateBytes, "state layout");
// one cell of a greedy: its walk, gain map, state and buffers
struct BatchGreedyCell {
  WalkArgs w;
  int32_t *map;
  void *st;                 // GreedyState (kGreedyStateBytes)
  long long *placed;
  long long *fresh;         // |B| words: those the last placement satisfied
  unsigned long long *ckey; // best key of each chunk of kGreedyChunk words
  const long long *code;    // words that are never placed (device)
  long long ncode;
  int max_add;
  int pats;                 // ball patterns per place block, <= kGreedyMaxPat
};
// the blocks of one cell in each launch, and its patterns per place block
inline long long greedy_chunks(long long space) {
  return (space + kGreedyChunk - 1) / kGreedyChunk;
}
inline int greedy_argmax_blocks(long long space) {
  return (int)((greedy_chunks(space) + kGreedyBlockChunks - 1) /
               kGreedyBlockChunks);
}
inline int greedy_pats(long long len, int blocks) {
  long long p = (len + blocks - 1) / blocks;
  if (p < 16) p = 16;
  if (p > kGreedyMaxPat) p = kGreedyMaxPat;
  return (int)p;
}
struct GreedyRun;         // barrier state of launch_greedy_run (device)
// takes each cell's code and the words placed so far out of its map (cells
// with rebuild[cell], or all)
int launch_greedy_exclude(const BatchGreedyCell *dcells, int ncells,
                          const int *rebuild, int32_t exclude,
                          cudaStream_t s);
// jobs: (cell, block of the cell) per block, or nullptr for one cell; par:
// parity of the step; all: read every chunk (a greedy's first step);
// rebuild[cell]: its gain map is left to a transform
int launch_greedy_argmax(const BatchGreedyCell *dcells, const int2 *jobs,
                         int njobs, int par, int all, cudaStream_t s);
int launch_greedy_place(const BatchGreedyCell *dcells, const int2 *jobs,
                        int njobs, int par, int32_t exclude, cudaStream_t s);
// the gains after a placement: `blocks` blocks per cell share its new words
int launch_greedy_refresh(const BatchGreedyCell *dcells, int ncells,
                          int blocks, const int *rebuild, cudaStream_t s);
// `steps` whole steps of one cell in a cooperative launch; run:
// kGreedyRunBytes of device state, zero before the first launch, whose second
// word is set when a barrier timed out
constexpr int kGreedyRunBytes = 16;
int launch_greedy_run(const BatchGreedyCell &cell, int par, int steps,
                      int32_t exclude, GreedyRun *run, cudaStream_t s);
// Whether a placement of gain `gain` is followed by a transform of
// `rebuild_us` microseconds rather than by gain * |B| gain updates
// (CC_GREEDY_REBUILD = 0 / 1 pins it).
bool greedy_rebuild_pays(long long gain, long long ball, double rebuild_us);
// swap evaluation fast path: per drop its loss and the list of its ball
// words at exactly mu (two walks and a segment scan), then per candidate
// the listed words of its drop within distance R
int launch_seg_scan(const int32_t *cnt, int n, long long cap, int32_t *offs,
                    int32_t *cursor, cudaStream_t s);
int launch_drop_walks(const WalkArgs &w, const long long *ddrops, int k,
                      int32_t *loss, int32_t *nmu, int32_t *offs,
                      int32_t *cursor, long long cap, long long *list,
                      cudaStream_t s);
int launch_swap_corr(const Geometry &g, int k, const long long *dcand,
                     const int32_t *dcoff, const int32_t *offs,
                     const long long *list, long long cap, int32_t *gain,
                     cudaStream_t s);
int launch_ball_hist(const WalkArgs &w, const long long *dwords, int nb,
                     const int32_t *map, int src, int nbins, int32_t *out,
                     cudaStream_t s);
int launch_layers_at(const int32_t *layers, long long plane, int R1,
                     const long long *idx, int k, int32_t *out,
                     cudaStream_t s);

// ------------------------------------------------------------ reductions
int launch_cnt_reduce(const uint16_t *cnt, long long N, int mode, int target,
                      int mu, long long *out, cudaStream_t s,
                      RedOut r = RedOut());
int launch_max(const int32_t *A, long long N, long long *out, cudaStream_t s,
               RedOut r = RedOut());
int launch_hist(const int32_t *A, long long N, int nbins, int32_t vmax,
                int32_t *hist, cudaStream_t s, RedOut r = RedOut());
int launch_extract(const int32_t *A, long long N, int32_t thr, void *oidx,
                   bool wide, int32_t *oval, long long cap, long long *ocount,
                   cudaStream_t s, RedOut r = RedOut());
int launch_read_at(const int32_t *A, const long long *idx, int k,
                   int32_t *out, cudaStream_t s);
int launch_scatter(int32_t *A, const long long *idx, long long M,
                   cudaStream_t s);

int sm_count();
// DCT_BLOCKS, read at each cell's init as coldcore's plugin reads it: when
// set, the grid of every persistent transform launch (at least 256 CTAs, at
// most one per tile; every such kernel strides its tiles by the grid); 0
// leaves the grids to the occupancy rule.
extern int g_dct_blocks;
inline int grid_knob(int grid, long long ntiles) {
  if (g_dct_blocks <= 0) return grid;
  long long g = g_dct_blocks;
  if (g > ntiles) g = ntiles;
  return (int)(g < 1 ? 1 : g);
}

}  // namespace cc

#define CC_CK(x)                                                            \
  do {                                                                      \
    cudaError_t e_ = (x);                                                   \
    if (e_ != cudaSuccess) {                                                \
      fprintf(stderr, "coldcore_b200: CUDA error %s at %s:%d\n",            \
              cudaGetErrorString(e_), __FILE__, __LINE__);                  \
      return -(100 + (int)e_);                                              \
    }                                                                       \
  } while (0)

namespace cc {
// Two timing events, destroyed on every way out of the scope that made
// them (error returns included).
struct EventPair {
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int create() {
    CC_CK(cudaEventCreate(&e0));
    CC_CK(cudaEventCreate(&e1));
    return 0;
  }
  ~EventPair() {
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  }
};
}  // namespace cc
