// walks.cu — exact incremental updates and per-candidate queries over a
// word's support set (its metric ball).
//
// Semantics of the reference's support walks
// (coldcore src/plugins/covering/dctcore_core.cuh:158-273, dctcore_grid.cuh
// :239-342, dctcore_mu.cuh:75-105, dctcore_fast.cuh:360-389): the ball of a
// centre w is the support table's patterns applied to w's digits, each
// pattern a set of (position, circular shift) pairs; the open grid rejects a
// pattern whose shift wraps past a board edge.  cnt is a uint16 plane,
// updated with packed 32-bit atomics on the aligned counter pair (the plane
// is padded, so the partner of the last counter exists and stays 0).
//
// The table is held as 32-bit (position, delta) slots instead of the v1
// nibble bytes, so axes of any width walk (the v1 format stops at 16).  A
// block owns one word (or a slice of its ball when the ball is large): the
// word's digits, axis sizes and strides sit in shared memory, and each
// thread resolves one pattern at a time with a few integer ops per slot.
#include <algorithm>
#include <cstdlib>

#include "engine.h"

namespace cc {

// Walk kinds: the table's slots resolved per pattern (kSlots; kGrid rejects
// patterns that leave the board), or the packed table (kPack): a word's
// (position, shift) offsets are computed once per block into shared memory,
// and a pattern is one 32-bit table read, four shared reads and three adds
// instead of up to four table reads with a digit, a wrap and a 64-bit
// multiply each.
enum Walk { kSlots = 0, kGridWalk = 1, kPack = 2 };

struct WordSmem {
  int dig[kMaxAxes];
  int ax[kMaxAxes];
  long long pw[kMaxAxes];
};
union WalkSmem {
  WordSmem s;
  int32_t off[kMaxPackOff + 1];
};

inline int walk_kind(const WalkArgs &w) {
  return w.g.prob == kGrid ? kGridWalk : w.pk ? kPack : kSlots;
}

template <int WALK>
__device__ __forceinline__ void word_setup(const WalkArgs &a, long long w,
                                           WalkSmem &m) {
  if (WALK == kPack) {
    for (int e = threadIdx.x; e <= a.noff; e += blockDim.x) {
      int v = 0;
      if (e < a.noff) {
        const int4 en = __ldg(a.ent + e);
        const int dg = (int)((unsigned)w / (unsigned)en.x % (unsigned)en.y);
        const int nd = dg + en.z >= en.y ? en.z - en.y : en.z;
        v = nd * en.x;
      }
      m.off[e] = v;
    }
  } else {
    for (int j = threadIdx.x; j < a.g.n; j += blockDim.x) {
      m.s.dig[j] = (int)((w / a.g.pw[j]) % a.g.ax[j]);
      m.s.ax[j] = a.g.ax[j];
      m.s.pw[j] = a.g.pw[j];
    }
  }
  __syncthreads();
}

// word index of pattern t around w; -1 when the open grid rejects it
template <int WALK>
__device__ __forceinline__ long long walk_word(const WalkArgs &a, long long w,
                                               long long t,
                                               const WalkSmem &m) {
  if (WALK == kPack) {
    const uint32_t p = __ldg(a.pk + t);
    return (int32_t)w + m.off[p & 255u] + m.off[(p >> 8) & 255u] +
           m.off[(p >> 16) & 255u] + m.off[p >> 24];
  }
  const WordSmem &s = m.s;
  long long x = w;
#pragma unroll 1
  for (int k = 0; k < a.slots; k++) {
    const int code = a.tbl[(long long)k * a.len + t];
    if (!code) break;
    const int p = code >> 24, dl = code & 0xFFFFFF;
    const int dg = s.dig[p];
    int nd = dg + dl;
    if (nd >= s.ax[p]) nd -= s.ax[p];
    const int sh = nd - dg;
    if (WALK == kGridWalk && (sh > a.g.R || sh < -a.g.R)) return -1;
    x += (long long)sh * s.pw[p];
  }
  return x;
}

bool metric_ball_table(const Geometry &g, const std::vector<int32_t> &soa,
                       int slots, long long len) {
  const bool sum = g.prob == kHamming || g.prob == kLee;
  auto weight = [&](int pos, int d) -> int {      // -1: inadmissible
    const int a = g.ax[pos], c = std::min(d, a - d);
    if (d < 1 || d >= a) return -1;
    if (g.prob == kHamming) return 1;
    return c > g.R ? -1 : sum ? c : 0;
  };
  static_assert(kMaxAxes <= 64, "one bit an axis");
  std::vector<long long> words((size_t)len);        // around word 0
  for (long long t = 0; t < len; t++) {
    unsigned long long moved = 0;
    long long x = 0;
    int w = 0;
    bool open = true;
    for (int k = 0; k < slots; k++) {
      const int32_t c = soa[(size_t)k * len + t];
      if (!c) { open = false; continue; }
      const int pos = c >> 24, d = c & 0xFFFFFF;
      // a walk stops at a gap
      if (!open || pos >= g.n || (moved >> pos & 1)) return false;
      moved |= 1ULL << pos;
      const int e = weight(pos, d);
      if (e < 0) return false;
      w += e;
      x += d * g.pw[pos];
    }
    if (w > g.R) return false;
    words[(size_t)t] = x;
  }
  std::sort(words.begin(), words.end());
  if (std::adjacent_find(words.begin(), words.end()) != words.end())
    return false;
  // |B|: coefficients 0..W of prod_j (1 + sum_d t^weight(j, d))
  const int W = sum ? g.R : 0;
  std::vector<long double> poly(W + 1, 0.0L);
  poly[0] = 1.0L;
  for (int j = 0; j < g.n; j++) {
    std::vector<long double> nx(poly);
    for (int w = 0; w <= W; w++)
      for (int d = 1; d < g.ax[j]; d++) {
        const int e = weight(j, d);
        if (e >= 0 && w + e <= W) nx[w + e] += poly[w];
      }
    poly.swap(nx);
  }
  long double tot = 0;
  for (long double v : poly) tot += v;
  return tot == (long double)len;
}

bool pack_walk(const Geometry &g, const std::vector<int32_t> &soa, int slots,
               long long len, std::vector<uint32_t> &pk,
               std::vector<int4> &ent) {
  if (g.prob == kGrid || g.space >= (1LL << 31) || slots > 4) return false;
  std::vector<int> base(g.n + 1, 0);
  for (int j = 0; j < g.n; j++) {
    if (g.ax[j] > kMaxPackOff) return false;
    base[j + 1] = base[j] + g.ax[j] - 1;
  }
  const int noff = base[g.n];
  if (noff > kMaxPackOff) return false;
  ent.clear();
  for (int j = 0; j < g.n; j++)
    for (int d = 1; d < g.ax[j]; d++)
      ent.push_back(make_int4((int)g.pw[j], g.ax[j], d, 0));
  pk.resize((size_t)len);
  for (long long t = 0; t < len; t++) {
    uint32_t v = 0;
    bool open = true;                     // slots after an empty one: unused
    for (int k = 0; k < 4; k++) {
      const int32_t c = open && k < slots ? soa[(size_t)k * len + t] : 0;
      open = open && c;
      const int e = c ? base[c >> 24] + (c & 0xFFFFFF) - 1 : noff;
      v |= (uint32_t)e << (8 * k);
    }
    pk[(size_t)t] = v;
  }
  return true;
}

__device__ __forceinline__ long long block_sum(long long v) {
  __shared__ long long red[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();                      // red may be in use by a prior call
  if (lane == 0) red[wid] = v;
  __syncthreads();
  v = threadIdx.x < (blockDim.x >> 5) ? red[lane] : 0;
  if (wid == 0)
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;                             // valid in thread 0
}

// cnt[x] += delta over each word's support set.  trans != nullptr also
// counts the deficit transitions read off the atomics' old values (an
// increment from c < mu, a decrement from c <= mu).
template <int WALK, bool PARAM>
__global__ void __launch_bounds__(256)
k_update(const WalkArgs a, const long long *words, const WordsParam pw,
         int split, int delta, unsigned long long *trans) {
  __shared__ WalkSmem s;
  const int wi = blockIdx.x / split, seg = blockIdx.x % split;
  const long long w = PARAM ? pw.w[wi] : words[wi];
  word_setup<WALK>(a, w, s);
  long long acc = 0;
  const long long step = (long long)split * blockDim.x;
  for (long long t = (long long)seg * blockDim.x + threadIdx.x; t < a.len;
       t += step) {
    const long long x = walk_word<WALK>(a, w, t, s);
    if (x < 0) continue;
    uint32_t *cell = reinterpret_cast<uint32_t *>(a.cnt + (x & ~1LL));
    const int sh = (x & 1) ? 16 : 0;
    const uint32_t add = 1u << sh;
    const uint32_t old = delta > 0 ? atomicAdd(cell, add) : atomicSub(cell, add);
    if (trans) {
      const int c = (int)((old >> sh) & 0xFFFFu);
      acc += delta > 0 ? (c < a.g.mu) : (c <= a.g.mu);
    }
  }
  if (trans) {
    acc = block_sum(acc);
    if (threadIdx.x == 0 && acc) atomicAdd(trans, (unsigned long long)acc);
  }
}

// out[wi] = #{x in B(w_i) : pred(cnt[x])}; split blocks per word add up
template <int WALK>
__global__ void __launch_bounds__(256)
k_gather(const WalkArgs a, const long long *words, int split, int mode,
         int target, int32_t *out) {
  __shared__ WalkSmem s;
  const int wi = blockIdx.x / split, seg = blockIdx.x % split;
  const long long w = words[wi];
  word_setup<WALK>(a, w, s);
  long long acc = 0;
  const long long step = (long long)split * blockDim.x;
  for (long long t = (long long)seg * blockDim.x + threadIdx.x; t < a.len;
       t += step) {
    const long long x = walk_word<WALK>(a, w, t, s);
    if (x >= 0) acc += cnt_pred(mode, (int)a.cnt[x], target, a.g.mu);
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) {
    if (split == 1) out[wi] = (int32_t)acc;
    else if (acc) atomicAdd(&out[wi], (int32_t)acc);
  }
}

// out[wi][b] = #{x in B(w_i) : bin(x) == b}.  src 0 bins the map in log2
// steps (0 for v <= 0, 1 for v == 1, 2 for 2..3, 3 for 4..7, ...), src 1
// bins cnt linearly (cnt == b); both clip to nbins - 1.
template <int WALK>
__global__ void __launch_bounds__(256)
k_ball_hist(const WalkArgs a, const long long *words, int split,
            const int32_t *map, int src, int nbins, int32_t *out) {
  __shared__ WalkSmem s;
  __shared__ int32_t hist[32];
  const int wi = blockIdx.x / split, seg = blockIdx.x % split;
  const long long w = words[wi];
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) hist[b] = 0;
  word_setup<WALK>(a, w, s);
  const long long step = (long long)split * blockDim.x;
  for (long long t = (long long)seg * blockDim.x + threadIdx.x; t < a.len;
       t += step) {
    const long long x = walk_word<WALK>(a, w, t, s);
    if (x < 0) continue;
    int b;
    if (src == 0) {
      const int32_t v = map[x];
      b = v <= 0 ? 0 : min(nbins - 1, 32 - __clz(v));
    } else {
      b = min(nbins - 1, (int)a.cnt[x]);
    }
    atomicAdd(&hist[b], 1);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nbins; b += blockDim.x)
    if (hist[b]) atomicAdd(&out[(long long)wi * nbins + b], hist[b]);
}

int launch_ball_hist(const WalkArgs &w, const long long *dwords, int nb,
                     const int32_t *map, int src, int nbins, int32_t *out,
                     cudaStream_t s) {
  if (nb <= 0) return 0;
  const int split = pick_split(w.len, nb);
  CC_CK(cudaMemsetAsync(out, 0, (size_t)nb * nbins * 4, s));
  const dim3 grid((unsigned)nb * split);
#define CC_BH(W)                                                            \
  case W:                                                                   \
    k_ball_hist<W><<<grid, 256, 0, s>>>(w, dwords, split, map, src, nbins,  \
                                        out);                               \
    break;
  switch (walk_kind(w)) { CC_BH(kSlots) CC_BH(kGridWalk) CC_BH(kPack) }
#undef CC_BH
  CC_CK(cudaGetLastError());
  return 0;
}

// the R + 1 layer values at each of k words: out[i][d]
__global__ void k_layers_at(const int32_t *layers, long long plane, int R1,
                            const long long *idx, int k, int32_t *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k) return;
  for (int d = 0; d < R1; d++) out[(long long)i * R1 + d] =
      layers[d * plane + idx[i]];
}

int launch_layers_at(const int32_t *layers, long long plane, int R1,
                     const long long *idx, int k, int32_t *out,
                     cudaStream_t s) {
  if (k <= 0) return 0;
  k_layers_at<<<(k + 255) / 256, 256, 0, s>>>(layers, plane, R1, idx, k, out);
  CC_CK(cudaGetLastError());
  return 0;
}

// swap evaluation, first walk: per drop word, its loss (critical ball words)
// and nmu = its ball words at exactly mu, the words that become deficient
// when one copy of the drop is removed
template <int WALK>
__global__ void __launch_bounds__(256)
k_drop_count(const WalkArgs a, const long long *drops, int split,
             int32_t *loss, int32_t *nmu) {
  __shared__ WalkSmem s;
  const int wi = blockIdx.x / split, seg = blockIdx.x % split;
  const long long w = drops[wi];
  word_setup<WALK>(a, w, s);
  long long lo = 0, at = 0;
  const long long step = (long long)split * blockDim.x;
  for (long long t = (long long)seg * blockDim.x + threadIdx.x; t < a.len;
       t += step) {
    const long long x = walk_word<WALK>(a, w, t, s);
    if (x < 0) continue;
    const int c = (int)a.cnt[x];
    lo += c >= 1 && c <= a.g.mu;
    at += c == a.g.mu;
  }
  lo = block_sum(lo);
  if (threadIdx.x == 0 && lo) atomicAdd(&loss[wi], (int32_t)lo);
  at = block_sum(at);
  if (threadIdx.x == 0 && at) atomicAdd(&nmu[wi], (int32_t)at);
}

// second walk: the words at exactly mu, into the drop's segment of `list`
// (cursor[i] starts at the segment's offset); slots past cap are dropped and
// the caller, seeing the total above cap, falls back
template <int WALK>
__global__ void __launch_bounds__(256)
k_drop_list(const WalkArgs a, const long long *drops, int split,
            int32_t *cursor, long long cap, long long *list) {
  __shared__ WalkSmem s;
  const int wi = blockIdx.x / split, seg = blockIdx.x % split;
  const long long w = drops[wi];
  word_setup<WALK>(a, w, s);
  const long long step = (long long)split * blockDim.x;
  for (long long t = (long long)seg * blockDim.x + threadIdx.x; t < a.len;
       t += step) {
    const long long x = walk_word<WALK>(a, w, t, s);
    if (x < 0 || (int)a.cnt[x] != a.g.mu) continue;
    const int slot = atomicAdd(&cursor[wi], 1);
    if (slot < cap) list[slot] = x;
  }
}

int launch_drop_walks(const WalkArgs &w, const long long *ddrops, int k,
                      int32_t *loss, int32_t *nmu, int32_t *offs,
                      int32_t *cursor, long long cap, long long *list,
                      cudaStream_t s) {
  if (k <= 0) return 0;
  const int split = pick_split(w.len, k);
  const dim3 grid((unsigned)k * split);
  const int kind = walk_kind(w);
#define CC_DC(W)                                                            \
  case W:                                                                   \
    k_drop_count<W><<<grid, 256, 0, s>>>(w, ddrops, split, loss, nmu);      \
    break;
  switch (kind) { CC_DC(kSlots) CC_DC(kGridWalk) CC_DC(kPack) }
#undef CC_DC
  CC_CK(cudaGetLastError());
  int rc = launch_seg_scan(nmu, k, cap, offs, cursor, s);
  if (rc) return rc;
#define CC_DL(W)                                                            \
  case W:                                                                   \
    k_drop_list<W><<<grid, 256, 0, s>>>(w, ddrops, split, cursor, cap,      \
                                        list);                              \
    break;
  switch (kind) { CC_DL(kSlots) CC_DL(kGridWalk) CC_DL(kPack) }
#undef CC_DL
  CC_CK(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------ device greedy
// The exact greedy over one cell (dct_b200_greedy_fill) or many at once (the
// batched engine's campaign repair), three launches a step:
//
//   k_greedy_argmax   the word of largest gain (ties: the smallest index).
//     The map is cut into chunks of kChunk words whose best keys are kept.
//     Gains never grow, so a kept key holds until its own word loses gain: a
//     step looks at that one word of each chunk and reads only the chunks
//     where it did, after a transform of the map too.  (A flag set by the
//     refresh where an updated word's gain equals its chunk's best costs a
//     second random read for each of the |fresh| x |B| updates, and ties
//     flag chunks for nothing: 14.0 us a step on K_3(14,3), 12.4 us this way.)
//   k_greedy_place    the word's ball, split over many blocks: cnt += 1 with
//     pair atomics; the words it satisfies (old count mu - 1) are listed.
//   k_greedy_refresh  lowers the gain of every candidate whose ball holds a
//     listed word, the list's balls shared out evenly in pieces.  (Blocks of
//     the place launch that refresh their own words need no list and no
//     third launch, but the words cluster: 46 us a step on K_3(14,3) near a
//     cover, against 16 us for the three.)
//
// When a placement satisfies many words, |fresh| x |B| gain updates cost more
// than a gain transform of the whole cell; the caller then leaves the map to
// a transform (rebuild), and the next argmax reads every chunk.  Gains never
// grow, so a cell leaves that regime for good.
//
// The state is committed by the NEXT argmax launch (block 0 of the cell), so
// every block of one place launch decides the same stop from values that the
// launch itself does not change.
struct GreedyState {
  // packed argmax keys of even and odd steps: (gain ^ sign) << 32 | ~index,
  // so the largest gain wins and ties go to the smallest index
  unsigned long long best[2];
  long long deficit;            // sum max(0, mu - cnt) before the last place
  unsigned long long served;    // the last placement's part of it
  int done;                     // no positive gain, or nothing uncovered
  int placed;                   // words placed before the last place
  int pend;                     // the last place launch placed a word
  int nnew;                     // words it satisfied (old count mu - 1)
};
static_assert(sizeof(GreedyState) == kGreedyStateBytes, "state layout");

constexpr int kChunk = kGreedyChunk;
// Updates a refresh makes in a microsecond, against a transform of the cell:
// 90,000 on K_3(14,3) (487 K of them in 5.4 us), whose map stays in L2, fewer
// on maps that pass it.  One line serves both because neither side is steep
// there: 64 mixed cells of up to 16.8 M words take 14.9 ms at any line from
// 36,000 to 90,000, and 24.7 ms at 130,000.
constexpr double kGreedyUpdatesPerUs = 36000.0;
constexpr int kBlockChunks = kGreedyBlockChunks;
constexpr int kArgmaxWarps = 8;

__device__ __forceinline__ unsigned long long greedy_key(int32_t v,
                                                         long long x) {
  return ((unsigned long long)((uint32_t)v ^ 0x80000000u) << 32) |
         (uint32_t)~(uint32_t)x;
}
__device__ __forceinline__ int32_t key_gain(unsigned long long k) {
  return (int32_t)((uint32_t)(k >> 32) ^ 0x80000000u);
}

// a chunk's kept key k, or 0 if its word has lost gain since
__device__ __forceinline__ unsigned long long fresh_key(
    const BatchGreedyCell &c, unsigned long long k) {
  return __ldcg(c.map + (uint32_t)~(uint32_t)k) == key_gain(k) ? k : 0;
}

// map[x] = exclude for a cell's code and placed words (they never re-enter);
// runs after a place launch, whose own word counts (pend)
__global__ void __launch_bounds__(256)
k_greedy_exclude(const BatchGreedyCell *__restrict__ cells,
                 const int *__restrict__ rebuild, int32_t exclude) {
  if (rebuild && !rebuild[blockIdx.y]) return;
  const BatchGreedyCell &c = cells[blockIdx.y];
  const GreedyState *st = reinterpret_cast<const GreedyState *>(c.st);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = t; i < c.ncode; i += step) c.map[c.code[i]] = exclude;
  const long long n = st->placed + (st->pend ? 1 : 0);
  for (long long i = t; i < n; i += step) c.map[c.placed[i]] = exclude;
}

// a warp: the key of chunk ch read from the map, and kept
__device__ __forceinline__ unsigned long long read_chunk(
    const BatchGreedyCell &c, long long ch) {
  const long long N = c.w.g.space, x0 = ch * kChunk;
  const int lane = threadIdx.x & 31;
  unsigned long long m = 0;
  if (x0 + kChunk <= N) {
    const int4 *v4 = reinterpret_cast<const int4 *>(c.map + x0);
    int4 q[kChunk / 128];
#pragma unroll
    for (int u = 0; u < kChunk / 128; u++) q[u] = __ldcg(v4 + lane + 32 * u);
#pragma unroll
    for (int u = 0; u < kChunk / 128; u++) {
      const long long x = x0 + 4 * (lane + 32 * u);
      m = max(m, greedy_key(q[u].x, x));
      m = max(m, greedy_key(q[u].y, x + 1));
      m = max(m, greedy_key(q[u].z, x + 2));
      m = max(m, greedy_key(q[u].w, x + 3));
    }
  } else {
    for (long long x = x0 + lane; x < N; x += 32)
      m = max(m, greedy_key(__ldcg(c.map + x), x));
  }
  for (int o = 16; o > 0; o >>= 1)
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) c.ckey[ch] = m;
  return m;
}

// jobs: (cell, block of the cell), or nullptr for cell 0 and blockIdx.x;
// block 0 of a cell also commits its last placement
__global__ void __launch_bounds__(32 * kArgmaxWarps)
k_greedy_argmax(const BatchGreedyCell *__restrict__ cells,
                const int2 *__restrict__ jobs, int par, int all) {
  const int2 job = jobs ? jobs[blockIdx.x] : make_int2(0, (int)blockIdx.x);
  const BatchGreedyCell &c = cells[job.x];
  GreedyState *st = reinterpret_cast<GreedyState *>(c.st);
  if (st->done) return;
  if (job.y == 0 && threadIdx.x == 0) {
    if (st->pend) {
      st->deficit -= (long long)st->served;
      st->placed += 1;
      st->pend = 0;
    }
    st->served = 0;
    st->nnew = 0;
    st->best[par ^ 1] = 0;
  }
  // lane j looks at the warp's chunk j, the warp reads the stale ones
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long first = (long long)job.y * kBlockChunks + warp;
  const long long mine = first + (long long)kArgmaxWarps * lane;
  unsigned long long m = 0;
  bool stale = false;
  if (lane < kBlockChunks / kArgmaxWarps && mine * kChunk < c.w.g.space) {
    if (!all) m = fresh_key(c, __ldcg(c.ckey + mine));
    stale = m == 0;
  }
  for (unsigned todo = __ballot_sync(0xffffffffu, stale); todo;
       todo &= todo - 1)
    m = max(m, read_chunk(c, first + kArgmaxWarps * (__ffs(todo) - 1)));
  for (int o = 16; o > 0; o >>= 1)
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  // one atomic a warp; most warps see a larger key already there
  if (lane == 0 && m > __ldcg(&st->best[par]))
    atomicMax(&st->best[par], m);
}

template <int WALK>
__device__ __forceinline__ void greedy_place(const BatchGreedyCell &c,
                                             int seg, int par,
                                             int32_t exclude) {
  __shared__ WalkSmem s;
  __shared__ long long fresh[kGreedyMaxPat];
  __shared__ long long w_s;
  __shared__ int stop;
  __shared__ int nfresh, base;
  GreedyState *st = reinterpret_cast<GreedyState *>(c.st);
  const WalkArgs &a = c.w;
  if (threadIdx.x == 0) {
    const unsigned long long k = __ldcg(&st->best[par]);
    const long long x = (long long)(uint32_t)~(uint32_t)k;
    const int done = __ldcg(&st->done), placed = __ldcg(&st->placed);
    stop = done || k == 0 || key_gain(k) <= 0 || __ldcg(&st->deficit) <= 0 ||
           placed >= c.max_add;
    w_s = x;
    nfresh = 0;
    if (seg == 0) {
      if (stop) {
        st->done = 1;
      } else {
        c.placed[placed] = x;
        st->pend = 1;
        c.map[x] = exclude;
      }
    }
  }
  __syncthreads();
  if (stop) return;
  word_setup<WALK>(a, w_s, s);
  int mine = 0;
  const long long t1 = min(a.len, (long long)(seg + 1) * c.pats);
  for (long long t = (long long)seg * c.pats + threadIdx.x; t < t1;
       t += blockDim.x) {
    const long long x = walk_word<WALK>(a, w_s, t, s);
    if (x < 0) continue;
    uint32_t *cell = reinterpret_cast<uint32_t *>(a.cnt + (x & ~1LL));
    const int sh = (x & 1) ? 16 : 0;
    const uint32_t old = atomicAdd(cell, 1u << sh);
    const int cv = (int)((old >> sh) & 0xFFFFu);
    mine += cv < a.g.mu;
    if (cv == a.g.mu - 1) fresh[atomicAdd(&nfresh, 1)] = x;
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine)
    atomicAdd(&st->served, (unsigned long long)mine);
  __syncthreads();
  if (threadIdx.x == 0 && nfresh) base = atomicAdd(&st->nnew, nfresh);
  __syncthreads();
  for (int i = threadIdx.x; i < nfresh; i += blockDim.x)
    c.fresh[base + i] = fresh[i];
}

__global__ void __launch_bounds__(256)
k_greedy_place(const BatchGreedyCell *__restrict__ cells,
               const int2 *__restrict__ jobs, int par, int32_t exclude) {
  const int2 job = jobs ? jobs[blockIdx.x] : make_int2(0, (int)blockIdx.x);
  const BatchGreedyCell &c = cells[job.x];
  if (c.w.g.prob == kGrid) greedy_place<kGridWalk>(c, job.y, par, exclude);
  else if (c.w.pk) greedy_place<kPack>(c, job.y, par, exclude);
  else greedy_place<kSlots>(c, job.y, par, exclude);
}

// every word satisfied by the placement stops counting towards the gain of
// the candidates whose balls hold it: map[y] -= 1 for y in B(u), in pieces
// of kRefreshPat patterns of one word shared out over the cell's blocks
constexpr int kRefreshPat = 1024;          // four a thread of 256

template <int WALK>
__device__ __forceinline__ void greedy_refresh(const BatchGreedyCell &c) {
  __shared__ WalkSmem s;
  const WalkArgs &a = c.w;
  const GreedyState *st = reinterpret_cast<const GreedyState *>(c.st);
  const long long nseg = (a.len + kRefreshPat - 1) / kRefreshPat;
  const long long n = st->nnew * nseg;
  for (long long p = blockIdx.x; p < n; p += gridDim.x) {
    const long long x0 = __ldcg(c.fresh + p / nseg);
    const long long t0 = p % nseg * kRefreshPat;
    const long long t1 = min(a.len, t0 + kRefreshPat);
    __syncthreads();                      // s is reused across words
    word_setup<WALK>(a, x0, s);
    long long y[4];
    const long long tt = t0 + threadIdx.x;
#pragma unroll
    for (int j = 0; j < 4; j++)
      y[j] = tt + 256 * j < t1 ? walk_word<WALK>(a, x0, tt + 256 * j, s) : -1;
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (y[j] >= 0) atomicSub(&c.map[y[j]], 1);
  }
}

__global__ void __launch_bounds__(256)
k_greedy_refresh(const BatchGreedyCell *__restrict__ cells,
                 const int *__restrict__ rebuild) {
  if (rebuild && rebuild[blockIdx.y]) return;
  const BatchGreedyCell &c = cells[blockIdx.y];
  if (c.w.g.prob == kGrid) greedy_refresh<kGridWalk>(c);
  else if (c.w.pk) greedy_refresh<kPack>(c);
  else greedy_refresh<kSlots>(c);
}

// ---------------------------------------------------- many steps, one launch
// `steps` whole steps of ONE cell in a cooperative launch, a grid barrier
// (1.2 us) between the phases.  Near a cover a phase is a few microseconds of
// dependent L2 round trips, so what does not change is kept close: the cell
// is a kernel parameter, the packed table and its entries sit in shared
// memory, the keys of its chunks beside them (7,500 -> 7,380 us for 640
// steps).  On K_3(14,3) a step takes 9 us at gains of 50 and 14 us at 160;
// the whole-map argmax, one-block place and refresh launches this replaces
// took 49 us, the three launches above 25 us (9 of them gaps).  The grid is
// resident as a whole (a cooperative launch) and every wait is bounded: a
// block that has waited 2 s sets the run's error and returns, and so do the
// others in their turn.
struct GreedyRun {
  unsigned arrived;             // blocks that reached a barrier so far
  int err;
  int pad[2];
};
static_assert(sizeof(GreedyRun) == kGreedyRunBytes, "run layout");

// barrier number `bar` (1, 2, ...)
__device__ __forceinline__ bool grid_barrier(GreedyRun *r, unsigned bar) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned target = bar * gridDim.x;
    int good = 1;
    unsigned seen;
    unsigned long long t0 = 0;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&r->arrived)
                 : "memory");
    for (unsigned polls = 0;; polls++) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];"
                   : "=r"(seen) : "l"(&r->arrived) : "memory");
      if (seen >= target) break;
      if ((polls & 1023u) != 1023u) continue;
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (!t0) t0 = now;
      if (now - t0 > 2000000000ULL) {
        atomicExch(&r->err, 1);
        good = 0;
        break;
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

constexpr int kRunThreads = 256;
constexpr int kRunWarps = kRunThreads / 32;
constexpr int kRunPat = 128;            // patterns of one refresh piece
constexpr int kRunTable = 8192;         // packed patterns kept in shared memory
// k_greedy_run's static shared memory (rounded up) with the longest table: it
// runs without an opt-in, so the sum stays within what every launch may use
constexpr size_t kRunStatic = kMaxPackOff * sizeof(int4) +
                              kRunWarps * sizeof(WalkSmem) +
                              (kRunWarps + kRunThreads) * 8 +
                              (kRunThreads + 1) * 4 + 128;
static_assert(kRunStatic + kRunTable * 4 <= 48 * 1024,
              "the persistent greedy's shared memory");

// one warp's form of word_setup
template <int WALK>
__device__ __forceinline__ void warp_setup(const WalkArgs &a, const int4 *ent,
                                           long long w, WalkSmem &m) {
  const int lane = threadIdx.x & 31;
  __syncwarp();                         // the warp's last walk is over
  if (WALK == kPack) {
    for (int e = lane; e <= a.noff; e += 32) {
      int v = 0;
      if (e < a.noff) {
        const int4 en = ent[e];
        const int dg = (int)((unsigned)w / (unsigned)en.x % (unsigned)en.y);
        v = (dg + en.z >= en.y ? en.z - en.y : en.z) * en.x;
      }
      m.off[e] = v;
    }
  } else {
    for (int j = lane; j < a.g.n; j += 32) {
      m.s.dig[j] = (int)((w / a.g.pw[j]) % a.g.ax[j]);
      m.s.ax[j] = a.g.ax[j];
      m.s.pw[j] = a.g.pw[j];
    }
  }
  __syncwarp();
}

// Argmax is shared out by chunks, whose stale ones a block's warps read side
// by side; place by whole warps of patterns (three lanes of every warp of the
// grid instead meant 2,368 atomics on two addresses, 1.5 us); refresh by
// pieces of kRunPat patterns of one new word, whose updates are all in flight
// together.  (A block refreshing its own new words saves a barrier,
// 1.4 us, but a word's 2,969 updates by one block take 8 us.)
template <int WALK>
__global__ void __launch_bounds__(kRunThreads)
k_greedy_run(const __grid_constant__ BatchGreedyCell c, int table_words,
             int par, int steps, int32_t exclude, GreedyRun *run) {
  extern __shared__ uint32_t table[];
  __shared__ int4 ent[WALK == kPack ? kMaxPackOff : 1];
  __shared__ WalkSmem smem[kRunWarps];
  __shared__ unsigned long long wbest[kRunWarps], keys[kRunThreads];
  __shared__ int stale[kRunThreads], nstale;
  GreedyState *st = reinterpret_cast<GreedyState *>(c.st);
  const WalkArgs &a = c.w;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  WalkSmem &s = smem[warp];
  // warps of the grid, the blocks' first warps first
  const long long W = (long long)gridDim.x * kRunWarps;
  const long long gw = (long long)warp * gridDim.x + blockIdx.x;
  if (__ldcg(&st->done)) return;        // nobody sets it before barrier 1
  if (WALK == kPack) {
    if (tid < a.noff) ent[tid] = a.ent[tid];
    for (int t = tid; t < table_words; t += kRunThreads) table[t] = a.pk[t];
    __syncthreads();
  }
  auto walk = [&](long long w, long long t) -> long long {
    if (WALK != kPack) return walk_word<WALK>(a, w, t, s);
    const uint32_t p = table_words ? table[t] : __ldg(a.pk + t);
    return (int32_t)w + s.off[p & 255u] + s.off[(p >> 8) & 255u] +
           s.off[(p >> 16) & 255u] + s.off[p >> 24];
  };
  const long long nch = (a.g.space + kChunk - 1) / kChunk;
  // the first kRunThreads of the block's chunks keep their keys here
  if (blockIdx.x + (long long)tid * gridDim.x < nch)
    keys[tid] = __ldcg(c.ckey + blockIdx.x + (long long)tid * gridDim.x);
  const long long nseg = (a.len + kRunPat - 1) / kRunPat;
  unsigned bar = 0;
  for (int i = 0; i < steps; i++, par ^= 1) {
    // -------- argmax; block 0 commits the last placement
    if (blockIdx.x == 0 && tid == 0) {
      if (__ldcg(&st->pend)) {
        st->deficit = __ldcg(&st->deficit) - (long long)__ldcg(&st->served);
        st->placed = __ldcg(&st->placed) + 1;
        st->pend = 0;
      }
      st->served = 0;
      st->nnew = 0;
      st->best[par ^ 1] = 0;
    }
    // a thread looks at each of the block's chunks, its warps share the
    // stale ones
    unsigned long long k = 0;
    for (long long b = blockIdx.x; b < nch; b += kRunThreads * gridDim.x) {
      const long long ch = b + (long long)tid * gridDim.x;
      __syncthreads();                  // the last round's list is read
      if (tid == 0) nstale = 0;
      __syncthreads();
      if (ch < nch) {
        const unsigned long long key = fresh_key(
            c, b == blockIdx.x ? keys[tid] : __ldcg(c.ckey + ch));
        if (key == 0) stale[atomicAdd(&nstale, 1)] = tid;
        k = max(k, key);
      }
      __syncthreads();
      for (int q = warp; q < nstale; q += kRunWarps) {
        const int own = stale[q];
        const unsigned long long key =
            read_chunk(c, b + (long long)own * gridDim.x);
        if (lane == 0 && b == blockIdx.x) keys[own] = key;
        k = max(k, key);
      }
    }
    for (int o = 16; o > 0; o >>= 1)
      k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
    if (lane == 0) wbest[warp] = k;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < kRunWarps; w++) k = max(k, wbest[w]);
      if (k) atomicMax(&st->best[par], k);
    }
    if (!grid_barrier(run, ++bar)) return;
    // -------- place: every thread of the grid reads the same verdict
    const unsigned long long best = __ldcg(&st->best[par]);
    const long long deficit = __ldcg(&st->deficit);
    const int placed = __ldcg(&st->placed);
    const long long x0 = (long long)(uint32_t)~(uint32_t)best;
    if (best == 0 || key_gain(best) <= 0 || deficit <= 0 ||
        placed >= c.max_add) {
      if (blockIdx.x == 0 && tid == 0) st->done = 1;
      return;
    }
    if (blockIdx.x == 0 && tid == 0) {
      c.placed[placed] = x0;
      st->pend = 1;
      c.map[x0] = exclude;
    }
    if (32 * gw < a.len) {
      warp_setup<WALK>(a, ent, x0, s);
      for (long long b = 32 * gw; b < a.len; b += 32 * W) {
        const long long t = b + lane;
        const long long x = t < a.len ? walk(x0, t) : -1;
        int cv = 0x10000;
        if (x >= 0) {
          uint32_t *cell = reinterpret_cast<uint32_t *>(a.cnt + (x & ~1LL));
          const int sh = (x & 1) ? 16 : 0;
          cv = (int)((atomicAdd(cell, 1u << sh) >> sh) & 0xFFFFu);
        }
        const int mine = __popc(__ballot_sync(0xffffffffu, cv < a.g.mu));
        const unsigned hit = __ballot_sync(0xffffffffu, cv == a.g.mu - 1);
        int at = 0;
        if (lane == 0 && mine) {
          atomicAdd(&st->served, (unsigned long long)mine);
          if (hit) at = atomicAdd(&st->nnew, __popc(hit));
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        if (cv == a.g.mu - 1)
          c.fresh[at + __popc(hit & ((1u << lane) - 1u))] = x;
      }
    }
    if (!grid_barrier(run, ++bar)) return;
    // -------- refresh
    const long long n = __ldcg(&st->nnew) * nseg;
    for (long long p0 = gw; p0 < n; p0 += 32 * W) {
      // the words of the warp's next 32 pieces in one read
      const long long pl = p0 + lane * W;
      const long long ul = pl < n ? __ldcg(c.fresh + pl / nseg) : 0;
      const int sl = (int)(pl % nseg);
      for (int r = 0; r < 32 && p0 + r * W < n; r++) {
        const long long u = __shfl_sync(0xffffffffu, ul, r);
        const long long t0 =
            (long long)__shfl_sync(0xffffffffu, sl, r) * kRunPat + lane;
        warp_setup<WALK>(a, ent, u, s);
        long long y[kRunPat / 32];
#pragma unroll
        for (int j = 0; j < kRunPat / 32; j++)
          y[j] = t0 + 32 * j < a.len ? walk(u, t0 + 32 * j) : -1;
#pragma unroll
        for (int j = 0; j < kRunPat / 32; j++)
          if (y[j] >= 0) atomicSub(&c.map[y[j]], 1);
      }
    }
    if (!grid_barrier(run, ++bar)) return;
  }
}

int launch_greedy_run(const BatchGreedyCell &cell, int par, int steps,
                      int32_t exclude, GreedyRun *run, cudaStream_t s) {
  const int kind = walk_kind(cell.w);
  const void *fn = kind == kGridWalk ? (const void *)k_greedy_run<kGridWalk>
                   : kind == kPack ? (const void *)k_greedy_run<kPack>
                                   : (const void *)k_greedy_run<kSlots>;
  // the packed table in shared memory where it is short
  int table = kind == kPack && cell.w.len <= kRunTable ? (int)cell.w.len : 0;
  // one block an SM: two or four measured slower (their barriers cost more
  // than their warps give: 11 us a step against 14 and 18 near a cover)
  const int grid = sm_count();
  BatchGreedyCell c = cell;
  // the barriers count from zero; err carries over
  CC_CK(cudaMemsetAsync(&run->arrived, 0, sizeof(unsigned), s));
  void *args[] = {&c, &table, &par, &steps, &exclude, &run};
  CC_CK(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kRunThreads), args,
                                    (size_t)table * 4, s));
  return 0;
}

int launch_greedy_refresh(const BatchGreedyCell *dcells, int ncells,
                          int blocks, const int *rebuild, cudaStream_t s) {
  k_greedy_refresh<<<dim3((unsigned)blocks, (unsigned)ncells), 256, 0, s>>>(
      dcells, rebuild);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_greedy_argmax(const BatchGreedyCell *dcells, const int2 *jobs,
                         int njobs, int par, int all, cudaStream_t s) {
  k_greedy_argmax<<<(unsigned)njobs, 32 * kArgmaxWarps, 0, s>>>(
      dcells, jobs, par, all);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_greedy_place(const BatchGreedyCell *dcells, const int2 *jobs,
                        int njobs, int par, int32_t exclude, cudaStream_t s) {
  k_greedy_place<<<(unsigned)njobs, 256, 0, s>>>(dcells, jobs, par, exclude);
  CC_CK(cudaGetLastError());
  return 0;
}

bool greedy_rebuild_pays(long long gain, long long ball, double rebuild_us) {
  const char *e = getenv("CC_GREEDY_REBUILD");
  if (e) return atoi(e) != 0;
  return (double)gain * (double)ball > kGreedyUpdatesPerUs * rebuild_us;
}

int launch_greedy_exclude(const BatchGreedyCell *dcells, int ncells,
                          const int *rebuild, int32_t exclude,
                          cudaStream_t s) {
  k_greedy_exclude<<<dim3(8, (unsigned)ncells), 256, 0, s>>>(dcells, rebuild,
                                                             exclude);
  CC_CK(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------ tiled gather
// Many candidates over a large ball: the per-word kernel above re-reads the
// whole support table for every candidate (|B| x slots x 4 bytes, 546 KB a
// candidate at ternary n=16, R=4), so a call with 10^5 candidates streams
// tens of GB of table through L2.  Here a block takes a tile of kTilePat
// patterns and a group of kTileCand candidates:
//   * the tile is decoded once into 16-bit offset indices, four to a 64-bit
//     shared word (a missing slot points at a zero entry, so every pattern
//     takes the same adds, branch-free);
//   * each candidate's index offsets per (position, shift) sit in shared
//     memory (32-bit: cells below 2^31 words);
//   * each warp walks the whole tile for one candidate at a time, 32
//     consecutive patterns a step and eight steps in flight, so one
//     candidate's loads stay close together in time and in address (the
//     table is sorted by offset) and reuse L1 like a per-word sweep.
// The table is read once per candidate group instead of once per candidate.
constexpr int kTilePat = 512;           // patterns per block
constexpr int kTileCand = 32;           // candidates per block
constexpr int kTileMaxOff = 128;        // offset entries per candidate

// The predicate of one gather call as a bit plane: bit x of bits is
// pred(cnt[x]).  Eight counters (one 16-byte load) per thread and byte.
__global__ void __launch_bounds__(256)
k_pred_bits(const uint16_t *cnt, long long n, int mode, int target, int mu,
            uint8_t *bits) {
  const long long nbytes = (n + 7) / 8;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
       i < nbytes; i += stride) {
    unsigned m = 0;
    if (8 * i + 8 <= n) {
      const uint4 v = __ldcs(reinterpret_cast<const uint4 *>(cnt) + i);
      const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        m |= (unsigned)cnt_pred(mode, (int)(w[k] & 0xFFFFu), target, mu)
             << (2 * k);
        m |= (unsigned)cnt_pred(mode, (int)(w[k] >> 16), target, mu)
             << (2 * k + 1);
      }
    } else {
      for (long long x = 8 * i; x < n; x++)
        m |= (unsigned)cnt_pred(mode, (int)cnt[x], target, mu)
             << (int)(x - 8 * i);
    }
    bits[i] = (uint8_t)m;
  }
}

template <int MAXS, bool BITS>
__global__ void __launch_bounds__(256, 6)
k_gather_tiled(const WalkArgs a, const long long *words, int nb, int mode,
               int target, int32_t *out, int noff, int group,
               const uint8_t *bits) {
  // MAXS 4: the packed table's own 8-bit indices, 32 bits a pattern; 8:
  // 16-bit indices, two 64-bit words
  constexpr int NQ = MAXS / 4;
  __shared__ int32_t off[kTileCand * kTileMaxOff];
  __shared__ unsigned long long idx[MAXS == 4 ? kTilePat / 2 : kTilePat * NQ];
  __shared__ int32_t base[kMaxAxes];
  __shared__ int32_t cand[kTileCand];
  uint32_t *idx4 = reinterpret_cast<uint32_t *>(idx);
  const int c0 = blockIdx.y * group;
  const int nc = min(group, nb - c0);
  const long long t0 = (long long)blockIdx.x * kTilePat;
  const int np = (int)min((long long)kTilePat, a.len - t0);
  if (MAXS != 4 && threadIdx.x == 0) {
    int b = 0;
    for (int j = 0; j < a.g.n; j++) { base[j] = b; b += a.g.ax[j] - 1; }
  }
  if (threadIdx.x < kTileCand)
    cand[threadIdx.x] = threadIdx.x < nc ? (int32_t)words[c0 + threadIdx.x]
                                         : 0;
  __syncthreads();
  // index offsets of every (position, shift) around each candidate; entry
  // noff is the zero a missing slot adds
  for (int i = threadIdx.x; i < nc * (noff + 1); i += blockDim.x) {
    const int c = i / (noff + 1), e = i % (noff + 1);
    int v = 0;
    if (e < noff) {
      int q, dl, pw;
      if (MAXS == 4) {
        const int4 en = __ldg(a.ent + e);
        pw = en.x; q = en.y; dl = en.z;
      } else {
        int j = 0;
        while (j + 1 < a.g.n && base[j + 1] <= e) j++;
        q = a.g.ax[j]; dl = e - base[j] + 1;
        pw = (int)a.g.pw[j];
      }
      const int dg = (cand[c] / pw) % q;
      const int nd = dg + dl >= q ? dg + dl - q : dg + dl;
      v = (nd - dg) * pw;
    }
    off[c * kTileMaxOff + e] = v;
  }
  // the tile's patterns as offset indices
  for (int p = threadIdx.x; p < np; p += blockDim.x) {
    if (MAXS == 4) {
      idx4[p] = __ldg(a.pk + t0 + p);
      continue;
    }
#pragma unroll
    for (int h = 0; h < NQ; h++) {
      unsigned long long wv = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int s = 4 * h + k;
        int code = 0;
        if (s < a.slots) code = a.tbl[(long long)s * a.len + t0 + p];
        const unsigned e = code ? (unsigned)(base[code >> 24] +
                                             (code & 0xFFFFFF) - 1)
                                : (unsigned)noff;
        wv |= (unsigned long long)e << (16 * k);
      }
      idx[p * NQ + h] = wv;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  for (int c = warp; c < nc; c += nwarps) {
    const int32_t *oc = off + c * kTileMaxOff;
    const int32_t w = cand[c];
    int hits = 0;
#pragma unroll 8
    for (int p = lane; p < np; p += 32) {
      int32_t x = w;
      if (MAXS == 4) {
        const uint32_t v = idx4[p];
        x += oc[v & 255u] + oc[(v >> 8) & 255u] + oc[(v >> 16) & 255u] +
             oc[v >> 24];
      } else {
#pragma unroll
        for (int h = 0; h < NQ; h++) {
          const unsigned long long wv = idx[p * NQ + h];
          x += oc[wv & 0xFFFF] + oc[(wv >> 16) & 0xFFFF] +
               oc[(wv >> 32) & 0xFFFF] + oc[wv >> 48];
        }
      }
      if (BITS)
        hits += (__ldg(bits + (x >> 3)) >> (x & 7)) & 1;
      else
        hits += cnt_pred(mode, (int)__ldg(a.cnt + x), target, a.g.mu);
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    if (lane == 0 && hits) atomicAdd(&out[c0 + c], hits);
  }
}

// the tiled gather applies: Hamming / Lee / torus cells below 2^31 words,
// offsets table within bounds, at most 8 slots, enough candidates to share
// a table tile (CC_GATHER_TILED=0 turns it off, =1 forces it on)
bool gather_tiled_ok(const WalkArgs &w, int nb, int *noff) {
  if (w.g.prob == kGrid || w.g.space >= (1LL << 31) || w.slots > 8 ||
      w.len >= (1LL << 31))
    return false;
  int n = 0;
  for (int j = 0; j < w.g.n; j++) n += w.g.ax[j] - 1;
  if (n >= kTileMaxOff) return false;          // entry n is the zero
  *noff = n;
  if ((long long)nb > 65535LL * kTileCand) return false;   // grid y
  const char *e = getenv("CC_GATHER_TILED");
  if (e) return atoi(e) != 0;
  return nb >= 16 && w.len >= 2048;
}

// A bit plane pays when the call reads more ball words than the plane
// costs to build (one pass over cnt): candidates x |B| >= |X|.
// CC_GATHER_BITS=0 turns it off, =1 forces it on.
bool gather_bits_pay(const WalkArgs &w, int nb) {
  int noff = 0;
  if (!gather_tiled_ok(w, nb, &noff)) return false;
  const char *e = getenv("CC_GATHER_BITS");
  if (e) return atoi(e) != 0;
  return (double)nb * (double)w.len >= (double)w.g.space;
}

// blocks per word so that single-word walks still fill the GPU
int pick_split(long long len, int nb) {
  long long cover = (len + 255) / 256;
  long long split = (long long)sm_count() * 64 / (nb > 0 ? nb : 1);
  if (split < 1) split = 1;
  if (split > cover) split = cover;
  if (split > 65535) split = 65535;
  return (int)split;
}

int launch_update(const WalkArgs &w, const long long *dwords,
                  const WordsParam *pw, int nb, int delta,
                  unsigned long long *trans, cudaStream_t s) {
  if (nb <= 0) return 0;
  const int split = pick_split(w.len, nb);
  const dim3 grid((unsigned)nb * split);
  static WordsParam empty;
#define CC_UP(W)                                                            \
  case W:                                                                   \
    if (dwords)                                                             \
      k_update<W, false><<<grid, 256, 0, s>>>(w, dwords, empty, split,      \
                                              delta, trans);                \
    else                                                                    \
      k_update<W, true><<<grid, 256, 0, s>>>(w, nullptr, *pw, split, delta, \
                                             trans);                        \
    break;
  switch (walk_kind(w)) { CC_UP(kSlots) CC_UP(kGridWalk) CC_UP(kPack) }
#undef CC_UP
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_gather(const WalkArgs &w, const long long *dwords, int nb,
                  int mode, int target, int32_t *out, bool zeroed,
                  cudaStream_t s, uint8_t *bits) {
  if (nb <= 0) return 0;
  int noff = 0;
  if (gather_tiled_ok(w, nb, &noff)) {
    if (!zeroed) CC_CK(cudaMemsetAsync(out, 0, (size_t)nb * 4, s));
    if (bits) {
      const long long nbytes = (w.g.space + 7) / 8;
      long long nbk = (nbytes + 255) / 256;
      if (nbk > (long long)sm_count() * 32) nbk = (long long)sm_count() * 32;
      k_pred_bits<<<(unsigned)nbk, 256, 0, s>>>(w.cnt, w.g.space, mode,
                                                target, w.g.mu, bits);
      CC_CK(cudaGetLastError());
    }
    // candidates a block shares its table tile with: 32, or a warp each when
    // that leaves too few blocks (64 candidates x 34,113 patterns: 134 blocks
    // of 32 candidates, 536 of 8)
    const long long tiles = (w.len + kTilePat - 1) / kTilePat;
    const int group = tiles * ((nb + kTileCand - 1) / kTileCand) <
                              (long long)sm_count() * 4 ? 8 : kTileCand;
    const dim3 tg((unsigned)tiles, (unsigned)((nb + group - 1) / group));
#define TG(M, B) k_gather_tiled<M, B><<<tg, 256, 0, s>>>(                  \
        w, dwords, nb, mode, target, out, noff, group, bits)
    if (w.pk) { if (bits) TG(4, true); else TG(4, false); }
    else { if (bits) TG(8, true); else TG(8, false); }
#undef TG
    CC_CK(cudaGetLastError());
    return 0;
  }
  const int split = pick_split(w.len, nb);
  if (split > 1 && !zeroed)
    CC_CK(cudaMemsetAsync(out, 0, (size_t)nb * 4, s));
  const dim3 grid((unsigned)nb * split);
#define CC_GA(W)                                                            \
  case W:                                                                   \
    k_gather<W><<<grid, 256, 0, s>>>(w, dwords, split, mode, target, out);  \
    break;
  switch (walk_kind(w)) { CC_GA(kSlots) CC_GA(kGridWalk) CC_GA(kPack) }
#undef CC_GA
  CC_CK(cudaGetLastError());
  return 0;
}

}  // namespace cc
