// group_rounds.cuh — the rounds of the register-blocked group transforms:
// the per-axis recurrences, one round over a tile, and a whole tile.  Shared
// by the one-launch-per-group kernels (transform_group.cu) and the batched
// engine's persistent kernels (batch_groups.cu).
#pragma once
#include "engine.h"

namespace cc {

template <int Q, int B>
struct IPow { static constexpr int v = Q * IPow<Q, B - 1>::v; };
template <int Q>
struct IPow<Q, 0> { static constexpr int v = 1; };

enum Op { kOpHamming = 0, kOpLee = 1, kOpTorus = 2, kOpGrid = 3 };

// ---------------------------------------------------------------- axis ops
// Hamming: newA_d[a] = A_d[a] + T_{d-1} - A_{d-1}[a], T = fibre sum.
// T_{d-1} - A_{d-1}[a] is the sum of the fibre's OTHER entries of layer
// d-1, which is how it is formed here: one add per entry for Q = 2, two for
// Q = 3, and T minus the entry above.  Descending d reads layer d-1 before
// it is rewritten, so every term is the old value, as in the recurrence.
template <int Q, int R1, int QB, int ST>
__device__ __forceinline__ void axis_hamming(int32_t (&v)[R1][QB]) {
#pragma unroll
  for (int e = 0; e < QB; e++) {
    if ((e / ST) % Q != 0) continue;
#pragma unroll
    for (int d = R1 - 1; d >= 1; d--) {
      if (Q == 2) {
        const int32_t a0 = v[d - 1][e], a1 = v[d - 1][e + ST];
        v[d][e] += a1;
        v[d][e + ST] += a0;
      } else if (Q == 3) {
        const int32_t a0 = v[d - 1][e], a1 = v[d - 1][e + ST],
                      a2 = v[d - 1][e + 2 * ST];
        v[d][e] += a1 + a2;
        v[d][e + ST] += a0 + a2;
        v[d][e + 2 * ST] += a0 + a1;
      } else {
        int32_t T = 0;
#pragma unroll
        for (int a = 0; a < Q; a++) T += v[d - 1][e + a * ST];
#pragma unroll
        for (int a = 0; a < Q; a++)
          v[d][e + a * ST] += T - v[d - 1][e + a * ST];
      }
    }
  }
}

// Lee: newA_d[a] = A_d[a] + sum_{w=1..min(d,Q/2)} (A_{d-w}[a-w] + A_{d-w}[a+w]),
// the two terms counted once when they coincide (even Q, w = Q/2)
template <int Q, int R1, int QB, int ST>
__device__ __forceinline__ void axis_lee(int32_t (&v)[R1][QB]) {
  constexpr int H = Q / 2;
#pragma unroll
  for (int e = 0; e < QB; e++) {
    if ((e / ST) % Q != 0) continue;
#pragma unroll
    for (int d = R1 - 1; d >= 1; d--) {
#pragma unroll
      for (int a = 0; a < Q; a++) {
        int32_t s = 0;
#pragma unroll
        for (int w = 1; w <= (d < H ? d : H); w++) {
          const int am = (a - w + Q) % Q, ap = (a + w) % Q;
          s += v[d - w][e + am * ST];
          if (ap != am) s += v[d - w][e + ap * ST];
        }
        v[d][e + a * ST] += s;       // only lower layers are read
      }
    }
  }
}

// torus / grid: newA[a] = sum over the circular (torus) or clamped (grid)
// window of radius R
template <int Q, int R1, int QB, int ST, bool GRID>
__device__ __forceinline__ void axis_window(int32_t (&v)[R1][QB], int R) {
#pragma unroll
  for (int e = 0; e < QB; e++) {
    if ((e / ST) % Q != 0) continue;
    int32_t nv[Q];
#pragma unroll
    for (int a = 0; a < Q; a++) {
      int32_t s = 0;
#pragma unroll
      for (int b = 0; b < Q; b++) {
        int dd = a > b ? a - b : b - a;
        if (!GRID && Q - dd < dd) dd = Q - dd;
        if (dd <= R) s += v[0][e + b * ST];
      }
      nv[a] = s;
    }
#pragma unroll
    for (int a = 0; a < Q; a++) v[0][e + a * ST] = nv[a];
  }
}

template <int OP, int Q, int R1, int QB, int ST>
__device__ __forceinline__ void apply_axis(int32_t (&v)[R1][QB], int R) {
  if (OP == kOpHamming) axis_hamming<Q, R1, QB, ST>(v);
  else if (OP == kOpLee) axis_lee<Q, R1, QB, ST>(v);
  else axis_window<Q, R1, QB, ST, OP == kOpGrid>(v, R);
}

template <int OP, int Q, int R1, int BM, int T>
struct AxisLoop {
  static __device__ __forceinline__ void run(
      int32_t (&v)[R1][IPow<Q, BM>::v], int rb, int R) {
    if (T < rb) apply_axis<OP, Q, R1, IPow<Q, BM>::v, IPow<Q, T>::v>(v, R);
    AxisLoop<OP, Q, R1, BM, T + 1>::run(v, rb, R);
  }
};
template <int OP, int Q, int R1, int BM>
struct AxisLoop<OP, Q, R1, BM, BM> {
  static __device__ __forceinline__ void run(
      int32_t (&)[R1][IPow<Q, BM>::v], int, int) {}
};

__device__ __forceinline__ int skewed(int p, int skew) {
  return skew ? p + (p >> skew) : p;
}

// Fill layer 0 of tile `tile` (shared memory) with the code multiplicities
// of its contiguous range [x0, x0 + len); other layers are implicit zeros.
// The tile's slice of the sorted code is code[bounds[tile], bounds[tile+1])
// (k_code_bounds, one binary search per tile boundary).
__device__ __forceinline__ void stage_code(const GroupArgs &g, int32_t *sm,
                                           long long tile, long long x0,
                                           int len) {
  for (int p = threadIdx.x; p < len; p += blockDim.x)
    sm[skewed(p, g.skew)] = 0;
  __syncthreads();
  const long long lo = g.code_bounds[tile], hi = g.code_bounds[tile + 1];
  for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x)
    atomicAdd(&sm[skewed((int)(g.code[t] - x0), g.skew)], 1);
  __syncthreads();
}

// The same for a first group whose words sit in pairs (inner == 2): word p
// of the range adds 1 to the half (p & 1) of packed lane p / 2.  Counts stay
// below 2^16 (the occurrence bound), so no add carries across halves.
__device__ __forceinline__ void stage_code_pairs(const GroupArgs &g,
                                                 int32_t *sm, long long tile,
                                                 long long x0, int len) {
  for (int P = threadIdx.x; P < (len + 1) / 2; P += blockDim.x)
    sm[skewed(P, g.skew)] = 0;
  __syncthreads();
  const long long lo = g.code_bounds[tile], hi = g.code_bounds[tile + 1];
  for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) {
    const int p = (int)(g.code[t] - x0);
    atomicAdd(&sm[skewed(p >> 1, g.skew)], 1 << (16 * (p & 1)));
  }
  __syncthreads();
}

// ------------------------------------------------------------------ kernel
// Where a round's block comes from and goes to: the first round reads HBM
// (layers, the cnt predicate) or the staged code, the last writes HBM
// (layers, map, cnt); every other side is shared memory.
enum RoundIo { kIoSmem = 0, kIoLayers = 1, kIoCnt = 2, kIoCode = 3,
               kIoMap = 4, kIoCntOut = 5, kIoCntSmem = 6 };

// One round over the whole tile: every thread takes register blocks of
// ne = Q^rb words (all layers), rb of the group's axes at local stride S.
// FULL: rb == BM (no per-word bound checks).  Addresses step linearly with
// the block word e: in HBM by S*inner words, in shared memory by sstep —
// the skew (one pad word per 2^skew) keeps that linear, because a round's
// stride S is 1 or a multiple of 2^skew and S == 1 blocks start on a
// multiple of 2^skew.
//
// PACK: every register, shared-memory word and lane carries TWO inner words
// (w, w+1) as 16-bit halves of one 32-bit value, so each add and each
// shared-memory access serves both.  Exact while every value stays below
// 2^16 (the planner's 16-bit bound) and the inner stride is even, so a pair
// never straddles a row; the group's HBM sides are u16 planes (one 32-bit
// access per pair), the int32 map and the u16 cnt (unpacked at the store).
//
// CG: global reads through L2 only (the batched engine, where other SMs of
// the same launch wrote them); otherwise streaming reads.
// Epilogue reductions of a launch's output (GroupArgs::red_mode): 2 the
// maximum of the map written (0 when no value is positive), 1 the deficit
// sum max(0, mu - c) of the cnt written.  Per thread, then per warp, one
// 64-bit atomic.
__device__ __forceinline__ void red_map(long long *acc, long long a,
                                        long long b) {
  const long long m = a > b ? a : b;
  if (m > *acc) *acc = m;
}
__device__ __forceinline__ void red_def(long long *acc, int mu, int c0,
                                        int c1) {
  *acc += (c0 < mu ? mu - c0 : 0) + (c1 < mu ? mu - c1 : 0);
}
__device__ __forceinline__ void red_flush(const GroupArgs &g, long long acc) {
  for (int o = 16; o > 0; o >>= 1) {
    const long long other = __shfl_down_sync(0xffffffffu, acc, o);
    acc = g.red_mode == 2 ? (other > acc ? other : acc) : acc + other;
  }
  if ((threadIdx.x & 31) == 0 && acc) {
    if (g.red_mode == 2)
      atomicMax((unsigned long long *)g.red, (unsigned long long)acc);
    else
      atomicAdd((unsigned long long *)g.red, (unsigned long long)acc);
  }
}

template <bool CG, typename T>
__device__ __forceinline__ T ld_stream(const T *p) {
  return CG ? __ldcg(p) : __ldcs(p);
}

template <int OP, int Q, int R1, int BM, bool FULL, bool PACK = false,
          bool CG = false>
__device__ __forceinline__ void run_round(const GroupArgs &g, int32_t *sm,
                                          int SD, long long o0, long long i0,
                                          int rb, int S, int src, int dst,
                                          int nl = R1,
                                          const uint16_t *cs = nullptr,
                                          long long *racc = nullptr) {
  constexpr int QB = IPow<Q, BM>::v;
  int ne = QB;
  if (!FULL) { ne = 1; for (int t = 0; t < rb; t++) ne *= Q; }
  const int W = PACK ? g.W >> 1 : g.W;         // lanes (pairs) per row
  const int nh = g.mid / (S * ne);
  const int nblk = W * S * nh * g.Bo;
  const long long imid = g.inner * (long long)g.mid;
  const long long gstep = (long long)S * g.inner;      // HBM word step of e
  const int sstep = g.skew == 0 ? S * W
                    : (S == 1 ? W : (S + (S >> g.skew)) * W);
  // predicate as a range: lo <= cnt <= hi
  const int plo = g.pmode == kPredDef ? 0 : g.pmode == kPredCrit ? 1
                  : g.ptarget;
  const int phi = g.pmode == kPredDef ? g.mu - 1 : g.pmode == kPredCrit
                  ? g.mu : g.ptarget;
  const unsigned pspan = (unsigned)(phi - plo);
  // blk = ((ob * nh + mhi) * S + mlo) * W + w, kept as mixed-radix digits
  // that advance by blockDim.x per trip (one compare per digit, no
  // division in the loop); every digit sum stays below twice its radix
  int w, mlo, mhi, ob, dw, dmlo, dmhi, dob;
  {
    int r = threadIdx.x;
    w = r % W; r /= W; mlo = r % S; r /= S; mhi = r % nh; ob = r / nh;
    r = blockDim.x;
    dw = r % W; r /= W; dmlo = r % S; r /= S; dmhi = r % nh; dob = r / nh;
  }
  for (int blk = threadIdx.x; blk < nblk; blk += blockDim.x) {
    const int wi = PACK ? 2 * w : w;                     // inner word
    const bool valid = (o0 + ob < g.outer) && (i0 + wi < g.inner);
    const int pb = ob * g.mid + mlo + S * ne * mhi;      // tile word, e = 0
    const int sp0 = skewed(pb, g.skew) * W + w;
    const long long xb = (o0 + ob) * imid + (long long)(mlo + S * ne * mhi)
                         * g.inner + i0 + wi;
    int32_t v[R1][QB];
#pragma unroll
    for (int d = 0; d < R1; d++)
#pragma unroll
      for (int e = 0; e < QB; e++) v[d][e] = 0;
    // -------- load
    if (src == kIoCntSmem) {                     // prefetched cnt window
      const uint16_t *p = cs + pb;
#pragma unroll
      for (int e = 0; e < QB; e++) {
        if (!FULL && e >= ne) break;
        v[0][e] = (unsigned)((int)p[e * S] - plo) <= pspan;
      }
    } else if (src == kIoSmem || src == kIoCode) {
      if (src == kIoCode) nl = 1;
#pragma unroll
      for (int d = 0; d < R1; d++) {
        if (d >= nl) break;
        const int32_t *p = sm + d * SD + sp0;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          v[d][e] = p[e * sstep];
        }
      }
    } else if (valid) {
      if (PACK && src == kIoLayers) {            // one u32 per word pair
#pragma unroll
        for (int d = 0; d < R1; d++) {
          if (d >= g.lin) break;
          const uint16_t *p = g.layers16 + d * g.plane + xb;
#pragma unroll
          for (int e = 0; e < QB; e++) {
            if (!FULL && e >= ne) break;
            v[d][e] = (int32_t)ld_stream<CG>(reinterpret_cast<const uint32_t *>(p));
            p += gstep;
          }
        }
      } else if (src == kIoLayers && g.in16) {
#pragma unroll
        for (int d = 0; d < R1; d++) {
          if (d >= g.lin) break;
          const uint16_t *p = g.layers16 + d * g.plane + xb;
#pragma unroll
          for (int e = 0; e < QB; e++) {
            if (!FULL && e >= ne) break;
            v[d][e] = ld_stream<CG>(p);
            p += gstep;
          }
        }
      } else if (src == kIoLayers) {
#pragma unroll
        for (int d = 0; d < R1; d++) {
          if (d >= g.lin) break;
          const int32_t *p = g.layers + d * g.plane + xb;
#pragma unroll
          for (int e = 0; e < QB; e++) {
            if (!FULL && e >= ne) break;
            v[d][e] = ld_stream<CG>(p);
            p += gstep;
          }
        }
      } else if (PACK) {                         // kIoCnt, a word pair
        const uint16_t *p = g.cnt + xb;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          const uint32_t c = ld_stream<CG>(reinterpret_cast<const uint32_t *>(p));
          const uint32_t lo = (unsigned)((int)(c & 0xFFFFu) - plo) <= pspan;
          const uint32_t hi = (unsigned)((int)(c >> 16) - plo) <= pspan;
          v[0][e] = (int32_t)(lo | (hi << 16));
          p += gstep;
        }
      } else {                                   // kIoCnt
        const uint16_t *p = g.cnt + xb;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          v[0][e] = (unsigned)((int)ld_stream<CG>(p) - plo) <= pspan;
          p += gstep;
        }
      }
    }
    // -------- axis 0 inside each pair (binary Hamming first group), once:
    // in the round that reads the code or cnt.  newA_d[a] = A_d[a] +
    // A_{d-1}[a ^ 1] is an add of the halves swapped, layers descending.
    if (PACK && OP == kOpHamming && Q == 2 && g.pair_axis &&
        (src == kIoCnt || src == kIoCode)) {
#pragma unroll
      for (int e = 0; e < QB; e++)
#pragma unroll
        for (int d = R1 - 1; d >= 1; d--)
          v[d][e] += (int32_t)__funnelshift_l((uint32_t)v[d - 1][e],
                                              (uint32_t)v[d - 1][e], 16);
    }
    // -------- rb axis recurrences in registers
    if (FULL) AxisLoop<OP, Q, R1, BM, 0>::run(v, BM, g.R);
    else AxisLoop<OP, Q, R1, BM, 0>::run(v, rb, g.R);
    // -------- store
    if (dst == kIoSmem) {
#pragma unroll
      for (int d = 0; d < R1; d++) {
        int32_t *p = sm + d * SD + sp0;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          p[e * sstep] = v[d][e];
        }
      }
    } else if (valid) {
      if (PACK && dst == kIoLayers) {            // one u32 per word pair
#pragma unroll
        for (int d = 0; d < R1; d++) {
          if (d >= g.lout) break;
          uint16_t *p = g.layers16 + d * g.plane + xb;
#pragma unroll
          for (int e = 0; e < QB; e++) {
            if (!FULL && e >= ne) break;
            __stcs(reinterpret_cast<uint32_t *>(p), (uint32_t)v[d][e]);
            p += gstep;
          }
        }
      } else if (PACK && dst == kIoMap) {        // both halves, widened
        int32_t *p = (g.map ? g.map : g.layers) + xb;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          uint32_t s = 0;
#pragma unroll
          for (int d = 0; d < R1; d++) s += (uint32_t)v[d][e];
          __stcs(reinterpret_cast<int2 *>(p),
                 make_int2((int)(s & 0xFFFFu), (int)(s >> 16)));
          if (racc) red_map(racc, (long long)(s & 0xFFFFu), (long long)(s >> 16));
          p += gstep;
        }
      } else if (PACK) {                         // cnt: both halves at once
        uint16_t *p = g.cnt + xb;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          uint32_t s = 0;
#pragma unroll
          for (int d = 0; d < R1; d++) s += (uint32_t)v[d][e];
          *reinterpret_cast<uint32_t *>(p) = s;
          if (racc) red_def(racc, g.mu, (int)(s & 0xFFFFu), (int)(s >> 16));
          p += gstep;
        }
      } else if (dst == kIoLayers && g.out16) {
        // a first group (inner 1) of a padded plan: the slab's row starts
        // at a pitch of g.pitch words
        const long long xo = g.pitch
            ? (o0 + ob) * g.pitch + (long long)(mlo + S * ne * mhi) *
                  g.inner + i0 + wi
            : xb;
#pragma unroll
        for (int d = 0; d < R1; d++) {
          if (d >= g.lout) break;
          uint16_t *p = g.layers16 + d * g.plane + xo;
#pragma unroll
          for (int e = 0; e < QB; e++) {
            if (!FULL && e >= ne) break;
            __stcs(p, (uint16_t)v[d][e]);
            p += gstep;
          }
        }
      } else if (dst == kIoLayers) {
#pragma unroll
        for (int d = 0; d < R1; d++) {
          if (d >= g.lout) break;
          int32_t *p = g.layers + d * g.plane + xb;
#pragma unroll
          for (int e = 0; e < QB; e++) {
            if (!FULL && e >= ne) break;
            __stcs(p, v[d][e]);
            p += gstep;
          }
        }
      } else if (dst == kIoMap) {
        int32_t *p = (g.map ? g.map : g.layers) + xb;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          int32_t s = 0;
#pragma unroll
          for (int d = 0; d < R1; d++) s += v[d][e];
          __stcs(p, s);
          if (racc) red_map(racc, (long long)s, 0);
          p += gstep;
        }
      } else {
        uint16_t *p = g.cnt + xb;
#pragma unroll
        for (int e = 0; e < QB; e++) {
          if (!FULL && e >= ne) break;
          int32_t s = 0;
#pragma unroll
          for (int d = 0; d < R1; d++) s += v[d][e];
          *p = (uint16_t)(s > 65535 ? 65535 : s);
          if (racc) red_def(racc, g.mu, s > 65535 ? 65535 : s, g.mu);
          p += gstep;
        }
      }
    }
    // advance the digits by blockDim.x
    w += dw;
    int c = w >= W;
    if (c) w -= W;
    mlo += dmlo + c;
    c = mlo >= S;
    if (c) mlo -= S;
    mhi += dmhi + c;
    c = mhi >= nh;
    if (c) mhi -= nh;
    ob += dob + c;
  }
}

// A round of rb axes runs with a register block of exactly Q^rb words: the
// kernel's own block size BM for full rounds, a compile-time smaller block
// for the group's last, partial round (no runtime bounds in the loops).
template <int OP, int Q, int R1, int B, bool PACK = false, bool CG = false>
struct RoundSel {
  static __device__ __forceinline__ void run(
      const GroupArgs &g, int32_t *sm, int SD, long long o0, long long i0,
      int rb, int S, int src, int dst, int nl, const uint16_t *cs,
      long long *racc = nullptr) {
    if (rb == B)
      run_round<OP, Q, R1, B, true, PACK, CG>(g, sm, SD, o0, i0, B, S, src,
                                              dst, nl, cs, racc);
    else
      RoundSel<OP, Q, R1, B - 1, PACK, CG>::run(g, sm, SD, o0, i0, rb, S,
                                                src, dst, nl, cs, racc);
  }
};
template <int OP, int Q, int R1, bool PACK, bool CG>
struct RoundSel<OP, Q, R1, 0, PACK, CG> {
  static __device__ __forceinline__ void run(
      const GroupArgs &, int32_t *, int, long long, long long, int, int, int,
      int, int, const uint16_t *, long long * = nullptr) {}
};
// Register kernels of packed word pairs: adds only, so no value carries
// across the halves (Hamming q <= 3, Lee).
template <int OP, int Q>
__host__ __device__ constexpr bool packable() {
  return (OP == kOpHamming && Q <= 3) || OP == kOpLee;
}

// All rounds of one tile of a group; ends with a barrier.  racc: the
// thread's running epilogue reduction, or nullptr.
template <int OP, int Q, int R1, int BM, bool CG>
__device__ __forceinline__ void group_tile(const GroupArgs &g, int32_t *sm,
                                           long long tile, long long *racc) {
  constexpr bool kPk = packable<OP, Q>();
  const int W = g.W;
  const int tile_words = g.Bo * g.mid;
  const bool pk = kPk && g.pack;
  const int SW = pk ? W >> 1 : W;                        // lanes per row
  const int SD = (skewed(tile_words, g.skew) + 1) * SW;  // layer stride
  const int first_src = g.src == kSrcLayers ? kIoLayers
                        : g.src == kSrcCnt ? kIoCnt : kIoCode;
  const int last_dst = g.dst == kDstLayers ? kIoLayers
                       : g.dst == kDstMap ? kIoMap : kIoCntOut;
  const long long o0 = (tile / g.nchunk) * g.Bo;
  const long long i0 = (tile % g.nchunk) * W;
  if (g.src == kSrcCode && pk) {
    // first group, axis 0 in pairs: inner == 2, the tile is contiguous
    const long long imid = g.inner * (long long)g.mid;
    const long long len = (g.outer - o0) * imid;
    const long long tw = (long long)tile_words * g.inner;
    stage_code_pairs(g, sm, tile, o0 * imid, (int)(len < tw ? len : tw));
  } else if (g.src == kSrcCode) {
    // first group only: W == 1, inner == 1, the tile is contiguous
    long long len = (g.outer - o0) * (long long)g.mid;
    stage_code(g, sm, tile, o0 * g.mid,
               (int)(len < tile_words ? len : tile_words));
  }
  for (int r = 0; r < g.nrounds; r++) {
    const int src = r == 0 ? first_src : kIoSmem;
    const int dst = r == g.nrounds - 1 ? last_dst : kIoSmem;
    if (pk)
      RoundSel<OP, Q, R1, BM, kPk, CG>::run(g, sm, SD, o0, i0, g.rb[r],
                                            g.rs[r], src, dst, R1, nullptr,
                                            racc);
    else
      RoundSel<OP, Q, R1, BM, false, CG>::run(g, sm, SD, o0, i0, g.rb[r],
                                              g.rs[r], src, dst, R1, nullptr,
                                              racc);
    __syncthreads();
  }
}

// the register-blocked kernels: axis operation, axis size, layers, axes of
// one register block.  A kernel's index in this list is GroupPlan::kernel.
#define CC_GROUP_KERNELS(KE)                                                \
 /* Hamming, binary: 16-word blocks up to 4 layers, 8-word above */         \
    KE(kOpHamming, 2, 2, 4) KE(kOpHamming, 2, 3, 4) KE(kOpHamming, 2, 4, 4) \
    KE(kOpHamming, 2, 4, 3) /* 8-word blocks: fewer registers per thread */ \
    KE(kOpHamming, 2, 5, 3) KE(kOpHamming, 2, 6, 3) KE(kOpHamming, 2, 7, 3) \
    KE(kOpHamming, 2, 8, 3)                                                 \
 /* Hamming, ternary: 9-word blocks; 3-word blocks for wider CTAs */        \
    KE(kOpHamming, 3, 2, 2) KE(kOpHamming, 3, 3, 2) KE(kOpHamming, 3, 4, 2) \
    KE(kOpHamming, 3, 5, 2) KE(kOpHamming, 3, 6, 2) KE(kOpHamming, 3, 7, 2) \
    KE(kOpHamming, 3, 4, 1) KE(kOpHamming, 3, 5, 1)                         \
 /* Hamming, quaternary */                                                  \
    KE(kOpHamming, 4, 2, 2) KE(kOpHamming, 4, 3, 2) KE(kOpHamming, 4, 4, 2) \
    KE(kOpHamming, 4, 5, 1)                                                 \
 /* Hamming, q = 5, 6: one axis per round (up to 5 layers) */               \
    KE(kOpHamming, 5, 2, 1) KE(kOpHamming, 5, 3, 1) KE(kOpHamming, 5, 4, 1) \
    KE(kOpHamming, 5, 5, 1)                                                 \
    KE(kOpHamming, 6, 2, 1) KE(kOpHamming, 6, 3, 1) KE(kOpHamming, 6, 4, 1) \
    KE(kOpHamming, 6, 5, 1)                                                 \
 /* Lee: one axis per round */                                              \
    KE(kOpLee, 7, 3, 1) KE(kOpLee, 7, 4, 1) KE(kOpLee, 7, 5, 1)             \
    KE(kOpLee, 5, 2, 1) KE(kOpLee, 5, 3, 1) KE(kOpLee, 5, 4, 1)             \
    KE(kOpLee, 5, 5, 1)                                                     \
    KE(kOpLee, 2, 2, 1) KE(kOpLee, 2, 3, 1) KE(kOpLee, 2, 4, 1)             \
    KE(kOpLee, 2, 5, 1)                                                     \
    KE(kOpLee, 3, 2, 1) KE(kOpLee, 3, 3, 1) KE(kOpLee, 3, 4, 1)             \
    KE(kOpLee, 3, 5, 1)                                                     \
    KE(kOpLee, 4, 2, 1) KE(kOpLee, 4, 3, 1) KE(kOpLee, 4, 4, 1)             \
    KE(kOpLee, 4, 5, 1)                                                     \
    KE(kOpLee, 6, 2, 1) KE(kOpLee, 6, 3, 1) KE(kOpLee, 6, 4, 1)             \
    KE(kOpLee, 6, 5, 1)                                                     \
 /* small-axis window sums (torus / grid) */                                \
    KE(kOpTorus, 3, 1, 3) KE(kOpTorus, 4, 1, 2) KE(kOpTorus, 5, 1, 2)      

}  // namespace cc
