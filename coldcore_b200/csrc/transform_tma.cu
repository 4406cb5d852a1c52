// transform_tma.cu — strided axis groups of the distance-layer families,
// streamed through shared memory by the Tensor Memory Accelerator.
//
// The group kernels of transform_group.cu load each tile into registers
// with ordinary loads, so the bytes a CTA keeps in flight are bounded by
// its register blocks: the large launches of H2(26,3) ran latency-bound at
// about half of the HBM bandwidth.  Here a group over 16-bit layer planes
// (two inner words per 32-bit lane) is split into a producer and the
// compute rounds:
//
//   * one thread issues, per tile, ONE tiled bulk tensor load (TMA) of the
//     tile's live layers — W inner words x mid x lin planes — into one of
//     S shared-memory stages, completing on that stage's mbarrier; the
//     loads of the next S-1 tiles are in flight while a tile computes;
//   * the rounds run in place on the stage (register blocks of Q^b words
//     per lane, every shared-memory offset a compile-time constant); the
//     last round writes HBM directly: the u16 layers, the int32 map or the
//     u16 cnt, 32 lanes x 4 bytes (or 8) per warp store;
//   * a stage is refilled once every thread has passed the barrier that
//     ends its last round.
//
// Every wait is bounded: a tile whose bytes have not landed within about
// two seconds (the GPU's global timer) stops the CTA, records a fault that
// the host sees in mapped host memory, and drains its own outstanding
// loads (again bounded) before returning.  No cluster multicast is used;
// the tensor maps cover this GPU's own layer planes only.
//
// Recurrence (coldcore src/plugins/covering/dctcore_hamming.cuh:4-8):
// newA_d[a] = A_d[a] + sum of the fibre's other entries of layer d-1.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <unordered_map>

#include "../../include/coldcore_b200/plugin.h"
#include "engine.h"
#include "rows_first.cuh"
#include "tma_group.cuh"

namespace cc {
namespace {

// ------------------------------------------------------------ first group
// The first group of a binary Hamming cell read from cnt: a tile is the
// contiguous range of 2^(KK+1) words; axis 0 is the word pair inside each
// 32-bit lane (a 16-bit rotate-and-add), axes 1..KK are bits 0..KK-1 of the
// lane index p.  One bulk copy stages the tile's cnt (2 bytes a word) per
// stage; the rounds work on one shared buffer of R1 layers, padded one word
// per 16 lanes (p + p/16), so that 16-lane register blocks are free of bank
// conflicts; the first round (lane bits BM..2BM-1) derives layer 0 from the
// staged cnt, the last round (the highest lane bits) stores to HBM with 32
// consecutive lanes per warp.
__device__ __forceinline__ void bulk_load(void *dst, const void *src,
                                          uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1], %2, [%3];\n" ::"r"(saddr(dst)),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(saddr(bar))
      : "memory");
}

__device__ __forceinline__ int pad16(int p) { return p + (p >> 4); }

// first-group rounds: BM-bit blocks; round order BM.., 0.., 2BM.., 3BM..
template <int KK, int BM, int I>
struct FirstRound {
  static constexpr int A = I == 0 ? BM : I == 1 ? 0 : I * BM;
  static constexpr int B = (KK - A) < BM ? (KK - A) : BM;
  static constexpr int N = (KK + BM - 1) / BM;
};

template <int KK, int R1, int OUT, int I, int SRC = 0>
__device__ __forceinline__ void first_round(uint32_t *work, int WS,
                                            const uint32_t *cnt32,
                                            const TmaArgs &a, long long x0,
                                            uint32_t plo, uint32_t pspan) {
  constexpr int BM = 4;
  using FR = FirstRound<KK, BM, I>;
  constexpr int A = FR::A, B = FR::B;
  constexpr int QB = 1 << B, QA = 1 << A;
  constexpr bool FIRST = I == 0, LAST = I == FR::N - 1;
  constexpr int NB = (1 << KK) / QB;
  for (int blk = threadIdx.x; blk < NB; blk += blockDim.x) {
    const int pb = (blk & (QA - 1)) | ((blk >> A) << (A + B));
    uint32_t v[R1][QB];
    if (FIRST) {
#pragma unroll
      for (int e = 0; e < QB; e++) {
        if (SRC == 0) {                       // the cnt predicate
          const uint32_t c = cnt32[pb + e * QA];
          const uint32_t lo = ((c & 0xFFFFu) - plo) <= pspan;
          const uint32_t hi = ((c >> 16) - plo) <= pspan;
          v[0][e] = lo | (hi << 16);
        } else {                              // code counts, staged
          v[0][e] = work[pad16(pb + e * QA)];
        }
#pragma unroll
        for (int d = 1; d < R1; d++) v[d][e] = 0;
        // axis 0, inside the pair: A_1 gains the other half of A_0
        if (R1 > 1) v[1][e] = __funnelshift_l(v[0][e], v[0][e], 16);
      }
    } else {
#pragma unroll
      for (int d = 0; d < R1; d++)
#pragma unroll
        for (int e = 0; e < QB; e++)
          v[d][e] = work[d * WS + pad16(pb + e * QA)];
    }
    Axes<2, R1, B, 0>::run(v);
    if (!LAST) {
#pragma unroll
      for (int d = 0; d < R1; d++)
#pragma unroll
        for (int e = 0; e < QB; e++)
          work[d * WS + pad16(pb + e * QA)] = v[d][e];
      continue;
    }
    const long long xb = x0 + 2LL * pb;
    if (OUT == 0) {
#pragma unroll
      for (int d = 0; d < R1; d++) {
        if (d >= a.lout) break;
        uint16_t *q = a.layers16 + d * a.plane + xb;
#pragma unroll
        for (int e = 0; e < QB; e++)
          __stcs(reinterpret_cast<unsigned *>(q + 2 * e * QA), v[d][e]);
      }
    } else if (OUT == 5) {
      // 8-bit planes: the low bytes of the pair's two halves (every value
      // below 256 by the planner's bound), one 16-bit store a lane
      uint8_t *q8 = reinterpret_cast<uint8_t *>(a.layers16) + a.off8;
#pragma unroll
      for (int d = 0; d < R1; d++) {
        if (d >= a.lout) break;
        uint8_t *q = q8 + d * a.plane + xb;
#pragma unroll
        for (int e = 0; e < QB; e++)
          __stcs(reinterpret_cast<unsigned short *>(q + 2 * e * QA),
                 (unsigned short)__byte_perm(v[d][e], 0u, 0x4420));
      }
    } else {
#pragma unroll
      for (int e = 0; e < QB; e++) {
        uint32_t s = 0;
#pragma unroll
        for (int d = 0; d < R1; d++) s += v[d][e];
        if (OUT == 1)
          __stcs(reinterpret_cast<int2 *>(a.map + xb + 2 * e * QA),
                 make_int2((int)(s & 0xFFFFu), (int)(s >> 16)));
        else
          *reinterpret_cast<unsigned *>(a.cnt + xb + 2 * e * QA) = s;
      }
    }
  }
}

template <int KK, int R1, int OUT, int I, int N>
struct FirstRounds {
  static __device__ __forceinline__ void run(uint32_t *work, int WS,
                                             const uint32_t *cnt32,
                                             const TmaArgs &a, long long x0,
                                             uint32_t plo, uint32_t pspan,
                                             uint64_t *refill_bar,
                                             const void *refill_src,
                                             void *refill_dst) {
    first_round<KK, R1, OUT, I>(work, WS, cnt32, a, x0, plo, pspan);
    __syncthreads();
    if (I == 0 && threadIdx.x == 0 && refill_src) {
      // the staged cnt has been read: refill its stage now
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      const uint32_t bytes = (uint32_t)((2LL << KK) * 2);
      mbar_expect(refill_bar, bytes);
      bulk_load(refill_dst, refill_src, bytes, refill_bar);
    }
    FirstRounds<KK, R1, OUT, I + 1, N>::run(work, WS, cnt32, a, x0, plo,
                                            pspan, refill_bar, refill_src,
                                            refill_dst);
  }
};
template <int KK, int R1, int OUT, int N>
struct FirstRounds<KK, R1, OUT, N, N> {
  static __device__ __forceinline__ void run(uint32_t *, int,
                                             const uint32_t *,
                                             const TmaArgs &, long long,
                                             uint32_t, uint32_t, uint64_t *,
                                             const void *, void *) {}
};

template <int KK, int R1, int OUT>
__global__ void __launch_bounds__(512)
tma_first(const TmaArgs a) {
  extern __shared__ __align__(128) uint8_t dyn[];
  constexpr int TW = 2 << KK;                 // words per tile
  constexpr int CW = TW / 2;                  // cnt stage, 32-bit words
  constexpr int WS = ((1 << KK) + (1 << KK) / 16 + 31) / 32 * 32;
  constexpr int NR = FirstRound<KK, 4, 0>::N;
  const int S = a.stages;
  uint8_t *base = dyn + ((1024u - (saddr(dyn) & 1023u)) & 1023u);
  uint32_t *cstage = reinterpret_cast<uint32_t *>(base);
  uint32_t *work = cstage + (size_t)S * CW;
  uint64_t *bar = reinterpret_cast<uint64_t *>(work + (size_t)R1 * WS);
  volatile int *stop = reinterpret_cast<volatile int *>(bar + kTmaMaxStages);
  const uint32_t bytes = (uint32_t)TW * 2;
  // predicate as a range: plo <= cnt <= plo + pspan
  const uint32_t plo = a.pmode == kPredDef ? 0u
                       : a.pmode == kPredCrit ? 1u : (uint32_t)a.ptarget;
  const uint32_t phi = a.pmode == kPredDef ? (uint32_t)(a.mu - 1)
                       : a.pmode == kPredCrit ? (uint32_t)a.mu
                       : (uint32_t)a.ptarget;
  const uint32_t pspan = phi - plo;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) mbar_init(&bar[s]);
    *stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  const long long grid = gridDim.x;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      const long long t = blockIdx.x + s * grid;
      if (t < a.ntiles) {
        mbar_expect(&bar[s], bytes);
        bulk_load(cstage + (size_t)s * CW, a.cnt_in + t * TW, bytes, &bar[s]);
      }
    }
  }
  long long it = 0;
  long long t = blockIdx.x;
  for (; t < a.ntiles; it++, t += grid) {
    const int s = (int)(it % S);
    const uint32_t parity = (uint32_t)((it / S) & 1);
    if (!mbar_wait(&bar[s], parity, kTmaWaitNs)) *stop = 1;
    __syncthreads();
    if (*stop) break;
    const long long nt = t + S * grid;
    FirstRounds<KK, R1, OUT, 0, NR>::run(
        work, WS, cstage + (size_t)s * CW, a, t * TW, plo, pspan, &bar[s],
        nt < a.ntiles ? (const void *)(a.cnt_in + nt * TW) : nullptr,
        cstage + (size_t)s * CW);
  }
  if (t < a.ntiles && threadIdx.x == 0) {
    *a.fault = 1;
    __threadfence_system();
    for (long long k = it; k < it + S; k++) {
      const long long tk = blockIdx.x + k * grid;
      if (tk >= a.ntiles) break;
      mbar_wait(&bar[k % S], (uint32_t)((k / S) & 1), kTmaDrainNs);
    }
  }
}

// The same first group read from the sorted code (a recount): per tile, the
// code slice [bounds[t], bounds[t+1]) is counted into layer 0 of the shared
// buffer (16-bit halves of the packed lanes, which the occurrence bound
// keeps below 2^16), then the rounds run as above.  No HBM reads but the
// slice; every byte written once.
template <int KK, int R1, int OUT, int I, int N>
struct CodeRounds {
  static __device__ __forceinline__ void run(uint32_t *work, int WS,
                                             const TmaArgs &a, long long x0) {
    first_round<KK, R1, OUT, I, 1>(work, WS, nullptr, a, x0, 0u, 0u);
    __syncthreads();
    CodeRounds<KK, R1, OUT, I + 1, N>::run(work, WS, a, x0);
  }
};
template <int KK, int R1, int OUT, int N>
struct CodeRounds<KK, R1, OUT, N, N> {
  static __device__ __forceinline__ void run(uint32_t *, int,
                                             const TmaArgs &, long long) {}
};

template <int KK, int R1, int OUT>
__global__ void __launch_bounds__(512)
code_first(const TmaArgs a) {
  extern __shared__ __align__(128) uint8_t dyn[];
  constexpr int TW = 2 << KK;
  constexpr int WS = ((1 << KK) + (1 << KK) / 16 + 31) / 32 * 32;
  constexpr int NR = FirstRound<KK, 4, 0>::N;
  uint32_t *work = reinterpret_cast<uint32_t *>(dyn);
  for (long long t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const long long x0 = t * TW;
    for (int i = threadIdx.x; i < WS; i += blockDim.x) work[i] = 0;
    __syncthreads();
    const long long lo = a.code_bounds[t], hi = a.code_bounds[t + 1];
    for (long long c = lo + threadIdx.x; c < hi; c += blockDim.x) {
      const int w = (int)(a.code[c] - x0);
      atomicAdd(&work[pad16(w >> 1)], 1u << (16 * (w & 1)));
    }
    __syncthreads();
    CodeRounds<KK, R1, OUT, 0, NR>::run(work, WS, a, x0);
  }
}

// ------------------------------------------------------------ dispatch
#define TE(Q, K, R1, L)                                                     \
  {Q, K, R1, L, 0, tma_group<Q, K, R1, L, 0>},                              \
  {Q, K, R1, L, 1, tma_group<Q, K, R1, L, 1>},                              \
  {Q, K, R1, L, 2, tma_group<Q, K, R1, L, 2>}
// ternary groups run only in the padded layout: OUT 0 (layers), 3 (map)
// and 4 (cnt), the last two back to the canonical index
// three axes a register round (8-word blocks): 512 blocks a round on
// 16-lane rows of an 8-axis group, one for each of 512 threads
#define TB(Q, K, R1, L, I8)                                                 \
  {Q, K, R1, L, 0, tma_group<Q, K, R1, L, 0, I8, 3>, I8 ? 1 : 0, 3},        \
  {Q, K, R1, L, 1, tma_group<Q, K, R1, L, 1, I8, 3>, I8 ? 1 : 0, 3},        \
  {Q, K, R1, L, 2, tma_group<Q, K, R1, L, 2, I8, 3>, I8 ? 1 : 0, 3}
// the launch after an 8-bit first group: its planes staged as bytes
#define TE8(Q, K, R1, L)                                                    \
  {Q, K, R1, L, 0, tma_group<Q, K, R1, L, 0, true>, 1},                     \
  {Q, K, R1, L, 1, tma_group<Q, K, R1, L, 1, true>, 1},                     \
  {Q, K, R1, L, 2, tma_group<Q, K, R1, L, 2, true>, 1}
#define TE3(Q, K, R1, L)                                                    \
  {Q, K, R1, L, 0, tma_group<Q, K, R1, L, 0>},                              \
  {Q, K, R1, L, 3, tma_group<Q, K, R1, L, 3>},                              \
  {Q, K, R1, L, 4, tma_group<Q, K, R1, L, 4>}
const TmaEntry kTma[] = {
    TE(2, 5, 4, 16), TE(2, 6, 4, 16), TE(2, 7, 4, 16), TE(2, 8, 4, 16),
    TE(2, 5, 4, 32), TE(2, 6, 4, 32), TE(2, 7, 4, 32),
    TE3(3, 3, 4, 16), TE3(3, 4, 4, 16), TE3(3, 5, 4, 16),
    TE3(3, 3, 4, 32), TE3(3, 4, 4, 32),
    TE3(3, 3, 5, 16), TE3(3, 4, 5, 16), TE3(3, 5, 5, 16),
    TE3(3, 3, 5, 32), TE3(3, 4, 5, 32),
    TE8(2, 5, 4, 16), TE8(2, 6, 4, 16), TE8(2, 7, 4, 16), TE8(2, 8, 4, 16),
    TE8(2, 5, 4, 32), TE8(2, 6, 4, 32), TE8(2, 7, 4, 32),
    TB(2, 8, 4, 16, false), TB(2, 8, 4, 16, true),
};
#undef TE
#undef TE3
#undef TE8
#undef TB

// src 0: the cnt predicate (tma_first), 1: the sorted code (code_first)
struct FirstEntry { int src, kk, r1, out; FirstFn fn; };
#define FE(KK, R1) {0, KK, R1, 0, tma_first<KK, R1, 0>},                 \
                   {0, KK, R1, 1, tma_first<KK, R1, 1>},                 \
                   {1, KK, R1, 0, code_first<KK, R1, 0>},                \
                   {1, KK, R1, 2, code_first<KK, R1, 2>}
// OUT 5: 8-bit layer planes (C(KK + 1, d) <= 255 for d <= 3)
#define FE8(KK) {0, KK, 4, 5, tma_first<KK, 4, 5>}
const FirstEntry kFirst[] = {FE(9, 4), FE(10, 4), FE(11, 4), FE(12, 4),
                             FE(13, 4), FE8(9), FE8(10), FE8(11)};
#undef FE
#undef FE8

// the first group over row pairs, this file's instances first
#define TF(KK, R1) {0, 3, KK, R1, rows_first<3, KK, R1, 0>},               \
                   {1, 3, KK, R1, rows_first<3, KK, R1, 1>}
const RowsEntry kRows[] = {TF(7, 4), TF(7, 5)};
#undef TF
constexpr int kRowsHere = sizeof(kRows) / sizeof(kRows[0]);
const RowsEntry &rows_entry(int i) {
  return i < kRowsHere ? kRows[i] : rows_table_q(nullptr)[i - kRowsHere];
}
int rows_entries() {
  int n = 0;
  rows_table_q(&n);
  return kRowsHere + n;
}
int axis_kind(int prob, int q) { return prob == kLee ? 32 + q : q; }

int find_rows(int src, int kind, int kk, int r1) {
  static const int n = rows_entries();
  for (int i = 0; i < n; i++) {
    const RowsEntry &e = rows_entry(i);
    if (e.src == src && e.kind == kind && e.kk == kk && e.r1 == r1) return i;
  }
  return -1;
}

const FirstEntry *find_first(int src, int kk, int r1, int out) {
  for (const auto &e : kFirst)
    if (e.src == src && e.kk == kk && e.r1 == r1 && e.out == out) return &e;
  return nullptr;
}

// the kernel's OUT: 0 layers, 1 map, 2 cnt; 3 map and 4 cnt of a padded
// plan (canonical stores)
int out_code(const GroupArgs &a) {
  const int out = a.dst == kDstLayers ? 0 : a.dst == kDstMap ? 1 : 2;
  return (a.pitch && out) ? out + 2 : out;
}

// every instance, this file's first
constexpr int kTmaHere = sizeof(kTma) / sizeof(kTma[0]);
const TmaEntry &tma_entry(int i) {
  return i < kTmaHere ? kTma[i] : tma_table_q(nullptr)[i - kTmaHere];
}
int tma_entries() {
  int n = 0;
  tma_table_q(&n);
  return kTmaHere + n;
}

// index of an instance, -1 when there is none
int find_tma(int kind, int k, int r1, int lanes, int out, int in8 = 0,
             int bm = 0) {
  static const int n = tma_entries();
  for (int i = 0; i < n; i++) {
    const TmaEntry &e = tma_entry(i);
    if (e.kind == kind && e.k == k && e.r1 == r1 && e.lanes == lanes &&
        e.out == out && e.in8 == (in8 ? 1 : 0) && e.bm == bm)
      return i;
  }
  return -1;
}

// the first group's OUT: 0 16-bit layers, 5 8-bit layers, 1 map, 2 cnt
int first_out(const GroupArgs &a) {
  return a.dst == kDstLayers ? (a.out8 ? 5 : 0) : a.dst == kDstMap ? 1 : 2;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p,
                                cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      cudaGetLastError();
  });
  return fn;
}

// the fault word: mapped pinned host memory the kernels write through
int *g_fault_host = nullptr;
int *g_fault_dev = nullptr;

int fault_word(int **dev) {
  static std::once_flag once;
  static int rc = 0;
  std::call_once(once, [] {
    void *h = nullptr;
    if (cudaHostAlloc(&h, sizeof(int), cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      rc = -1;
      return;
    }
    g_fault_host = static_cast<int *>(h);
    *g_fault_host = 0;
    void *d = nullptr;
    if (cudaHostGetDevicePointer(&d, h, 0) != cudaSuccess) {
      cudaGetLastError();
      rc = -1;
      return;
    }
    g_fault_dev = static_cast<int *>(d);
  });
  *dev = g_fault_dev;
  return rc;
}

}  // namespace

size_t tma_smem_bytes(int q, int k, int r1, int lanes, int stages,
                      int in8) {
  long long mid = 1;
  for (int i = 0; i < k; i++) mid *= q;
  const long long words = (r1 * mid * lanes + 255) / 256 * 256;
  if (in8) {                    // byte stages and one 32-bit work buffer
    const long long sb = (r1 * mid * 2 * lanes + 1023) / 1024 * 1024;
    return (size_t)(stages * sb + words * 4) + 1024 + kTmaMaxStages * 8 + 16;
  }
  return (size_t)stages * words * 4 + 1024 + kTmaMaxStages * 8 + 16;
}

// The groups the streamed form serves: Hamming (q <= 6) and Lee (q <= 7)
// groups over 16-bit planes in packed pairs (an even inner stride), 16-bit
// planes, the map or cnt out, one tile per W inner words x the whole group, an
// instantiated (q, k, layers, lanes) and its stages within 227 KB of shared
// memory.
bool tma_group_ok(const GroupArgs &a, int q, int r1, int lanes, int stages) {
  // one stage: a CTA small enough for two a SM, whose loads then overlap
  // the other CTA's rounds
  if (stages < 1 || stages > kTmaMaxStages || !encode_fn()) return false;
  const int out = out_code(a);
  if (find_tma(axis_kind(a.prob, q), a.k, r1, lanes, out, a.in8, a.tbm) < 0)
    return false;
  if ((a.prob != kHamming && a.prob != kLee) || !a.pack || !a.in16 || a.pair_axis ||
      a.src != kSrcLayers || a.R + 1 != r1)
    return false;
  if (out == 0 && !a.out16) return false;
  // 8-bit planes: the tensor map's byte strides are multiples of 16
  if (a.in8 && (a.plane % 16 || a.inner % 16 || a.pitch || a.off8 % 16))
    return false;
  if (a.inner % (2 * lanes) || a.plane % 8 || a.lin < 1 || a.lin > r1)
    return false;
  if ((reinterpret_cast<uintptr_t>(a.layers16) & 15) != 0) return false;
  if (a.outer >= (1LL << 31) || a.inner >= (1LL << 31)) return false;
  return tma_smem_bytes(q, a.k, r1, lanes, stages, a.in8) <= kTmaSmemMax;
}

// The same group as a streamed launch: W = 2 x lanes inner words a tile.
GroupPlan tma_first_variant(const GroupPlan &p, int stages, int threads) {
  GroupPlan v = p;
  v.a.tma = 2;
  v.a.stages = stages;
  v.a.pipe = 0;
  v.threads = threads;
  v.smem = tma_first_smem_bytes(v.a.k, v.a.R + 1, stages);
  v.grid = 0;
  return v;
}

GroupPlan tma_variant(const GroupPlan &p, int lanes, int stages,
                      int threads) {
  GroupPlan v = p;
  v.a.tma = 1;
  v.a.stages = stages;
  v.a.pipe = 0;
  v.a.W = 2 * lanes;
  v.a.Bo = 1;
  v.a.nchunk = (v.a.inner + v.a.W - 1) / v.a.W;
  v.a.ntiles = v.a.outer * v.a.nchunk;
  v.threads = threads;
  v.smem = tma_smem_bytes(v.a.rq[0] ? v.a.rq[0] : v.a.qax[0], v.a.k,
                          v.a.R + 1, lanes, stages, v.a.in8);
  v.grid = 0;
  return v;
}

size_t tma_first_smem_bytes(int kk, int r1, int stages) {
  const long long lanes = 1LL << kk;
  const long long ws = (lanes + lanes / 16 + 31) / 32 * 32;
  if (stages == 0)                        // code source: the buffer alone
    return (size_t)r1 * ws * 4;
  return (size_t)stages * (4LL << kk) + (size_t)r1 * ws * 4 + 1024 +
         kTmaMaxStages * 8 + 16;
}

// The first group of a binary Hamming cell read from cnt, its axis 0 inside
// the pair, one contiguous tile of 2^(k+1) words (Bo = 1).
// (stages 0: the code-sourced form of a recount's first group)
bool tma_first_ok(const GroupArgs &a, int r1, int stages) {
  const int src = a.src == kSrcCnt ? 0 : a.src == kSrcCode ? 1 : -1;
  if (src < 0 || (src == 0 && (stages < 2 || stages > kTmaMaxStages)) ||
      (src == 1 && stages != 0))
    return false;
  const int out = first_out(a);
  if (!find_first(src, a.k, r1, out)) return false;
  if (a.prob != kHamming || !a.pair_axis || !a.pack || a.W != 2 ||
      a.inner != 2 || a.Bo != 1 || a.R + 1 != r1 || a.nchunk != 1)
    return false;
  if ((out == 0 || out == 5) && !a.out16) return false;
  if (a.plane % 8 || (reinterpret_cast<uintptr_t>(a.cnt) & 15) != 0)
    return false;
  return tma_first_smem_bytes(a.k, r1, stages) <= kTmaSmemMax;
}

size_t rows_first_smem_bytes(int q, int kk, int r1) {
  long long t0 = 1;
  for (int i = 0; i < kk; i++) t0 *= q;
  return (size_t)r1 * ((t0 + 31) / 32 * 32) * 4;
}

// The first groups rows_first serves: Hamming or Lee axes of one size, inner
// stride 1, row pairs (Bo = 2) as the tiles, 16-bit layers out (at the plan's
// pitch, or T0), the cnt or the code as the source.
bool rows_first_ok(const GroupArgs &a, int r1) {
  const int src = a.src == kSrcCnt ? 0 : a.src == kSrcCode ? 1 : -1;
  if (src < 0 || (a.prob != kHamming && a.prob != kLee) ||
      a.dst != kDstLayers || !a.out16 || a.inner != 1 || a.W != 1 ||
      a.Bo != 2 || a.pair_axis || a.pack || a.R + 1 != r1 || a.lin != 1 ||
      a.k < 1)
    return false;
  const int q = a.qax[0];
  long long t0 = 1;
  for (int i = 0; i < a.k; i++) {
    if (a.qax[i] != q) return false;
    t0 *= q;
  }
  if (t0 != a.mid || find_rows(src, axis_kind(a.prob, q), a.k, r1) < 0)
    return false;
  if (a.pitch && (a.pitch < t0 || a.t0 != t0)) return false;
  if (a.outer < 1 || a.ntiles != (a.outer + 1) / 2) return false;
  return rows_first_smem_bytes(q, a.k, r1) <= kTmaSmemMax;
}

GroupPlan rows_first_variant(const GroupPlan &p, int threads) {
  GroupPlan v = p;
  v.a.tma = 3;
  v.a.stages = 0;
  v.a.pipe = 0;
  v.threads = threads;
  v.smem = rows_first_smem_bytes(v.a.qax[0], v.a.k, v.a.R + 1);
  v.grid = 0;
  return v;
}

int tma_fault_take() {
  volatile int *f = g_fault_host;
  if (!f || !*f) return 0;
  *f = 0;
  fprintf(stderr, "coldcore_b200: a streamed group launch timed out "
          "waiting for its tensor loads\n");
  return -8;
}

static std::atomic<int> g_inject[kFaultKinds];

bool fault_due(int kind) {
  std::atomic<int> &c = g_inject[kind];
  return c.load() > 0 && c.fetch_sub(1) == 1;
}

namespace {

const FirstEntry *first_of(const GroupPlan &p) {
  const GroupArgs &a = p.a;
  return find_first(a.src == kSrcCode ? 1 : 0, a.k, a.R + 1, first_out(a));
}

int first_opt_in(const FirstEntry *e) {
  static std::mutex mu;
  static bool done[sizeof(kFirst) / sizeof(kFirst[0])];
  std::lock_guard<std::mutex> g(mu);
  const size_t idx = (size_t)(e - kFirst);
  if (!done[idx]) {
    CC_CK(cudaFuncSetAttribute((const void *)e->fn,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kTmaSmemMax));
    done[idx] = true;
  }
  return 0;
}

int rows_of(const GroupPlan &p) {
  return find_rows(p.a.src == kSrcCode ? 1 : 0,
                   axis_kind(p.a.prob, p.a.qax[0]), p.a.k, p.a.R + 1);
}

int rows_opt_in(int idx) {
  static std::mutex mu;
  static std::vector<bool> done;
  std::lock_guard<std::mutex> g(mu);
  if (done.empty()) done.resize(rows_entries(), false);
  if (!done[idx]) {
    CC_CK(cudaFuncSetAttribute((const void *)rows_entry(idx).fn,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kTmaSmemMax));
    done[idx] = true;
  }
  return 0;
}

int entry_of(const GroupPlan &p) {
  const GroupArgs &a = p.a;
  const int out = out_code(a);
  return find_tma(axis_kind(a.prob, a.rq[0] ? a.rq[0] : a.qax[0]), a.k,
                  a.R + 1, a.W / 2, out, a.in8, a.tbm);
}

// opt every streamed kernel in to the largest dynamic shared memory once
int opt_in(int idx) {
  static std::mutex mu;
  static std::vector<bool> done;
  std::lock_guard<std::mutex> g(mu);
  if (done.empty()) done.resize(tma_entries(), false);
  if (!done[idx]) {
    CC_CK(cudaFuncSetAttribute((const void *)tma_entry(idx).fn,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kTmaSmemMax));
    done[idx] = true;
  }
  return 0;
}

}  // namespace

int tma_prepare(const GroupPlan &p) {
  // the mapped fault word is allocated here, ahead of any stream capture
  int *fault = nullptr;
  if (fault_word(&fault)) return -9;
  if (p.a.tma == 3) {
    const int f = rows_of(p);
    return f < 0 ? -9 : rows_opt_in(f);
  }
  if (p.a.tma == 2) {
    const FirstEntry *f = first_of(p);
    return f ? first_opt_in(f) : -9;
  }
  const int e = entry_of(p);
  return e < 0 ? -9 : opt_in(e);
}

int tma_blocks_per_sm(const GroupPlan &p) {
  const void *fn = nullptr;
  if (p.a.tma == 3) {
    const int f = rows_of(p);
    if (f < 0 || rows_opt_in(f)) return 0;
    fn = (const void *)rows_entry(f).fn;
  } else if (p.a.tma == 2) {
    const FirstEntry *f = first_of(p);
    if (!f || first_opt_in(f)) return 0;
    fn = (const void *)f->fn;
  } else {
    const int e = entry_of(p);
    if (e < 0 || opt_in(e)) return 0;
    fn = (const void *)tma_entry(e).fn;
  }
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &n, fn, p.threads, p.smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int launch_rows_first(const GroupPlan &p, cudaStream_t s) {
  const GroupArgs &a = p.a;
  const int f = rows_of(p);
  const bool from_code = a.src == kSrcCode;
  if (f < 0 || !rows_first_ok(a, a.R + 1) ||
      (from_code && (!a.code_bounds || (!a.code && a.ncode > 0))))
    return -9;
  int rc = rows_opt_in(f);
  if (rc) return rc;
  TmaArgs t{};
  t.layers16 = a.layers16;
  t.plane = a.plane;
  t.cnt_in = a.cnt;
  t.pmode = a.pmode;
  t.ptarget = a.ptarget;
  t.mu = a.mu;
  t.ntiles = a.ntiles;
  t.lin = 1;
  t.lout = a.lout;
  t.code = a.code;
  t.code_bounds = a.code_bounds;
  t.pitch = a.pitch ? a.pitch : a.mid;
  t.t0 = a.mid;
  t.rows = a.outer;
  const size_t smem = rows_first_smem_bytes(a.qax[0], a.k, a.R + 1);
  int grid = p.grid;
  if (grid < 1) {
    const int per_sm = tma_blocks_per_sm(p);
    long long gr = (long long)sm_count() * (per_sm < 1 ? 1 : per_sm);
    if (gr > a.ntiles) gr = a.ntiles;
    grid = (int)(gr < 1 ? 1 : gr);
  }
  grid = grid_knob(grid, a.ntiles);
  rows_entry(f).fn<<<grid, p.threads, smem, s>>>(t);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_tma_first(const GroupPlan &p, cudaStream_t s) {
  const GroupArgs &a = p.a;
  const FirstEntry *f = first_of(p);
  const bool from_code = a.src == kSrcCode;
  if (!f || (!from_code && (a.stages < 2 || a.stages > kTmaMaxStages)) ||
      (from_code && (!a.code_bounds || (!a.code && a.ncode > 0))))
    return -9;
  int *fault = nullptr;
  if (fault_word(&fault)) return -9;
  int rc = first_opt_in(f);
  if (rc) return rc;
  TmaArgs t{};
  t.layers16 = a.layers16;
  t.plane = a.plane;
  t.map = a.map ? a.map : a.layers;
  t.cnt = a.cnt;
  t.cnt_in = a.cnt;
  t.pmode = a.pmode;
  t.ptarget = a.ptarget;
  t.mu = a.mu;
  t.inner = a.inner;
  t.nchunk = 1;
  t.ntiles = a.ntiles;
  t.lin = 1;
  t.lout = a.lout;
  t.stages = a.stages;
  t.fault = fault;
  t.code = a.code;
  t.code_bounds = a.code_bounds;
  t.off8 = a.off8;
  const size_t smem = tma_first_smem_bytes(a.k, a.R + 1,
                                           from_code ? 0 : a.stages);
  int grid = p.grid;
  if (grid < 1) {
    const int per_sm = tma_blocks_per_sm(p);
    long long gr = (long long)sm_count() * (per_sm < 1 ? 1 : per_sm);
    if (gr > a.ntiles) gr = a.ntiles;
    grid = (int)(gr < 1 ? 1 : gr);
  }
  grid = grid_knob(grid, a.ntiles);
  f->fn<<<grid, p.threads, smem, s>>>(t);
  CC_CK(cudaGetLastError());
  return 0;
}

namespace {

// tensor-map parameters of one streamed launch (the map is a pure function
// of them)
struct MapKey {
  const void *base;
  cuuint64_t dims[4], strides[3];
  cuuint32_t box[4];
  int dt;
  bool operator==(const MapKey &o) const {
    return std::memcmp(this, &o, sizeof(MapKey)) == 0;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey &k) const {
    const unsigned char *b = reinterpret_cast<const unsigned char *>(&k);
    size_t h = 1469598103934665603ULL;
    for (size_t i = 0; i < sizeof(MapKey); i++) {
      h ^= b[i];
      h *= 1099511628211ULL;
    }
    return h;
  }
};
std::mutex g_map_mu;
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_maps;

bool map_cache_get(const MapKey &k, CUtensorMap *m) {
  std::lock_guard<std::mutex> g(g_map_mu);
  auto it = g_maps.find(k);
  if (it == g_maps.end()) return false;
  *m = it->second;
  return true;
}

void map_cache_put(const MapKey &k, const CUtensorMap &m) {
  std::lock_guard<std::mutex> g(g_map_mu);
  if (g_maps.size() >= 4096) g_maps.clear();   // freed planes' stale keys
  g_maps[k] = m;
}

}  // namespace

int launch_tma_group(const GroupPlan &p, cudaStream_t s) {
  if (p.a.tma == 3) return launch_rows_first(p, s);
  if (p.a.tma == 2) return launch_tma_first(p, s);
  const GroupArgs &a = p.a;
  const int q = a.rq[0] ? a.rq[0] : a.qax[0];
  const int lanes = a.W / 2;
  const int e = entry_of(p);
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
  if (e < 0 || !enc || a.stages < 1 || a.stages > kTmaMaxStages) return -9;
  int *fault = nullptr;
  if (fault_word(&fault)) return -9;
  int rc = opt_in(e);
  if (rc) return rc;
  long long mid = 1;
  for (int i = 0; i < a.k; i++) mid *= q;
  // the live layers as a 4-D u16 (or, 8-bit planes, u8) tensor: inner
  // word, mid, outer, layer
  CUtensorMap map;
  const cuuint64_t esz = a.in8 ? 1 : 2;
  const cuuint64_t dims[4] = {(cuuint64_t)a.inner, (cuuint64_t)mid,
                              (cuuint64_t)a.outer, (cuuint64_t)a.lin};
  const cuuint64_t strides[3] = {(cuuint64_t)a.inner * esz,
                                 (cuuint64_t)(a.inner * mid) * esz,
                                 (cuuint64_t)a.plane * esz};
  const cuuint32_t box[4] = {(cuuint32_t)(2 * lanes), (cuuint32_t)mid, 1,
                             (cuuint32_t)a.lin};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  void *gbase = a.in8 ? (void *)(reinterpret_cast<uint8_t *>(a.layers16) +
                                 a.off8)
                      : (void *)a.layers16;
  // the encoded maps of earlier launches, by their parameters: a plan's
  // launches repeat every transform, and the encode is host work
  MapKey key{};
  key.base = gbase;
  key.dt = a.in8 ? 1 : 2;
  for (int i = 0; i < 4; i++) key.dims[i] = dims[i], key.box[i] = box[i];
  for (int i = 0; i < 3; i++) key.strides[i] = strides[i];
  if (!map_cache_get(key, &map)) {
    const CUresult cr = enc(&map, a.in8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                        : CU_TENSOR_MAP_DATA_TYPE_UINT16, 4,
                            gbase, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
      fprintf(stderr, "coldcore_b200: tensor map encode failed (%d)\n",
              (int)cr);
      return -9;
    }
    map_cache_put(key, map);
  }
  TmaArgs t{};
  t.layers16 = a.layers16;
  t.plane = a.plane;
  t.map = a.map ? a.map : a.layers;
  t.cnt = a.cnt;
  t.inner = a.inner;
  t.nchunk = a.nchunk;
  t.ntiles = a.ntiles;
  t.lin = a.lin;
  t.lout = a.lout;
  t.stages = a.stages;
  t.fault = fault;
  t.pitch = a.pitch;
  t.t0 = a.t0;
  t.inner_c = a.pitch ? a.inner / a.pitch * a.t0 : a.inner;
  t.mu = a.mu;
  t.red = a.red;
  t.red_mode = a.dst != kDstLayers && a.red ? a.red_mode : 0;
  const size_t smem = tma_smem_bytes(q, a.k, a.R + 1, lanes, a.stages,
                                     a.in8);
  int grid = p.grid;
  if (grid < 1) {
    const int per_sm = tma_blocks_per_sm(p);
    long long gr = (long long)sm_count() * (per_sm < 1 ? 1 : per_sm);
    if (gr > a.ntiles) gr = a.ntiles;
    grid = (int)(gr < 1 ? 1 : gr);
  }
  grid = grid_knob(grid, a.ntiles);
  tma_entry(e).fn<<<grid, p.threads, smem, s>>>(map, t);
  CC_CK(cudaGetLastError());
  if (fault_due(kFaultStreamed)) *(volatile int *)g_fault_host = 1;
  return 0;
}

}  // namespace cc

extern "C" int dct_b200_fault_inject(int kind, int nth) {
  if (kind < 0 || kind >= cc::kFaultKinds || nth < 0) return -1;
  cc::g_inject[kind] = nth;
  return 0;
}
