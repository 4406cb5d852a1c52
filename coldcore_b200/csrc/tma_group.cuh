// tma_group.cuh — the streamed strided groups: mbarrier and tensor-load
// helpers, the axis recurrences on packed lanes, and the kernel.
// transform_tma.cu has the binary and ternary Hamming instances, the dispatch
// and the first groups; transform_tma_q.cu the other axis sizes and Lee.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include "engine.h"

namespace cc {

typedef void (*TmaFn)(const CUtensorMap, const TmaArgs);
// an instance: axis kind, axes, layers, lanes (half a tile's row), output
struct TmaEntry { int kind, k, r1, lanes, out; TmaFn fn; int in8 = 0;
                  int bm = 0; };
// the instances of transform_tma_q.cu
const TmaEntry *tma_table_q(int *n);

namespace {

constexpr size_t kTmaSmemMax = 227 * 1024;
constexpr unsigned long long kTmaWaitNs = 2000000000ULL;   // 2 s
constexpr unsigned long long kTmaDrainNs = 200000000ULL;   // 0.2 s

template <int Q, int E>
struct P { static constexpr int v = Q * P<Q, E - 1>::v; };
template <int Q>
struct P<Q, 0> { static constexpr int v = 1; };

// ------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t saddr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile(
      "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
          saddr(bar)),
      "r"(bytes)
      : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(saddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// true once the phase of `parity` has completed; false after `limit` ns
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          unsigned long long limit) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  for (unsigned it = 1;; it++) {
    if (mbar_test(bar, parity)) return true;
    if ((it & 255) == 0 && now_ns() - t0 > limit) return false;
  }
}
__device__ __forceinline__ void tma_load4(void *dst, const CUtensorMap *map,
                                          uint64_t *bar, int c0, int c1,
                                          int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::"
      "complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(
          saddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2),
      "r"(c3), "r"(saddr(bar))
      : "memory");
}

// ------------------------------------------------------------ axis math
// The axis kinds of the streamed groups: Hamming of size q is kind q, Lee of
// size q is kind 32 + q.
__host__ __device__ constexpr int axis_size(int kind) { return kind & 31; }
__host__ __device__ constexpr bool axis_lee(int kind) { return kind >= 32; }

// One axis over a register block: the fibres are the Q entries at element
// stride ST; layers descend so a lower layer is read before it changes.
// Every form is made of adds whose partial sums are parts of a layer value,
// so two 16-bit words ride in each 32-bit register and no add carries from
// one to the other.  Hamming: the other entries of layer d-1 (for Q >= 4 from
// shared partial sums: 14 adds a fibre of 5, as many as the fibre sum less
// each entry, which can pass 16 bits, would take).  Lee: the entries w steps
// away of layer d-w, w up to Q / 2, one term where the two coincide.
template <int C, int R1, int QB, int ST>
__device__ __forceinline__ void axis_op(uint32_t (&v)[R1][QB]) {
  constexpr int Q = axis_size(C);
#pragma unroll
  for (int e = 0; e < QB; e++) {
    if ((e / ST) % Q != 0) continue;
#pragma unroll
    for (int d = R1 - 1; d >= 1; d--) {
      if constexpr (axis_lee(C)) {
        constexpr int H = Q / 2;
#pragma unroll
        for (int a = 0; a < Q; a++) {
          uint32_t s = 0;
#pragma unroll
          for (int w = 1; w <= (d < H ? d : H); w++) {
            const int am = (a - w + Q) % Q, ap = (a + w) % Q;
            s += v[d - w][e + am * ST];
            if (ap != am) s += v[d - w][e + ap * ST];
          }
          v[d][e + a * ST] += s;
        }
      } else {
        uint32_t a[Q];
#pragma unroll
        for (int k = 0; k < Q; k++) a[k] = v[d - 1][e + k * ST];
        uint32_t o[Q];                      // the sum of the others
        if constexpr (Q == 2) {
          o[0] = a[1];
          o[1] = a[0];
        } else if constexpr (Q == 3) {
          o[0] = a[1] + a[2];
          o[1] = a[0] + a[2];
          o[2] = a[0] + a[1];
        } else if constexpr (Q == 4) {
          const uint32_t l = a[0] + a[1], h = a[2] + a[3];
          o[0] = a[1] + h;
          o[1] = a[0] + h;
          o[2] = a[3] + l;
          o[3] = a[2] + l;
        } else if constexpr (Q == 5) {
          const uint32_t l = a[0] + a[1], h = a[3] + a[4];
          const uint32_t lm = l + a[2], mh = a[2] + h;
          o[0] = a[1] + mh;
          o[1] = a[0] + mh;
          o[2] = l + h;
          o[3] = lm + a[4];
          o[4] = lm + a[3];
        } else {
          static_assert(Q <= 6, "Hamming axes of 2..6");
          const uint32_t l = a[0] + a[1], h = a[3] + a[4];
          const uint32_t lo = l + a[2], hi = h + a[5];
          o[0] = a[1] + a[2] + hi;
          o[1] = a[0] + a[2] + hi;
          o[2] = l + hi;
          o[3] = a[4] + a[5] + lo;
          o[4] = a[3] + a[5] + lo;
          o[5] = h + lo;
        }
#pragma unroll
        for (int k = 0; k < Q; k++) v[d][e + k * ST] += o[k];
      }
    }
  }
}

template <int C, int R1, int B, int T>
struct Axes {
  static __device__ __forceinline__ void run(
      uint32_t (&v)[R1][P<axis_size(C), B>::v]) {
    axis_op<C, R1, P<axis_size(C), B>::v, P<axis_size(C), T>::v>(v);
    Axes<C, R1, B, T + 1>::run(v);
  }
};
template <int C, int R1, int B>
struct Axes<C, R1, B, B> {
  static __device__ __forceinline__ void run(
      uint32_t (&)[R1][P<axis_size(C), B>::v]) {}
};

// axes per register round: Q^b x R1 registers at most 64
template <int C, int R1>
struct RoundAxes {
  static constexpr int v = (P<axis_size(C), 4>::v * R1 <= 64) ? 4
                           : (P<axis_size(C), 3>::v * R1 <= 64) ? 3
                           : (P<axis_size(C), 2>::v * R1 <= 64) ? 2 : 1;
};

// Epilogue reductions of a streamed launch's output (TmaArgs::red_mode): 2
// the map maximum, 1 the deficit sum max(0, mu - c) of the cnt written; a
// packed lane's two words, each only where it is a word of the cell.
__device__ __forceinline__ void tma_red(long long *acc, const TmaArgs &a,
                                        int w0, int w1, bool ok0, bool ok1) {
  if (a.red_mode == 2) {
    if (ok0 && w0 > *acc) *acc = w0;
    if (ok1 && w1 > *acc) *acc = w1;
  } else {
    if (ok0 && w0 < a.mu) *acc += a.mu - w0;
    if (ok1 && w1 < a.mu) *acc += a.mu - w1;
  }
}

// ------------------------------------------------------------ one round
// Round over axes [A, A + B) of the group on a stage of L lanes x MID mid
// positions x R1 layers (32-bit packed lanes, layer-major as the tensor
// load lays it down).  FIRST: layers >= lin start at zero.  LAST: the
// block goes to HBM (OUT 0 layers, 1 map, 2 cnt) instead of the stage.
template <int C, int K, int R1, int L, int OUT, int A, int B, bool FIRST,
          bool LAST, bool IN8 = false>
__device__ __forceinline__ void tma_round(uint32_t *st, const TmaArgs &a,
                                          long long o, long long i0,
                                          const uint16_t *s8 = nullptr,
                                          long long *racc = nullptr) {
  constexpr int MID = P<axis_size(C), K>::v;
  constexpr int QB = P<axis_size(C), B>::v;
  constexpr int QA = P<axis_size(C), A>::v;
  constexpr int NB = L * MID / QB;            // register blocks in the tile
  for (int blk = threadIdx.x; blk < NB; blk += blockDim.x) {
    const int l = blk % L;
    const int rest = blk / L;                 // mid digits outside [A, A+B)
    const int mb = rest % QA + (rest / QA) * (QA * QB);
    uint32_t *p = st + mb * L + l;
    uint32_t v[R1][QB];
    if (IN8 && FIRST) {
      // the staged 8-bit planes: one 16-bit read gives the lane's two
      // words, widened to the two 16-bit halves of the packed lane
      const uint16_t *p8 = s8 + mb * L + l;
#pragma unroll
      for (int d = 0; d < R1; d++) {
        const bool live = d < a.lin;
#pragma unroll
        for (int e = 0; e < QB; e++)
          v[d][e] = live ? __byte_perm((uint32_t)p8[(d * MID + e * QA) * L],
                                       0u, 0x4140)
                         : 0u;
      }
    } else {
#pragma unroll
      for (int d = 0; d < R1; d++) {
        const bool live = !FIRST || d < a.lin;
#pragma unroll
        for (int e = 0; e < QB; e++)
          v[d][e] = live ? p[(d * MID + e * QA) * L] : 0u;
      }
    }
    Axes<C, R1, B, 0>::run(v);
    if (!LAST) {
#pragma unroll
      for (int d = 0; d < R1; d++)
#pragma unroll
        for (int e = 0; e < QB; e++) p[(d * MID + e * QA) * L] = v[d][e];
      continue;
    }
    // HBM word of element e: o*(MID*inner) + (mb + e*QA)*inner + i0 + 2l
    const long long x0 = (o * MID + mb) * a.inner + i0 + 2 * l;
    const long long step = (long long)QA * a.inner;
    if (OUT == 0) {
#pragma unroll
      for (int d = 0; d < R1; d++) {
        if (d >= a.lout) break;
        uint16_t *q = a.layers16 + d * a.plane + x0;
#pragma unroll
        for (int e = 0; e < QB; e++)
          __stcs(reinterpret_cast<unsigned *>(q + e * step), v[d][e]);
      }
    } else if (OUT == 1 || OUT == 2) {
#pragma unroll
      for (int e = 0; e < QB; e++) {
        uint32_t s = 0;
#pragma unroll
        for (int d = 0; d < R1; d++) s += v[d][e];
        if (OUT == 1)
          __stcs(reinterpret_cast<int2 *>(a.map + x0 + e * step),
                 make_int2((int)(s & 0xFFFFu), (int)(s >> 16)));
        else
          *reinterpret_cast<unsigned *>(a.cnt + x0 + e * step) = s;
        if (racc)
          tma_red(racc, a, (int)(s & 0xFFFFu), (int)(s >> 16), true, true);
      }
    } else {
      // OUT 3 (map) / 4 (cnt) of a padded plan: the pair's words j', j'+1
      // of the padded inner go back to the canonical index, padding dropped
      const long long jp = i0 + 2 * l;
      const long long r = jp / a.pitch, i = jp - r * a.pitch;
      const bool ok0 = i < a.t0, ok1 = i + 1 < a.t0;
      const long long xc = (o * MID + mb) * a.inner_c + r * a.t0 + i;
      const long long stepc = (long long)QA * a.inner_c;
#pragma unroll
      for (int e = 0; e < QB; e++) {
        uint32_t s = 0;
#pragma unroll
        for (int d = 0; d < R1; d++) s += v[d][e];
        const long long x = xc + e * stepc;
        if (OUT == 3) {
          if (ok0) __stcs(a.map + x, (int)(s & 0xFFFFu));
          if (ok1) __stcs(a.map + x + 1, (int)(s >> 16));
        } else {
          if (ok0) a.cnt[x] = (uint16_t)(s & 0xFFFFu);
          if (ok1) a.cnt[x + 1] = (uint16_t)(s >> 16);
        }
        if (racc) tma_red(racc, a, (int)(s & 0xFFFFu), (int)(s >> 16), ok0, ok1);
      }
    }
  }
}

// The rounds of a K-axis group: RoundAxes-sized rounds from axis 0 up (or
// BMX axes a round: smaller register blocks, twice the blocks a round, for
// twice the threads), the remainder last.
template <int C, int K, int R1, int L, int OUT, int A, bool IN8 = false,
          int BMX = 0>
struct Rounds {
  static constexpr int BM = BMX ? BMX : RoundAxes<C, R1>::v;
  static constexpr int B = (K - A) < BM ? (K - A) : BM;
  static __device__ __forceinline__ void run(uint32_t *st, const TmaArgs &a,
                                             long long o, long long i0,
                                             const uint16_t *s8 = nullptr,
                                             long long *racc = nullptr) {
    tma_round<C, K, R1, L, OUT, A, B, A == 0, A + B == K, IN8>(st, a, o, i0,
                                                              s8, racc);
    if (A + B < K) __syncthreads();
    Rounds<C, K, R1, L, OUT, (A + B < K ? A + B : K), IN8, BMX>::run(
        st, a, o, i0, s8, racc);
  }
};
template <int C, int K, int R1, int L, int OUT, bool IN8, int BMX>
struct Rounds<C, K, R1, L, OUT, K, IN8, BMX> {
  static __device__ __forceinline__ void run(uint32_t *, const TmaArgs &,
                                             long long, long long,
                                             const uint16_t *,
                                             long long * = nullptr) {}
};

// stage stride: the tile's words rounded up to 1 KB (tensor loads land on
// 128-byte-aligned shared addresses)
template <int C, int K, int R1, int L>
struct Stage {
  static constexpr int words = (R1 * P<axis_size(C), K>::v * L + 255) / 256 * 256;
};
// 8-bit staged planes: a stage is R1 x mid x 2L bytes (1 KB multiples),
// and the rounds run on one 32-bit work buffer of the Stage size
template <int C, int K, int R1, int L>
struct Stage8 {
  static constexpr int bytes = (R1 * P<axis_size(C), K>::v * 2 * L + 1023) / 1024 * 1024;
};

template <int C, int K, int R1, int L, int OUT, bool IN8 = false,
          int BMX = 0>
__global__ void __launch_bounds__(512)
tma_group(const __grid_constant__ CUtensorMap map, const TmaArgs a) {
  extern __shared__ __align__(128) uint8_t dyn[];
  constexpr int MID = P<axis_size(C), K>::v;
  constexpr int SW = Stage<C, K, R1, L>::words;
  // bytes a stage: the 16-bit planes' tile, or the 8-bit planes' tile
  constexpr int SB = IN8 ? Stage8<C, K, R1, L>::bytes : SW * 4;
  const int S = a.stages;
  // stages on a 1 KB boundary, then (8-bit planes) the work buffer, then
  // the barriers and the stop flag
  uint8_t *base = dyn + ((1024u - (saddr(dyn) & 1023u)) & 1023u);
  uint8_t *stage = base;
  uint32_t *work = IN8 ? reinterpret_cast<uint32_t *>(base + (size_t)S * SB)
                       : nullptr;
  uint64_t *bar = reinterpret_cast<uint64_t *>(
      base + (size_t)S * SB + (IN8 ? (size_t)SW * 4 : 0));
  volatile int *stop = reinterpret_cast<volatile int *>(bar + kTmaMaxStages);
  const uint32_t bytes = (uint32_t)(2 * L * (IN8 ? 1 : 2)) * MID * a.lin;
  long long acc = 0;                    // epilogue reduction (red_mode)
  long long *racc = (OUT != 0 && a.red_mode) ? &acc : nullptr;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) mbar_init(&bar[s]);
    *stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  const long long grid = gridDim.x;
  auto issue = [&](long long t, int s) {
    const int i0 = (int)((t % a.nchunk) * (2 * L));
    const int o = (int)(t / a.nchunk);
    mbar_expect(&bar[s], bytes);
    tma_load4(stage + (size_t)s * SB, &map, &bar[s], i0, 0, o, 0);
  };
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(
                     reinterpret_cast<uint64_t>(&map))
                 : "memory");
    for (int s = 0; s < S; s++) {
      const long long t = blockIdx.x + s * grid;
      if (t < a.ntiles) issue(t, s);
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
    const long long o = t / a.nchunk;
    const long long i0 = (t % a.nchunk) * (2 * L);
    if (IN8)
      Rounds<C, K, R1, L, OUT, 0, IN8, BMX>::run(
          work, a, o, i0,
          reinterpret_cast<const uint16_t *>(stage + (size_t)s * SB), racc);
    else
      Rounds<C, K, R1, L, OUT, 0, false, BMX>::run(
          reinterpret_cast<uint32_t *>(stage + (size_t)s * SB), a, o, i0,
          nullptr, racc);
    __syncthreads();                          // stage s is free again
    if (threadIdx.x == 0) {
      const long long nt = t + S * grid;
      if (nt < a.ntiles) {
        // the rounds wrote the stage through the generic proxy; order those
        // writes before the tensor load overwrites it
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        issue(nt, s);
      }
    }
  }
  if (t < a.ntiles && threadIdx.x == 0) {
    // a load never completed: report, then wait (bounded) for every load
    // this CTA still has outstanding before the CTA's memory goes away
    *a.fault = 1;
    __threadfence_system();
    for (long long k = it; k < it + S; k++) {
      const long long tk = blockIdx.x + k * grid;
      if (tk >= a.ntiles) break;
      mbar_wait(&bar[k % S], (uint32_t)((k / S) & 1), kTmaDrainNs);
    }
  }
  if (racc) {
    for (int o2 = 16; o2 > 0; o2 >>= 1) {
      const long long other = __shfl_down_sync(0xffffffffu, acc, o2);
      acc = a.red_mode == 2 ? (other > acc ? other : acc) : acc + other;
    }
    if ((threadIdx.x & 31) == 0 && acc) {
      if (a.red_mode == 2)
        atomicMax((unsigned long long *)a.red, (unsigned long long)acc);
      else
        atomicAdd((unsigned long long *)a.red, (unsigned long long)acc);
    }
  }
}

}  // namespace
}  // namespace cc
