// rows_first.cuh — the first group of a cell whose rows have no word pairs to
// pack (Hamming q >= 3, Lee): two rows packed in each lane.
// transform_tma.cu has the ternary instances and the dispatch,
// transform_first_q.cu the other axis sizes and Lee.
#pragma once
#include "tma_group.cuh"

namespace cc {

// src 0 the cnt predicate, 1 the code; axis kind; KK axes; R1 layers
typedef void (*FirstFn)(const TmaArgs);
struct RowsEntry { int src, kind, kk, r1; FirstFn fn; };
// the instances of transform_first_q.cu
const RowsEntry *rows_table_q(int *n);

namespace {

// Axes 0..KK-1, T0 = Q^KK words a row at inner stride 1.  A tile is TWO
// consecutive rows, and the 32-bit lane of row position m carries row 2t in
// its low half and row 2t+1 in its high half.  The recurrences are adds only,
// every partial sum part of a layer value and so below 2^16 by the planner's
// 16-bit bound, and one add serves both rows.  Rounds of BM axes (register
// blocks of Q^BM words) run on one shared buffer of R1 x T0 lanes: the first
// round takes the highest axes and reads the cnt predicate (or the code
// counts) with consecutive threads on consecutive words; the last takes those
// below them and stores both rows' u16 layers at the plan's row pitch (the
// padded layout, or T0); the low axes run in between.  No waits: plain loads,
// one CTA buffer, a barrier between rounds.
//
// Bound by the rounds' shared-memory traffic: H3(16,4)'s axes 0..6 take 164 us
// in a recount and 176 in a gain (183 and 190 with every layer in every round
// and 4-byte copies out), where their bytes alone would take 66 and 79; Lee
// 7^8's axes 0..3 take 28.5 us (31; the register kernel 65).
//
// Axes a round: two for Q = 3 (9-word blocks), and for Q = 4 up to four
// layers (64 registers); one otherwise.
template <int C, int R1>
struct RowAxes {
  static constexpr int Q = axis_size(C);
  static constexpr int v = Q == 3 || (Q == 4 && R1 <= 4) ? 2 : 1;
};
template <int KK, int BM, int I>
struct RowRound {
  static_assert(KK > BM, "at least two rounds");
  static constexpr int N = (KK + BM - 1) / BM;
  static constexpr int LOW = KK > 2 * BM ? KK - 2 * BM : 0;   // middle axes
  static constexpr int A = I == 0 ? KK - BM : I == N - 1 ? LOW : BM * (I - 1);
  static constexpr int B = I == 0 ? BM : I == N - 1 ? KK - BM - LOW
                           : (LOW - A < BM ? LOW - A : BM);
  // axes applied by the rounds before this one
  static constexpr int DONE = I == 0 ? 0 : I == N - 1 ? BM + LOW
                              : BM + BM * (I - 1);
};
// Distance layers that can be nonzero after `axes` axes of kind C: a Hamming
// axis adds at most 1 to the distance, a Lee axis Q / 2.  The early rounds
// neither write nor read the others.
template <int C, int R1>
__host__ __device__ constexpr int live_after(int axes) {
  const int reach = axes * (axis_lee(C) ? axis_size(C) / 2 : 1);
  return reach + 1 < R1 ? reach + 1 : R1;
}

template <int C, int KK, int R1, int SRC, int I>
__device__ __forceinline__ void rows_round(uint32_t *work, const TmaArgs &a,
                                           long long r0, bool two, bool wide,
                                           uint32_t plo, uint32_t pspan) {
  constexpr int Q = axis_size(C);
  using TR = RowRound<KK, RowAxes<C, R1>::v, I>;
  constexpr int A = TR::A, B = TR::B;
  constexpr int T0 = P<axis_size(C), KK>::v;
  constexpr int WS = (T0 + 31) / 32 * 32;
  constexpr int QA = P<Q, A>::v, QB = P<Q, B>::v;
  constexpr bool FIRST = I == 0, LAST = I == TR::N - 1;
  constexpr int NB = T0 / QB;
  constexpr int LIN = live_after<C, R1>(TR::DONE);
  constexpr int LOUT = live_after<C, R1>(TR::DONE + B);
  for (int blk = threadIdx.x; blk < NB; blk += blockDim.x) {
    const int pb = blk % QA + (blk / QA) * (QA * QB);
    uint32_t v[R1][QB];
    if (FIRST) {
#pragma unroll
      for (int e = 0; e < QB; e++) {
        const int m = pb + e * QA;
        if (SRC == 0) {                       // the cnt predicate, two rows
          const uint16_t *c = a.cnt_in + r0 * T0 + m;
          const uint32_t lo = ((uint32_t)__ldcs(c) - plo) <= pspan;
          const uint32_t hi =
              two ? (((uint32_t)__ldcs(c + T0) - plo) <= pspan) : 0u;
          v[0][e] = lo | (hi << 16);
        } else {                              // code counts, staged
          v[0][e] = work[m];
        }
#pragma unroll
        for (int d = 1; d < R1; d++) v[d][e] = 0;
      }
    } else {
#pragma unroll
      for (int d = 0; d < R1; d++)
#pragma unroll
        for (int e = 0; e < QB; e++)
          v[d][e] = d < LIN ? work[d * WS + pb + e * QA] : 0u;
    }
    Axes<C, R1, B, 0>::run(v);
    if (!LAST) {
#pragma unroll
      for (int d = 0; d < LOUT; d++)
#pragma unroll
        for (int e = 0; e < QB; e++) work[d * WS + pb + e * QA] = v[d][e];
      continue;
    }
    if (wide) {                 // back to the buffer; rows_copy_out stores
#pragma unroll
      for (int d = 0; d < R1; d++)
#pragma unroll
        for (int e = 0; e < QB; e++) work[d * WS + pb + e * QA] = v[d][e];
      continue;
    }
    const long long x0 = r0 * a.pitch + pb;
#pragma unroll
    for (int d = 0; d < R1; d++) {
      if (d >= a.lout) break;
      uint16_t *q = a.layers16 + d * a.plane + x0;
#pragma unroll
      for (int e = 0; e < QB; e++) {
        __stcs(q + e * QA, (uint16_t)(v[d][e] & 0xFFFFu));
        if (two) __stcs(q + a.pitch + e * QA, (uint16_t)(v[d][e] >> 16));
      }
    }
  }
}

template <int C, int KK, int R1, int SRC, int I, int N>
struct RowRounds {
  static __device__ __forceinline__ void run(uint32_t *work,
                                             const TmaArgs &a, long long r0,
                                             bool two, bool wide,
                                             uint32_t plo, uint32_t pspan) {
    rows_round<C, KK, R1, SRC, I>(work, a, r0, two, wide, plo, pspan);
    __syncthreads();
    RowRounds<C, KK, R1, SRC, I + 1, N>::run(work, a, r0, two, wide, plo,
                                           pspan);
  }
};
template <int C, int KK, int R1, int SRC, int N>
struct RowRounds<C, KK, R1, SRC, N, N> {
  static __device__ __forceinline__ void run(uint32_t *, const TmaArgs &,
                                             long long, bool, bool, uint32_t,
                                             uint32_t) {}
};

// Wide stores of a tile's layers (a row pitch that is a multiple of 8 words
// and at least T0 rounded up to 8): each thread takes 4 positions of one layer
// from the buffer (a 16-byte shared load of packed lanes, consecutive across
// the warp, so free of bank conflicts) and stores each row's 4 words with one
// 8-byte store.  Positions from T0 to the next multiple of 4 land in the
// row's padding.
template <int C, int KK, int R1>
__device__ __forceinline__ void rows_copy_out(const uint32_t *work,
                                              const TmaArgs &a, long long r0,
                                              bool two) {
  constexpr int T0 = P<axis_size(C), KK>::v;
  constexpr int WS = (T0 + 31) / 32 * 32;
  constexpr int C4 = (T0 + 3) / 4;
  static_assert(C4 * 4 <= WS, "the buffer covers the rounded row");
  const int n = a.lout * C4;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int d = i / C4, m = (i - d * C4) * 4;
    const uint4 x = *reinterpret_cast<const uint4 *>(work + d * WS + m);
    uint16_t *q = a.layers16 + d * a.plane + r0 * a.pitch + m;
    __stcs(reinterpret_cast<uint2 *>(q),
           make_uint2(__byte_perm(x.x, x.y, 0x5410),
                      __byte_perm(x.z, x.w, 0x5410)));
    if (two)
      __stcs(reinterpret_cast<uint2 *>(q + a.pitch),
             make_uint2(__byte_perm(x.x, x.y, 0x7632),
                        __byte_perm(x.z, x.w, 0x7632)));
  }
}

// SRC 0: the cnt predicate (gain, loss); 1: the sorted code (a recount),
// the tile's slice [bounds[t], bounds[t+1]) counted into layer 0 first
template <int C, int KK, int R1, int SRC>
__global__ void __launch_bounds__(512)
rows_first(const TmaArgs a) {
  extern __shared__ __align__(16) uint8_t dyn[];
  constexpr int T0 = P<axis_size(C), KK>::v;
  constexpr int NR = RowRound<KK, RowAxes<C, R1>::v, 0>::N;
  uint32_t *work = reinterpret_cast<uint32_t *>(dyn);
  const uint32_t plo = a.pmode == kPredDef ? 0u
                       : a.pmode == kPredCrit ? 1u : (uint32_t)a.ptarget;
  const uint32_t phi = a.pmode == kPredDef ? (uint32_t)(a.mu - 1)
                       : a.pmode == kPredCrit ? (uint32_t)a.mu
                       : (uint32_t)a.ptarget;
  const uint32_t pspan = phi - plo;
  constexpr int C8 = (T0 + 7) / 8;
  const bool wide = (a.pitch & 7) == 0 && a.pitch >= C8 * 8 &&
                    (a.plane & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(a.layers16) & 15) == 0;
  for (long long t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
    const long long r0 = 2 * t;
    const bool two = r0 + 1 < a.rows;
    if (SRC == 1) {
      for (int i = threadIdx.x; i < T0; i += blockDim.x) work[i] = 0;
      __syncthreads();
      const long long lo = a.code_bounds[t], hi = a.code_bounds[t + 1];
      const long long x0 = r0 * T0;
      for (long long c = lo + threadIdx.x; c < hi; c += blockDim.x) {
        const long long w = a.code[c] - x0;
        if (w < 0 || w >= 2 * T0) continue;   // outside this tile's rows
        const int h = w >= T0 ? 1 : 0;
        atomicAdd(&work[(int)w - h * T0], 1u << (16 * h));
      }
      __syncthreads();
    }
    RowRounds<C, KK, R1, SRC, 0, NR>::run(work, a, r0, two, wide, plo, pspan);
    if (wide) {
      rows_copy_out<C, KK, R1>(work, a, r0, two);
      __syncthreads();                  // the buffer is the next tile's
    }
  }
}

}  // namespace
}  // namespace cc
