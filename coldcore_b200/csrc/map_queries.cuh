// map_queries.cuh — the maximum, the histogram and the extraction of an int32
// map: 16-byte loads, four in flight a thread, warp shuffles or warp-claimed
// slots, and the result straight to the host (RedOut).  Shared by the two
// engines (reduce.cu and sparse/sparse_abi.cu).
#pragma once
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

#include "query_out.h"

namespace cc {

// blocks of a streaming pass: 1,536 threads an SM in blocks of 512 (every
// block ends with an add to one ticket word: 1,184 blocks of 256 took 2 us
// for that on a map that is read in 5)
constexpr int kQueryThreads = 512;
inline int query_blocks(long long nvec, int sms) {
  const long long b = (nvec + kQueryThreads - 1) / kQueryThreads;
  const long long cap = (long long)sms * 3;
  return (int)(b < 1 ? 1 : b < cap ? b : cap);
}

__device__ __forceinline__ long long warp_sum(long long v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// True in every thread of the last block of the launch to get here, with
// every block's earlier atomics visible to it.
__device__ __forceinline__ bool last_block(const RedOut &r) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(r.ticket, 1u) + 1 == gridDim.x;
    if (last) {
      *r.ticket = 0;
      __threadfence();
    }
  }
  __syncthreads();
  return last != 0;
}

__global__ void __launch_bounds__(kQueryThreads)
k_max(const int32_t *A, long long N, long long *out, RedOut r) {
  const long long nvec = N >> 2;
  const long long gs = (long long)gridDim.x * blockDim.x;
  const int4 *v = reinterpret_cast<const int4 *>(A);
  int32_t m = 0;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * gs < nvec; i += 4 * gs) {
    int4 q[4];
#pragma unroll
    for (int u = 0; u < 4; u++) q[u] = v[i + u * gs];
#pragma unroll
    for (int u = 0; u < 4; u++)
      m = max(m, max(max(q[u].x, q[u].y), max(q[u].z, q[u].w)));
  }
  for (; i < nvec; i += gs) {
    const int4 q = v[i];
    m = max(m, max(max(q.x, q.y), max(q.z, q.w)));
  }
  if (blockIdx.x == 0 && threadIdx.x < (N & 3))
    m = max(m, A[nvec * 4 + threadIdx.x]);
  for (int o = 16; o > 0; o >>= 1)
    m = max(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax((int *)out, m);
  if (r.host && last_block(r) && threadIdx.x == 0)
    *r.host = (long long)atomicExch((unsigned long long *)out, 0ULL);
}

// Bin of a positive value v <= vmax: (v - 1) * nbins / vmax.  With vmax *
// nbins below 2^31 the division is a multiplication by m = ceil(2^(31 + l) /
// vmax), l = ceil(log2(vmax)), exact for 31-bit numerators (with a
// 64-bit division a value the histogram of 67 M words took 139 us, now 56;
// reading it takes 41).
struct BinArgs {
  int nbins;
  int32_t vmax;
  uint32_t m;                   // 0: divide
  int shift;
};

inline BinArgs bin_args(int nbins, int32_t vmax) {
  BinArgs b{nbins, vmax, 0, 0};
  if ((long long)vmax * nbins < (1LL << 31) && vmax > 1) {
    int l = 0;
    while ((1LL << l) < vmax) l++;
    b.m = (uint32_t)(((1ULL << (31 + l)) + vmax - 1) / vmax);
    b.shift = l - 1;
  }
  return b;
}

__device__ __forceinline__ void hist_one(int32_t v, const BinArgs &b,
                                         int32_t *sh) {
  if (v <= 0) return;
  int k = b.nbins - 1;
  if (v <= b.vmax)
    k = b.m ? (int)(__umulhi((uint32_t)(v - 1) * (uint32_t)b.nbins, b.m) >>
                    b.shift)
            : (int)((long long)(v - 1) * b.nbins / b.vmax);
  atomicAdd(&sh[k], 1);
}

__global__ void __launch_bounds__(kQueryThreads)
k_hist(const int32_t *A, long long N, const BinArgs b, int32_t *hist,
       RedOut r) {
  extern __shared__ int32_t sh[];
  for (int i = threadIdx.x; i < b.nbins; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const long long nvec = N >> 2;
  const long long gs = (long long)gridDim.x * blockDim.x;
  const int4 *v = reinterpret_cast<const int4 *>(A);
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * gs < nvec; i += 4 * gs) {
    int4 q[4];
#pragma unroll
    for (int u = 0; u < 4; u++) q[u] = v[i + u * gs];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      hist_one(q[u].x, b, sh);
      hist_one(q[u].y, b, sh);
      hist_one(q[u].z, b, sh);
      hist_one(q[u].w, b, sh);
    }
  }
  for (; i < nvec; i += gs) {
    const int4 q = v[i];
    hist_one(q.x, b, sh);
    hist_one(q.y, b, sh);
    hist_one(q.z, b, sh);
    hist_one(q.w, b, sh);
  }
  if (blockIdx.x == 0 && threadIdx.x < (N & 3))
    hist_one(A[nvec * 4 + threadIdx.x], b, sh);
  __syncthreads();
  for (int k = threadIdx.x; k < b.nbins; k += blockDim.x)
    if (sh[k]) atomicAdd(&hist[k], sh[k]);
  if (r.host && last_block(r)) {
    int32_t *out = reinterpret_cast<int32_t *>(r.host);
    for (int k = threadIdx.x; k < b.nbins; k += blockDim.x)
      out[k] = atomicExch(&hist[k], 0);
  }
}

// The words of q[0..NV) (vectors at word index x[u]) that reach thr, into
// output slots claimed with one atomic for the warp's whole batch; a warp
// that has seen the output full only counts.
template <typename IDX, int NV>
__device__ __forceinline__ void extract_batch(
    const int4 (&q)[NV], const long long (&x)[NV], int32_t thr, IDX *oidx,
    int32_t *oval, long long cap, unsigned long long *ctr, bool &full,
    long long &tally) {
  unsigned hits = 0;                            // bit 4 u + h: word h of q[u]
#pragma unroll
  for (int u = 0; u < NV; u++)
    if (x[u] >= 0)
      hits |= ((unsigned)(q[u].x >= thr) | (unsigned)(q[u].y >= thr) << 1 |
               (unsigned)(q[u].z >= thr) << 2 | (unsigned)(q[u].w >= thr) << 3)
              << (4 * u);
  if (!__any_sync(0xffffffffu, hits)) return;
  const int n = __popc(hits), lane = threadIdx.x & 31;
  if (full) {
    tally += n;
    return;
  }
  int before = n;                               // inclusive scan
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += v;
  }
  unsigned long long base = 0;
  if (lane == 31) base = atomicAdd(ctr, (unsigned long long)before);
  base = __shfl_sync(0xffffffffu, base, 31);
  full = (long long)base >= cap;
  long long s = (long long)base + before - n;
#pragma unroll
  for (int u = 0; u < NV; u++) {
    const int32_t e[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
    for (int h = 0; h < 4; h++)
      if (hits >> (4 * u + h) & 1) {
        if (s < cap) { oidx[s] = (IDX)(x[u] + h); oval[s] = e[h]; }
        s++;
      }
  }
}

template <typename IDX>
__global__ void __launch_bounds__(kQueryThreads)
k_extract(const int32_t *A, long long N, int32_t thr, IDX *oidx,
          int32_t *oval, long long cap, unsigned long long *ctr, RedOut r) {
  const long long nvec = N >> 2;                // whole vectors
  const long long gs = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int4 *v = reinterpret_cast<const int4 *>(A);
  const long long trips = (nvec + gs - 1) / gs; // uniform per warp
  long long tally = 0;
  bool full = false;
  for (long long k = 0; k < trips; k += 4) {
    int4 q[4];
    long long x[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const long long i = t0 + (k + u) * gs;
      x[u] = i < nvec ? 4 * i : -1;
      q[u] = i < nvec ? v[i] : make_int4(0, 0, 0, 0);
    }
    extract_batch(q, x, thr, oidx, oval, cap, ctr, full, tally);
  }
  if (blockIdx.x == 0 && threadIdx.x < 32) {    // the last, partial vector
    const long long w = nvec * 4 + threadIdx.x;
    if (w < N && A[w] >= thr) {
      const long long s = (long long)atomicAdd(ctr, 1ULL);
      if (s < cap) { oidx[s] = (IDX)w; oval[s] = A[w]; }
    }
  }
  tally = warp_sum(tally);
  if ((threadIdx.x & 31) == 0 && tally)
    atomicAdd(ctr, (unsigned long long)tally);
  if (r.host && last_block(r) && threadIdx.x == 0)
    *r.host = (long long)atomicExch(ctr, 0ULL);
}

}  // namespace cc
