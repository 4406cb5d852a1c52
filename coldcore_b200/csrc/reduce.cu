// reduce.cu — whole-field reductions and map queries.
//
// Semantics of the reference's queries (coldcore
// src/plugins/covering/dctcore_core.cuh:284-371, dctcore_fast.cuh:191-327,
// dctcore_mu.cuh:53-73): sum [cnt == t] or sum max(0, mu - cnt) with int64
// accumulation; the map maximum (0 when every value is <= 0); a histogram of
// positive values v at bin (v-1)*nbins/vmax clipped to the last bin; the
// unordered extraction of every map value >= thr, storing at most `cap`
// entries but counting all of them.
//
// These are HBM streaming passes: 16-byte loads (8 counters or 4 map values
// per load), four in flight a thread, warp shuffles then one atomic per
// warp.  A query that returns to the host (RedOut) is ONE launch: the last
// block to finish writes the result to mapped host memory and clears the
// accumulators for the next query, in place of a clearing, a launch and a
// copy.
#include "engine.h"
#include "map_queries.cuh"

namespace cc {

static int stream_blocks(long long nvec) {
  return query_blocks(nvec, sm_count());
}

__device__ __forceinline__ long long cnt_term(int mode, int c, int target,
                                              int mu) {
  if (mode == kPredDef) { int d = mu - c; return d > 0 ? d : 0; }
  return c == target;
}

// mode kPredEq: sum [cnt == target]; kPredDef: sum max(0, mu - cnt)
__global__ void __launch_bounds__(kQueryThreads)
k_cnt_reduce(const uint16_t *cnt, long long N, int mode, int target, int mu,
             unsigned long long *out, RedOut r) {
  const long long nvec = N >> 3;
  const long long gs = (long long)gridDim.x * blockDim.x;
  const uint4 *v = reinterpret_cast<const uint4 *>(cnt);
  long long acc = 0;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  // four independent 16-byte loads in flight per thread, then the rest
  for (; i + 3 * gs < nvec; i += 4 * gs) {
    uint4 q[4];
#pragma unroll
    for (int u = 0; u < 4; u++) q[u] = v[i + u * gs];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t w4[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
      for (int h = 0; h < 8; h++)
        acc += cnt_term(mode,
                        (int)((w4[h >> 1] >> (16 * (h & 1))) & 0xFFFFu),
                        target, mu);
    }
  }
  for (; i < nvec; i += gs) {
    const uint4 q = v[i];
    const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int h = 0; h < 8; h++)
      acc += cnt_term(mode, (int)((w4[h >> 1] >> (16 * (h & 1))) & 0xFFFFu),
                      target, mu);
  }
  if (blockIdx.x == 0 && threadIdx.x < (N & 7))
    acc += cnt_term(mode, (int)cnt[nvec * 8 + threadIdx.x], target, mu);
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0 && acc)
    atomicAdd(out, (unsigned long long)acc);
  if (r.host && last_block(r) && threadIdx.x == 0)
    *r.host = (long long)atomicExch(out, 0ULL);
}

__global__ void k_read_at(const int32_t *A, const long long *idx, int k,
                          int32_t *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < k) out[i] = A[idx[i]];
}

__global__ void k_scatter(int32_t *A, const long long *idx, long long M) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < M) atomicAdd(&A[idx[i]], 1);
}

int launch_cnt_reduce(const uint16_t *cnt, long long N, int mode, int target,
                      int mu, long long *out, cudaStream_t s, RedOut r) {
  k_cnt_reduce<<<stream_blocks(N >> 3), kQueryThreads, 0, s>>>(
      cnt, N, mode, target, mu, reinterpret_cast<unsigned long long *>(out),
      r);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_max(const int32_t *A, long long N, long long *out,
               cudaStream_t s, RedOut r) {
  k_max<<<stream_blocks(N >> 2), kQueryThreads, 0, s>>>(A, N, out, r);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_hist(const int32_t *A, long long N, int nbins, int32_t vmax,
                int32_t *hist, cudaStream_t s, RedOut r) {
  const BinArgs b = bin_args(nbins, vmax);
  k_hist<<<stream_blocks(N >> 2), kQueryThreads, nbins * 4, s>>>(A, N, b, hist, r);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_extract(const int32_t *A, long long N, int32_t thr, void *oidx,
                   bool wide, int32_t *oval, long long cap, long long *ocount,
                   cudaStream_t s, RedOut r) {
  const int nb = stream_blocks((N + 3) >> 2);
  auto *ctr = reinterpret_cast<unsigned long long *>(ocount);
  if (wide)
    k_extract<int64_t><<<nb, kQueryThreads, 0, s>>>(A, N, thr, (int64_t *)oidx, oval,
                                          cap, ctr, r);
  else
    k_extract<uint32_t><<<nb, kQueryThreads, 0, s>>>(A, N, thr, (uint32_t *)oidx, oval,
                                           cap, ctr, r);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_read_at(const int32_t *A, const long long *idx, int k,
                   int32_t *out, cudaStream_t s) {
  if (k <= 0) return 0;
  k_read_at<<<(k + 255) / 256, 256, 0, s>>>(A, idx, k, out);
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_scatter(int32_t *A, const long long *idx, long long M,
                   cudaStream_t s) {
  if (M <= 0) return 0;
  k_scatter<<<(unsigned)((M + 255) / 256), 256, 0, s>>>(A, idx, M);
  CC_CK(cudaGetLastError());
  return 0;
}

}  // namespace cc
