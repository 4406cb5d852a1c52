// batch_groups.cu — the batched engine's small cells on the register-blocked
// group kernels: one persistent launch per kernel over a table of
// (pass, tile) work items of every cell that kernel serves.
//
// The runtime-size tiles of batch_kernel (transform_group.cu) spend their
// time on divisions, 32-bit shared words and local arrays: 6.8 ms for a step
// of 256 cells of 10^3..10^5 words, whose shared-memory traffic alone would
// take 0.1 ms.  The same tiles on the kernels of group_rounds.cuh keep every
// size but the tile's a compile-time constant.  Cells share a launch when
// they share the kernel (axis operation, axis size, layers), so a campaign
// of uneven cells is some twenty concurrent launches on forked streams.
//
// Items are claimed in table order, level by level, and wait only for items
// before them in the same table, so the schedule cannot deadlock; the wait
// is bounded as in batch_kernel.  A cell whose passes all are single tiles
// is one chained item: its recount, gain and loss run back to back in one
// CTA.  The passes are read through a const restrict pointer: they do not
// change during a launch, so their fields stay in registers.
#include "engine.h"
#include "group_rounds.cuh"

namespace cc {

constexpr int kBatchThreads = 256;
constexpr long long kItemSpinLimit = 1LL << 22;

template <int OP, int Q, int R1, int BM>
__global__ void __launch_bounds__(kBatchThreads)
batch_group_kernel(const GroupArgs *__restrict__ passes,
                   const int *__restrict__ pass_dep,
                   const unsigned *__restrict__ pass_need,
                   const int4 *__restrict__ items, long long nitems,
                   unsigned *done, unsigned long long *next, int *err,
                   const int *__restrict__ pass_cell,
                   const int *__restrict__ active) {
  extern __shared__ int32_t sm[];
  __shared__ long long s_it;
  __shared__ int s_bad;
  for (;;) {
    if (threadIdx.x == 0) {
      s_it = (long long)atomicAdd(next, 1ULL);
      s_bad = 0;
    }
    __syncthreads();
    const long long it = s_it;
    if (it >= nitems) return;
    const int4 item = items[it];
    const int chain = item.w > 1 ? item.w : 1;
    for (int c = 0; c < chain; c++) {
      const int pass = item.x + c;
      if (active && !active[pass_cell[pass]]) break;
      if (threadIdx.x == 0) {
        const int dep = pass_dep[pass];
        if (dep >= 0) {
          const unsigned need = pass_need[dep];
          long long spins = 0;
          while (*(volatile unsigned *)(done + dep) < need) {
            if (++spins > kItemSpinLimit) {
              atomicExch(err, 1);
              s_bad = 1;
              break;
            }
            __nanosleep(128);
          }
          __threadfence();
        }
      }
      __syncthreads();
      if (s_bad) return;
      const GroupArgs &g = passes[pass];
      long long acc = 0;                // epilogue reduction (red_mode)
      long long *racc = g.red_mode && g.dst != kDstLayers ? &acc : nullptr;
      for (int t = 0; t < item.z; t++)
        group_tile<OP, Q, R1, BM, true>(g, sm, (long long)item.y + t, racc);
      if (racc) red_flush(g, acc);
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(done + pass, (unsigned)item.z);
      }
    }
    __syncthreads();
  }
}

typedef void (*BatchGroupFn)(const GroupArgs *, const int *, const unsigned *,
                             const int4 *, long long, unsigned *,
                             unsigned long long *, int *, const int *,
                             const int *);
#define KE(OP, Q, R1, BM) batch_group_kernel<OP, Q, R1, BM>,
static const BatchGroupFn kBatchTable[] = {CC_GROUP_KERNELS(KE)};
#undef KE
static const int kBatchTableLen = sizeof(kBatchTable) / sizeof(kBatchTable[0]);
static_assert(sizeof(kBatchTable) / sizeof(kBatchTable[0]) <= 64,
              "the shared-memory opt-in cache holds 64 kernels");

int batch_groups_grid(int kernel, size_t smem) {
  if (kernel < 0 || kernel >= kBatchTableLen) return 1;
  static size_t attr[64];
  const void *fn = (const void *)kBatchTable[kernel];
  if (smem > 48 * 1024 && smem > attr[kernel] &&
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) == cudaSuccess)
    attr[kernel] = smem;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kBatchThreads,
                                                smem);
  if (per_sm < 1) per_sm = 1;
  return per_sm * sm_count();
}

int launch_batch_groups(const BatchLaunch &b, cudaStream_t s) {
  if (b.kernel < 0 || b.kernel >= kBatchTableLen) return -2;
  if (b.nitems <= 0) return 0;
  kBatchTable[b.kernel]<<<b.grid, kBatchThreads, b.smem, s>>>(
      b.passes, b.dep, b.need, b.items, b.nitems, b.done, b.next, b.err,
      b.pass_cell, b.active);
  CC_CK(cudaGetLastError());
  return 0;
}

}  // namespace cc
