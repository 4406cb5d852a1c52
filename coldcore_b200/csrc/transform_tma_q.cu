// transform_tma_q.cu — the streamed groups of Hamming axes of 4 to 6, Lee axes
// of 4 to 7 and ternary cells of R = 2 (tma_group.cuh), all in a padded plan's
// layout: OUT 0 writes layers, 3 the map and 4 the cnt at their canonical
// index.  Lee 7^8's two strided launches take 16 us each, 45 and 41 with the
// register kernels.
//
// A group takes as many axes as keep its tile's middle extent within 256, the
// tensor map's box limit, and two stages within shared memory; tiles of up to
// 64 middle positions are 64 words wide, larger ones 32.
#include "tma_group.cuh"

namespace cc {
namespace {

#define TQ1(C, K, R1, L)                                                    \
  {C, K, R1, L, 0, tma_group<C, K, R1, L, 0>},                              \
  {C, K, R1, L, 3, tma_group<C, K, R1, L, 3>},                              \
  {C, K, R1, L, 4, tma_group<C, K, R1, L, 4>}
#define TQ(C, K, L)                                                         \
  TQ1(C, K, 2, L), TQ1(C, K, 3, L), TQ1(C, K, 4, L), TQ1(C, K, 5, L)
const TmaEntry kTmaQ[] = {
    // ternary cells of three layers (four and five: transform_tma.cu)
    TQ1(3, 3, 3, 32), TQ1(3, 4, 3, 32), TQ1(3, 5, 3, 16),
    TQ(4, 1, 32), TQ(4, 2, 32), TQ(4, 3, 32), TQ(4, 4, 16),
    TQ(5, 1, 32), TQ(5, 2, 32), TQ(5, 3, 16),
    TQ(6, 1, 32), TQ(6, 2, 32), TQ(6, 3, 16),
    TQ(32 + 4, 1, 32), TQ(32 + 4, 2, 32), TQ(32 + 4, 3, 32),
    TQ(32 + 4, 4, 16),
    TQ(32 + 5, 1, 32), TQ(32 + 5, 2, 32), TQ(32 + 5, 3, 16),
    TQ(32 + 6, 1, 32), TQ(32 + 6, 2, 32), TQ(32 + 6, 3, 16),
    TQ(32 + 7, 1, 32), TQ(32 + 7, 2, 32),
};
#undef TQ
#undef TQ1

}  // namespace

const TmaEntry *tma_table_q(int *n) {
  if (n) *n = (int)(sizeof(kTmaQ) / sizeof(kTmaQ[0]));
  return kTmaQ;
}

}  // namespace cc
