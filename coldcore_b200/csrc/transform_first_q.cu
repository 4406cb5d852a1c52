// transform_first_q.cu — the first groups over row pairs of Hamming axes of 4
// to 6, Lee axes of 4 to 7 and ternary cells of R = 2 (rows_first.cuh): rows
// of up to 4,096 words, so that two to four CTAs of R1 x T0 lanes share an SM.
#include "rows_first.cuh"

namespace cc {
namespace {

#define RF1(C, KK, R1) {0, C, KK, R1, rows_first<C, KK, R1, 0>},            \
                       {1, C, KK, R1, rows_first<C, KK, R1, 1>}
#define RF(C, KK) RF1(C, KK, 2), RF1(C, KK, 3), RF1(C, KK, 4), RF1(C, KK, 5)
const RowsEntry kRowsQ[] = {
    RF1(3, 7, 3), RF1(3, 8, 3),
    RF(4, 5), RF(4, 6), RF(5, 4), RF(5, 5), RF(6, 4),
    RF(32 + 4, 5), RF(32 + 4, 6), RF(32 + 5, 4), RF(32 + 5, 5),
    RF(32 + 6, 4), RF(32 + 7, 3), RF(32 + 7, 4),
};
#undef RF
#undef RF1

}  // namespace

const RowsEntry *rows_table_q(int *n) {
  if (n) *n = (int)(sizeof(kRowsQ) / sizeof(kRowsQ[0]));
  return kRowsQ;
}

}  // namespace cc
