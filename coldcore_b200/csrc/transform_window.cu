// transform_window.cu — window-sum passes over one or two axes of any width
// (torus / grid).
//
// Recurrence of the reference's torus and open-grid plugins
// (coldcore src/plugins/covering/dctcore_torus.cuh:1-12,
//  dctcore_grid.cuh:1-30): newA[a] = sum of A over the circular (torus) or
// clamped (grid) window [a-R, a+R] along one axis.  The reference keeps the
// fibre in a 16-entry register array (axes <= 16); this pass has no width
// limit (the king 2048x2048 torus), runs out of place, and maps one thread
// to one output word so that a warp's 2R+1 reads and its write are 128-byte
// coalesced along the contiguous inner index; the 2R neighbours of a word
// are re-read from L1/L2, not HBM.
#include "engine.h"

namespace cc {

// The word x = (o * q + a) * stride + i of the pass's axis position a:
// with the space below 2^31 words the digit comes from two 32-bit
// divisions (a 64-bit division costs several times more instructions, and
// the pass is issue-bound: one read of each of 2R+1 neighbours a word).
template <bool GRID, int SRC16, int DST16, bool I32>
__global__ void __launch_bounds__(256) window_axis(const WindowArgs w) {
  const long long gs = (long long)gridDim.x * blockDim.x;
  for (long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
       x < w.space; x += gs) {
    int a;
    long long base;
    if (I32) {
      const unsigned xs = (unsigned)x, st = (unsigned)w.stride;
      const unsigned hi = xs / st;
      a = (int)(hi % (unsigned)w.q);
      base = (long long)(xs - (unsigned)a * st);
    } else {
      const long long hi = x / w.stride;
      a = (int)(hi % w.q);
      base = x - (long long)a * w.stride;
    }
    int lo = a - w.R, up = a + w.R;
    if (GRID) { if (lo < 0) lo = 0; if (up > w.q - 1) up = w.q - 1; }
    int32_t s = 0;
    for (int b = lo; b <= up; b++) {
      int bb = b;
      if (!GRID) { if (bb < 0) bb += w.q; else if (bb >= w.q) bb -= w.q; }
      const long long y = base + (long long)bb * w.stride;
      if (SRC16) s += cnt_pred(w.pmode, (int)w.src16[y], w.ptarget, w.mu);
      else s += w.src32[y];
    }
    if (DST16) w.dst16[x] = (uint16_t)(s > 65535 ? 65535 : s);
    else w.dst32[x] = s;
  }
}

// Two consecutive axes in one pass.  The words of the lower axis and below are
// a row of L = stride * q words, in which the lower axis' window is the words
// k * stride away, wrapped at L (torus) or cut at its ends (grid).  A thread
// takes one position of a row and walks `rows` steps of the upper axis,
// keeping the row sums of the 2R + 1 rows of its window in registers: a word
// costs 2R + 1 reads (L1 serves all but one), one row sum and one write, and
// the pass between the axes is gone.  King 2048 x 2048: 43 us for two passes,
// 14 us for one.
template <bool GRID, int SRC16, int DST16, int R>
__global__ void __launch_bounds__(256)
window_pair(const WindowArgs w, int L, int rows, long long nthreads) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nthreads) return;
  const int nseg = (w.q2 + rows - 1) / rows;
  const int x = (int)(t % L);
  const long long rest = t / L;
  const int b0 = (int)(rest % nseg) * rows;
  const int b1 = min(w.q2, b0 + rows);
  const long long base = rest / nseg * ((long long)L * w.q2);
  // predicate as a range: lo <= cnt <= hi
  const int plo = w.pmode == kPredDef ? 0 : w.pmode == kPredCrit ? 1
                  : w.ptarget;
  const int phi = w.pmode == kPredDef ? w.mu - 1 : w.pmode == kPredCrit
                  ? w.mu : w.ptarget;
  const unsigned pspan = (unsigned)(phi - plo);
  const int st = (int)w.stride;
  int xo[2 * R + 1];
  bool in[2 * R + 1];
#pragma unroll
  for (int k = -R; k <= R; k++) {
    int y = x + k * st;
    in[k + R] = !GRID || (y >= 0 && y < L);
    if (!GRID) { if (y < 0) y += L; else if (y >= L) y -= L; }
    xo[k + R] = y;
  }
  auto row = [&](int b) -> int32_t {
    if (GRID) { if (b < 0 || b >= w.q2) return 0; }
    else { if (b < 0) b += w.q2; else if (b >= w.q2) b -= w.q2; }
    const long long p = base + (long long)b * L;
    int32_t s = 0;
#pragma unroll
    for (int k = 0; k < 2 * R + 1; k++)
      if (in[k]) {
        if (SRC16)
          s += (unsigned)((int)__ldg(w.src16 + p + xo[k]) - plo) <= pspan;
        else
          s += __ldg(w.src32 + p + xo[k]);
      }
    return s;
  };
  int32_t h[2 * R + 1];
#pragma unroll
  for (int k = 0; k < 2 * R; k++) h[k + 1] = row(b0 - R + k);
#pragma unroll 2
  for (int b = b0; b < b1; b++) {
#pragma unroll
    for (int k = 0; k < 2 * R; k++) h[k] = h[k + 1];
    h[2 * R] = row(b + R);
    int32_t s = 0;
#pragma unroll
    for (int k = 0; k <= 2 * R; k++) s += h[k];
    const long long y = base + (long long)b * L + x;
    if (DST16) w.dst16[y] = (uint16_t)(s > 65535 ? 65535 : s);
    else w.dst32[y] = s;
  }
}

// the pair form: rows that fit 32-bit positions, windows that fit registers
bool window_pair_ok(long long stride, int q, int R) {
  return R <= kWindowPairMaxR && stride * q < (1LL << 30);
}

template <int R>
static int launch_pair(const WindowArgs &w, cudaStream_t s) {
  const int L = (int)(w.stride * w.q);
  // rows a thread walks: few enough for two waves of threads, 4 to 32
  const long long want = w.space / ((long long)sm_count() * 2048);
  const int rows = (int)(want < 4 ? 4 : want > 32 ? 32 : want);
  const long long nseg = (w.q2 + rows - 1) / rows;
  const long long threads = w.space / w.q2 * nseg;
  const long long nb = (threads + 255) / 256;
#define WP(G, A, B)                                                         \
  window_pair<G, A, B, R><<<(unsigned)nb, 256, 0, s>>>(w, L, rows, threads)
  const bool s16 = w.src16 != nullptr, d16 = w.dst16 != nullptr;
  if (w.grid) {
    if (s16 && d16) WP(true, 1, 1); else if (s16) WP(true, 1, 0);
    else if (d16) WP(true, 0, 1); else WP(true, 0, 0);
  } else {
    if (s16 && d16) WP(false, 1, 1); else if (s16) WP(false, 1, 0);
    else if (d16) WP(false, 0, 1); else WP(false, 0, 0);
  }
#undef WP
  CC_CK(cudaGetLastError());
  return 0;
}

int launch_window(const WindowArgs &w, cudaStream_t s) {
  if (w.q2) {
    switch (w.R) {
      case 1: return launch_pair<1>(w, s);
      case 2: return launch_pair<2>(w, s);
      case 3: return launch_pair<3>(w, s);
      default: return -2;
    }
  }
  const long long nblk = (w.space + 255) / 256;
  long long nb = nblk;
  const long long cap = (long long)sm_count() * 16;
  if (nb > cap) nb = cap;
  if (nb < 1) nb = 1;
  nb = grid_knob((int)nb, nblk);
  const bool s16 = w.src16 != nullptr, d16 = w.dst16 != nullptr;
  const bool i32 = w.space < (1LL << 31);
#define WL(G, A, B)                                                         \
  (i32 ? window_axis<G, A, B, true><<<(int)nb, 256, 0, s>>>(w)              \
       : window_axis<G, A, B, false><<<(int)nb, 256, 0, s>>>(w))
  if (w.grid) {
    if (s16 && d16) WL(true, 1, 1); else if (s16) WL(true, 1, 0);
    else if (d16) WL(true, 0, 1); else WL(true, 0, 0);
  } else {
    if (s16 && d16) WL(false, 1, 1); else if (s16) WL(false, 1, 0);
    else if (d16) WL(false, 0, 1); else WL(false, 0, 0);
  }
#undef WL
  CC_CK(cudaGetLastError());
  return 0;
}

}  // namespace cc
