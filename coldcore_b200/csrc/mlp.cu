// mlp.cu — the learned ruin proposal's scorer: a 32-128-128-1 MLP with
// ReLU hidden layers, trained and evaluated on the GPU by this file's own
// kernels.  BF16 operands, FP32 accumulation: the two hidden-layer GEMMs and
// the three backward GEMMs run on the tensor cores through warp-level
// mma.sync m16n8k16 (bf16 x bf16 -> f32); the 128-wide output layer, the
// loss and the Adam step are FP32 SIMT.
//
// A CTA takes blocks of 64 samples and holds every weight (the whole net is
// 20,865 parameters: W1 and W2 sit in shared memory as bf16).  Forward:
//   h1 = bf16(relu(bf16(x) W1b + b1)), h2 = bf16(relu(h1 W2b + b2)),
//   y = h2 . w3 + b3;
// training loss: binary cross-entropy with logits against t in {0,1},
// averaged over the n samples of the batch; backward (ReLU masks from the
// stored bf16 activations):
//   dy = (sigmoid(y) - t) / n, dw3 = sum dy h2, db3 = sum dy,
//   dz2 = bf16(dy w3 [h2 > 0]), dW2 = h1^T dz2, db2 = sum dz2,
//   dz1 = bf16((dz2 W2b^T) [h1 > 0]), dW1 = bf16(x)^T dz1, db1 = sum dz1;
// per-CTA partial gradients are added into one FP32 gradient vector.
// oracle/mlp_oracle.py restates the same arithmetic in float64 for the
// gradient check.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "../../include/coldcore_b200/plugin.h"
#include "engine.h"

namespace {

constexpr int kIn = 32, kHid = 128, kRows = 64;
// flat parameter vector (fp32 master copy)
constexpr int kW1 = 0, kB1 = kW1 + kIn * kHid, kW2 = kB1 + kHid,
              kB2 = kW2 + kHid * kHid, kW3 = kB2 + kHid, kB3 = kW3 + kHid,
              kParams = kB3 + 1;

// Rows of the shared tiles are padded by 8 bf16 (272 and 80 bytes): the eight
// rows of an 8 x 8 matrix start in different banks, so every ldmatrix is free
// of conflicts.  h2 becomes dz2 and h1 becomes dz1 in place, each after its
// last reader.
constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kLdH = kHid + 8, kLdX = kIn + 8;
struct MlpSmem {
  __nv_bfloat16 w1[kIn * kLdH];      // [in][hid]
  __nv_bfloat16 w2[kHid * kLdH];     // [in][out]
  __nv_bfloat16 x[kRows * kLdX];
  __nv_bfloat16 h1[kRows * kLdH];    // then dz1
  __nv_bfloat16 h2[kRows * kLdH];    // then dz2
  float b1[kHid], b2[kHid], w3[kHid];
  float dy[kRows];
  float b3;
};

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}

// four 8 x 8 matrices; lane l gives the address of row l % 8 of matrix l / 8
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const void *p) {
  asm volatile(
      "ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
      : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const void *p) {
  asm volatile(
      "ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
      : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4],
                                    uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One warp: C[16 x 8 NT] += A[16 x K] B[K x 8 NT], from shared memory.
// TA: A(i, k) is stored [k][i], else [i][k]; TB: B(k, j) is stored [j][k],
// else [k][j].  A and B point at the warp's first row and column.
template <int K, int NT, bool TA, bool TB>
__device__ __forceinline__ void warp_gemm(const __nv_bfloat16 *A, int lda,
                                          const __nv_bfloat16 *B, int ldb,
                                          float (&c)[NT][4]) {
  static_assert(NT % 2 == 0, "B comes two column tiles at a time");
  const int lane = threadIdx.x & 31, r = lane & 7, q = lane >> 3;
#pragma unroll
  for (int k = 0; k < K; k += 16) {
    uint32_t a[4];
    // matrices: (i 0-7, k 0-7), (i 8-15, k 0-7), (i 0-7, k 8-15), (8-15, 8-15)
    if (TA) ldm4t(a, A + (k + (q >> 1) * 8 + r) * lda + (q & 1) * 8);
    else ldm4(a, A + ((q & 1) * 8 + r) * lda + k + (q >> 1) * 8);
#pragma unroll
    for (int n = 0; n < NT; n += 2) {
      uint32_t b[4];
      // matrices: (k 0-7, n 0-7), (k 8-15, n 0-7), and both for n 8-15
      if (TB) ldm4(b, B + (8 * n + (q >> 1) * 8 + r) * ldb + k + (q & 1) * 8);
      else ldm4t(b, B + (k + (q & 1) * 8 + r) * ldb + 8 * n + (q >> 1) * 8);
      mma(c[n], a, b[0], b[1]);
      mma(c[n + 1], a, b[2], b[3]);
    }
  }
}

// c[n][2 h + v] is row g + 8 h, column 8 n + 2 t + v of the warp's block
template <int NT, typename F>
__device__ __forceinline__ void each_pair(const float (&c)[NT][4], F f) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int n = 0; n < NT; n++)
#pragma unroll
    for (int h = 0; h < 2; h++)
      f(g + 8 * h, 8 * n + 2 * t, c[n][2 * h], c[n][2 * h + 1]);
}

// h[rows m0.., cols n0..] = bf16(relu(A W + b)), 16 x 32 of it per warp
template <int K>
__device__ __forceinline__ void hidden_layer(const __nv_bfloat16 *A, int lda,
                                             const __nv_bfloat16 *W,
                                             const float *bias,
                                             __nv_bfloat16 *h) {
  const int warp = threadIdx.x >> 5;
  const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * 32;
  float c[4][4] = {};
  warp_gemm<K, 4, false, false>(A + m0 * lda, lda, W + n0, kLdH, c);
  each_pair(c, [&](int i, int j, float u, float v) {
    u += bias[n0 + j];
    v += bias[n0 + j + 1];
    *reinterpret_cast<uint32_t *>(h + (m0 + i) * kLdH + n0 + j) =
        pack2(u > 0.f ? u : 0.f, v > 0.f ? v : 0.f);
  });
}

__device__ __forceinline__ void add2(float *p, float u, float v) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(p), "f"(u),
               "f"(v)
               : "memory");
}

// One CTA of 16 warps takes blocks of 64 samples, one an SM at most, with the
// weights in shared memory throughout; the weight gradients stay in registers
// (40 a thread) until its last block, so a gradient vector is added to memory
// once per CTA.  Fragments are loaded with ldmatrix: built from two-byte
// shared loads, as they were, the gradient over 20,000 samples took 172 us
// (two CTAs an SM, 313 of them, 6.5 M atomics); it takes 28 us.
template <bool TRAIN>
__global__ void __launch_bounds__(kThreads, 1)
k_mlp(const float *P, const __nv_bfloat16 *w1b, const __nv_bfloat16 *w2b,
      const float *X, const float *T, int n, float scale, float *out_y,
      float *G) {
  extern __shared__ __align__(16) unsigned char smraw[];
  MlpSmem &s = *reinterpret_cast<MlpSmem *>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < kIn * kHid / 8; i += kThreads)
    *reinterpret_cast<uint4 *>(s.w1 + (i / 16) * kLdH + (i % 16) * 8) =
        reinterpret_cast<const uint4 *>(w1b)[i];
  for (int i = tid; i < kHid * kHid / 8; i += kThreads)
    *reinterpret_cast<uint4 *>(s.w2 + (i / 16) * kLdH + (i % 16) * 8) =
        reinterpret_cast<const uint4 *>(w2b)[i];
  for (int i = tid; i < kHid; i += kThreads) {
    s.b1[i] = P[kB1 + i];
    s.b2[i] = P[kB2 + i];
    s.w3[i] = P[kW3 + i];
  }
  if (tid == 0) s.b3 = P[kB3];
  // gradients of this CTA's blocks: dW2 rows 16 (warp % 8), columns
  // 64 (warp / 8); dW1 rows 16 (warp % 2), columns 16 (warp / 2); a column
  // and a quarter of the rows a thread for the vectors
  float gw2[8][4] = {}, gw1[2][4] = {};
  float gw3 = 0.f, gb2 = 0.f, gb1 = 0.f, gb3 = 0.f;
  const int m2 = (warp & 7) * 16, n2 = (warp >> 3) * 64;
  const int m1 = (warp & 1) * 16, n1 = (warp >> 1) * 16;
  const int col = tid & (kHid - 1), rq = tid / kHid * (kRows / 4);
  const int blocks = (n + kRows - 1) / kRows;
  for (int blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
    const int r0 = blk * kRows;
    {
      const int r = tid >> 3, c = (tid & 7) * 4;       // 64 rows x 8 float4
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r0 + r < n)
        v = *reinterpret_cast<const float4 *>(X + (long long)(r0 + r) * kIn +
                                              c);
      *reinterpret_cast<uint2 *>(s.x + r * kLdX + c) =
          make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
    }
    __syncthreads();
    hidden_layer<kIn>(s.x, kLdX, s.w1, s.b1, s.h1);
    __syncthreads();
    hidden_layer<kHid>(s.h1, kLdH, s.w2, s.b2, s.h2);
    __syncthreads();
    // output layer and the loss gradient: a warp per row
    for (int r = warp; r < kRows; r += kWarps) {
      float acc = 0.f;
#pragma unroll
      for (int c = 0; c < kHid; c += 64) {
        const int j = c + 2 * lane;
        const float2 h = __bfloat1622float2(
            *reinterpret_cast<const __nv_bfloat162 *>(s.h2 + r * kLdH + j));
        acc += h.x * s.w3[j] + h.y * s.w3[j + 1];
      }
      for (int o = 16; o > 0; o >>= 1)
        acc += __shfl_down_sync(0xffffffffu, acc, o);
      if (lane == 0) {
        const float y = acc + s.b3;
        const bool in = r0 + r < n;
        if (in && out_y) out_y[r0 + r] = y;
        if (TRAIN)
          s.dy[r] = in ? (1.f / (1.f + expf(-y)) - T[r0 + r]) * scale : 0.f;
      }
    }
    __syncthreads();
    if (!TRAIN) continue;
    // dw3, db2, db3; dz2 in place of h2
    for (int r = rq; r < rq + kRows / 4; r++) {
      __nv_bfloat16 *p = s.h2 + r * kLdH + col;
      const float h = __bfloat162float(*p), d = s.dy[r];
      gw3 += d * h;
      const __nv_bfloat16 dz = __float2bfloat16(h > 0.f ? d * s.w3[col] : 0.f);
      *p = dz;
      gb2 += __bfloat162float(dz);
      if (col == 0) gb3 += d;
    }
    __syncthreads();
    // dW2 += h1^T dz2, and dz1 = dz2 W2^T where h1 > 0
    warp_gemm<kRows, 8, true, false>(s.h1 + m2, kLdH, s.h2 + n2, kLdH, gw2);
    const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * 32;
    float c[4][4] = {};
    warp_gemm<kHid, 4, false, true>(s.h2 + m0 * kLdH, kLdH, s.w2 + n0 * kLdH,
                                    kLdH, c);
    __syncthreads();                     // h1's last readers are through
    each_pair(c, [&](int i, int j, float u, float v) {
      __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(
          s.h1 + (m0 + i) * kLdH + n0 + j);
      const float2 h = __bfloat1622float2(*p);
      *reinterpret_cast<uint32_t *>(p) =
          pack2(h.x > 0.f ? u : 0.f, h.y > 0.f ? v : 0.f);
    });
    __syncthreads();
    // db1, dW1 += x^T dz1
    for (int r = rq; r < rq + kRows / 4; r++)
      gb1 += __bfloat162float(s.h1[r * kLdH + col]);
    warp_gemm<kRows, 2, true, false>(s.x + m1, kLdX, s.h1 + n1, kLdH, gw1);
    __syncthreads();                     // the next block's x, h1, h2
  }
  if (!TRAIN) return;
  each_pair(gw2, [&](int i, int j, float u, float v) {
    add2(G + kW2 + (m2 + i) * kHid + n2 + j, u, v);
  });
  each_pair(gw1, [&](int i, int j, float u, float v) {
    add2(G + kW1 + (m1 + i) * kHid + n1 + j, u, v);
  });
  atomicAdd(G + kW3 + col, gw3);
  atomicAdd(G + kB2 + col, gb2);
  atomicAdd(G + kB1 + col, gb1);
  if (col == 0) atomicAdd(G + kB3, gb3);
}

// Adam on the fp32 master copy; refreshes the bf16 copies of W1 / W2 and
// clears the gradient
__global__ void k_adam(float *P, float *G, float *M, float *V, int np,
                       float lr, float b1, float b2, float eps, float c1,
                       float c2, __nv_bfloat16 *w1b, __nv_bfloat16 *w2b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const float g = G[i];
  const float m = b1 * M[i] + (1.f - b1) * g;
  const float v = b2 * V[i] + (1.f - b2) * g * g;
  M[i] = m;
  V[i] = v;
  const float p = P[i] - lr * (m / c1) / (sqrtf(v / c2) + eps);
  P[i] = p;
  G[i] = 0.f;
  if (i >= kW1 && i < kW1 + kIn * kHid) w1b[i - kW1] = __float2bfloat16(p);
  if (i >= kW2 && i < kW2 + kHid * kHid) w2b[i - kW2] = __float2bfloat16(p);
}

__global__ void k_refresh_bf16(const float *P, __nv_bfloat16 *w1b,
                               __nv_bfloat16 *w2b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kIn * kHid) w1b[i] = __float2bfloat16(P[kW1 + i]);
  if (i < kHid * kHid) w2b[i] = __float2bfloat16(P[kW2 + i]);
}

struct Mlp {
  float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr;
  __nv_bfloat16 *w1b = nullptr, *w2b = nullptr;
  float *dX = nullptr, *dT = nullptr, *dY = nullptr;
  long long cap = 0;
  long long step = 0;
  cudaStream_t s = nullptr;
};

std::unordered_map<long long, Mlp *> g_mlps;
long long g_mlp_next = 1;

Mlp *get(long long h) {
  auto it = g_mlps.find(h);
  return it == g_mlps.end() ? nullptr : it->second;
}

int ensure_cap(Mlp *m, long long n) {
  if (n <= m->cap) return 0;
  if (m->dX) cudaFree(m->dX);
  if (m->dT) cudaFree(m->dT);
  if (m->dY) cudaFree(m->dY);
  m->dX = m->dT = m->dY = nullptr;
  CC_CK(cudaMalloc(&m->dX, (size_t)n * kIn * 4));
  CC_CK(cudaMalloc(&m->dT, (size_t)n * 4));
  CC_CK(cudaMalloc(&m->dY, (size_t)n * 4));
  m->cap = n;
  return 0;
}

int launch_mlp(Mlp *m, bool train, const float *X, const float *T, int n,
               float scale, float *Y) {
  const size_t smem = sizeof(MlpSmem);
  static bool attr = false;
  if (!attr) {
    CC_CK(cudaFuncSetAttribute((const void *)k_mlp<true>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
    CC_CK(cudaFuncSetAttribute((const void *)k_mlp<false>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
    attr = true;
  }
  const int grid = std::min((n + kRows - 1) / kRows, cc::sm_count());
  if (train)
    k_mlp<true><<<grid, kThreads, smem, m->s>>>(m->P, m->w1b, m->w2b, X, T, n,
                                           scale, Y, m->G);
  else
    k_mlp<false><<<grid, kThreads, smem, m->s>>>(m->P, m->w1b, m->w2b, X, T, n,
                                            scale, Y, m->G);
  CC_CK(cudaGetLastError());
  return 0;
}

// splitmix64: deterministic host initialisation
uint64_t mix(uint64_t &x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

}  // namespace

extern "C" {

long long dct_mlp_create(unsigned long long seed) {
  Mlp *m = new Mlp();
  if (cudaStreamCreateWithFlags(&m->s, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&m->P, kParams * 4) != cudaSuccess ||
      cudaMalloc(&m->G, kParams * 4) != cudaSuccess ||
      cudaMalloc(&m->M, kParams * 4) != cudaSuccess ||
      cudaMalloc(&m->V, kParams * 4) != cudaSuccess ||
      cudaMalloc(&m->w1b, kIn * kHid * 2) != cudaSuccess ||
      cudaMalloc(&m->w2b, kHid * kHid * 2) != cudaSuccess) {
    delete m;
    return -1;
  }
  // He-uniform weights, zero biases
  std::vector<float> p(kParams, 0.f);
  uint64_t st = seed;
  auto uni = [&](float a) {
    return (float)((mix(st) >> 11) * (1.0 / 9007199254740992.0) * 2 - 1) * a;
  };
  for (int i = 0; i < kIn * kHid; i++) p[kW1 + i] = uni(sqrtf(6.f / kIn));
  for (int i = 0; i < kHid * kHid; i++) p[kW2 + i] = uni(sqrtf(6.f / kHid));
  for (int i = 0; i < kHid; i++) p[kW3 + i] = uni(sqrtf(6.f / kHid) * 0.5f);
  // on the net's own stream, which does not wait for the default one
  cudaMemcpyAsync(m->P, p.data(), kParams * 4, cudaMemcpyHostToDevice, m->s);
  for (float *z : {m->G, m->M, m->V})
    cudaMemsetAsync(z, 0, kParams * 4, m->s);
  k_refresh_bf16<<<(kHid * kHid + 255) / 256, 256, 0, m->s>>>(m->P, m->w1b,
                                                             m->w2b);
  cudaStreamSynchronize(m->s);
  const long long h = g_mlp_next++;
  g_mlps[h] = m;
  return h;
}

int dct_mlp_params(long long h, float *get_out, const float *set_in) {
  Mlp *m = get(h);
  if (!m) return -1;
  if (set_in) {
    CC_CK(cudaMemcpyAsync(m->P, set_in, kParams * 4, cudaMemcpyHostToDevice,
                          m->s));
    k_refresh_bf16<<<(kHid * kHid + 255) / 256, 256, 0, m->s>>>(m->P, m->w1b,
                                                               m->w2b);
    CC_CK(cudaGetLastError());
  }
  if (get_out)
    CC_CK(cudaMemcpyAsync(get_out, m->P, kParams * 4, cudaMemcpyDeviceToHost,
                          m->s));
  CC_CK(cudaStreamSynchronize(m->s));
  return kParams;
}

int dct_mlp_grad(long long h, const float *X, const float *T, int n,
                 float *grad_out) {
  Mlp *m = get(h);
  if (!m || n < 1 || !X || !T || !grad_out) return -1;
  int rc = ensure_cap(m, n);
  if (rc) return rc;
  CC_CK(cudaMemcpyAsync(m->dX, X, (size_t)n * kIn * 4,
                        cudaMemcpyHostToDevice, m->s));
  CC_CK(cudaMemcpyAsync(m->dT, T, (size_t)n * 4, cudaMemcpyHostToDevice,
                        m->s));
  CC_CK(cudaMemsetAsync(m->G, 0, kParams * 4, m->s));
  rc = launch_mlp(m, true, m->dX, m->dT, n, 1.f / n, m->dY);
  if (rc) return rc;
  CC_CK(cudaMemcpyAsync(grad_out, m->G, kParams * 4, cudaMemcpyDeviceToHost,
                        m->s));
  CC_CK(cudaMemsetAsync(m->G, 0, kParams * 4, m->s));
  CC_CK(cudaStreamSynchronize(m->s));
  return kParams;
}

int dct_mlp_train(long long h, const float *X, const float *T, int n,
                  int epochs, int batch, float lr, unsigned long long seed) {
  Mlp *m = get(h);
  if (!m || n < 1 || !X || !T || epochs < 1 || batch < 1) return -1;
  int rc = ensure_cap(m, n);
  if (rc) return rc;
  // shuffle once per epoch on the host, upload the permuted set
  std::vector<int> perm(n);
  for (int i = 0; i < n; i++) perm[i] = i;
  std::vector<float> xs((size_t)n * kIn), ts(n);
  uint64_t st = seed;
  for (int e = 0; e < epochs; e++) {
    for (int i = n - 1; i > 0; i--) {
      const int j = (int)(mix(st) % (uint64_t)(i + 1));
      std::swap(perm[i], perm[j]);
    }
    for (int i = 0; i < n; i++) {
      memcpy(&xs[(size_t)i * kIn], X + (size_t)perm[i] * kIn, kIn * 4);
      ts[i] = T[perm[i]];
    }
    CC_CK(cudaMemcpyAsync(m->dX, xs.data(), xs.size() * 4,
                          cudaMemcpyHostToDevice, m->s));
    CC_CK(cudaMemcpyAsync(m->dT, ts.data(), ts.size() * 4,
                          cudaMemcpyHostToDevice, m->s));
    for (int b0 = 0; b0 < n; b0 += batch) {
      const int nb = n - b0 < batch ? n - b0 : batch;
      rc = launch_mlp(m, true, m->dX + (size_t)b0 * kIn, m->dT + b0, nb,
                      1.f / nb, nullptr);
      if (rc) return rc;
      m->step++;
      const float b1 = 0.9f, b2 = 0.999f;
      const float c1 = 1.f - powf(b1, (float)m->step);
      const float c2 = 1.f - powf(b2, (float)m->step);
      k_adam<<<(kParams + 255) / 256, 256, 0, m->s>>>(
          m->P, m->G, m->M, m->V, kParams, lr, b1, b2, 1e-8f, c1, c2, m->w1b,
          m->w2b);
      CC_CK(cudaGetLastError());
    }
    CC_CK(cudaStreamSynchronize(m->s));      // xs / ts reused next epoch
  }
  return 0;
}

int dct_mlp_predict(long long h, const float *X, int n, float *out) {
  Mlp *m = get(h);
  if (!m || n < 0 || (n && (!X || !out))) return -1;
  if (!n) return 0;
  int rc = ensure_cap(m, n);
  if (rc) return rc;
  CC_CK(cudaMemcpyAsync(m->dX, X, (size_t)n * kIn * 4,
                        cudaMemcpyHostToDevice, m->s));
  rc = launch_mlp(m, false, m->dX, nullptr, n, 0.f, m->dY);
  if (rc) return rc;
  CC_CK(cudaMemcpyAsync(out, m->dY, (size_t)n * 4, cudaMemcpyDeviceToHost,
                        m->s));
  CC_CK(cudaStreamSynchronize(m->s));
  return 0;
}

int dct_mlp_free(long long h) {
  Mlp *m = get(h);
  if (!m) return -1;
  cudaStreamSynchronize(m->s);
  cudaFree(m->P); cudaFree(m->G); cudaFree(m->M); cudaFree(m->V);
  cudaFree(m->w1b); cudaFree(m->w2b);
  if (m->dX) cudaFree(m->dX);
  if (m->dT) cudaFree(m->dT);
  if (m->dY) cudaFree(m->dY);
  cudaStreamDestroy(m->s);
  g_mlps.erase(h);
  delete m;
  return 0;
}

}  // extern "C"
