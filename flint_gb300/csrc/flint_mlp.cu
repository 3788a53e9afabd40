// flint_mlp.cu -- BF16 tensor-core MLP kernels of the learned reactor surrogate.
//
// The surrogate is a multilayer perceptron (33 -> 256 -> 256 -> 256 -> 256 -> 32,
// GELU) with BF16 MMA operands and FP32 accumulation, master weights and
// activations in FP32.  One tiled GEMM serves the per-layer forward and both
// backward products; its operands are FP32 matrices staged as BF16 tiles in
// shared memory and multiplied by mma.sync.m16n8k16; epilogues: +bias and GELU
// (writes the pre-activation and the activation), +bias, plain FP32, or (for
// back-propagation) C * GELU'(Z).
//
// What bounds it: a training step of 4,096 samples is 5 GFLOP (15 with the
// forward's split operands), a few microseconds of the tensor cores, so what
// counts is the number of dependent launches and the latency inside each.
// Tiles of 64 x 64 (8 warps of 32 x 16) give 256 blocks for 4,096 x 256; the
// next K step's 16-byte loads are in flight while a step is multiplied (two
// shared-memory stages); the weight and bias gradients of all layers are one
// launch (k_weight_grad).  A forward layer takes 15 us (20 with 4 warps a tile), a
// backward one 17, the weight gradients 79; a step 0.26 ms, where it took 3.4 with
// a scalar load and conversion per element, weight gradients one layer at a time
// on 16 blocks and one thread per column sum.  Sums keep their order (samples in
// order, 16 to an MMA): the result does not depend on the tiling.
//
// Split mode (the forward pass): every operand x is staged as the BF16 pair
// hi = bf16(x), lo = bf16(x - hi), and each fragment product is accumulated as
// lo*hi + hi*lo + hi*hi in FP32.  A single BF16 operand carries 8 significant
// bits; the pair carries about 16, which moves the network's rounding floor
// from ~1e-3 to ~1e-5 of its output scale at three times the MMA work (the
// lo*lo term is below the FP32 accumulation error and is skipped).
#include <cstdint>
#include <algorithm>
#include <cuda_bf16.h>
#include "flint_host.h"
#include "flint_mlp.h"

namespace flint {

constexpr int GBM = 64, GBN = 64, GBK = 32, GTHREADS = 256;
// A staged tile holds its 64 x 32 elements by rows of k (an operand contiguous in
// k; rows padded to 40 elements) or by rows of n (contiguous in n; padded to
// 72): fragments are then read without bank conflicts, in the second case by
// ldmatrix.trans.
constexpr int KPAD = 40, MPAD = 72, TILE = GBM * KPAD;

__device__ __forceinline__ float gelu_f(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * x * (1.0f + tanhf(k0 * (x + k1 * x * x * x)));
}
__device__ __forceinline__ float gelu_grad(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float u = k0 * (x + k1 * x * x * x);
  const float t = tanhf(u);
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * k0 * (1.0f + 3.0f * k1 * x * x);
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void ldmatrix_trans(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
}

// The 8 elements of a 64 x 32 operand tile that a thread stages: two groups of
// four along the contiguous dimension.  KC: X[mn][k] (k contiguous), else
// X[k][mn].  vec: 16-byte loads are aligned.
template <bool KC>
__device__ __forceinline__ void load_tile(float (&v)[8], const float* __restrict__ X, int64_t ld, bool vec, int mn0,
                                          int mn_end, int k0, int k_end, int tid) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = KC ? mn0 + (tid >> 3) + 32 * i : k0 + (tid >> 4) + 16 * i;
    const int c = KC ? k0 + (tid & 7) * 4 : mn0 + (tid & 15) * 4;
    const int r_end = KC ? mn_end : k_end, c_end = KC ? k_end : mn_end;
    const float* p = X + (int64_t)r * ld + c;
    if (r < r_end && vec && c + 3 < c_end) {
      const float4 q = *reinterpret_cast<const float4*>(p);
      v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) v[4 * i + u] = r < r_end && c + u < c_end ? p[u] : 0.f;
    }
  }
}

template <bool KC, int NP>
__device__ __forceinline__ void store_tile(__nv_bfloat16* s, const float (&v)[8], int tid) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int o = KC ? ((tid >> 3) + 32 * i) * KPAD + (tid & 7) * 4 : ((tid >> 4) + 16 * i) * MPAD + (tid & 15) * 4;
    uint32_t h[2], l[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float x = v[4 * i + 2 * u], y = v[4 * i + 2 * u + 1];
      const __nv_bfloat16 a = __float2bfloat16_rn(x), b = __float2bfloat16_rn(y);
      h[u] = (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
      const __nv_bfloat16 c = __float2bfloat16_rn(x - __bfloat162float(a)), d = __float2bfloat16_rn(y - __bfloat162float(b));
      l[u] = (uint32_t)__bfloat16_as_ushort(c) | ((uint32_t)__bfloat16_as_ushort(d) << 16);
    }
    *reinterpret_cast<uint2*>(s + o) = make_uint2(h[0], h[1]);
    if (NP == 2) *reinterpret_cast<uint2*>(s + TILE + o) = make_uint2(l[0], l[1]);
  }
}

template <bool SPLIT, bool B_KC>
__global__ void __launch_bounds__(GTHREADS) k_gemm(const __grid_constant__ GemmArgs g) {
  constexpr int NP = SPLIT ? 2 : 1;   // hi (and lo) planes
  __shared__ __align__(16) __nv_bfloat16 sA[2][NP * TILE];
  __shared__ __align__(16) __nv_bfloat16 sB[2][NP * TILE];
  const int n0 = blockIdx.x * GBN, m0 = blockIdx.y * GBM, ke = g.K;
  const bool va = (g.lda & 3) == 0 && (reinterpret_cast<uintptr_t>(g.A) & 15) == 0;
  const bool vb = (g.ldb & 3) == 0 && (reinterpret_cast<uintptr_t>(g.B) & 15) == 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
  const int grp = lane >> 2, tig = lane & 3;
  float acc[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;

  float ra[8], rb[8];
  load_tile<true>(ra, g.A, g.lda, va, m0, g.M, 0, ke, tid);
  load_tile<B_KC>(rb, g.B, g.ldb, vb, n0, g.N, 0, ke, tid);
  int buf = 0;
  for (int k0 = 0; k0 < ke; k0 += GBK, buf ^= 1) {
    store_tile<true, NP>(sA[buf], ra, tid);
    store_tile<B_KC, NP>(sB[buf], rb, tid);
    __syncthreads();   // (the other stage was read before the previous one of these)
    if (k0 + GBK < ke) {
      load_tile<true>(ra, g.A, g.lda, va, m0, g.M, k0 + GBK, ke, tid);
      load_tile<B_KC>(rb, g.B, g.ldb, vb, n0, g.N, k0 + GBK, ke, tid);
    }
#pragma unroll
    for (int kk = 0; kk < GBK; kk += 16) {
      uint32_t af[NP][2][4], bfr[NP][2][2];
#pragma unroll
      for (int pl = 0; pl < NP; ++pl) {
        const __nv_bfloat16 *a = sA[buf] + pl * TILE, *b = sB[buf] + pl * TILE;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int r = wm + i * 16 + grp;
          af[pl][i][0] = *reinterpret_cast<const uint32_t*>(a + r * KPAD + kk + tig * 2);
          af[pl][i][1] = *reinterpret_cast<const uint32_t*>(a + (r + 8) * KPAD + kk + tig * 2);
          af[pl][i][2] = *reinterpret_cast<const uint32_t*>(a + r * KPAD + kk + tig * 2 + 8);
          af[pl][i][3] = *reinterpret_cast<const uint32_t*>(a + (r + 8) * KPAD + kk + tig * 2 + 8);
        }
#pragma unroll
        for (int j = 0; j < 2; j += 2) {
          if (B_KC) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int n = wn + (j + u) * 8 + grp;
              bfr[pl][j + u][0] = *reinterpret_cast<const uint32_t*>(b + n * KPAD + kk + tig * 2);
              bfr[pl][j + u][1] = *reinterpret_cast<const uint32_t*>(b + n * KPAD + kk + tig * 2 + 8);
            }
          } else {
            // matrices (k, n): (0,0) (8,0) of column tile j, then of j + 1
            uint32_t r[4];
            ldmatrix_trans(r, b + (kk + ((lane >> 3) & 1) * 8 + (lane & 7)) * MPAD + wn + (j + (lane >> 4)) * 8);
            bfr[pl][j][0] = r[0]; bfr[pl][j][1] = r[1];
            bfr[pl][j + 1][0] = r[2]; bfr[pl][j + 1][1] = r[3];
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (SPLIT) {
            mma_bf16(acc[i][j], af[NP - 1][i], bfr[0][j]);
            mma_bf16(acc[i][j], af[0][i], bfr[NP - 1][j]);
          }
          mma_bf16(acc[i][j], af[0][i], bfr[0][j]);
        }
    }
  }
  // epilogue
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int m = m0 + wm + i * 16 + grp + (c >= 2 ? 8 : 0);
        const int n = n0 + wn + j * 8 + tig * 2 + (c & 1);
        if (m >= g.M || n >= g.N) continue;
        float v = acc[i][j][c];
        if (g.epi == EPI_BIAS || g.epi == EPI_BIAS_GELU) v += g.bias[n];
        if (g.epi == EPI_GELU_BWD) v *= gelu_grad(g.Zprev[(int64_t)m * g.ldz + n]);
        if (g.C) g.C[(int64_t)m * g.ldc + n] = v;
        if (g.Cf) g.Cf[(int64_t)m * g.ldcf + n] = g.epi == EPI_BIAS_GELU ? gelu_f(v) : v;
      }
}

// ---------------------------------------------------------------- weight gradients
// Every layer's weight gradient C = A^T B (A: gradients by its pre-activations
// [sample][M], B: its inputs [sample][N]) and bias gradient (column sums of A), all
// layers in one launch.  A block owns a 32 x 64 tile of one layer and walks the
// samples in order, 16 to an MMA, so an element's sum has one order whatever the
// tiling; blocks of their own add the columns, sample by sample.  What bounds it is
// the latency of a step (64 samples: copy, barrier, fragment reads, conversion,
// MMA) on two warps per scheduler: 79 us for 4,096 samples, 106 with steps of 32 and
// the column sums in the first tiles' blocks, 138 with 4 warps a block; 64 x 64
// tiles would leave 56 blocks for 152 SMs.  The FP32 tiles arrive by cp.async three
// steps ahead and are rounded to BF16 as fragments are read: element (k, m) at
// k ld + m with ld = 4 mod 16 puts the 32 lanes of a fragment read on 32 banks.
constexpr int WBM = 32, WBN = 64, WBK = 64, WTHREADS = 256, WSTAGES = 4, WLDA = 36, WLDB = 68;
constexpr int WSTAGE = WBK * (WLDA + WLDB);                    // floats
constexpr size_t WGRAD_SMEM = (size_t)WSTAGES * WSTAGE * sizeof(float);

struct WeightGrads {
  WeightGrad g[GRAD_BATCH];
  int first[GRAD_BATCH + 1];   // first block of each layer
};

// 16 bytes to shared memory, the last ones zero where fewer are there.
__device__ __forceinline__ void copy_async(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}

// Rows k0 .. k0 + WBK - 1 of X[K][W], columns c0 .. c0 + BW - 1, zero outside, to dst with
// a row stride of LD; W a multiple of 4, X aligned.  flat: W <= BW and the rows go
// as they lie, with a stride of W (any W; what lies beyond column W is not used).
// Neither: element by element.
template <int BW, int LD>
__device__ __forceinline__ void copy_tile(float* dst, const float* __restrict__ X, int K, int W, int k0, int c0, int tid,
                                          bool wide, bool flat) {
  if (flat) {
    const int64_t base = (int64_t)k0 * W, end = (int64_t)K * W;
    for (int e = tid * 4; e < WBK * W; e += WTHREADS * 4) {
      const int64_t left = end - base - e;
      copy_async(dst + e, left > 0 ? X + base + e : X, left >= 4 ? 16 : (left > 0 ? (int)left * 4 : 0));
    }
  } else if (wide) {
#pragma unroll
    for (int i = 0; i < WBK * BW / 4 / WTHREADS; ++i) {
      const int e = tid + i * WTHREADS, r = e / (BW / 4), c = (e % (BW / 4)) * 4;
      const bool on = k0 + r < K && c0 + c < W;
      copy_async(dst + r * LD + c, on ? X + (int64_t)(k0 + r) * W + c0 + c : X, on ? 16 : 0);
    }
  } else {
#pragma unroll 4
    for (int i = 0; i < WBK * BW / WTHREADS; ++i) {
      const int e = tid + i * WTHREADS, r = e / BW, c = e % BW;
      dst[r * LD + c] = k0 + r < K && c0 + c < W ? X[(int64_t)(k0 + r) * W + c0 + c] : 0.f;
    }
  }
}

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  const __nv_bfloat16 a = __float2bfloat16_rn(lo), b = __float2bfloat16_rn(hi);
  return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}

__global__ void __launch_bounds__(WTHREADS) k_weight_grad(const __grid_constant__ WeightGrads batch) {
  extern __shared__ __align__(16) float wsm[];
  int id = blockIdx.x, p = 0;
  while (id >= batch.first[p + 1]) ++p;
  const WeightGrad& g = batch.g[p];
  id -= batch.first[p];
  // the last column of tiles of a layer forms the column sums
  const int nt = (g.N + WBN - 1) / WBN + 1;
  const int n0 = (id % nt) * WBN, m0 = (id / nt) * WBM;
  const bool sums = n0 >= g.N;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 16, wn = (warp & 3) * 16, grp = lane >> 2, tig = lane & 3;
  const int steps = (g.K + WBK - 1) / WBK;
  const bool aa = (reinterpret_cast<uintptr_t>(g.A) & 15) == 0, ab = (reinterpret_cast<uintptr_t>(g.B) & 15) == 0;
  const bool wa = (g.M & 3) == 0 && aa, wb = (g.N & 3) == 0 && ab;
  const bool fb = !wb && ab && g.N <= WBN;
  const int ldb = fb ? g.N : WLDB;
  float acc[2][4], cs = 0.f;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;
  auto fetch = [&](int s) {
    if (s < steps) {
      float* st = wsm + (s % WSTAGES) * WSTAGE;
      copy_tile<WBM, WLDA>(st, g.A, g.K, g.M, s * WBK, m0, tid, wa, false);
      if (!sums) copy_tile<WBN, WLDB>(st + WBK * WLDA, g.B, g.K, g.N, s * WBK, n0, tid, wb, fb);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < WSTAGES - 1; ++s) fetch(s);
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(WSTAGES - 2) : "memory");
    __syncthreads();               // step s has arrived for all; step s - 1 is no longer read
    fetch(s + WSTAGES - 1);
    const float* a = wsm + (s % WSTAGES) * WSTAGE;
    const float* b = a + WBK * WLDA;
    if (sums) {
      if (warp == 0)
#pragma unroll 16
        for (int k = 0; k < WBK; ++k) cs += a[k * WLDA + lane];
      continue;
    }
#pragma unroll
    for (int kk = 0; kk < WBK; kk += 16) {
      uint32_t af[4], bf[2][2];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float* q = a + (kk + tig * 2 + (h >> 1) * 8) * WLDA + wm + grp + (h & 1) * 8;
        af[h] = bf16_pair(q[0], q[WLDA]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float* q = b + (kk + tig * 2 + h * 8) * ldb + wn + j * 8 + grp;
          bf[j][h] = bf16_pair(q[0], q[ldb]);
        }
#pragma unroll
      for (int j = 0; j < 2; ++j) mma_bf16(acc[j], af, bf[j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (sums) {
    if (warp == 0 && m0 + lane < g.M) g.colsum[m0 + lane] = cs;
    return;
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int m = m0 + wm + grp + (c >= 2 ? 8 : 0), n = n0 + wn + j * 8 + tig * 2 + (c & 1);
      if (m < g.M && n < g.N) g.C[(int64_t)m * g.N + n] = acc[j][c];
    }
}

// MSE over an (M x N) output: grad = 2 (yhat - y) / (M N); loss partial sums per block.
__global__ void k_mse(const float* __restrict__ yhat, const float* __restrict__ y, int64_t total, float scale,
                      float* __restrict__ grad, double* __restrict__ loss_acc) {
  double part = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const float d = yhat[i] - y[i];
    grad[i] = 2.f * d * scale;
    part += (double)d * d;
  }
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss_acc, part * scale);
}

// Adam on FP32 master weights.
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ gw, float* __restrict__ m1,
                       float* __restrict__ m2, int64_t n, float lr, float b1, float b2, float eps, float bc1, float bc2,
                       float wd) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float g = gw[i] + wd * w[i];
    const float a = b1 * m1[i] + (1.f - b1) * g;
    const float b = b2 * m2[i] + (1.f - b2) * g * g;
    m1[i] = a;
    m2[i] = b;
    const float upd = lr * (a / bc1) / (sqrtf(b / bc2) + eps);
    const float nw = w[i] - upd;
    w[i] = nw;
  }
}

cudaError_t launch_gemm(GemmForm form, const GemmArgs& g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0) return cudaSuccess;
  const dim3 grid((g.N + GBN - 1) / GBN, (g.M + GBM - 1) / GBM);
  if (form == GEMM_FORWARD) k_gemm<true, true><<<grid, GTHREADS, 0, st>>>(g);
  else k_gemm<false, false><<<grid, GTHREADS, 0, st>>>(g);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_weight_grads(const WeightGrad* g, int count, cudaStream_t st) {
  if (count < 1 || count > GRAD_BATCH) return cudaErrorInvalidValue;
  WeightGrads b{};
  int blocks = 0;
  for (int i = 0; i < count; ++i) {
    b.g[i] = g[i];
    b.first[i] = blocks;
    blocks += ((g[i].N + WBN - 1) / WBN + 1) * ((g[i].M + WBM - 1) / WBM);
  }
  for (int i = count; i <= GRAD_BATCH; ++i) b.first[i] = blocks;
  cudaError_t e = set_smem((const void*)k_weight_grad, WGRAD_SMEM);
  if (e != cudaSuccess) return e;
  k_weight_grad<<<blocks, WTHREADS, WGRAD_SMEM, st>>>(b);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_mse(const float* yhat, const float* y, int64_t total, float scale, float* grad, double* loss,
                       cudaStream_t st) {
  int blocks = (int)std::min<int64_t>((total + 255) / 256, 4 * device_sms());
  k_mse<<<blocks, 256, 0, st>>>(yhat, y, total, scale, grad, loss);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_adam(float* w, const float* gw, float* m1, float* m2, int64_t n, float lr, float b1, float b2,
                        float eps, float bc1, float bc2, float wd, cudaStream_t st) {
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 8 * device_sms());
  k_adam<<<blocks, 256, 0, st>>>(w, gw, m1, m2, n, lr, b1, b2, eps, bc1, bc2, wd);
  count_launch();
  return cudaGetLastError();
}

}  // namespace flint
