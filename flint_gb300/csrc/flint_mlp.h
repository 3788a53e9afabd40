// flint_mlp.h -- the BF16 tensor-core GEMM and elementwise kernels of the
// surrogate MLP (flint_mlp.cu), shared with the surrogate driver.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace flint {

enum { EPI_STORE = 0, EPI_BIAS = 1, EPI_BIAS_GELU = 2, EPI_GELU_BWD = 3 };

// C[m][n] = sum_k A(m,k) B(k,n) of FP32 operands, staged as BF16.
enum GemmForm {
  GEMM_FORWARD,   // A[m][k], B[n][k], operands as BF16 hi + lo pairs (three MMAs per fragment)
  GEMM_INPUT      // A[m][k], B[k][n]: the gradient by a layer's input
};

struct GemmArgs {
  int M, N, K;
  const float* A; int64_t lda;       // leading dimension of the stored matrix
  const float* B; int64_t ldb;
  const float* bias;                 // [N]
  float* C; int64_t ldc;             // FP32 output (pre-activation or result); may be null
  float* Cf; int64_t ldcf;           // optional FP32 activation output (GELU applied for EPI_BIAS_GELU)
  const float* Zprev; int64_t ldz;   // GELU_BWD: pre-activation of the previous layer (may be C itself)
  int epi;
};

// A layer's weight gradient C[m][n] = sum_k A[k][m] B[k][n] and bias gradient
// colsum[m] = sum_k A[k][m], k over the samples.
struct WeightGrad {
  int M, N, K;
  const float* A;   // [K][M]
  const float* B;   // [K][N]
  float* C;         // [M][N]
  float* colsum;
};

constexpr int GRAD_BATCH = 8;        // layers of one launch

cudaError_t launch_gemm(GemmForm form, const GemmArgs& g, cudaStream_t st);
cudaError_t launch_weight_grads(const WeightGrad* g, int count, cudaStream_t st);
cudaError_t launch_mse(const float* yhat, const float* y, int64_t total, float scale, float* grad, double* loss,
                       cudaStream_t st);
cudaError_t launch_adam(float* w, const float* gw, float* m1, float* m2, int64_t n, float lr, float b1, float b2,
                        float eps, float bc1, float bc2, float wd, cudaStream_t st);

}  // namespace flint
