// Parameters shared by the FP32 MLP kernels: the CUDA-core kernels of
// mlp_f32.cu and the split-operand tensor-core kernels of mlp_f32_split.cu.
#pragma once
#include "common.cuh"

namespace vx {
namespace mf {

struct RowGemmParams {
  const float* A;            // [M, lda]
  int64_t lda;
  int64_t M;
  const int64_t* m_dev;      // optional device row count (<= M)
  int K;                     // columns of A used
  const float* Bt;           // [Kp][Np] (Kp = round_up(K, 16), zero rows beyond K)
  int Np;
  int mode;                  // 0: relu(acc + bias); 1: acc * [H > 0] + column sums; 2: acc
  const float* bias;         // mode 0: [Np]
  const float* H;            // mode 1: [M, ldh] post-ReLU activation of the layer
  int64_t ldh;
  float* C;                  // [M, ldc], columns < n_store
  int64_t ldc;
  int n_store;
  float* colsum;             // mode 1: [n_colsum][Np] column sums, one row per CTA
  int64_t n_colsum;          // vx_mlp_f32_rowgemm_grid(M) rows, those beyond the CTAs zero
};

struct WgradParams {
  const float* A;            // [rows, lda] (dz of the layer's output), columns < M
  int64_t lda;
  const float* B;            // [rows, ldb] (the layer's input), columns < N
  int64_t ldb;
  int M, N;                  // padded widths MP >= M, NP >= N
  int64_t rows;
  const int64_t* rows_dev;
  float* part;               // [grid][MP][NP]
};

__device__ __forceinline__ int64_t rows_of(int64_t n, const int64_t* n_dev) {
  if (n_dev) {
    const int64_t d = *n_dev;
    if (d < n) n = d < 0 ? 0 : d;
  }
  return n;
}

// The backward GEMMs on the tensor cores; false when the shapes or the
// alignment of the buffers are not theirs (the CUDA-core kernels run then).
bool split_rowgemm_takes(const RowGemmParams& P);
unsigned split_rowgemm_grid(int64_t M);
int split_rowgemm_launch(const RowGemmParams& P, cudaStream_t st);
bool split_wgrad_takes(const WgradParams& P, int MP, int NP);
int split_wgrad_launch(const WgradParams& P, int MP, int NP, unsigned grid, cudaStream_t st);

}  // namespace mf
}  // namespace vx
