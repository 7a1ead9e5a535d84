// GEMM with few rows of A (generation, short prompts): gemm_skinny_tcgen05.cu.
#pragma once
#include "common.h"
#include "ptx.cuh"

namespace nx {

constexpr int SKINNY_MAX_M = 128;

struct SkinnyParams {
  int M, N, K;
  h16* C;
  long long ldc;
  const h16* bias;
  h16* aux_out;
  const h16* residual;
  long long ld_aux;
  int flags;           // the EPI_* bits of gemm_tcgen05.cu that the call sets
  float alpha;
  int* err;
};

// C[M, N] = epilogue(A[M, K] * B[N, K]^T), both K-contiguous.  `flags` without any of the accumulate, fp32-output and
// multiply-by-aux bits.
int gemm_skinny_launch(const void* A, const void* B, long long lda, long long ldb, const SkinnyParams& p,
                       cudaStream_t stream);

}  // namespace nx
