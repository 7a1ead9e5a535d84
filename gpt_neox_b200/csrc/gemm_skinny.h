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

// A product and where its operands lie (row-major, K-contiguous).
struct SkinnyProduct {
  const void *A, *B;
  long long lda, ldb;
  SkinnyParams p;
};
// Whether a product of these sizes and flags goes to the few-rows kernel (gemm_tcgen05.cu).
bool skinny_better(int M, int N, int K, int transA, int transB, int flags);
// Two products of the same number of rows in one launch, each with the bits that it has by itself.
int gemm_skinny_launch_pair(const SkinnyProduct (&q)[2], cudaStream_t stream);
// C[M, N] = epilogue(A[M, K] * B[N, K]^T), both K-contiguous.  `flags` without any of the accumulate, fp32-output and
// multiply-by-aux bits.
int gemm_skinny_launch(const void* A, const void* B, long long lda, long long ldb, const SkinnyParams& p,
                       cudaStream_t stream);

}  // namespace nx
