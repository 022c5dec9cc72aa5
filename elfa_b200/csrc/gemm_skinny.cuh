// Products of a few rows (gemm_skinny.cu), reached through elfa_gemm_bf16.
#pragma once
#include "common.cuh"

namespace elfa {

constexpr int SKINNY_ROWS = 8;

struct SkinnyParams {
  const __nv_bfloat16 *A, *B, *bias;
  __nv_bfloat16 *C, *preact;
  long long lda, ldb, ldc, ldpre;
  int M, N, K;
  float alpha;
  unsigned flags;                          // ELFA_EPI_BIAS, ELFA_EPI_GELU, ELFA_EPI_STORE_PREACT
};

// How a [K, N] matrix is cut: column tiles of 64 (narrow) or 128, `shares` slices of the contraction of `ks` rows each
struct SkinnyPlan {
  bool narrow;
  int shares;
  int tiles(int N) const { return narrow ? (N + 63) / 64 : (N + 127) / 128; }
  int ks(int K) const { return ((K + shares - 1) / shares + 15) / 16 * 16; }
};

bool gemm_skinny_better(int M, int N, int K);
SkinnyPlan skinny_plan(int N, int K);
int launch_gemm_skinny(const SkinnyParams& p, bool b_mn, cudaStream_t s);

}  // namespace elfa
