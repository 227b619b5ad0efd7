// The projections of layers that run in one call (dense_rows.cu).
#pragma once
#include "small_rows.cuh"

namespace llb {

// y[m][n] = x[m] . w[n], m < M, n < N, over K numbers; head_cols > 0: w is [N / head_cols][K][head_cols] instead of [N][K].  Sizes and strides in
// multiples of 8, head_cols of 64, x and w on 16-byte boundaries.
int dense_rows(const void* x, long long ldx, const void* w, int head_cols, void* y, int ldy, int M, int N, int K, cudaStream_t st);

namespace {

// a projection of any number of rows: one or two on CUDA cores, up to 32 in blocks of 16 weight rows (small_rows.cuh).
// early: w was written before a kernel that this stream ran without overlap after it
inline int rows_linear(const void* x, int ldx, const void* w, void* y, int ldy, int M, int N, int K, bool early, cudaStream_t st) {
  if (M <= SR_MAX) return small_linear(x, ldx, w, y, ldy, M, N, K, st);
  if (M <= 16 || (M <= FR_MAX && N <= 4096)) return few_rows(x, ldx, w, y, ldy, M, N, K, early, st);
  return dense_rows(x, ldx, w, 0, y, ldy, M, N, K, st);
}

}  // namespace
}  // namespace llb
