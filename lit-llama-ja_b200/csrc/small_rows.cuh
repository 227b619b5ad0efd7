// Products of a few rows with bf16 weights that are read once: bound by the weights' way from memory, so what counts is 16-byte loads in flight.  Three
// forms: one or two rows with weights [N][K] on CUDA cores (a warp per output row), 3 to 32 rows with the same weights on mma.sync (few_rows_kernel), and
// weights [K][N] per head on CUDA cores (partial sums over k in a block, four rows at most).  All start under the kernel before them and wait for it before
// they read what it makes; few_rows_kernel reads weights before that wait where its caller knows whoever wrote them to have ended (early).
// The first form takes one or two rows only: every weight meets every row's sums in registers, and from three rows on the conversions cost more than the loads.  Both
// projections of an attention layer, us, here / the library's products: one row of width 2048 12.7 / 12.7, of 4096 21.7 / 27.3; four rows (when
// this form still took them) 21.4 / 11.4 and 51.9 / 27.1.  Two rows of w a warp halve the warps in flight: 8.4 for the first projection against 5.5.
#pragma once
#include "row_loads.cuh"

namespace llb {
namespace {

constexpr int SR_MAX = 2, SR_THREADS = 256, SR_WARPS = SR_THREADS / 32;

// y[m][n] = x[m] . w[n], m < MT: a warp per row of w, eight 16-byte loads of it in flight; in the last round a lane past the end of k takes the last
// piece again and zeros in its place (zero times an infinite weight would be no number; a check in every round costs the layer 2 %).
// K, ldx multiples of 8, rows on 16-byte boundaries.
template <int MT>
__global__ void __launch_bounds__(SR_THREADS) small_linear_kernel(const __nv_bfloat16* x, int ldx, const __nv_bfloat16* __restrict__ w,
                                                                  __nv_bfloat16* __restrict__ y, int ldy, int N, int K) {
  constexpr int U = 8;
  pdl_wait();
  pdl_launch_dependents();
  x = after_wait(x);
  const int n = (int)blockIdx.x * SR_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31, pieces = K / 8;
  if (n >= N) return;
  const __nv_bfloat16* row = w + (size_t)n * K;
  float acc[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m] = 0.f;
  auto round = [&](int i, bool whole) {        // whole: no lane's pieces lie past the end
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = sr_ld(row, whole ? i + 32 * u : min(i + 32 * u, pieces - 1));
    uint4 xq[MT][U];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int m = 0; m < MT; ++m) xq[m][u] = sr_ldx(x + (size_t)m * ldx, whole ? i + 32 * u : min(i + 32 * u, pieces - 1));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = whole || i + 32 * u < pieces;
      float wf[8];
      sr_floats(in ? q[u] : make_uint4(0u, 0u, 0u, 0u), wf);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        float xf[8];
        sr_floats(in ? xq[m][u] : make_uint4(0u, 0u, 0u, 0u), xf);
        sr_dot(acc[m], wf, xf);
      }
    }
  };
  int i = lane;
  for (const int end = pieces / (32 * U) * (32 * U); i < end; i += 32 * U) round(i, true);
  if (i < pieces) round(i, false);
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const float v = warp_sum(acc[m]);
    if (lane == 0) y[(size_t)m * ldy + n] = __float2bfloat16_rn(v);
  }
}

// y[m][n] = x[m] . w[n] for 3 to 32 rows: a block takes 16 rows of w, its warps share k in pieces of 32, and the products are m16n8k16 with w as the
// 16 rows and eight rows of x as the columns.  Which k a lane's numbers stand for is the same on both sides and otherwise free, so a lane loads
// 16 bytes of a row (four lanes 64) and uses them for two products.  Bound by the weights' way from memory; those of the first pieces are asked
// for before the kernel waits for the one before it where whatever wrote them is known to have ended (early: a kernel that was launched without
// overlap stands between).  The warps' sums meet in shared memory, in the order of the warps.
// us, graphed, here / the library's product: 1024 x 1024 with 8, 16 and 32 rows 2.6 / 4.3, 3.5 / 4.2, 3.4 / 3.8; 2048 x 2048 4.7 / 6.9, 6.4 / 5.6,
// 6.1 / 5.7; 5120 x 2048 6.9 / 6.3, 7.5 / 7.3, 12.3 / 7.5 (more than 16 rows of that many weights go to dense_rows.cu, 9.6).  K a multiple of 8, rows on 16-byte boundaries.
// RT: tiles of 16 rows a block (two where rows of x are many: every block reads them all).
constexpr int FR_MAX = 32, FR_U = 4;
template <int NT, int RT>
__global__ void __launch_bounds__(SR_THREADS) few_rows_kernel(const __nv_bfloat16* x, int ldx, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                              int ldy, int M, int N, int K, int early) {
  constexpr int ROWS = 16 * RT;
  __shared__ float part[SR_WARPS][NT * 8][ROWS + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, n0 = (int)blockIdx.x * ROWS;
  const int pieces = (K + 31) / 32, last = K / 8 - 1;      // last: the last 16 bytes of a row
  const __nv_bfloat16* row[2 * RT];
#pragma unroll
  for (int r = 0; r < 2 * RT; ++r) row[r] = w + (size_t)min(n0 + g + 8 * r, N - 1) * K;
  uint4 a[2 * RT][FR_U];
  auto weights = [&](int c0) {
#pragma unroll
    for (int u = 0; u < FR_U; ++u)
#pragma unroll
      for (int r = 0; r < 2 * RT; ++r) a[r][u] = sr_ld(row[r], min((c0 + u * SR_WARPS) * 4 + t, last));
  };
  if (early) weights(warp);
  pdl_wait();
  pdl_launch_dependents();
  x = after_wait(x);
  if (!early) weights(warp);
  float acc[RT][NT][4];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  for (int c0 = warp; c0 < pieces; c0 += FR_U * SR_WARPS) {
#pragma unroll
    for (int u = 0; u < FR_U; ++u) {
      const int at = (c0 + u * SR_WARPS) * 4 + t;
      uint4 b[NT];
#pragma unroll
      for (int j = 0; j < NT; ++j)
        b[j] = at <= last && 8 * j + g < M ? *reinterpret_cast<const uint4*>(x + (size_t)(8 * j + g) * ldx + at * 8) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const uint4 z = make_uint4(0u, 0u, 0u, 0u), p = at <= last ? a[2 * i][u] : z, q = at <= last ? a[2 * i + 1][u] : z;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          mma_bf16_16816(acc[i][j], p.x, q.x, p.y, q.y, b[j].x, b[j].y);
          mma_bf16_16816(acc[i][j], p.z, q.z, p.w, q.w, b[j].z, b[j].w);
        }
      }
    }
    if (c0 + FR_U * SR_WARPS < pieces) weights(c0 + FR_U * SR_WARPS);
  }
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) part[warp][8 * j + 2 * t + (e & 1)][16 * i + g + 8 * (e >> 1)] = acc[i][j][e];
  __syncthreads();
  for (int i = threadIdx.x; i < NT * 8 * ROWS; i += SR_THREADS) {
    const int m = i / ROWS, r = i - m * ROWS;
    float v = 0.f;
#pragma unroll
    for (int z = 0; z < SR_WARPS; ++z) v += part[z][m][r];
    if (m < M && n0 + r < N) y[(size_t)m * ldy + n0 + r] = __float2bfloat16_rn(v);
  }
}

// y(h, m, n) = sum_k x(h, m, k) w[h][k][n]: a block takes 32 columns of a head, four threads side by side eight columns each, 64 of them one
// k apart; their sums meet by shuffles and in shared memory.  N a multiple of 8 (K of any size), rows of w on 16-byte boundaries.  Rows
// beyond MT go to further blocks, which read the head's weights again (from L2).
template <int MT>
__global__ void __launch_bounds__(SR_THREADS) small_heads_kernel(const __nv_bfloat16* x, long long xs_h, long long xs_m,
                                                                 const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y, long long ys_h,
                                                                 long long ys_m, int M, int N, int K) {
  extern __shared__ float sr_x[];                      // [MT][K]
  __shared__ float part[SR_WARPS][MT][32];
  pdl_wait();
  pdl_launch_dependents();
  x = after_wait(x) + (long long)blockIdx.z * MT * xs_m, y += (long long)blockIdx.z * MT * ys_m, M -= (int)blockIdx.z * MT;
  const int h = blockIdx.y, tid = threadIdx.x, n = (int)blockIdx.x * 32 + (tid & 3) * 8, kg = tid >> 2, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < MT * K; i += SR_THREADS) {
    const int m = i / K, k = i - m * K;
    sr_x[i] = m < M ? __bfloat162float(x[h * xs_h + m * xs_m + k]) : 0.f;
  }
  const __nv_bfloat16* wh = w + (size_t)h * K * N + min(n, N - 8);
  float acc[MT][8];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[m][e] = 0.f;
  constexpr int U = 8;
  bool first = true;
  for (int k0 = kg; k0 < K + kg; k0 += 64 * U) {       // (the same number of turns for every thread: a barrier lies in the first)
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = sr_ld(wh + (size_t)min(k0 + 64 * u, K - 1) * N, 0);
    if (first) __syncthreads();
    first = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + 64 * u;
      if (k >= K) break;
      float wf[8];
      sr_floats(q[u], wf);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const float xv = sr_x[m * K + k];
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[m][e] = fmaf(xv, wf[e], acc[m][e]);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float v = acc[m][e];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < 4) part[warp][m][lane * 8 + e] = v;
    }
  __syncthreads();
  for (int i = tid; i < MT * 32; i += SR_THREADS) {
    const int m = i / 32, c = i & 31;
    float v = 0.f;
#pragma unroll
    for (int z = 0; z < SR_WARPS; ++z) v += part[z][m][c];
    if (m < M && (int)blockIdx.x * 32 + c < N) y[h * ys_h + m * ys_m + blockIdx.x * 32 + c] = __float2bfloat16_rn(v);
  }
}

inline int small_linear(const void* x, int ldx, const void* w, void* y, int ldy, int M, int N, int K, cudaStream_t st) {
  typedef const __nv_bfloat16* B;
  const dim3 grid((N + SR_WARPS - 1) / SR_WARPS);
  if (M == 1)
    LL_CUDA(launch(small_linear_kernel<1>, grid, dim3(SR_THREADS), 0, st, true, (B)x, ldx, (B)w, (__nv_bfloat16*)y, ldy, N, K));
  else
    LL_CUDA(launch(small_linear_kernel<2>, grid, dim3(SR_THREADS), 0, st, true, (B)x, ldx, (B)w, (__nv_bfloat16*)y, ldy, N, K));
  LL_LAUNCH_OK("small_linear_kernel");
  return LL_OK;
}

inline int few_rows(const void* x, int ldx, const void* w, void* y, int ldy, int M, int N, int K, bool early, cudaStream_t st) {
  typedef const __nv_bfloat16* B;
#define LL_FR(NT, RT)                                                                                                                        \
  LL_CUDA(launch(few_rows_kernel<NT, RT>, dim3((N + 16 * RT - 1) / (16 * RT)), dim3(SR_THREADS), 0, st, true, (B)x, ldx, (B)w, (__nv_bfloat16*)y, \
                 ldy, M, N, K, (int)early))
  const bool wide = N >= 32 * sm_count();      // two tiles of rows a block still leave every SM one
  if (M <= 8) LL_FR(1, 1);
  else if (M <= 16 && !wide) LL_FR(2, 1);
  else if (M <= 16) LL_FR(2, 2);
  else if (!wide) LL_FR(4, 1);
  else LL_FR(4, 2);
#undef LL_FR
  LL_LAUNCH_OK("few_rows_kernel");
  return LL_OK;
}

inline int small_heads(const void* x, long long xs_h, long long xs_m, const void* w, void* y, long long ys_h, long long ys_m, int H, int M, int N, int K,
                       cudaStream_t st) {
  typedef const __nv_bfloat16* B;
  const int mt = M == 1 ? 1 : M == 2 ? 2 : 4;
  const dim3 grid((N + 31) / 32, H, (M + mt - 1) / mt);
#define LL_SH(MT)                                                                                                                               \
  LL_CUDA(launch(small_heads_kernel<MT>, grid, dim3(SR_THREADS), sizeof(float) * MT * K, st, true, (B)x, xs_h, xs_m, (B)w, (__nv_bfloat16*)y, ys_h, \
                 ys_m, M, N, K))
  if (mt == 1) LL_SH(1);
  else if (mt == 2) LL_SH(2);
  else LL_SH(4);
#undef LL_SH
  LL_LAUNCH_OK("small_heads_kernel");
  return LL_OK;
}

}  // namespace
}  // namespace llb
