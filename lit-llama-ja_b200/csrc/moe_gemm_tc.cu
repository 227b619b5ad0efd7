// Grouped expert GEMM of the mixture-of-experts feed-forward on the tcgen05 tensor cores (pair_rows.cuh), and the whole layer for more than a
// few tokens.
//
// The (token, choice) pairs are sorted by expert (ll_moe_route) and the rows of the activations are gathered into that order once
// (ll_moe_gather_rows), so every operand is a matrix that TMA can tile:
//   mode 1 (GLU) : h[r][n] = glu(xs[r] . gate_e[n], xs[r] . up_e[n])     w [X][2N][K] = [gate; up]
//   mode 3 (relu^2): h[r][n] = relu(xs[r] . up_e[n])^2                    w [X][N][K]
//   mode 0 (down): y[perm[r]][n] = h[r] . down_e[n]                       w [X][N][K]
// for the sorted rows r of expert e (found from the device-side offsets: no host synchronisation).
// 64 tokens, 32 experts of 2048 x 1024: 5.7 TB/s of weights while all pairs have a tile, and 3.6 rounds of tiles dealt out in four.  8192 rows:
// first projections 97 us with 128-row tiles of one CTA, 72 so; second ones 57 and 45.
// ll_moe_prompt chains the whole layer by programmatic launches; the shared expert's tiles stand before the experts' in the same launch, which
// fills rounds and starts while the router and the sort still run.  Rows brought by gather4 copies instead of a gathering kernel: 301 us a layer
// where it takes 188 (2048 tokens; 128-byte pieces are too many copies).
#include "pair_rows.cuh"

namespace llb {

// moe_ops.cu: the router alone, and the combination, as parts of a chain of launches
int moe_route_only(const void* x, const float* w_router, const float* bias, int M, int dim, int n_experts, int top, int score, const float* correction,
                   float out_scale, int n_groups, int keep_groups, int group_top, int32_t* expert_idx, float* expert_w, int32_t* counts, int32_t* rank,
                   const void* gate_row, float* gate, cudaStream_t st);
int moe_permute(const int32_t* expert_idx, const int32_t* rank, const int32_t* counts, int n_pairs, int X, int32_t* offsets, int32_t* perm, cudaStream_t st);
int moe_combine_rows(const void* y, const float* expert_w, int top, const void* shared_y, const float* gate, void* out, int M, int dim, cudaStream_t st);

namespace {

// xs[r][:] = x[perm[r] / top][:] for the sorted rows r (16-byte pieces): a warp a row, eight pieces a lane on their way
constexpr int GR_WARPS = 8;
__global__ void __launch_bounds__(32 * GR_WARPS) moe_gather_rows_kernel(const uint4* __restrict__ x, long long ldx16, const int32_t* perm,
                                                                        int top, uint4* __restrict__ out, int k16, int n_rows) {
  const int r = blockIdx.x * GR_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_launch_dependents();
  pdl_wait();
  if (r >= n_rows) return;
  const uint4* src = x + (long long)(after_wait(perm)[r] / top) * ldx16;
  uint4* dst = out + (long long)r * k16;
  for (int i0 = lane; i0 < k16; i0 += 256) {
    uint4 u[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (i0 + 32 * j < k16) u[j] = src[i0 + 32 * j];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (i0 + 32 * j < k16) dst[i0 + 32 * j] = u[j];
  }
}

// The (token, choice) pairs of a prompt in the order of their experts, the experts in the order of their tiles' size, and how many row tiles stand before
// each of them in that order: one block, counts and places in shared memory (8192 pairs of 32 experts: 4 us; the pairs of an expert come in no
// fixed order, which no result depends on).  Pairs in registers: up to SORT_PAIRS.  More are counted by the router and placed by a grid of their own
// (moe_permute; counts not null), which leaves the experts to this kernel: in one block
// the rest of 131072 pairs of four experts took a layer of 64 x 64 358 us instead of 282.
constexpr int SORT_THREADS = 1024, SORT_KEPT = 16, SORT_PAIRS = SORT_THREADS * SORT_KEPT, SORT_EXPERTS = 4;      // SORT_EXPERTS: of a thread
__global__ void __launch_bounds__(SORT_THREADS) moe_sort_kernel(const int32_t* expert_idx, const int32_t* counts, int n_pairs, int X,
                                                                int32_t* __restrict__ offsets, int32_t* __restrict__ order, int32_t* __restrict__ first,
                                                                int32_t* __restrict__ perm) {
  extern __shared__ int32_t sort_smem[];
  int32_t *count = sort_smem, *at = count + X, *size = at + X;      // [X] each
  const int tid = threadIdx.x, lane = tid & 31;
  pdl_launch_dependents();
  for (int e = tid; e < X; e += SORT_THREADS) count[e] = 0;
  __syncthreads();
  pdl_wait();
  int32_t mine[SORT_KEPT], rank[SORT_KEPT];
  if (counts == nullptr) {
    expert_idx = after_wait(expert_idx);
#pragma unroll
    for (int j = 0; j < SORT_KEPT; ++j) mine[j] = j * SORT_THREADS + tid < n_pairs ? expert_idx[j * SORT_THREADS + tid] : -1;
#pragma unroll
    for (int j = 0; j < SORT_KEPT; ++j)
      if (mine[j] >= 0) rank[j] = atomicAdd(&count[mine[j]], 1);
  } else {
    counts = after_wait(counts);
    for (int e = tid; e < X; e += SORT_THREADS) count[e] = counts[e];
  }
  __syncthreads();
  // exclusive sums of numbers in shared memory, by the first warp
  auto sums = [&](const int32_t* v, int32_t* keep, int32_t* out) {
    int before = 0;
    for (int e0 = 0; e0 < X; e0 += 32) {
      const int e = e0 + lane, c = e < X ? v[e] : 0;
      int incl = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += u;
      }
      if (e < X) {
        out[e] = before + incl - c;
        if (keep != nullptr) keep[e] = before + incl - c;
      }
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) out[X] = before;
  };
  auto row_tiles = [&](int e) { return (count[e] + MT_NMAX - 1) / MT_NMAX; };
  for (int e = tid; e < X; e += SORT_THREADS) size[e] = count[e] > 0 ? MtWalk::columns(count[e], row_tiles(e)) : 0;
  if (tid < 32) sums(count, at, offsets);
  __syncthreads();
  int place[SORT_EXPERTS];
#pragma unroll
  for (int j = 0; j < SORT_EXPERTS; ++j) {
    const int e = j * SORT_THREADS + tid;
    if (e >= X) break;
    const int own = size[e];
    int n = 0;
#pragma unroll 4
    for (int o = 0; o < X; ++o) n += size[o] > own || (size[o] == own && o < e);
    order[n] = e;
    place[j] = n;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < SORT_EXPERTS; ++j)
    if (j * SORT_THREADS + tid < X) size[place[j]] = row_tiles(j * SORT_THREADS + tid);
  __syncthreads();
  if (tid < 32) sums(size, nullptr, first);
  if (counts == nullptr)
#pragma unroll
    for (int j = 0; j < SORT_KEPT; ++j)
      if (mine[j] >= 0) perm[at[mine[j]] + rank[j]] = j * SORT_THREADS + tid;
}

struct MpScratch {
  int32_t *idx, *offsets, *order, *first, *perm, *counts, *rank;      // counts, rank: of more pairs than the sort keeps
  float *weight, *gate;
  __nv_bfloat16 *xs, *h, *y, *hs, *ys;
  size_t total;
};
MpScratch mp_carve(void* base, int M, int X, int top, int width, int ff, int sff) {
  MpScratch s;
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o += (b + 127) & ~(size_t)127; return r; };
  uint8_t* p = (uint8_t*)base;
  const size_t n = (size_t)M * top;
  s.idx = (int32_t*)(p + take(n * 4)), s.weight = (float*)(p + take(n * 4)), s.perm = (int32_t*)(p + take(n * 4));
  s.offsets = (int32_t*)(p + take((size_t)(X + 1) * 4)), s.order = (int32_t*)(p + take((size_t)X * 4)), s.gate = (float*)(p + take((size_t)M * 4));
  s.first = (int32_t*)(p + take((size_t)(X + 1) * 4));
  s.counts = (int32_t*)(p + take(n > SORT_PAIRS ? (size_t)X * 4 : 0)), s.rank = (int32_t*)(p + take(n > SORT_PAIRS ? n * 4 : 0));
  s.xs = (__nv_bfloat16*)(p + take(n * width * 2)), s.h = (__nv_bfloat16*)(p + take(n * ff * 2)), s.y = (__nv_bfloat16*)(p + take(n * width * 2));
  s.hs = (__nv_bfloat16*)(p + take((size_t)M * sff * 2)), s.ys = (__nv_bfloat16*)(p + take(sff ? (size_t)M * width * 2 : 0));
  s.total = o;
  return s;
}

}  // namespace
}  // namespace llb

using namespace llb;

extern "C" {

int ll_moe_gather_rows(const void* x, int ldx, const int32_t* perm, int top, int n_rows, int K, void* out, ll_stream stream) {
  LL_CHECK_ARG(x && perm && out && top > 0 && n_rows >= 0 && K > 0, "bad moe_gather_rows arguments");
  LL_CHECK_ARG(K % 8 == 0 && ldx % 8 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)out & 15) == 0,
               "moe_gather_rows: rows must be 16-byte aligned bf16");
  if (n_rows == 0) return LL_OK;
  moe_gather_rows_kernel<<<(n_rows + GR_WARPS - 1) / GR_WARPS, 32 * GR_WARPS, 0, (cudaStream_t)stream>>>((const uint4*)x, ldx / 8, perm, top, (uint4*)out,
                                                                                                      K / 8, n_rows);
  LL_LAUNCH_OK("moe_gather_rows_kernel");
  return LL_OK;
}

int ll_moe_grouped_gemm_tc(const void* a, const void* w, const int32_t* offsets, const int32_t* perm, int mode, int n_rows,
                           int n_experts, int N, int K, float limit, float alpha, void* c, int ldc, ll_stream stream) {
  LL_CHECK_ARG(a && w && offsets && perm && c, "moe_grouped_gemm_tc: null pointer");
  LL_CHECK_ARG(n_rows >= 0 && n_experts > 0 && N > 0 && K > 0 && ldc >= N && mode >= 0 && mode <= 3, "bad moe_grouped_gemm_tc arguments");
  const float shift = mode == 2 ? 0.f : 1.f;     // mode 2: the up branch enters as it is
  if (mode == 2) mode = 1;
  LL_CHECK_ARG(K % 8 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)c & 15) == 0,
               "moe_grouped_gemm_tc: K must be a multiple of 8 and the operands 16-byte aligned (TMA rows)");
  if (n_rows == 0) return LL_OK;
  const long long wrows = (long long)n_experts * (mode == 1 ? 2 : 1) * N;
  LL_CHECK_ARG(wrows < (1ll << 31), "moe_grouped_gemm_tc: weight stack too tall for one tensor map");
  MtMaps maps;
  if (int r = mt_maps(w, mode, n_experts, N, K, a, n_rows, &maps)) return r;
  MtParams p{};
  p.part[0] = p.part[1] = mt_part(c, mode, N, K, ldc, limit);
  p.offsets = offsets, p.perm = perm, p.X = n_experts, p.alpha = alpha, p.shift = shift, p.word = wait_word();
  cudaStream_t st = (cudaStream_t)stream;
  if (mode == 1) return launch_moe_pair<1>(maps, maps, p, n_rows, st);
  if (mode == 3) return launch_moe_pair<3>(maps, maps, p, n_rows, st);
  return launch_moe_pair<0>(maps, maps, p, n_rows, st);
}

int ll_moe_prompt_supported(int M, int width, int n_experts, int ff, int shared_ff) {
  return M >= 1 && M < (1 << 24) && width > 0 && width % 8 == 0 && ff > 0 && ff % 8 == 0 && shared_ff >= 0 && shared_ff % 8 == 0 &&
         n_experts <= SORT_THREADS * SORT_EXPERTS &&
         (long long)n_experts * 2 * ff < (1ll << 31) && (long long)n_experts * width < (1ll << 31);
}

size_t ll_moe_prompt_scratch_bytes(int M, int width, int n_experts, int top, int ff, int shared_ff) {
  return mp_carve(nullptr, M, n_experts, top, width, ff, shared_ff).total;
}

int ll_moe_prompt(const void* x, const float* w_router, const float* bias, const float* correction, int score, float out_scale, int n_groups,
                  int keep_groups, int group_top, const void* w_gu, const void* w_down, const void* ws_in, const void* ws_down, int M, int width,
                  int n_experts, int top, int ff, int shared_ff, int shared_gate, int mode, float limit, float alpha, float shared_limit, void* out,
                  void* scratch, ll_stream stream) {
  LL_CHECK_ARG(x && w_router && w_gu && w_down && out && scratch && (shared_ff == 0 || (ws_in && ws_down)), "moe_prompt: null pointer");
  LL_CHECK_ARG(n_experts > 0 && top > 0 && top <= n_experts && mode >= 1 && mode <= 3 && (long long)M * top < (1ll << 30), "bad moe_prompt arguments");
  if (!ll_moe_prompt_supported(M, width, n_experts, ff, shared_ff)) {
    set_error("moe_prompt takes widths in multiples of 8 (M=%d width=%d experts=%d ff=%d shared=%d)", M, width, n_experts, ff, shared_ff);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG((((uintptr_t)x | (uintptr_t)w_gu | (uintptr_t)w_down | (uintptr_t)ws_in | (uintptr_t)ws_down | (uintptr_t)scratch | (uintptr_t)out) & 15) == 0,
               "moe_prompt: rows must be 16-byte aligned bf16");
  cudaStream_t st = (cudaStream_t)stream;
  const MpScratch s = mp_carve(scratch, M, n_experts, top, width, ff, shared_ff);
  const int n = M * top, up = mode == 2 ? 1 : mode;
  const __nv_bfloat16* gate_row = shared_ff && shared_gate ? (const __nv_bfloat16*)ws_in + (size_t)(up == 1 ? 2 : 1) * shared_ff * width : nullptr;
  int32_t* const counts = n > SORT_PAIRS ? s.counts : nullptr;
  if (counts != nullptr) LL_CUDA(cudaMemsetAsync(counts, 0, sizeof(int32_t) * n_experts, st));
  if (int r = moe_route_only(x, w_router, bias, M, width, n_experts, top, score, correction, out_scale, n_groups, keep_groups, group_top, s.idx, s.weight,
                             counts, counts != nullptr ? s.rank : nullptr, gate_row, s.gate, st))
    return r;
  if (counts != nullptr)
    if (int r = moe_permute(s.idx, s.rank, counts, n, n_experts, s.offsets, s.perm, st)) return r;
  LL_CUDA(launch(moe_sort_kernel, dim3(1), dim3(SORT_THREADS), 3 * sizeof(int32_t) * n_experts, st, true, (const int32_t*)s.idx, (const int32_t*)counts, n,
                 n_experts, s.offsets, s.order, s.first, s.perm));
  LL_LAUNCH_OK("moe_sort_kernel");
  LL_CUDA(launch(moe_gather_rows_kernel, dim3((n + GR_WARPS - 1) / GR_WARPS), dim3(32 * GR_WARPS), 0, st, true, (const uint4*)x, (long long)(width / 8),
                 (const int32_t*)s.perm, top, (uint4*)s.xs, width / 8, n));
  LL_LAUNCH_OK("moe_gather_rows_kernel");
  // first projections with their unit
  MtMaps experts, shared;
  if (int r = mt_maps(w_gu, up, n_experts, ff, width, s.xs, n, &experts)) return r;
  shared = experts;
  if (shared_ff)
    if (int r = mt_maps(ws_in, up, 1, shared_ff, width, x, M, &shared)) return r;
  MtParams p{};
  p.part[0] = mt_part(s.h, up, ff, width, ff, limit), p.part[1] = mt_part(s.hs, up, shared_ff, width, shared_ff, shared_limit);
  p.offsets = s.offsets, p.perm = s.perm, p.order = s.order, p.first = s.first, p.X = n_experts, p.M = shared_ff ? M : 0, p.cuts = (p.M + MT_NMAX - 1) / MT_NMAX, p.early = 1;
  p.alpha = alpha, p.shift = mode == 2 ? 0.f : 1.f, p.word = wait_word();
  if (int r = up == 1 ? launch_moe_pair<1>(experts, shared, p, n, st) : launch_moe_pair<3>(experts, shared, p, n, st)) return r;
  // second ones
  if (int r = mt_maps(w_down, 0, n_experts, width, ff, s.h, n, &experts)) return r;
  shared = experts;
  if (shared_ff)
    if (int r = mt_maps(ws_down, 0, 1, width, shared_ff, s.hs, M, &shared)) return r;
  p.part[0] = mt_part(s.y, 0, width, ff, width, 0.f), p.part[1] = mt_part(s.ys, 0, width, shared_ff, width, 0.f);
  p.early = 0;
  if (int r = launch_moe_pair<0>(experts, shared, p, n, st)) return r;
  return moe_combine_rows(s.y, s.weight, top, shared_ff ? s.ys : nullptr, gate_row ? s.gate : nullptr, out, M, width, st);
}

// 0, or the code of the first bounded wait that ran out in a kernel of this file (1: ring slot, 2: operands, 3: accumulator,
// 4: accumulator to be free).
// Synchronises the device.
int ll_moe_tc_error(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_pair_rows_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // extern "C"
