// Mixture-of-experts feed-forward of a few tokens (decoding): route, then two kernels that read the chosen experts' weights once, a warp per
// output, and the combination as the second one's epilogue.  No sort by expert: a token's choices are walked as they are.
//
//   up    h[m][c][f] = unit(x[m] . W_gate[f], x[m] . W_up[f]) for the token's choices c < top, and for the shared expert, whose gate logit is
//         one more row of its weights
//   down  out[m][n] = sum_c w[m][c] * bf16(h[m][c] . W_down[n])  (+ sigmoid(gate) * bf16(hs[m] . W_sdown[n]))
//
// Bound by the weights' way from memory: 69 MB for one token of width 2048 (4 of 32 experts of 1024, a shared one of 1536), 10.6 us at the
// copy rate.  The shared expert's blocks come first and do not wait for the router.
// us a call (graphed), sorted and grouped with dense layers for the shared expert / here: that size at 1, 2, 4, 8 tokens 98 (72) / 25 (23),
// 97 (77) / 34 (32), 99 (80) / 51 (49), 122 (108) / 80 (77).  Which steps come here: by what they read again (the module's rule).
#include "row_loads.cuh"

namespace llb {

// moe_ops.cu: the router alone
int moe_route_only(const void* x, const float* w_router, const float* bias, int M, int dim, int n_experts, int top, int score, const float* correction,
                   float out_scale, int n_groups, int keep_groups, int group_top, int32_t* expert_idx, float* expert_w, int32_t* counts, int32_t* rank,
                   const void* gate_row, float* gate, cudaStream_t st);

namespace {

constexpr int MS_THREADS = 256, MS_WARPS = MS_THREADS / 32;

struct MsParams {
  const __nv_bfloat16 *x, *w_gu, *w_down, *ws_in, *ws_down;      // ws_*: shared expert, or null
  const int32_t* idx;
  const float* weight;
  __nv_bfloat16 *h, *hs, *gate, *out;
  int M, width, top, ff, sff, mode, shared_gate;            // mode: 1, 2 gated unit with / without the up branch's shift, 3 relu^2
  float limit, alpha, slimit;
};

__device__ __forceinline__ float ms_unit(float g, float u, const MsParams& p, float limit) {
  if (p.mode == 3) return fmaxf(u, 0.f) * fmaxf(u, 0.f);
  g = fminf(g, limit), u = fminf(fmaxf(u, -limit), limit);
  return g / (1.f + expf(-p.alpha * g)) * (u + (p.mode == 1 ? 1.f : 0.f));
}
// This lane's part of the dot products of R rows with R vectors (or all with the first: SAME) of n numbers; U 16-byte loads of every row in
// flight.  Past the end a lane takes the last piece again and drops its sum.
template <int R, int U, bool SAME>
__device__ __forceinline__ void ms_rows(const __nv_bfloat16* const (&row)[R], const __nv_bfloat16* const (&x)[R], int n, float (&part)[R]) {
  const int lane = threadIdx.x & 31, pieces = n / 8;
#pragma unroll
  for (int r = 0; r < R; ++r) part[r] = 0.f;
  for (int i = lane; i < pieces; i += 32 * U) {
    uint4 w[R][U];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) w[r][u] = sr_ld(row[r], min(i + 32 * u, pieces - 1));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = i + 32 * u < pieces;
      float xf[8];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r == 0 || !SAME) sr_floats(in ? reinterpret_cast<const uint4*>(x[r])[i + 32 * u] : make_uint4(0u, 0u, 0u, 0u), xf);
        float wf[8];
        sr_floats(w[r][u], wf);
        float sum = part[r];
        sr_dot(sum, wf, xf);
        part[r] = in ? sum : part[r];
      }
    }
  }
}

// blockIdx.y: token and choice, the shared expert's first; blockIdx.x: 2 outputs a warp
__global__ void __launch_bounds__(MS_THREADS) moe_step_up_kernel(const MsParams p) {
  pdl_launch_dependents();
  const int shared = p.ws_in != nullptr ? p.M : 0, lane = threadIdx.x & 31;
  const bool is_shared = (int)blockIdx.y < shared;
  const int pair = (int)blockIdx.y - shared, m = is_shared ? (int)blockIdx.y : pair / p.top;
  const int ff = is_shared ? p.sff : p.ff, f = ((int)blockIdx.x * MS_WARPS + (threadIdx.x >> 5)) * 2;
  const bool gated = p.mode != 3;
  const __nv_bfloat16* x = p.x + (size_t)m * p.width;
  const __nv_bfloat16* w = p.ws_in;
  if (!is_shared) {
    pdl_wait();                                // the router's choice
    w = p.w_gu + (size_t)p.idx[pair] * (gated ? 2 : 1) * ff * p.width;
  }
  if (f < ff) {
    const __nv_bfloat16* wu = gated ? w + (size_t)ff * p.width : w;
    const size_t at0 = (size_t)f * p.width, at1 = (size_t)min(f + 1, ff - 1) * p.width;
    const __nv_bfloat16* const row[4] = {w + at0, wu + at0, w + at1, wu + at1};
    const __nv_bfloat16* const xs[4] = {x, x, x, x};
    float a[4];
    ms_rows<4, 4, true>(row, xs, p.width, a);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      a[r] = warp_sum(a[r]);
      if (is_shared) a[r] = bf16r(a[r]);       // (there the projection's outputs are bf16 numbers before the unit)
    }
    const float limit = is_shared ? p.slimit : p.limit, o0 = ms_unit(a[0], a[1], p, limit), o1 = ms_unit(a[2], a[3], p, limit);
    __nv_bfloat16* h = (is_shared ? p.hs + (size_t)m * ff : p.h + (size_t)pair * ff) + f;
    if (lane == 0) {
      h[0] = __float2bfloat16_rn(o0);
      if (f + 1 < ff) h[1] = __float2bfloat16_rn(o1);
    }
  } else if (is_shared && p.shared_gate && f < ff + 2) {
    const __nv_bfloat16* const row[1] = {w + (size_t)(gated ? 2 : 1) * ff * p.width};
    const __nv_bfloat16* const xs[1] = {x};
    float a[1];
    ms_rows<1, 4, true>(row, xs, p.width, a);
    a[0] = warp_sum(a[0]);
    if (lane == 0) p.gate[m] = __float2bfloat16_rn(a[0]);
  }
}

// blockIdx.y: token; an output a warp
__global__ void __launch_bounds__(MS_THREADS) moe_step_down_kernel(const MsParams p) {
  pdl_wait();
  const int m = blockIdx.y, n = (int)blockIdx.x * MS_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (n >= p.width) return;
  float ys = 0.f;
  if (p.ws_down != nullptr) {
    const __nv_bfloat16* const row[1] = {p.ws_down + (size_t)n * p.sff};
    const __nv_bfloat16* const xs[1] = {p.hs + (size_t)m * p.sff};
    float a[1];
    ms_rows<1, 6, true>(row, xs, p.sff, a);
    ys = a[0];
  }
  float v = 0.f;
  for (int c = 0; c < p.top; c += 4) {       // four choices side by side
    const __nv_bfloat16 *row[4], *xs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t pr = (size_t)m * p.top + min(c + j, p.top - 1);
      row[j] = p.w_down + ((size_t)p.idx[pr] * p.width + n) * p.ff, xs[j] = p.h + pr * p.ff;
    }
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    if (c + 2 < p.top) {
      const __nv_bfloat16* const r4[4] = {row[0], row[1], row[2], row[3]};
      const __nv_bfloat16* const x4[4] = {xs[0], xs[1], xs[2], xs[3]};
      ms_rows<4, 4, false>(r4, x4, p.ff, a);
    } else {
      const __nv_bfloat16* const r2[2] = {row[0], row[1]};
      const __nv_bfloat16* const x2[2] = {xs[0], xs[1]};
      float b[2];
      ms_rows<2, 4, false>(r2, x2, p.ff, b);
      a[0] = b[0], a[1] = b[1];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = warp_sum(a[j]);
      if (c + j < p.top) v += p.weight[(size_t)m * p.top + c + j] * bf16r(a[j]);
    }
  }
  if (p.ws_down != nullptr) v += (p.shared_gate ? 1.f / (1.f + expf(-__bfloat162float(p.gate[m]))) : 1.f) * bf16r(warp_sum(ys));
  if (lane == 0) p.out[(size_t)m * p.width + n] = __float2bfloat16_rn(v);
}

struct MsScratch {
  int32_t* idx;
  float* weight;
  __nv_bfloat16 *h, *hs, *gate;
  size_t total;
};
MsScratch ms_carve(void* base, int M, int top, int ff, int sff) {
  MsScratch s;
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o += (b + 127) & ~(size_t)127; return r; };
  uint8_t* p = (uint8_t*)base;
  s.idx = (int32_t*)(p + take((size_t)M * top * 4));
  s.weight = (float*)(p + take((size_t)M * top * 4));
  s.h = (__nv_bfloat16*)(p + take((size_t)M * top * ff * 2));
  s.hs = (__nv_bfloat16*)(p + take((size_t)M * sff * 2));
  s.gate = (__nv_bfloat16*)(p + take((size_t)M * 2));
  s.total = o;
  return s;
}

}  // namespace
}  // namespace llb

using namespace llb;

extern "C" {

int ll_moe_step_supported(int M, int width, int ff, int shared_ff) {
  return M >= 1 && M <= 8 && width > 0 && width % 8 == 0 && ff > 0 && ff % 8 == 0 && shared_ff >= 0 && shared_ff % 8 == 0;
}

size_t ll_moe_step_scratch_bytes(int M, int n_experts, int top, int ff, int shared_ff) { return ms_carve(nullptr, M, top, ff, shared_ff).total; }

int ll_moe_step(const void* x, const float* w_router, const float* bias, const float* correction, int score, float out_scale, int n_groups,
                int keep_groups, int group_top, const void* w_gu, const void* w_down, const void* ws_in, const void* ws_down, int M, int width,
                int n_experts, int top, int ff, int shared_ff, int shared_gate, int mode, float limit, float alpha, float shared_limit, void* out,
                void* scratch, ll_stream stream) {
  LL_CHECK_ARG(x && w_router && w_gu && w_down && out && scratch && (shared_ff == 0 || (ws_in && ws_down)), "moe_step: null pointer");
  LL_CHECK_ARG(n_experts > 0 && top > 0 && top <= n_experts && mode >= 1 && mode <= 3, "bad moe_step arguments");
  if (!ll_moe_step_supported(M, width, ff, shared_ff)) {
    set_error("moe_step takes 1 to 8 tokens and widths in multiples of 8 (M=%d width=%d ff=%d shared=%d)", M, width, ff, shared_ff);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG((((uintptr_t)x | (uintptr_t)w_gu | (uintptr_t)w_down | (uintptr_t)ws_in | (uintptr_t)ws_down | (uintptr_t)scratch) & 15) == 0,
               "moe_step: rows must be 16-byte aligned bf16");
  cudaStream_t st = (cudaStream_t)stream;
  const MsScratch s = ms_carve(scratch, M, top, ff, shared_ff);
  if (int r = moe_route_only(x, w_router, bias, M, width, n_experts, top, score, correction, out_scale, n_groups, keep_groups, group_top, s.idx, s.weight,
                             nullptr, nullptr, nullptr, nullptr, st))
    return r;
  typedef const __nv_bfloat16* B;
  const MsParams p{(B)x, (B)w_gu, (B)w_down, shared_ff ? (B)ws_in : nullptr, shared_ff ? (B)ws_down : nullptr, s.idx, s.weight, s.h, s.hs, s.gate,
                   (__nv_bfloat16*)out, M, width, top, ff, shared_ff, mode, shared_gate, limit, alpha, shared_limit};
  const int most = ff > shared_ff + 2 ? ff : shared_ff + 2;      // (+ 2: the shared expert's gate row)
  LL_CUDA(launch(moe_step_up_kernel, dim3((most + 2 * MS_WARPS - 1) / (2 * MS_WARPS), M * top + (shared_ff ? M : 0)), dim3(MS_THREADS), 0, st, true, p));
  LL_LAUNCH_OK("moe_step_up_kernel");
  LL_CUDA(launch(moe_step_down_kernel, dim3((width + MS_WARPS - 1) / MS_WARPS, M), dim3(MS_THREADS), 0, st, true, p));
  LL_LAUNCH_OK("moe_step_down_kernel");
  return LL_OK;
}

}  // extern "C"
