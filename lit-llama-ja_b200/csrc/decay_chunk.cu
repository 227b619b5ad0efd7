// The linear recurrence of decay_scan.cu for prompts in bf16, on tensor cores: with one decay per head and token (or one constant
// per head) the walk over tokens can be cut into chunks of 64 whose work is matrix products.  Per (sequence, head), G_t the sum of
// log a over the chunk up to token t:
//
//   collect   D_c = sum_s e^(G_last - G_s) (ks_s k_s) v_s^T             what a chunk adds to the state      (a block per chunk)
//   pass      S_c = e^(G_last) S_(c-1) + D_c                            the state before every chunk        (fp32, element by element)
//   read      y_t = qs ( sum_(s <= t) e^(G_t - G_s) ks_s (q_t.k_s) v_s + e^(G_t) S_(c-1)^T q_t ) + skip v_t     (a block per chunk)
//
// q, k and v are bf16 as they stand, so only the fp32 factors have to be split for the bf16 tensor cores (fp32 accumulation):
// e^(..) ks k enters D as three bf16 terms (24 bits: what is carried on is as exact as the walk's fp32), the chunk's weights and
// the state meet v and q as two terms (16 bits, the sum of both products in fp32).  Sums of log a are formed in fp64, so that the
// difference of two of them keeps its digits whatever lies before it in the chunk.  The state handed on is fp32.
//
// UNIT: the last of the p columns of every head is the constant 1 and not part of v (the normaliser of a matrix memory rides in the same
// products).  p is then one more than a multiple of 8: the chunks' states are kept with rows of p + 3 numbers, the caller's state and y are
// read and written one number at a time, and what meets v and q has three terms (24 bits), as the walk this form replaces is fp32.
// 2048 tokens, 8 heads of 128 x 257: the walk took 496 us (a chain of 2048 steps), collect + pass + read take 24 + 14 + 51.  Column tiles of
// 64: with three terms of the state a tile of 128 leaves one block per SM.
#include "chunk_mma.cuh"
#include "dense_rows.cuh"

namespace llb {

// Blocks of eight warps: four rows of 16 x two halves of the block's PT value columns (64, or 128 for wide heads).  Everything a
// block reads is requested before anything is worked on, so that a block waits for memory about once.

// G[t] = sum over the chunk's tokens up to t of log a (tokens past the end: a = 1), by the first warp, two tokens a lane
__device__ __forceinline__ void dc_log_sums(const float* __restrict__ a, int a_row, int h, size_t m0, int len, double* G) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  double v[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = 2 * lane + e;
    v[e] = t < len ? fmax((double)logf(a[(m0 + t) * a_row + h]), DC_LOG_MIN) : 0.0;
  }
  dc_running_sums(v, G);
}

// grid (chunks * p tiles, H, B): D_c into dst[((b * H + h) * chunks + c)][n][p], e^(G_last) into total[(b * H + h) * chunks + c].
// NP: n rounded up to 16, 32, 64 or 128.
template <int NP, int PT, bool SILU, bool UNIT>
__global__ void __launch_bounds__(DC_THREADS, 2) decay_collect_kernel(const __nv_bfloat16* __restrict__ k, int k_stride,
                                                                      const __nv_bfloat16* __restrict__ v, int v_stride,
                                                                      const float* __restrict__ a, int a_row, const float* __restrict__ ks,
                                                                      float* __restrict__ dst, float* __restrict__ total, int Tn, int H,
                                                                      int qk_heads, int n, int p, int ptiles) {
  constexpr int LK = NP + 8, LV = PT + 8, NF = PT / 16;        // NF: 8-column fragments of a warp's half
  const int pv = UNIT ? p - 1 : p, pp = UNIT ? p + 3 : p;      // columns of v; numbers in a row of a chunk's state
  extern __shared__ __align__(16) unsigned char dc_smem[];
  __nv_bfloat16* Ks = (__nv_bfloat16*)dc_smem;                // [3 terms][64][LK]
  __nv_bfloat16* Vs = Ks + 3 * DC_L * LK;                     // [64][LV]
  __shared__ double G[DC_L];
  __shared__ float wgt[DC_L];
  const int c = blockIdx.x / ptiles, p0 = (blockIdx.x - c * ptiles) * PT, h = blockIdx.y, b = blockIdx.z, g = h / (H / qk_heads);
  const int chunks = gridDim.x / ptiles, t0 = c * DC_L, len = min(DC_L, Tn - t0), tid = threadIdx.x;
  const size_t m0 = (size_t)b * Tn + t0;
  DcTile<NP> kt;
  DcTile<PT> vt;
  kt.load(k + m0 * k_stride + (size_t)g * n, k_stride, len, n);
  vt.load(v + m0 * v_stride + (size_t)h * pv + p0, v_stride, len, pv - p0);
  if (UNIT) vt.one(pv - p0, len);
  const float ksv = (tid < len && ks) ? ks[(m0 + tid) * H + h] : 1.f;
  dc_log_sums(a, a_row, h, m0, len, G);
  vt.template store<SILU>(Vs, LV);
  __syncthreads();
  if (tid < DC_L) wgt[tid] = tid < len ? expf((float)(G[DC_L - 1] - G[tid])) * ksv : 0.f;
  if (tid == 0 && p0 == 0) total[((size_t)b * H + h) * chunks + c] = expf((float)G[DC_L - 1]);
  __syncthreads();
#pragma unroll
  for (int it = 0; it < DcTile<NP>::IT; ++it) {
    const int i = it * DC_THREADS + tid, s = i / (NP / 8), ch = (i % (NP / 8)) * 8;
    if (i >= DcTile<NP>::UNITS) break;
    const uint4 u = dc_in8<SILU>(kt.u[it]);
    const float w = wgt[s];
    const uint32_t in[4] = {u.x, u.y, u.z, u.w};
    uint32_t out[3][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float x0 = bf16_bits_to_f32(in[q] & 0xffffu) * w, x1 = bf16_bits_to_f32(in[q] >> 16) * w;
      out[0][q] = dc_term(x0, x1);
      out[1][q] = dc_term(x0, x1);
      out[2][q] = pack_bf16(x0, x1);
    }
#pragma unroll
    for (int z = 0; z < 3; ++z) *(uint4*)&Ks[(z * DC_L + s) * LK + ch] = make_uint4(out[z][0], out[z][1], out[z][2], out[z][3]);
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31, c0 = (warp >> 2) * (PT / 2);
  float* D = dst + (((size_t)b * H + h) * chunks + c) * (size_t)n * pp;
#pragma unroll 1
  for (int mt = warp & 3; mt < NP / 16; mt += 4) {
    if (mt * 16 >= n) break;
    float acc[NF][4];
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[f][0] = acc[f][1] = acc[f][2] = acc[f][3] = 0.f;
#pragma unroll
    for (int st = 0; st < DC_L / 16; ++st) {
      uint32_t bf[NF / 2][4];
#pragma unroll
      for (int d = 0; d < NF / 2; ++d)
        dc_ldmatrix_trans(bf[d], &Vs[(st * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LV + c0 + d * 16 + (lane >> 4) * 8]);
#pragma unroll
      for (int z = 2; z >= 0; --z) {                          // the smallest term first
        uint32_t af[4];
        dc_ldmatrix_trans(af, &Ks[(z * DC_L + st * 16 + (lane & 7) + (lane >> 4) * 8) * LK + mt * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
        for (int d = 0; d < NF / 2; ++d) {
          mma_bf16_16816(acc[2 * d], af[0], af[1], af[2], af[3], bf[d][0], bf[d][1]);
          mma_bf16_16816(acc[2 * d + 1], af[0], af[1], af[2], af[3], bf[d][2], bf[d][3]);
        }
      }
    }
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = mt * 16 + (lane >> 2) + e * 8, col = p0 + c0 + f * 8 + (lane & 3) * 2;
        if (i < n && col < p) *(float2*)(D + (size_t)i * pp + col) = make_float2(acc[f][2 * e], acc[f][2 * e + 1]);
      }
  }
}

// Per (sequence, head), two neighbouring elements of the state a thread: D_c is replaced by the state before chunk c, the state
// after the last chunk goes back to `state`.
template <bool UNIT>
__global__ void __launch_bounds__(128) decay_pass_kernel(float* __restrict__ chunk_state, const float* __restrict__ total,
                                                         float* __restrict__ state, const int32_t* __restrict__ pos_ids, int chunks,
                                                         int np2, int n, int p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np2) return;
  const size_t bh = blockIdx.y;
  float2* D = (float2*)chunk_state + bh * chunks * np2 + i;
  // UNIT: where the pair sits in the caller's rows of p numbers, and whether its two numbers are there at all
  const int r = UNIT ? (2 * i) / (p + 3) : 0, c = UNIT ? 2 * i - r * (p + 3) : 0;
  float* S = UNIT ? state + bh * ((size_t)n * p) + (size_t)r * p + c : state + (bh * np2 + i) * 2;
  const bool in0 = !UNIT || c < p, in1 = !UNIT || c + 1 < p;
  if (!in0) return;
  const float* tot = total + bh * chunks;
  float2 s = make_float2(0.f, 0.f);
  if (pos_ids[0] != 0) {
    if (UNIT) s = make_float2(S[0], in1 ? S[1] : 0.f);
    else s = *(const float2*)S;
  }
  constexpr int AHEAD = 16;                                   // chunks whose loads are in flight together
  for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
    float2 d[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) d[j] = c0 + j < chunks ? D[(size_t)(c0 + j) * np2] : make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (c0 + j < chunks) {
        const float w = tot[c0 + j];
        D[(size_t)(c0 + j) * np2] = s;
        s = make_float2(w * s.x + d[j].x, w * s.y + d[j].y);
      }
  }
  if (UNIT) {
    S[0] = s.x;
    if (in1) S[1] = s.y;
  } else {
    *(float2*)S = s;
  }
}

// grid (chunks * p tiles, H, B).  A warp owns 16 consecutive tokens and half of the block's columns; its queries come from global
// memory straight into fragments.
template <int NP, int PT, bool SILU, bool UNIT>
__global__ void __launch_bounds__(DC_THREADS, 2) decay_read_kernel(
    const __nv_bfloat16* __restrict__ q, int q_stride, const __nv_bfloat16* __restrict__ k, int k_stride, const __nv_bfloat16* __restrict__ v,
    int v_stride, const float* __restrict__ a, int a_row, const float* __restrict__ ks, const float* __restrict__ skip, float qs,
    const float* __restrict__ chunk_state, const int32_t* __restrict__ pos_ids, float* __restrict__ y, int Tn, int H, int qk_heads, int n,
    int p, int ptiles) {
  constexpr int LK = NP + 8, LV = PT + 8, NF = PT / 16, ZT = UNIT ? 3 : 2;      // ZT: bf16 terms of a weight and of the state
  const int pv = UNIT ? p - 1 : p, pp = UNIT ? p + 3 : p;
  extern __shared__ __align__(16) unsigned char dc_smem[];
  __nv_bfloat16* Ks = (__nv_bfloat16*)dc_smem;                // [64][LK]
  __nv_bfloat16* Vs = Ks + DC_L * LK;                         // [64][LV]
  __nv_bfloat16* Ss = Vs + DC_L * LV;                         // [ZT terms][NP][LV]
  __shared__ double G[DC_L];
  __shared__ float kw[DC_L];
  const int c = blockIdx.x / ptiles, p0 = (blockIdx.x - c * ptiles) * PT, h = blockIdx.y, b = blockIdx.z, g = h / (H / qk_heads);
  const int chunks = gridDim.x / ptiles, t0 = c * DC_L, len = min(DC_L, Tn - t0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, row0 = (warp & 3) * 16, c0 = (warp >> 2) * (PT / 2);
  const size_t m0 = (size_t)b * Tn + t0;
  const bool has_state = c > 0 || pos_ids[0] != 0;
  const float* S = chunk_state + (((size_t)b * H + h) * chunks + c) * (size_t)n * pp;
  DcTile<NP> kt;
  DcTile<PT> vt;
  kt.load(k + m0 * k_stride + (size_t)g * n, k_stride, len, n);
  vt.load(v + m0 * v_stride + (size_t)h * pv + p0, v_stride, len, pv - p0);
  if (UNIT) vt.one(pv - p0, len);
  const float ksv = (tid < len && ks) ? ks[(m0 + tid) * H + h] : 1.f;
  // the state's rows in rounds of eight 16-byte units per thread: the first round is requested with the keys and values
  constexpr int SU = NP * (PT / 4), SR = (SU + 8 * DC_THREADS - 1) / (8 * DC_THREADS);
  float4 sv[8];
  auto state_load = [&](int rd) {
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int i = (rd * 8 + it) * DC_THREADS + tid, r = i / (PT / 4), col = (i % (PT / 4)) * 4;
      sv[it] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < SU && r < n && p0 + col < p) sv[it] = *(const float4*)(S + (size_t)r * pp + p0 + col);
    }
  };
  if (has_state) state_load(0);
  kt.template store<SILU>(Ks, LK);
  vt.template store<SILU>(Vs, LV);
  if (has_state) {
#pragma unroll
    for (int rd = 0; rd < SR; ++rd) {
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int i = (rd * 8 + it) * DC_THREADS + tid, r = i / (PT / 4), col = (i % (PT / 4)) * 4;
        if (i >= SU) break;
        float4 f = sv[it];
        uint32_t z0[ZT], z1[ZT];
        dc_terms<ZT>(f.x, f.y, z0);
        dc_terms<ZT>(f.z, f.w, z1);
#pragma unroll
        for (int z = 0; z < ZT; ++z) *(uint2*)&Ss[(z * NP + r) * LV + col] = make_uint2(z0[z], z1[z]);
      }
      if (rd + 1 < SR) state_load(rd + 1);
    }
  }
  if (tid < DC_L) kw[tid] = tid < len ? ksv * qs : 0.f;
  dc_log_sums(a, a_row, h, m0, len, G);
  // query fragments: rows (lane / 4) and + 8 of the warp's 16, columns (lane % 4) * 2 and + 8 of every 16
  uint32_t qf[NP / 16][4];
  const int r0 = row0 + (lane >> 2);
#pragma unroll
  for (int kk = 0; kk < NP / 16; ++kk)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = r0 + (e & 1) * 8, col = kk * 16 + (lane & 3) * 2 + (e >> 1) * 8;
      qf[kk][e] = (r < len && col < n) ? dc_in2<SILU>(*(const uint32_t*)(q + (m0 + r) * q_stride + (size_t)g * n + col)) : 0u;
    }
  __syncthreads();
  if (row0 >= len) return;
  float o[NF][4];
#pragma unroll
  for (int f = 0; f < NF; ++f) o[f][0] = o[f][1] = o[f][2] = o[f][3] = 0.f;
  const double g0 = G[r0], g1 = G[r0 + 8];
  if (has_state) {
#pragma unroll
    for (int kk = 0; kk < NP / 16; ++kk)
#pragma unroll
      for (int z = ZT - 1; z >= 0; --z)
#pragma unroll
        for (int d = 0; d < NF / 2; ++d) {
          uint32_t bf[4];
          dc_ldmatrix_trans(bf, &Ss[(z * NP + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LV + c0 + d * 16 + (lane >> 4) * 8]);
          mma_bf16_16816(o[2 * d], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], bf[0], bf[1]);
          mma_bf16_16816(o[2 * d + 1], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], bf[2], bf[3]);
        }
    const float e0 = expf((float)g0) * qs, e1 = expf((float)g1) * qs;
#pragma unroll
    for (int f = 0; f < NF; ++f) o[f][0] *= e0, o[f][1] *= e0, o[f][2] *= e1, o[f][3] *= e1;
  }
#pragma unroll
  for (int st = 0; st < DC_L / 16; ++st) {                    // 16 keys at a time, none that lie after all of the warp's tokens
    if (st * 16 > row0) break;
    float sc[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) sc[j][0] = sc[j][1] = sc[j][2] = sc[j][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < NP / 16; ++kk) {
      uint32_t bf[4];
      dc_ldmatrix(bf, &Ks[(st * 16 + (lane & 7) + (lane >> 4) * 8) * LK + kk * 16 + ((lane >> 3) & 1) * 8]);
      mma_bf16_16816(sc[0], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], bf[0], bf[1]);
      mma_bf16_16816(sc[1], qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], bf[2], bf[3]);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int s = st * 16 + j * 8 + (lane & 3) * 2 + (e & 1), r = r0 + (e >> 1) * 8;
        sc[j][e] = s <= r ? sc[j][e] * (expf((float)((e >> 1 ? g1 : g0) - G[s])) * kw[s]) : 0.f;
      }
    uint32_t at[ZT][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t z0[ZT];
        dc_terms<ZT>(sc[j][2 * e], sc[j][2 * e + 1], z0);
#pragma unroll
        for (int z = 0; z < ZT; ++z) at[z][2 * j + e] = z0[z];
      }
#pragma unroll
    for (int d = 0; d < NF / 2; ++d) {
      uint32_t bf[4];
      dc_ldmatrix_trans(bf, &Vs[(st * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LV + c0 + d * 16 + (lane >> 4) * 8]);
#pragma unroll
      for (int z = ZT - 1; z >= 0; --z) {
        mma_bf16_16816(o[2 * d], at[z][0], at[z][1], at[z][2], at[z][3], bf[0], bf[1]);
        mma_bf16_16816(o[2 * d + 1], at[z][0], at[z][1], at[z][2], at[z][3], bf[2], bf[3]);
      }
    }
  }
  const float sk = skip ? skip[h] : 0.f;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = r0 + e * 8;
    if (r >= len) continue;
    float* yr = y + (m0 + r) * (size_t)H * p + (size_t)h * p + p0 + c0;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const int col = f * 8 + (lane & 3) * 2;
      if (p0 + c0 + col >= p) continue;
      float v0 = o[f][2 * e], v1 = o[f][2 * e + 1];
      if (skip) {
        v0 += sk * __bfloat162float(Vs[r * LV + c0 + col]);
        v1 += sk * __bfloat162float(Vs[r * LV + c0 + col + 1]);
      }
      if (UNIT) {
        yr[col] = v0;
        if (p0 + c0 + col + 1 < p) yr[col + 1] = v1;
      } else {
        *(float2*)(yr + col) = make_float2(v0, v1);
      }
    }
  }
}

template <int NP, int PT, bool SILU, bool UNIT = false>
static int decay_chunked_launch(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, const float* a,
                                int a_row, const float* ks, const float* skip, float qs, float* state, const int32_t* pos_ids, float* y,
                                int B, int Tn, int H, int qk_heads, int n, int p, float* scratch, cudaStream_t st) {
  const int chunks = (Tn + DC_L - 1) / DC_L, ptiles = (p + PT - 1) / PT, pp = UNIT ? p + 3 : p, np2 = n * pp / 2;
  float* chunk_state = scratch;
  float* total = scratch + (size_t)B * H * chunks * n * pp;
  const dim3 grid(chunks * ptiles, H, B);
  constexpr int smem_c = (3 * DC_L * (NP + 8) + DC_L * (PT + 8)) * 2, smem_r = (DC_L * (NP + 8) + DC_L * (PT + 8) + (UNIT ? 3 : 2) * NP * (PT + 8)) * 2;
  static PerDevice sized;
  if (!sized) {
    LL_CUDA(cudaFuncSetAttribute(decay_collect_kernel<NP, PT, SILU, UNIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_c));
    LL_CUDA(cudaFuncSetAttribute(decay_read_kernel<NP, PT, SILU, UNIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_r));
    sized.mark();
  }
  typedef const __nv_bfloat16* in_t;
  decay_collect_kernel<NP, PT, SILU, UNIT><<<grid, DC_THREADS, smem_c, st>>>((in_t)k, k_stride, (in_t)v, v_stride, a, a_row, ks, chunk_state, total, Tn, H,
                                                                  qk_heads, n, p, ptiles);
  LL_LAUNCH_OK("decay_collect_kernel");
  decay_pass_kernel<UNIT><<<dim3((np2 + 127) / 128, B * H), 128, 0, st>>>(chunk_state, total, state, pos_ids, chunks, np2, n, p);
  LL_LAUNCH_OK("decay_pass_kernel");
  decay_read_kernel<NP, PT, SILU, UNIT><<<grid, DC_THREADS, smem_r, st>>>((in_t)q, q_stride, (in_t)k, k_stride, (in_t)v, v_stride, a, a_row, ks, skip, qs,
                                                               chunk_state, pos_ids, y, Tn, H, qk_heads, n, p, ptiles);
  LL_LAUNCH_OK("decay_read_kernel");
  return LL_OK;
}

}  // namespace llb

using namespace llb;

extern "C" {

int ll_decay_chunked_supported(int dtype, int T, int n, int p, int q_stride, int k_stride, int v_stride) {
  return dtype == LL_BF16 && T >= DC_L && n % 8 == 0 && n <= 128 && p % 8 == 0 && ((q_stride | k_stride | v_stride) & 7) == 0;
}

size_t ll_decay_chunked_scratch_bytes(int B, int T, int H, int n, int p) {
  const size_t chunks = (T + DC_L - 1) / DC_L;
  return (size_t)B * H * chunks * ((size_t)n * p + 1) * sizeof(float);
}

int ll_decay_chunked(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, int dtype, const float* a,
                     int a_constant, int act_silu, const float* ks, const float* skip, float qs, float* state, const int32_t* pos_ids,
                     float* y, int B, int T, int H, int qk_heads, int n, int p, float* scratch, ll_stream stream) {
  LL_CHECK_ARG(q && k && v && a && state && pos_ids && y && scratch, "decay_chunked: null pointer");
  LL_CHECK_ARG(B >= 0 && T >= 0 && H > 0 && qk_heads > 0 && H % qk_heads == 0 && n > 0 && p > 0, "bad decay_chunked arguments");
  if (B == 0 || T == 0) return LL_OK;
  const uintptr_t at = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state | (uintptr_t)y | (uintptr_t)scratch;
  if (!ll_decay_chunked_supported(dtype, T, n, p, q_stride, k_stride, v_stride) || (at & 15) != 0 || (long long)B * H > 65535) {
    set_error("decay_chunked: bf16, at least %d tokens, n and p in multiples of 8 (n up to 128), rows on 16-byte boundaries", DC_L);
    return LL_ERR_UNSUPPORTED;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int a_row = a_constant ? 0 : H;
#define LL_DC_S(NP, SILU)                                                                                                              \
  return p <= 64 ? decay_chunked_launch<NP, 64, SILU>(q, q_stride, k, k_stride, v, v_stride, a, a_row, ks, skip, qs, state, pos_ids, y, B, T, \
                                                      H, qk_heads, n, p, scratch, st)                                                        \
                 : decay_chunked_launch<NP, 128, SILU>(q, q_stride, k, k_stride, v, v_stride, a, a_row, ks, skip, qs, state, pos_ids, y, B, T, \
                                                       H, qk_heads, n, p, scratch, st)
#define LL_DC(NP)                  \
  if (n <= NP) {                   \
    if (act_silu) LL_DC_S(NP, true); \
    LL_DC_S(NP, false);            \
  }
  LL_DC(16) LL_DC(32) LL_DC(64) LL_DC(128)
#undef LL_DC
#undef LL_DC_S
  return LL_ERR_UNSUPPORTED;
}

size_t ll_decay_chunked_unit_scratch_bytes(int B, int T, int H, int n, int p) {
  return ll_decay_chunked_scratch_bytes(B, T, H, n, p + 3);
}

int ll_decay_chunked_unit(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, int dtype, const float* a,
                          const float* ks, float qs, float* state, const int32_t* pos_ids, float* y, int B, int T, int H, int qk_heads, int n,
                          int p, float* scratch, ll_stream stream) {
  LL_CHECK_ARG(q && k && v && a && state && pos_ids && y && scratch, "decay_chunked_unit: null pointer");
  LL_CHECK_ARG(B >= 0 && T >= 0 && H > 0 && qk_heads > 0 && H % qk_heads == 0 && n > 0 && p > 1, "bad decay_chunked_unit arguments");
  if (B == 0 || T == 0) return LL_OK;
  const uintptr_t at = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch;
  if (!ll_decay_chunked_supported(dtype, T, n, p - 1, q_stride, k_stride, v_stride) || (at & 15) != 0 || (long long)B * H > 65535) {
    set_error("decay_chunked_unit: bf16, at least %d tokens, n and p - 1 in multiples of 8 (n up to 128), rows on 16-byte boundaries", DC_L);
    return LL_ERR_UNSUPPORTED;
  }
  cudaStream_t st = (cudaStream_t)stream;
#define LL_DCU(NP)                                                                                                                        \
  if (n <= NP)                                                                                                                            \
    return decay_chunked_launch<NP, 64, false, true>(q, q_stride, k, k_stride, v, v_stride, a, H, ks, nullptr, qs, state, pos_ids, y, B, T, H, \
                                                     qk_heads, n, p, scratch, st);
  LL_DCU(16) LL_DCU(32) LL_DCU(64) LL_DCU(128)
#undef LL_DCU
  return LL_ERR_UNSUPPORTED;
}

namespace {
struct MatrixLayerScratch {
  void *proj, *normed;
  float *keep, *take, *stab, *y, *chunks;
  size_t total;
};
MatrixLayerScratch matrix_layer_carve(void* base, int B, int T, int n_in, int H, int n, int p) {
  MatrixLayerScratch s;
  size_t o = 0;
  auto take = [&](size_t b) { void* r = (uint8_t*)base + o; o += (b + 255) & ~(size_t)255; return r; };
  const size_t M = (size_t)B * T;
  s.proj = take(M * n_in * 2);
  s.keep = (float*)take(M * H * 4), s.take = (float*)take(M * H * 4), s.stab = (float*)take(M * H * 4);
  s.y = (float*)take(M * H * p * 4);
  s.normed = take(M * H * (p - 1) * 2);
  s.chunks = (float*)take(T >= DC_L ? ll_decay_chunked_unit_scratch_bytes(B, T, H, n, p) : 0);
  s.total = o;
  return s;
}
}  // namespace

size_t ll_matrix_memory_layer_scratch_bytes(int B, int T, int n_in, int H, int n, int p) { return matrix_layer_carve(nullptr, B, T, n_in, H, n, p).total; }

int ll_matrix_memory_layer(const void* x, const void* w_in, int n_in, const void* w_o, int q_col, int k_col, int v_col, int g_col, int i_col, int f_col,
                           const float* bias_i, const float* bias_f, float gate_cap, const float* norm, float eps, float qs, float* memory, float* stabiliser,
                           const int32_t* pos_ids, int B, int T, int width, int H, int n, int p, int chunks, void* out, void* scratch, ll_stream stream) {
  LL_CHECK_ARG(x && w_in && w_o && bias_i && bias_f && norm && memory && stabiliser && pos_ids && out && scratch, "matrix_memory_layer: null pointer");
  LL_CHECK_ARG(B > 0 && T > 0 && H > 0 && n > 0 && p > 1 && q_col >= 0 && k_col >= 0 && v_col >= 0 && g_col >= 0 && i_col >= 0 && f_col >= 0,
               "bad matrix_memory_layer arguments");
  const int hv = H * (p - 1), M = B * T;
  if (width % 8 != 0 || n_in % 8 != 0 || hv % 8 != 0) {
    set_error("matrix_memory_layer takes widths in multiples of 8 (width=%d rows %d heads %d x %d)", width, n_in, H, p - 1);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG((((uintptr_t)x | (uintptr_t)w_in | (uintptr_t)w_o | (uintptr_t)scratch) & 15) == 0, "matrix_memory_layer: rows must be 16-byte aligned bf16");
  cudaStream_t st = (cudaStream_t)stream;
  const MatrixLayerScratch s = matrix_layer_carve(scratch, B, T, n_in, H, n, p);
  const __nv_bfloat16* proj = (const __nv_bfloat16*)s.proj;
  if (int r = rows_linear(x, width, w_in, s.proj, n_in, M, n_in, width, false, st)) return r;
  if (int r = ll_matrix_memory_gates(proj + i_col, proj + f_col, LL_BF16, n_in, bias_i, bias_f, gate_cap, stabiliser, pos_ids, s.keep, s.take, s.stab, B, T, H,
                                     stream))
    return r;
  if (chunks) {
    if (int r = ll_decay_chunked_unit(proj + q_col, n_in, proj + k_col, n_in, proj + v_col, n_in, LL_BF16, s.keep, s.take, qs, memory, pos_ids, s.y, B, T, H, H, n,
                                      p, s.chunks, stream))
      return r;
  } else if (int r = ll_decay_scan(proj + q_col, n_in, proj + k_col, n_in, proj + v_col, n_in, LL_BF16, s.keep, 0, s.take, nullptr, qs, memory, pos_ids, s.y, B,
                                   T, H, H, n, p, 1, stream)) {
    return r;
  }
  if (int r = ll_gated_group_norm_rows(s.y, p, s.stab, proj + g_col, n_in, norm, 0, eps, H, 0, 1, s.normed, hv, LL_BF16, M, hv, stream)) return r;
  return rows_linear(s.normed, hv, w_o, out, width, M, width, hv, true, st);
}

}  // extern "C"
