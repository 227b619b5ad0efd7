// y[m][n] = sum_k x[m][k] w[n][k] for any number of rows on the tcgen05 tensor cores (pair_rows.cuh): the projections of layers that run in one
// call.  Rows are cut into as many tiles as take the least time by the kernel's own measure (a round of tiles costs 256 + n clocks a stage of k).
// us, graphed, weights from memory, here / the library's product: 5120 x 2048 with 64, 300, 1500 and 2048 rows 9.6 / 6.9, 12.4 / 9.9, 24.4 / 24.1,
// 31.4 / 32.7; 1024 x 1024 6.7 / 4.2, 6.9 / 4.4, 7.3 / 5.7, 7.5 / 6.3; 10240 x 4096 22 / 18, 39 / 27, 85 / 86, 113 / 109.  A library call costs the host
// 15 us, so a layer that makes its products itself is the faster one where the host's time is what a call takes (_native.layer_rows).
#include "dense_rows.cuh"

#include "pair_rows.cuh"

namespace llb {
namespace {

// A tile's k shared by S pairs of one cluster, for products with fewer tiles than the chip has pairs: each pair sums its part in tensor memory; then
// all but the first hand their sums (fp32) to the first one's shared memory, which its ring no longer needs, and it adds them in order.
// Otherwise as moe_gemm_pair_kernel, one tile a cluster.
struct SpParams {
  __nv_bfloat16* y;
  int M, N, nkb, ldy, vec, across, step, cuts;
  int* word;
};
constexpr int SP_PITCH = 132;      // floats from one token's sums to the next: a quarter's rows and four pairs of tokens fall on 32 banks
static_assert(MT_NMAX * SP_PITCH * 4 <= MT_STAGES * (MT_A_BYTES + MT_B_BYTES), "a tile's sums in the ring's place (two pairs a tile)");

// 32 lanes x 32 columns to the same place of another CTA's shared memory: v[c] of lane l at (c * SP_PITCH + l) floats
__device__ __forceinline__ void sp_store(uint32_t at, const uint32_t (&v)[32]) {
#pragma unroll
  for (int c = 0; c < 32; ++c) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at + (uint32_t)(c * SP_PITCH * 4)), "r"(v[c]) : "memory");
}
__device__ __forceinline__ float sp_load(uint32_t at) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
  return v;
}

template <int S>
__global__ void __cluster_dims__(2 * S, 1, 1) __launch_bounds__(MT_THREADS, 1)
    dense_split_kernel(const __grid_constant__ MtMaps maps, const __grid_constant__ SpParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* sa = base;
  uint8_t* sb = sa + MT_STAGES * MT_A_BYTES;
  uint8_t* so = sb + MT_STAGES * MT_B_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(so + MT_EPI_WARPS * MT_OUT);
  uint64_t* empty = full + MT_STAGES;
  uint64_t* acc_full = empty + MT_STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_full + 4);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int crank = (int)cluster_rank(), j = crank >> 1, rank = crank & 1, lead = crank & ~1;
  if (threadIdx.x == 0) {
    prefetch_tensormap(&maps.w);
    prefetch_tensormap(&maps.t64);
    prefetch_tensormap(&maps.t16);
    for (int i = 0; i < MT_STAGES; ++i) mbar_init(&full[i], 1), mbar_init(&empty[i], 1);
    mbar_init(acc_full, 1);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) pair_tmem_alloc(tmem_ptr, MT_NMAX);
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const MtFail fail{s_fail, cluster_addr(s_fail, (uint32_t)(crank ^ 1)), p.word};
  const int t = (int)blockIdx.x / (2 * S), ct = t / p.cuts, r0 = (t - ct * p.cuts) * p.step, cnt = min(p.step, p.M - r0);
  const int n = (cnt + MT_NSTEP - 1) / MT_NSTEP * MT_NSTEP, half = n / 2, n0 = (ct * 2 + rank) * 128;
  const int k0 = p.nkb * j / S, k1 = p.nkb * (j + 1) / S;
  const int quarter = warp & 3, part = (warp - 2) >> 2;
  pdl_wait();
  pdl_launch_dependents();
  bool ok = true;
  if (warp == 0) {
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 1;
      for (int kb = k0; kb < k1; ++kb) {
        if (!(ok = mt_wait(&empty[s], ph, fail, 1))) break;
        if (rank == 0) mbar_expect_tx(&full[s], (uint32_t)(2 * (MT_A_BYTES + half * BK * 2)));
        const uint32_t bar = cluster_addr(&full[s], (uint32_t)lead);
        uint8_t *da = sa + s * MT_A_BYTES, *db = sb + s * MT_B_BYTES;
        if (p.across) {
          for (int q = 0; q < 2; ++q) {
            const int blk = (n0 >> 6) + q, head = blk / p.across;
            pair_box3(da + q * (MT_A_BYTES / 2), &maps.w, (blk - head * p.across) * 64, kb * BK, head, bar);
          }
        } else {
          pair_box3(da, &maps.w, kb * BK, n0, 0, bar);
        }
        int r = 0;
        for (; r + 64 <= half; r += 64) pair_box(db + r * BK * 2, &maps.t64, kb * BK, r0 + rank * half + r, bar);
        for (; r < half; r += 16) pair_box(db + r * BK * 2, &maps.t16, kb * BK, r0 + rank * half + r, bar);
        if (++s == MT_STAGES) s = 0, ph ^= 1u;
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      const bool across = p.across != 0;
      const uint64_t ad = across ? mt_desc_across(smem_u32(sa)) : smem_desc_sw128(smem_u32(sa)), astep = across ? 128 : 2, bd = smem_desc_sw128(smem_u32(sb));
      const uint32_t idesc = instr_desc_bf16(256, 0) | ((uint32_t)(n >> 3) << 17) | (across ? 1u << 15 : 0u);
      int s = 0;
      uint32_t ph = 0;
      for (int kb = k0; kb < k1; ++kb) {
        if (!(ok = mt_wait(&full[s], ph, fail, 2))) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          mt_mma(tmem, ad + (uint64_t)(s * (MT_A_BYTES >> 4)) + astep * (uint64_t)k, bd + (uint64_t)(s * (MT_B_BYTES >> 4) + 2 * k), idesc,
                 (kb > k0 || k > 0) ? 1u : 0u);
        mt_commit(&empty[s], j);
        if (++s == MT_STAGES) s = 0, ph ^= 1u;
      }
      if (ok) mt_commit(acc_full, j);
      else let_issued_work_end();
    }
  } else {
    ok = __all_sync(0xffffffffu, mt_wait(acc_full, 0, fail, 3));
    tc_fence_after();
  }
  __syncwarp();
  cluster_sync();                          // every pair's products have ended: the first pair's ring is free
  const uint32_t td = tmem + ((uint32_t)(quarter * 32) << 16);
  if (j > 0 && warp >= 2) {
    const uint32_t to = cluster_addr(sa, (uint32_t)rank) + (uint32_t)((((j - 1) * n) * SP_PITCH + quarter * 32 + lane) * 4);
    for (int c0 = part * 32; ok && c0 < n; c0 += 64) {
      uint32_t v[32];
      tmem_ld_32x32(td + (uint32_t)c0, v);
      sp_store(to + (uint32_t)(c0 * SP_PITCH * 4), v);
    }
  }
  __syncwarp();
  cluster_sync();
  if (j == 0 && warp >= 2 && ok) {
    const uint32_t stage = smem_u32(so + (warp - 2) * MT_OUT), mine = stage + (uint32_t)(lane * 64), sums = smem_u32(sa);
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll 1
    for (int c0 = part * 32; c0 < cnt; c0 += 64) {
#pragma unroll
      for (int hl = 0; hl < 2; ++hl) {
        uint32_t v[16];
        tmem_ld_16x32(td + ((uint32_t)(16 * hl) << 16) + (uint32_t)c0, v);
        float f[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) f[e] = __uint_as_float(v[e]);
#pragma unroll
        for (int z = 0; z < S - 1; ++z)
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int tok = c0 + 8 * (e >> 2) + 2 * tq + (e & 1), row = quarter * 32 + 16 * hl + g + 8 * ((e >> 1) & 1);
            f[e] += sp_load(sums + (uint32_t)(((z * n + tok) * SP_PITCH + row) * 4));
          }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = pack_bf16(f[4 * i + 2 * q], f[4 * i + 2 * q + 1]);
          store_tokens(mine + (uint32_t)(((2 * hl + q) ^ ((lane >> 1) & 3)) * 16), o[0], o[1], o[2], o[3]);
        }
      }
      __syncwarp();
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        const int at = it * 32 + lane, tk = at / 4, ch = at % 4, col = n0 + quarter * 32 + 8 * ch;
        const uint4 u = lds128(stage + (uint32_t)(tk * 64 + ((ch ^ ((tk >> 1) & 3)) * 16)));
        if (c0 + tk < cnt && col < p.N) {
          __nv_bfloat16* out = p.y + (size_t)(r0 + c0 + tk) * p.ldy + col;
          if (p.vec) {
            *reinterpret_cast<uint4*>(out) = u;
          } else {
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
            for (int i = 0; i < 8 && col + i < p.N; ++i) out[i] = __ushort_as_bfloat16((uint16_t)(w[i >> 1] >> (16 * (i & 1))));
          }
        }
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem, MT_NMAX);
  }
}

template <int S>
int launch_split(const MtMaps& maps, const SpParams& p, int tiles, cudaStream_t st) {
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(dense_split_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MT_SMEM));
    configured.mark();
  }
  LL_CUDA(launch(dense_split_kernel<S>, dim3((unsigned)(tiles * 2 * S)), dim3(MT_THREADS), MT_SMEM, st, true, maps, p));
  LL_LAUNCH_OK("dense_split_kernel");
  return LL_OK;
}

int token_map(const void* x, long long ldx, int M, int K, int box_rows, CUtensorMap* out) {
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M}, strides[1] = {(cuuint64_t)ldx * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  return mt_encode(x, 2, dims, strides, box, out);
}

}  // namespace

int dense_rows(const void* x, long long ldx, const void* w, int head_cols, void* y, int ldy, int M, int N, int K, cudaStream_t st) {
  MtMaps maps;
  if (head_cols > 0) {
    const cuuint64_t dims[3] = {(cuuint64_t)head_cols, (cuuint64_t)K, (cuuint64_t)(N / head_cols)}, row = (cuuint64_t)head_cols * 2, strides[2] = {row, row * K};
    const cuuint32_t box[3] = {64, (cuuint32_t)BK, 1};
    if (int r = mt_encode(w, 3, dims, strides, box, &maps.w)) return r;
  } else if (int r = mt_weight_map(w, 0, 1, N, K, &maps.w)) {
    return r;
  }
  if (int r = token_map(x, ldx, M, K, 64, &maps.t64)) return r;
  if (int r = token_map(x, ldx, M, K, 16, &maps.t16)) return r;
  // the cheapest way by the kernels' own measure: clocks of a stage of k, rounds of tiles, and for k shared by S pairs the handing over
  const int pairs = sm_count() > 1 ? sm_count() / 2 : 1, wt = (N + 255) / 256, nkb = (K + BK - 1) / BK;
  long long best = -1;
  int cuts = 1, split = 1;
  for (int step = MT_NMAX; step >= MT_NSTEP; step -= MT_NSTEP) {
    const int c = (M + step - 1) / step;
    for (int sp = 1; sp <= 2; ++sp) {
      // (clusters of four CTAs: an eighth of the pairs is left for what does not fit a GPC.  Four pairs a tile: clusters of eight ran in two waves,
      // 2048 x 2048 with 64 rows 13.0 where two pairs take 8.8 and one 10.3)
      if (sp > 1 && ((long long)wt * c * sp > pairs - pairs / 8 || nkb < 8)) continue;
      const long long rounds = ((long long)wt * c + pairs - 1) / pairs, cost = rounds * (256 + step) * ((nkb + sp - 1) / sp) + (sp > 1 ? 2000 + 16 * step : 0);
      if (best < 0 || cost < best) best = cost, cuts = c, split = sp;
    }
  }
  const int step = MtWalk::columns(M, cuts);
  cuts = (M + step - 1) / step;          // (no tile without a row)
  if (split > 1) {
    const SpParams p{(__nv_bfloat16*)y, M, N, nkb, ldy, ldy % 8 == 0 && N % 8 == 0 && ((uintptr_t)y & 15) == 0, head_cols / 64, step, cuts, wait_word()};
    return launch_split<2>(maps, p, wt * cuts, st);
  }
  MtParams p{};
  p.cuts = cuts;
  p.part[0] = p.part[1] = mt_part(y, 0, N, K, ldy, 0.f);
  p.part[1].across = head_cols / 64;
  p.M = M, p.word = wait_word();
  return launch_moe_pair<0>(maps, maps, p, 0, st);
}

}  // namespace llb

using namespace llb;

extern "C" {

int ll_dense_rows(const void* x, int ldx, const void* w, int head_cols, void* y, int ldy, int M, int N, int K, ll_stream stream) {
  LL_CHECK_ARG(x && w && y, "dense_rows: null pointer");
  LL_CHECK_ARG(M >= 0 && N > 0 && K > 0 && ldx >= K && ldy >= N && head_cols >= 0 && (head_cols == 0 || N % head_cols == 0), "bad dense_rows arguments");
  LL_CHECK_ARG(K % 8 == 0 && ldx % 8 == 0 && head_cols % 64 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0,
               "dense_rows: rows in multiples of 8 numbers on 16-byte boundaries, heads in multiples of 64");
  if (M == 0) return LL_OK;
  return dense_rows(x, ldx, w, head_cols, y, ldy, M, N, K, (cudaStream_t)stream);
}

// as a layer's projections choose among the forms
int ll_rows_linear(const void* x, int ldx, const void* w, void* y, int ldy, int M, int N, int K, ll_stream stream) {
  LL_CHECK_ARG(x && w && y, "rows_linear: null pointer");
  LL_CHECK_ARG(M >= 0 && N > 0 && K > 0 && ldx >= K && ldy >= N && K % 8 == 0 && ldx % 8 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0,
               "rows_linear: rows in multiples of 8 numbers on 16-byte boundaries");
  return M == 0 ? LL_OK : rows_linear(x, ldx, w, y, ldy, M, N, K, false, (cudaStream_t)stream);
}

// 0, or the code of the first bounded wait that ran out in a kernel of this file.  Synchronises the device.
int ll_dense_rows_error(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_pair_rows_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // extern "C"
