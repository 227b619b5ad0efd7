// Grouped expert GEMM of the mixture-of-experts feed-forward on the 5th-generation tensor cores
// (tcgen05 + TMEM + TMA), for steps with many rows per expert (prefill).
//
// The (token, choice) pairs are sorted by expert (ll_moe_route) and the rows of the activations are
// gathered into that order once (ll_moe_gather_rows), so every operand is a plain row-major matrix
// that TMA can tile:
//   mode 1 (GLU) : h[r][n] = glu(xs[r] . gate_e[n], xs[r] . up_e[n])     w [X][2N][K] = [gate; up]
//   mode 3 (relu^2): h[r][n] = relu(xs[r] . up_e[n])^2                    w [X][N][K]
//   mode 0 (down): y[perm[r]][n] = h[r] . down_e[n]                       w [X][N][K]
// for the sorted rows r of expert e.  A CTA owns 128 sorted rows of ONE expert (found from the device-side
// offsets, as in the mma.sync form: no host synchronisation) x 256 accumulator columns in TMEM:
//   GLU : columns 0..127 = gate tile, 128..255 = up tile of the same 128 outputs; the clamped gated unit is
//         the epilogue, applied to the two accumulators as they are read back from TMEM;
//   relu^2: columns 0..255 = 256 outputs, squared as they are read back;
//   down: columns 0..255 = 256 outputs, scattered to (token, choice) order by the epilogue.
// A row tile may run past its expert's last row: those rows (the next expert's, or zero fill) are
// computed and never stored.
// One CTA per SM walks the tiles t = blockIdx.x, + gridDim.x, ... (column tiles first, so the tiles in flight share their
// experts' weights and their rows in L2):
//   warp 0   : TMA producer (A box 128 x 64, two B boxes 128 x 64, 128-byte swizzle) into a 4-stage ring that runs on across
//              tiles
//   warp 1   : TMEM allocation, one elected thread issues tcgen05.mma 128 x 256 x 16 (bf16 in, fp32 accumulate)
//   warps 2-9: epilogue, one accumulator row and half of its columns per thread
// Two accumulators of 256 TMEM columns alternate, so the epilogue of a tile (an exponential, a division and scattered rows
// of stores, about half as long as the main loop) and the search for the next one run under the main loop of the next.  One
// tile per CTA, two CTAs per SM, left both in the open and dealt out whole tiles in three rounds where 2.2 would do:
// 8192 rows of 32 experts, width 2048, ff 1024: gate and up 137 us -> 96 (0.72 PFLOP/s of rows that count), down 73 -> 56.
// What bounds it now: 128-row tiles that are not full (a fifth of the products) and the operands' way from L2 (96 bytes a
// clock and SM at the full rate of the products).
// Every wait on an mbarrier is bounded; a wait that runs out records a code in g_moe_tc_error, the roles
// stop, the CTA waits for its copies and products in flight (bounded), frees its TMEM and returns.
#include <algorithm>

#include "tcgen05.cuh"

namespace llb {
namespace {

constexpr int MT_BN = 128;                 // rows of one B box
constexpr int MT_STAGES = 4;
constexpr int MT_A_BYTES = BM * BK * 2, MT_B_BYTES = 2 * MT_BN * BK * 2;
constexpr int MT_COLS = 256, MT_TMEM_COLS = 2 * MT_COLS;      // two accumulators
constexpr int MT_EPI_WARPS = 8, MT_THREADS = 64 + 32 * MT_EPI_WARPS;
constexpr uint32_t MT_WAIT_LIMIT = 1u << 22;

__device__ int g_moe_tc_error = 0;

// A wait that ends: on its phase, when another role has given up, or after the limit.
__device__ __forceinline__ bool mt_wait(uint64_t* bar, uint32_t parity, volatile int* fail, int* word, int code) {
  for (uint32_t i = 0; i < MT_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  atomicCAS(&g_moe_tc_error, 0, code);
  wait_ran_out(word, 400 + code);
  return false;
}

// Walk over the row tiles (128 sorted rows of one expert) in rising order; every role that needs them keeps its own.
struct MtWalk {
  int e = -1, first = 0, next = 0;      // expert, its first row tile, the one after its last
  int row = 0, end = 0;                 // its sorted rows
  __device__ __forceinline__ bool seek(const int32_t* __restrict__ offsets, int X, int rt) {
    while (rt >= next) {
      if (++e >= X) return false;
      row = __ldg(offsets + e);
      end = __ldg(offsets + e + 1);
      first = next;
      next += (end - row + BM - 1) / BM;
    }
    return true;
  }
  __device__ __forceinline__ int r0(int rt) const { return row + (rt - first) * BM; }
};

// 2-D tiled TMA load, default L2 policy (both operands are re-read by other CTAs through L2)
__device__ __forceinline__ void tma_box(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                   smem_u32(dst)),
               "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(MT_THREADS, 1) moe_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a,
                                                                    const __grid_constant__ CUtensorMap map_b,
                                                                    const int32_t* __restrict__ offsets, const int32_t* __restrict__ perm,
                                                                    int X, int N, int K, float limit, float alpha, float shift,
                                                                    __nv_bfloat16* __restrict__ c, int ldc, int* word) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* sa = base;                              // [STAGES][128][64] bf16, swizzled
  uint8_t* sb = base + MT_STAGES * MT_A_BYTES;     // [STAGES][256][64]
  uint64_t* full = reinterpret_cast<uint64_t*>(sb + MT_STAGES * MT_B_BYTES);
  uint64_t* empty = full + MT_STAGES;
  uint64_t* acc_full = empty + MT_STAGES;          // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2]
  uint64_t* drained = acc_empty + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(drained + 1);
  int* s_tiles = reinterpret_cast<int*>(tmem_ptr + 1);
  volatile int* s_fail = s_tiles + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NCOL = MODE == 1 ? MT_BN : MT_COLS;      // outputs of a tile
  const int ncol = (N + NCOL - 1) / NCOL;
  const int nkb = (K + BK - 1) / BK;
  if (warp == 0) {
    int n = 0;
    for (int e = lane; e < X; e += 32) n += (offsets[e + 1] - offsets[e] + BM - 1) / BM;
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) {
      *s_tiles = n * ncol;
      *s_fail = 0;
      prefetch_tensormap(&map_a);
      prefetch_tensormap(&map_b);
      for (int i = 0; i < MT_STAGES; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&empty[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&acc_full[i], 1);
        mbar_init(&acc_empty[i], MT_EPI_WARPS);
      }
      mbar_init(drained, 1);
      fence_barrier_init();
    }
  }
  if (warp == 1) tmem_alloc(tmem_ptr, MT_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = *tmem_ptr;
  const int tiles = *s_tiles;

  if (warp == 0) {
    if (elect_one()) {
      MtWalk walk;
      int s = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        const int rt = t / ncol, n0 = (t - rt * ncol) * NCOL;
        if (!walk.seek(offsets, X, rt)) break;
        const int r0 = walk.r0(rt);
        // rows of the expert's weight matrix under the two B boxes
        const int brow0 = MODE == 1 ? walk.e * 2 * N + n0 : walk.e * N + n0;
        const int brow1 = MODE == 1 ? brow0 + N : brow0 + MT_BN;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mt_wait(&empty[s], phase ^ 1, s_fail, word, 1)) { ok = false; break; }
          mbar_expect_tx(&full[s], MT_A_BYTES + MT_B_BYTES);
          tma_box(sa + s * MT_A_BYTES, &map_a, kb * BK, r0, &full[s]);
          tma_box(sb + s * MT_B_BYTES, &map_b, kb * BK, brow0, &full[s]);
          tma_box(sb + s * MT_B_BYTES + MT_BN * BK * 2, &map_b, kb * BK, brow1, &full[s]);
          issued = 1;
          if (++s == MT_STAGES) { s = 0; phase ^= 1u; }
        }
      }
      if (!ok && issued) {   // give the copies already issued time to land before the CTA leaves
        for (int w = 0; w < 2048; ++w) __nanosleep(512);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc_bf16(BM, 2 * MT_BN);
      int s = 0, i = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++i) {
        const uint32_t d = tmem_d + (uint32_t)((i & 1) * MT_COLS);
        if (!mt_wait(&acc_empty[i & 1], ((i >> 1) & 1) ^ 1, s_fail, word, 4)) break;
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mt_wait(&full[s], phase, s_fail, word, 2)) { ok = false; break; }
          tc_fence_after();
          const uint64_t adesc = smem_desc_sw128(smem_u32(sa + s * MT_A_BYTES));
          const uint64_t bdesc = smem_desc_sw128(smem_u32(sb + s * MT_B_BYTES));
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16(d, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit(&empty[s]);
          if (++s == MT_STAGES) { s = 0; phase ^= 1u; }
        }
        if (ok) umma_commit(&acc_full[i & 1]);
      }
      umma_commit(drained);      // on every path: nothing is in flight when the TMEM goes back
      for (uint32_t w = 0; w < MT_WAIT_LIMIT && !mbar_try_wait(drained, 0); ++w) {
      }
    }
  } else {
    const int quarter = warp & 3, part = (warp - 2) >> 2;   // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
    const int rt_row = quarter * 32 + lane;
    MtWalk walk;
    int i = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++i) {
      const int rt = t / ncol, n0 = (t - rt * ncol) * NCOL;
      if (!walk.seek(offsets, X, rt)) break;
      const int row = walk.r0(rt) + rt_row;
      const bool row_ok = row < walk.end;
      const long long dst_row = !row_ok || MODE != 0 ? (long long)row : (long long)perm[row];
      __nv_bfloat16* dst = c + dst_row * ldc;
      if (!__all_sync(0xffffffffu, mt_wait(&acc_full[i & 1], (i >> 1) & 1, s_fail, word, 3))) break;
      tc_fence_after();
      const uint32_t trow = tmem_d + (uint32_t)((i & 1) * MT_COLS) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c0 = part * (NCOL / 2); c0 < (part + 1) * (NCOL / 2); c0 += 32) {
        if (n0 + c0 >= N) break;            // uniform over the warp
        uint32_t v[32];
        tmem_ld_32x32(trow + (uint32_t)c0, v);
        float f[32];
        if (MODE == 1) {
          uint32_t u[32];
          tmem_ld_32x32(trow + (uint32_t)(MT_BN + c0), u);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float g = fminf(__uint_as_float(v[j]), limit);
            const float up = fminf(fmaxf(__uint_as_float(u[j]), -limit), limit);
            f[j] = g / (1.f + expf(-alpha * g)) * (up + shift);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            f[j] = __uint_as_float(v[j]);
            if (MODE == 3) f[j] = fmaxf(f[j], 0.f) * fmaxf(f[j], 0.f);
          }
        }
        const int col = n0 + c0;
        if (row_ok && col + 32 <= N && (ldc & 7) == 0) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t pk[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              pk[q] = (uint32_t)f32_to_bf16_bits(f[j * 8 + 2 * q]) | ((uint32_t)f32_to_bf16_bits(f[j * 8 + 2 * q + 1]) << 16);
            *reinterpret_cast<uint4*>(dst + col + j * 8) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          }
        } else if (row_ok) {
          for (int j = 0; j < 32 && col + j < N; ++j) dst[col + j] = __float2bfloat16_rn(f[j]);
        }
        __syncwarp();
      }
      __syncwarp();
      tc_fence_before();
      if (lane == 0) mbar_arrive(&acc_empty[i & 1]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_d, MT_TMEM_COLS);
  }
}

// xs[r][:] = x[perm[r] / top][:] for the sorted rows r (16-byte pieces)
__global__ void moe_gather_rows_kernel(const uint4* __restrict__ x, long long ldx16, const int32_t* __restrict__ perm, int top,
                                       uint4* __restrict__ out, int k16) {
  const int r = blockIdx.x;
  const uint4* src = x + (long long)(perm[r] / top) * ldx16;
  uint4* dst = out + (long long)r * k16;
  for (int i = threadIdx.x; i < k16; i += blockDim.x) dst[i] = src[i];
}

template <int MODE>
int launch_moe_tc(const CUtensorMap& ma, const CUtensorMap& mb, const int32_t* offsets, const int32_t* perm, int X, int N, int K,
                  float limit, float alpha, float shift, void* c, int ldc, int n_rows, cudaStream_t st) {
  constexpr size_t smem = (size_t)MT_STAGES * (MT_A_BYTES + MT_B_BYTES) + (2 * MT_STAGES + 5) * 8 + 32 + 1024;
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(moe_gemm_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured.mark();
  }
  const int ncols = MODE == 1 ? MT_BN : MT_COLS;
  const long long most = (long long)((N + ncols - 1) / ncols) * ((n_rows + BM - 1) / BM + X);
  LL_CHECK_ARG(most < (1ll << 30), "moe_grouped_gemm_tc: too many tiles");
  const int grid = (int)std::min<long long>(most, sm_count() > 0 ? sm_count() : 148);
  moe_gemm_tc_kernel<MODE><<<grid, MT_THREADS, smem, st>>>(ma, mb, offsets, perm, X, N, K, limit, alpha, shift, (__nv_bfloat16*)c, ldc, wait_word());
  LL_LAUNCH_OK("moe_gemm_tc_kernel");
  return LL_OK;
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
  moe_gather_rows_kernel<<<n_rows, K / 8 >= 256 ? 256 : 128, 0, (cudaStream_t)stream>>>((const uint4*)x, ldx / 8, perm, top, (uint4*)out,
                                                                                     K / 8);
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
  CUtensorMap ma, mb;
  if (int r = make_map(a, n_rows, K, BM, &ma)) return r;
  if (int r = make_map(w, (int)wrows, K, MT_BN, &mb)) return r;
  cudaStream_t st = (cudaStream_t)stream;
  if (mode == 1) return launch_moe_tc<1>(ma, mb, offsets, perm, n_experts, N, K, limit, alpha, shift, c, ldc, n_rows, st);
  if (mode == 3) return launch_moe_tc<3>(ma, mb, offsets, perm, n_experts, N, K, limit, alpha, shift, c, ldc, n_rows, st);
  return launch_moe_tc<0>(ma, mb, offsets, perm, n_experts, N, K, limit, alpha, shift, c, ldc, n_rows, st);
}

// 0, or the code of the first bounded wait that ran out in a kernel of this file (1: ring slot, 2: operands, 3: accumulator,
// 4: accumulator to be free).
// Synchronises the device.
int ll_moe_tc_error(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_moe_tc_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // extern "C"
