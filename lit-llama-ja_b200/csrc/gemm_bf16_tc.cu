// Large-M path of the quantized Linear on the 5th-generation tensor cores (tcgen05 + TMEM + TMA):
//   C[M][N] (bf16) = X[M][K] (bf16) . W[N][K]^T (bf16, fp32 accumulate in TMEM) (+ bias)
// W is the bit-exact bf16 de-quantisation of the packed int4 layer (ll_get_weight: the reference's
// get_weight(dtype=bf16), quantization.py:390-409), so the result is the reference's fallback branch
// F.linear(inp, get_weight(inp.dtype)) (quantization.py:420-421) with fp32 accumulation - the branch the
// reference takes for every grouped checkpoint and the semantics of its Triton kernel for per-row ones.
// Used for prefill of layers the many-row kernel (int4_rows.cu) does not take and for steps of more than 6144 rows; replaces Triton's mma.sync kernel
// (quantization.py:185-280).
//
#include "tcgen05.cuh"

namespace llb {
namespace {


// ==================================================================================== pairs of CTAs
// Tiles of 256 rows x BN columns a pair (tcgen05 cta_group::2: a CTA has 128 rows of x, half of the tile's rows of W and
// the sums of its 128 rows), persistent, with two accumulators in tensor memory, so that a tile's epilogue runs under the next one's products.
// A CTA of its own takes 128 x 256 and reads 1.5 times the operand bytes per product from L2; one tile per CTA leaves its prologue and
// epilogue in the open.
//   GP_GATED: the two layers of a gated feed-forward that read the same x: the tile's columns are 128 of W1 (brought by rank 0) and the same
//   128 of W2 (rank 1), and y = silu(x W1^T) * (x W2^T), each step rounded as the separate kernels round it.
//   warp 0   : TMA producer;  warp 1 : in rank 0, one thread issues the products;  warps 2-5: epilogue, a row per thread, boxes of 32 rows x
//   64 columns stored by TMA from a staging place per warp
// Bound by the products: us, a tile of 128 x 256 per CTA / pairs: 13824 x 5120 at 512, 2048, 16384 rows 86 / 56, 277 / 182, 2161 / 1452
// (1.60 PFLOP/s, as the library's); 4096 x 11008 at 512 rows 51 / 38.  The gated form of 16384 rows: 2864 for both layers and their product.
// Tiles are walked in blocks of GP_BAND row tiles, columns outermost within a block: what the pairs work on at a time is about as many row
// tiles as column tiles, so that W and x come from HBM once a block, not once a row tile.
// Every wait is bounded, as in the other tcgen05 kernels.
constexpr int GP_BAND = 8, GP_OUT = 32 * 128, GP_SMEM = 192 * 1024 + 4 * 2 * GP_OUT + 512 + 1024;
constexpr uint32_t GP_WAIT_LIMIT = 1u << 22;
__device__ int g_gp_error = 0;

struct GpParams {
  __nv_bfloat16* y;
  const __nv_bfloat16* bias[2];
  int M, N, nkb, mtiles, ntiles, boxes;      // boxes: y's rows are multiples of 16 bytes, TMA can store them
  int* word;
};
struct GpFail {
  volatile int* here;
  uint32_t there;
  int* word;
};
__device__ __forceinline__ bool gp_wait(uint64_t* bar, uint32_t parity, const GpFail& f, int code) {
  for (uint32_t i = 0; i < GP_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *f.here) return false;
  }
  *f.here = 1;
  store_cluster_u32(f.there, 1u);
  atomicCAS(&g_gp_error, 0, code);
  wait_ran_out(f.word, 600 + code);
  return false;
}
__device__ __forceinline__ void gp_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void gp_tile(const GpParams& p, int t, int& mt, int& nt) {
  const int per = GP_BAND * p.ntiles, blk = t / per, r = t - blk * per, rows = min(GP_BAND, p.mtiles - blk * GP_BAND);
  nt = r / rows;
  mt = blk * GP_BAND + (r - nt * rows);
}

template <int BN, bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                     const __grid_constant__ CUtensorMap map_y, const GpParams p) {
  constexpr int A_BYTES = 128 * BK * 2, B_BYTES = BN / 2 * BK * 2, STAGES = 192 * 1024 / (A_BYTES + B_BYTES);
  constexpr int COLS = GATED ? BN / 2 : BN;            // outputs of a tile
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t *sa = base, *sb = base + STAGES * A_BYTES, *so = base + 192 * 1024;
  uint64_t* full = reinterpret_cast<uint64_t*>(so + 4 * 2 * GP_OUT);        // used in rank 0
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;                 // [2]
  uint64_t* acc_empty = acc_full + 2;                  // [2], used in rank 0: both CTAs' warps arrive
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_x);
    prefetch_tensormap(&map_w0);
    prefetch_tensormap(&map_w1);
    prefetch_tensormap(&map_y);
    for (int i = 0; i < STAGES; ++i) mbar_init(&full[i], 1), mbar_init(&empty[i], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&acc_full[i], 1), mbar_init(&acc_empty[i], 8);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) pair_tmem_alloc(tmem_ptr, 2 * BN);
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const GpFail fail{s_fail, cluster_addr(s_fail, (uint32_t)(rank ^ 1)), p.word};
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, tiles = p.mtiles * p.ntiles, nkb = p.nkb;
  pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      int s = 0;
      uint32_t ph = 1;
      for (int t = pair; ok && t < tiles; t += pairs) {
        int mt, nt;
        gp_tile(p, t, mt, nt);
        const int m0 = mt * 256 + rank * 128, n0 = nt * COLS + (GATED ? 0 : rank * (BN / 2));
        const CUtensorMap* mw = GATED && rank == 1 ? &map_w1 : &map_w0;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = gp_wait(&empty[s], ph, fail, 1))) break;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * (A_BYTES + B_BYTES));      // both CTAs' operands
          const uint32_t bar = cluster_addr(&full[s], 0);
          pair_box(sa + s * A_BYTES, &map_x, kb * BK, m0, bar);
          pair_box(sb + s * B_BYTES, mw, kb * BK, n0, bar);
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc_bf16(256, BN);
      const uint64_t ad = smem_desc_sw128(smem_u32(sa)), bd = smem_desc_sw128(smem_u32(sb));
      bool ok = true;
      int s = 0, i = 0;
      uint32_t ph = 0;
      for (int t = pair; rank == 0 && ok && t < tiles; t += pairs, ++i) {
        const uint32_t d = tmem + (uint32_t)((i & 1) * BN);
        if (!(ok = gp_wait(&acc_empty[i & 1], (uint32_t)((i >> 1) & 1) ^ 1u, fail, 4))) break;
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = gp_wait(&full[s], ph, fail, 2))) break;
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            gp_mma(d, ad + (uint64_t)(s * (A_BYTES >> 4) + 2 * k), bd + (uint64_t)(s * (B_BYTES >> 4) + 2 * k), idesc, (kb | k) != 0 ? 1u : 0u);
          pair_commit(&empty[s]);
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
        if (ok) pair_commit(&acc_full[i & 1]);
      }
      if (!ok) let_issued_work_end();
    }
  } else {
    const int quarter = warp & 3;
    uint8_t* out = so + quarter * 2 * GP_OUT;
    int i = 0;
    uint32_t boxes = 0;
    for (int t = pair; t < tiles; t += pairs, ++i) {
      int mt, nt;
      gp_tile(p, t, mt, nt);
      const int r0 = mt * 256 + rank * 128 + quarter * 32, n0 = nt * COLS;
      if (!__all_sync(0xffffffffu, gp_wait(&acc_full[i & 1], (uint32_t)(i >> 1) & 1u, fail, 3))) break;
      tc_fence_after();
      const uint32_t td = tmem + (uint32_t)((i & 1) * BN) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c0 = 0; c0 < COLS; c0 += 64) {
        uint32_t o[32];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int cc = c0 + 32 * h;
          uint32_t v[32];
          tmem_ld_32x32(td + (uint32_t)cc, v);
          if (p.bias[0] != nullptr) {
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) + (n0 + cc + e < p.N ? __bfloat162float(p.bias[0][n0 + cc + e]) : 0.f));
          }
          if (GATED) {
            uint32_t u[32];
            tmem_ld_32x32(td + (uint32_t)(BN / 2 + cc), u);
            if (p.bias[1] != nullptr) {
#pragma unroll
              for (int e = 0; e < 32; ++e) u[e] = __float_as_uint(__uint_as_float(u[e]) + (n0 + cc + e < p.N ? __bfloat162float(p.bias[1][n0 + cc + e]) : 0.f));
            }
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              v[e] = __float_as_uint(__fmul_rn(silu_act<__nv_bfloat16>(bf16r(__uint_as_float(v[e]))), bf16r(__uint_as_float(u[e]))));
            }
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) o[16 * h + e] = pack_bf16(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
        }
        if (c0 + 64 >= COLS) {               // the sums have left tensor memory
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[i & 1], 0));
        }
        if (p.boxes) {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the box before the last has left
          __syncwarp();
          uint8_t* box = out + (boxes & 1u) * GP_OUT;
          ++boxes;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(box + lane * 128 + ((j ^ (lane & 7)) * 16)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            if (r0 < p.M && n0 + c0 < p.N)
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&map_y), "r"(n0 + c0), "r"(r0),
                           "r"(smem_u32(box))
                           : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        } else if (r0 + lane < p.M) {
          __nv_bfloat16* dst = p.y + (size_t)(r0 + lane) * p.N + n0 + c0;
#pragma unroll
          for (int e = 0; e < 64; ++e)
            if (n0 + c0 + e < p.N) dst[e] = __ushort_as_bfloat16((uint16_t)(o[e >> 1] >> (16 * (e & 1))));
        }
        __syncwarp();                        // the next load from tensor memory is the whole warp's
      }
    }
    tc_fence_before();
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem, 2 * BN);
  }
}

template <int BN, bool GATED>
int launch_pair(const void* x, const void* w0, const void* w1, const void* b0, const void* b1, void* y, int M, int N, int K, cudaStream_t st) {
  constexpr int COLS = GATED ? BN / 2 : BN;
  GpParams p;
  p.y = (__nv_bfloat16*)y, p.bias[0] = (const __nv_bfloat16*)b0, p.bias[1] = (const __nv_bfloat16*)b1;
  p.M = M, p.N = N, p.nkb = (K + BK - 1) / BK, p.mtiles = (M + 255) / 256, p.ntiles = (N + COLS - 1) / COLS, p.boxes = N % 8 == 0;
  p.word = wait_word();
  const long long tiles = (long long)p.mtiles * p.ntiles;
  LL_CHECK_ARG(tiles < (1ll << 30), "gemm_pair: too many tiles");
  CUtensorMap mx, m0, m1, my;
  if (int r = make_map(x, M, K, 128, &mx)) return r;
  if (int r = make_map(w0, N, K, BN / 2, &m0)) return r;
  if (int r = make_map(w1, N, K, BN / 2, &m1)) return r;
  if (p.boxes) {
    if (int r = make_map(y, M, N, 32, &my)) return r;
  } else {
    my = mx;
  }
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<BN, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM));
    configured.mark();
  }
  const int pairs = sm_count() > 1 ? sm_count() / 2 : 1;
  LL_CUDA(launch(gemm_pair_kernel<BN, GATED>, dim3(2 * (unsigned)(tiles < pairs ? tiles : pairs)), dim3(192), GP_SMEM, st, true, mx, m0, m1, my, p));
  LL_LAUNCH_OK("gemm_pair_kernel");
  return LL_OK;
}

// ==================================================================================== fused int4 dequant-GEMM, M <= 128
// (The layers of this package run int4_batch.cu; this kernel takes the packed stream of callers that hold nothing else, and layers whose
// checkpoint bytes that one does not take.)
// y[M][N] = x[M][K] . dequant(W)^T for 9 <= M <= 128 (batched decode, short prefill): the regime where the weights are
// the traffic (HBM-bound), so they are streamed ONCE in their packed form and de-quantised inside the main loop - what the
// reference's Triton kernel does (ref quantization.py:259-267: load nibble, (q - zero) * scale, tl.dot) - instead of
// writing a bf16 copy of W to HBM and reading it back.  (More rows: int4_rows.cu.)
//
//  * operand roles are swapped: the WEIGHTS are the A operand (128 output columns = the 128 TMEM lanes) and live in TENSOR
//    MEMORY: each of 128 de-quantising threads owns one output column, reads its nibbles from the packed stream (kind 1,
//    the batch-1 GEMV's stream: no second copy of the weights), forms bf16((q - zero) * scale) with the reference's two
//    bf16 roundings (HSUB2.BF16 exact for integer zeros, HMUL2.BF16 rounded) and writes 16 k per tcgen05.st;
//    the ACTIVATIONS are the B operand, TMA-loaded [M_pad][64 k] tiles (128-byte swizzle); D[128][M_pad] fp32 in TMEM.
//    Eight de-quantising warps: two per TMEM lane quarter, each takes half of a block's k (the arithmetic is ALU-bound).
//  * one thread issues tcgen05.mma (128 x M_pad x 16, A from TMEM); A is double-buffered (2 x 64 columns) so that
//    de-quantising k-block i + 1 overlaps the MMAs of block i; a 4-stage TMA ring feeds packed blocks and x tiles.
//  * work unit = (128-column tile, k-range): K is split so that the units fill the SMs; partial sums go to a scratch
//    buffer and a second small kernel adds them in split order (deterministic), adds the bias and rounds to bf16.
constexpr int W4_BN = 128;          // output columns per unit = TMEM lanes
constexpr int W4_KB = 128;          // k per block of the packed stream
constexpr int W4_BLK = W4_KB * 8 + 64;
__host__ __device__ constexpr int w4_stages(int) { return 4; }

__device__ __forceinline__ void umma_ts_bf16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ uint32_t w4_prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ uint32_t w4_sub2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t w4_mul2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void w4_bulk_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

struct W4Params {
  const uint8_t* w;       // stream kind 1: [N/16][K/128] blocks of 1088 B
  __nv_bfloat16* y;       // [M][N] (written directly when ksplit == 1)
  float* scratch;         // [tiles][ksplit][M_pad][128] partial sums (ksplit > 1)
  int32_t* counters;      // [tiles] arrivals of a tile's k-splits (left zero)
  const __nv_bfloat16* bias;
  int M, N, K, G, ksplit, mpad;
};

constexpr bool W4_REDUCE_IN_KERNEL = false;
constexpr int W4_DW = 8;  // de-quantising warps: two per TMEM lane quarter, each takes half of a block's k
template <int MPAD>
__global__ void __launch_bounds__(64 + 32 * W4_DW, 1) gemm_w4_tc_kernel(const __grid_constant__ CUtensorMap map_x, const W4Params p) {
  constexpr int W4_STAGES = w4_stages(MPAD);
  __shared__ int s_last;
  constexpr int W_BYTES = 8 * W4_BLK;        // eight 16-column blocks of the stream = 128 columns x 128 k
  constexpr int X_ATOM = MPAD * 128;         // [MPAD][64 k] bf16, swizzled
  constexpr int X_BYTES = 2 * X_ATOM;
  constexpr int STAGE = ((W_BYTES + 1023) / 1024) * 1024 + X_BYTES;
  constexpr int X_OFF = ((W_BYTES + 1023) / 1024) * 1024;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + W4_STAGES * STAGE);
  uint64_t* empty = full + W4_STAGES;
  uint64_t* a_ready = empty + W4_STAGES;   // [2] A buffer written (4 warps)
  uint64_t* a_free = a_ready + 2;          // [2] A buffer consumed (commit)
  uint64_t* tmem_full = a_free + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tmem_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / p.ksplit, ks = blockIdx.x - tile * p.ksplit;
  const int kb0 = (int)(((long long)p.G * ks) / p.ksplit), kb1 = (int)(((long long)p.G * (ks + 1)) / p.ksplit);
  const int nkb = kb1 - kb0;

  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&map_x);
    for (int i = 0; i < W4_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], W4_DW + 1);  // the de-quantising warps + the MMA commit
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&a_ready[i], W4_DW);
      mbar_init(&a_free[i], 1);
    }
    mbar_init(tmem_full, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_ptr, 256);  // D: columns [0, MPAD); A buffers: [128, 192) and [192, 256)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  if (warp == 0) {
    // ===================== TMA producer: eight packed blocks + two x atoms per 128 k =====================
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nkb; ++i) {
        const int kb = kb0 + i;
        mbar_wait_parity(&empty[s], phase ^ 1);
        mbar_expect_tx(&full[s], W_BYTES + X_BYTES);
        uint8_t* st = base + s * STAGE;
#pragma unroll
        for (int t = 0; t < 8; ++t)
          w4_bulk_1d(st + t * W4_BLK, p.w + ((size_t)(tile * 8 + t) * p.G + kb) * W4_BLK, W4_BLK, &full[s]);
#pragma unroll
        for (int a = 0; a < 2; ++a)
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                  smem_u32(st + X_OFF + a * X_ATOM)),
              "l"(&map_x), "r"(kb * W4_KB + a * 64), "r"(0), "r"(smem_u32(&full[s]))
              : "memory");
        if (++s == W4_STAGES) {
          s = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    if (lane == 0) {
      constexpr uint32_t idesc = instr_desc_bf16(128, MPAD);
      int s = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nkb; ++i) {
        const int buf = i & 1;
        mbar_wait_parity(&full[s], phase);                   // the x atoms of this stage have landed
        mbar_wait_parity(&a_ready[buf], (uint32_t)(i >> 1) & 1u);  // the weights of this block are in tensor memory
        tc_fence_after();
        const uint32_t xs = smem_u32(base + s * STAGE + X_OFF);
        const uint32_t ta = tmem_base + 128u + (uint32_t)buf * 64u;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint64_t bdesc = smem_desc_sw128(xs + (uint32_t)(k >> 2) * X_ATOM) + (uint64_t)(2 * (k & 3));
          umma_ts_bf16(tmem_base, ta + (uint32_t)(8 * k), bdesc, idesc, (i | k) != 0 ? 1u : 0u);
        }
        umma_commit(&a_free[buf]);
        umma_commit(&empty[s]);
        if (++s == W4_STAGES) {
          s = 0;
          phase ^= 1u;
        }
      }
      umma_commit(tmem_full);
    }
  } else {
    // ===================== de-quantising warps 2.., then the epilogue =====================
    const int quarter = warp & 3;            // a warp may only touch TMEM lanes [32 * (warpid % 4), +32)
    const int khalf = (warp - 2) >> 2;       // which half of a block's k this warp de-quantises (W4_DW = 8)
    const int t = quarter * 32 + lane;       // TMEM lane = output column n0 + t
    const int t16 = t >> 4, g = t & 7, hi = (t >> 3) & 1;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t sh = 4u * (uint32_t)hi;
    int s = 0;
    uint32_t phase = 0;
    for (int i = 0; i < nkb; ++i) {
      const int buf = i & 1;
      mbar_wait_parity(&full[s], phase);
      if (i >= 2) mbar_wait_parity(&a_free[buf], (uint32_t)((i >> 1) - 1) & 1u);
      tc_fence_after();
      const uint32_t blk = smem_u32(base + s * STAGE + t16 * W4_BLK);
      uint32_t sz;
      asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sz) : "r"(blk + 1024u + (uint32_t)(2 * g + hi) * 4u));
      const uint32_t s2 = (sz & 0xffffu) * 0x00010001u;  // bf16x2 (scale, scale)
      const uint32_t z2 = ((sz >> 16) ^ 0x8000u) * 0x00010001u;  // tail holds -zero: bf16x2 (zero, zero)
      // an integer zero (every RTN / GPTQ checkpoint): (128 + q) - (128 + zero) in ONE exact subtraction
      const float zf = __uint_as_float((sz & 0xffff0000u) ^ 0x80000000u);
      const bool zint = zf == floorf(zf) && zf >= 0.f && zf <= 64.f;
      const uint32_t zc2 = zint ? (uint32_t)(0x4300u + (uint32_t)zf) * 0x00010001u : 0x43004300u;
      // a column's zero may be whole and its neighbour's not: the warp goes one way (the store below is the whole warp's), a whole zero
      // then subtracts 0
      const bool one_step = __all_sync(0xffffffffu, zint);
      const uint32_t zr2 = zint ? 0u : z2;
      const uint32_t ta = lane_addr + 128u + (uint32_t)buf * 64u;
      constexpr int MPW = 8 * 4 / W4_DW;  // 16-k slices per warp per block
#pragma unroll
      for (int mm = 0; mm < MPW; ++mm) {  // m = 2 tig + q: k = 32 tig + 16 q + 0..15 of the block -> TMEM columns 16 tig + 8 q + 0..7
        const int m = (W4_DW == 8 ? khalf * 4 : 0) + mm;
        const int tig = m >> 1, q = m & 1;
        uint4 wq;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(wq.x), "=r"(wq.y), "=r"(wq.z), "=r"(wq.w)
                     : "r"(blk + (uint32_t)(q * 512 + (g * 4 + tig) * 16)));
        const uint32_t w[4] = {wq.x, wq.y, wq.z, wq.w};
        uint32_t r[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t nib = (w[j] >> sh) & 0x0F0F0F0Fu;          // this column's four nibbles (k, k+1, k+2, k+3)
          // bf16 (128 + q) = 0x4300 | q; minus 128, minus zero (both exact for integer zeros), times scale (rounded):
          // the reference's get_weight in bf16 (quantization.py:399-408)
          uint32_t a = w4_sub2(w4_prmt(nib, 0x43434343u, 0x5140u), zc2);
          uint32_t b = w4_sub2(w4_prmt(nib, 0x43434343u, 0x5342u), zc2);
          if (!one_step) {
            a = w4_sub2(a, zr2);
            b = w4_sub2(b, zr2);
          }
          r[2 * j] = w4_mul2(a, s2);
          r[2 * j + 1] = w4_mul2(b, s2);
        }
        tmem_st_x8(ta + (uint32_t)(16 * tig + 8 * q), r);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&a_ready[buf]);
        mbar_arrive(&empty[s]);
      }
      if (++s == W4_STAGES) {
        s = 0;
        phase ^= 1u;
      }
    }
    // ---- epilogue: D[t][m] for m < M: thread t holds output column n0 + t; the two warps of a lane quarter share the
    //      M_pad accumulator columns
    mbar_wait_parity(tmem_full, 0);
    tc_fence_after();
    const int n = tile * W4_BN + t;
    constexpr int EW = W4_DW / 4;  // warps per lane quarter
    const float bias = (p.bias != nullptr && p.ksplit == 1) ? __bfloat162float(p.bias[n]) : 0.f;
#pragma unroll 1
    for (int c0 = 16 * khalf; c0 < MPAD; c0 += 16 * EW) {
      uint32_t v[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
            "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
          : "r"(lane_addr + (uint32_t)c0)
          : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int m = c0 + j;
        if (m < p.M) {
          if (p.ksplit == 1) p.y[(size_t)m * p.N + n] = __float2bfloat16_rn(__uint_as_float(v[j]) + bias);
          else p.scratch[(((size_t)tile * p.ksplit + ks) * MPAD + m) * W4_BN + t] = __uint_as_float(v[j]);
        }
      }
      __syncwarp();
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
  // (Measured: reducing inside the kernel - the last k-split to arrive sums the tile - and two
  // CTAs per SM were both SLOWER than a separate reduce kernel and one CTA per SM: 2.95 -> 3.76 ms per 161 Linears at
  // batch 32.  The code stays behind a constant for the record.)
  if (W4_REDUCE_IN_KERNEL && p.ksplit > 1) {
    // the k-split that arrives last adds the tile's partial sums in SPLIT order (the same bits whoever is last), adds the
    // bias, rounds and stores; the counter goes back to zero for the next launch
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(&p.counters[tile], 1) == p.ksplit - 1);
    __syncthreads();
    if (s_last) {
      __threadfence();
      const float* base_t = p.scratch + (size_t)tile * p.ksplit * MPAD * W4_BN;
      for (int e = threadIdx.x; e < p.M * W4_BN; e += blockDim.x) {
        const int m = e / W4_BN, tt = e - m * W4_BN;
        float acc = 0.f;
        for (int k2 = 0; k2 < p.ksplit; ++k2) acc += __ldcg(base_t + ((size_t)k2 * MPAD + m) * W4_BN + tt);
        const int n = tile * W4_BN + tt;
        if (p.bias != nullptr) acc += __bfloat162float(p.bias[n]);
        p.y[(size_t)m * p.N + n] = __float2bfloat16_rn(acc);
      }
      if (threadIdx.x == 0) p.counters[tile] = 0;
    }
  }
}

// y[m][n] = bf16(sum over the k-splits, in split order, + bias)   
__global__ void w4_reduce_kernel(const float* __restrict__ scratch, const __nv_bfloat16* __restrict__ bias,
                                 __nv_bfloat16* __restrict__ y, int M, int N, int ksplit, int mpad) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)M * N) return;
  const int m = (int)(i / N), n = (int)(i - (size_t)m * N);
  const int tile = n / W4_BN, t = n - tile * W4_BN;
  float acc = 0.f;
  for (int ks = 0; ks < ksplit; ++ks) acc += scratch[(((size_t)tile * ksplit + ks) * mpad + m) * W4_BN + t];
  if (bias != nullptr) acc += __bfloat162float(bias[n]);
  y[i] = __float2bfloat16_rn(acc);
}

template <int MPAD>
int launch_w4(const CUtensorMap& mx, const W4Params& p, cudaStream_t st) {
  constexpr int W4_STAGES = w4_stages(MPAD);
  constexpr size_t stage = ((8 * W4_BLK + 1023) / 1024) * 1024 + 2 * MPAD * 128;
  constexpr size_t smem = W4_STAGES * stage + (2 * W4_STAGES + 5) * 8 + 16 + 1024;
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(gemm_w4_tc_kernel<MPAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured.mark();
  }
  gemm_w4_tc_kernel<MPAD><<<(p.N / W4_BN) * p.ksplit, 64 + 32 * W4_DW, smem, st>>>(mx, p);
  LL_LAUNCH_OK("gemm_w4_tc_kernel");
  return LL_OK;
}

// k-split that fills the SMs best (whole waves of one CTA per SM), each unit at least four k-blocks long
int w4_pick_ksplit(int tiles, int G, int sms) {
  int best = 1;
  double best_eff = 0.0;
  for (int ks = 1; ks <= 16 && G / ks >= 4; ++ks) {
    const int units = tiles * ks;
    const double eff = (double)units / ((double)((units + sms - 1) / sms) * sms);
    if (eff > best_eff + 0.03) {
      best_eff = eff;
      best = ks;
    }
  }
  return best;
}

}  // namespace
}  // namespace llb

using namespace llb;

extern "C" {

int ll_gemm_bf16_tc(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, ll_stream stream) {
  return ll_gemm_bf16_tc_form(x, w, bias, y, M, N, K, 0, stream);
}

int ll_gemm_bf16_gated(const void* x, const void* w1, const void* bias1, const void* w2, const void* bias2, void* h, int M, int N, int K,
                       ll_stream stream) {
  LL_CHECK_ARG(x && w1 && w2 && h, "null pointer");
  LL_CHECK_ARG(M > 0 && N > 0 && K > 0, "bad shape M=%d N=%d K=%d", M, N, K);
  LL_CHECK_ARG(K % 8 == 0, "K must be a multiple of 8 (16-byte rows for TMA), got %d", K);
  LL_CHECK_ARG((((uintptr_t)x | (uintptr_t)w1 | (uintptr_t)w2 | (uintptr_t)h) & 15) == 0, "x, the weights and h must be 16-byte aligned");
  return launch_pair<256, true>(x, w1, w2, bias1, bias2, h, M, N, K, (cudaStream_t)stream);
}

int ll_gemm_bf16_tc_error(void) {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, g_gp_error, sizeof(int)) == cudaSuccess ? v : -1;
}

int ll_gemm_bf16_tc_form(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, int tile_columns, ll_stream stream) {
  LL_CHECK_ARG(x && w && y, "null pointer");
  LL_CHECK_ARG(M > 0 && N > 0 && K > 0, "bad shape M=%d N=%d K=%d", M, N, K);
  LL_CHECK_ARG(K % 8 == 0, "K must be a multiple of 8 (16-byte rows for TMA), got %d", K);
  LL_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)y & 15) == 0, "x/w/y must be 16-byte aligned");
  LL_CHECK_ARG(tile_columns == 0 || tile_columns == 128 || tile_columns == 256, "gemm_bf16_tc: tiles of 128 or 256 columns");
  if (tile_columns == 0) {
    // a tile of 128 columns takes 0.53 (many tiles a pair) to 0.67 (one) of the time of 256: what the waves cost.  us, 256 / 128 columns:
    // 11008 x 4096 at 512 rows 45 / 42 (2 waves / 3), 2048 rows 119 / 133 (5 / 10); 4096 x 11008 at 512 rows 57 / 38 (1 / 1).
    const long long pairs = sm_count() > 1 ? sm_count() / 2 : 1, mt = (M + 255) / 256;
    const long long wide = (mt * ((N + 255) / 256) + pairs - 1) / pairs, narrow = (mt * ((N + 127) / 128) + pairs - 1) / pairs;
    tile_columns = 3 * narrow < 5 * wide ? 128 : 256;
  }
  if (tile_columns == 256) return launch_pair<256, false>(x, w, w, bias, nullptr, y, M, N, K, (cudaStream_t)stream);
  return launch_pair<128, false>(x, w, w, bias, nullptr, y, M, N, K, (cudaStream_t)stream);
}

size_t ll_int4_gemm_tc_scratch_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || N % W4_BN != 0 || K % W4_KB != 0) return 0;
  const int mpad = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  const int ks = w4_pick_ksplit(N / W4_BN, K / W4_KB, sm_count() > 0 ? sm_count() : 148);
  return ks == 1 ? 0 : (size_t)(N / W4_BN) * ks * mpad * W4_BN * sizeof(float);
}

namespace {
// per-device arrival counters of the k-splits (one int per 128-column tile; the kernels leave them zero), allocated on
// first use outside stream capture
int32_t* w4_counters(int tiles, cudaStream_t st) {
  static int32_t* buf[16] = {};
  static int cap[16] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return nullptr;
  if (cap[dev] < tiles) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return nullptr;
    const int n = tiles < 4096 ? 4096 : tiles;
    int32_t* nb = nullptr;
    if (cudaMalloc(&nb, (size_t)n * sizeof(int32_t)) != cudaSuccess) return nullptr;
    cudaMemset(nb, 0, (size_t)n * sizeof(int32_t));
    buf[dev] = nb;   // (an older, smaller buffer stays alive: captured graphs may hold it)
    cap[dev] = n;
  }
  return buf[dev];
}
}  // namespace

int ll_int4_gemm_tc(const uint8_t* w_stream, const void* x, const void* bias, void* y, float* scratch, int M, int N, int K,
                    int group, ll_stream stream) {
  LL_CHECK_ARG(w_stream && x && y, "null pointer");
  LL_CHECK_ARG(M >= 1 && M <= 128, "ll_int4_gemm_tc serves 1 <= M <= 128 rows (got %d); larger M: ll_get_weight + ll_gemm_bf16_tc", M);
  if (N <= 0 || K <= 0 || group <= 0 || N % W4_BN != 0 || group % W4_KB != 0 || K % group != 0) {
    set_error("ll_int4_gemm_tc needs N %% 128 == 0 and group %% 128 == 0 (N=%d K=%d group=%d)", N, K, group);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)w_stream & 15) == 0, "x / stream must be 16-byte aligned");
  const int sms = sm_count();
  W4Params p;
  p.w = w_stream; p.y = (__nv_bfloat16*)y; p.scratch = scratch; p.bias = (const __nv_bfloat16*)bias;
  p.M = M; p.N = N; p.K = K; p.G = K / W4_KB;
  p.mpad = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  p.ksplit = w4_pick_ksplit(N / W4_BN, p.G, sms > 0 ? sms : 148);
  LL_CHECK_ARG(p.ksplit == 1 || scratch != nullptr, "this shape splits K %d ways: pass ll_int4_gemm_tc_scratch_bytes() of scratch", p.ksplit);
  CUtensorMap mx;
  if (int r = make_map(x, M, K, p.mpad, &mx)) return r;
  cudaStream_t st = (cudaStream_t)stream;
  p.counters = nullptr;
  if (W4_REDUCE_IN_KERNEL && p.ksplit > 1) {
    p.counters = w4_counters(N / W4_BN, st);
    if (p.counters == nullptr) {
      set_error("ll_int4_gemm_tc: could not allocate the split counters (first call under stream capture?)");
      return LL_ERR_CUDA;
    }
  }
  int r;
  if (p.mpad == 16) r = launch_w4<16>(mx, p, st);
  else if (p.mpad == 32) r = launch_w4<32>(mx, p, st);
  else if (p.mpad == 64) r = launch_w4<64>(mx, p, st);
  else r = launch_w4<128>(mx, p, st);
  if (r) return r;
  if (!W4_REDUCE_IN_KERNEL && p.ksplit > 1) {
    const size_t n = (size_t)M * N;
    w4_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(scratch, p.bias, p.y, M, N, p.ksplit, p.mpad);
    LL_LAUNCH_OK("w4_reduce_kernel");
  }
  return LL_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------------------
// No-allocation variant of ll_int4_gemm_tc (no counterpart in the reference; added at the request of the run's operators
// for callers that cannot call cudaMalloc: code under CUDA-graph capture, tight serving loops, harnesses that forbid it).
// The split-K partial sums live in a file-scope device array instead of a caller-provided buffer.  Every GPU that loads
// this library holds LL_INT4_GEMM_TC_STATIC_SCRATCH_BYTES until exit.  All calls on a device share the array: two calls
// that overlap on the GPU (different streams, or graphs replayed concurrently) race on it.  Nothing in it has to start at
// zero: every (tile, k-split) unit writes rows m < M of its block of partial sums, and w4_reduce_kernel (after it on
// the stream) reads exactly those rows, so the previous call's contents are never observed.
// ---------------------------------------------------------------------------------------------------------------------
static_assert(!llb::W4_REDUCE_IN_KERNEL, "the static-scratch entry point has no arrival counters: it needs the two-kernel reduce");
static __device__ __align__(256) float g_w4_static_scratch[LL_INT4_GEMM_TC_STATIC_SCRATCH_BYTES / sizeof(float)];

namespace {
// In host code `g_w4_static_scratch` is only a stand-in for the symbol: its device address comes from
// cudaGetSymbolAddress, asked once per device with that device current.
float* w4_static_scratch(void) {
  constexpr int MAX_DEV = 64;
  static float* ptr[MAX_DEV] = {};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= MAX_DEV) {
    set_error("ll_int4_gemm_tc_static: cudaGetDevice: %s (device %d)", cudaGetErrorString(e), dev);
    return nullptr;
  }
  if (ptr[dev] == nullptr) {
    void* d = nullptr;
    e = cudaGetSymbolAddress(&d, g_w4_static_scratch);
    if (e != cudaSuccess || d == nullptr) {
      set_error("ll_int4_gemm_tc_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      return nullptr;
    }
    ptr[dev] = static_cast<float*>(d);
  }
  return ptr[dev];
}
}  // namespace

extern "C" int ll_int4_gemm_tc_static(const uint8_t* w_stream, const void* x, const void* bias, void* y, int M, int N, int K,
                                      int group, ll_stream stream) {
  LL_CHECK_ARG(w_stream && x && y, "null pointer");
  LL_CHECK_ARG(M >= 1 && M <= 128, "ll_int4_gemm_tc_static serves 1 <= M <= 128 rows (got %d)", M);
  if (N <= 0 || K <= 0 || group <= 0 || N % llb::W4_BN != 0 || group % llb::W4_KB != 0 || K % group != 0) {
    set_error("ll_int4_gemm_tc_static needs N %% 128 == 0 and group %% 128 == 0 (N=%d K=%d group=%d)", N, K, group);
    return LL_ERR_UNSUPPORTED;
  }
  const size_t need = ll_int4_gemm_tc_scratch_bytes(M, N, K);
  if (need > (size_t)LL_INT4_GEMM_TC_STATIC_SCRATCH_BYTES) {
    set_error("ll_int4_gemm_tc_static: M=%d N=%d K=%d needs %zu bytes of split-K scratch, the built-in array holds %zu: "
              "use ll_int4_gemm_tc with a caller-provided buffer", M, N, K, need, (size_t)LL_INT4_GEMM_TC_STATIC_SCRATCH_BYTES);
    return LL_ERR_UNSUPPORTED;
  }
  float* scratch = nullptr;
  if (need != 0) {
    scratch = w4_static_scratch();
    if (scratch == nullptr) return LL_ERR_CUDA;
  }
  return ll_int4_gemm_tc(w_stream, x, bias, y, scratch, M, N, K, group, stream);
}
