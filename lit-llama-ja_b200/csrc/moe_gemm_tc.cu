// Grouped expert GEMM of the mixture-of-experts feed-forward on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// The (token, choice) pairs are sorted by expert (ll_moe_route) and the rows of the activations are gathered into that order once
// (ll_moe_gather_rows), so every operand is a matrix that TMA can tile:
//   mode 1 (GLU) : h[r][n] = glu(xs[r] . gate_e[n], xs[r] . up_e[n])     w [X][2N][K] = [gate; up]
//   mode 3 (relu^2): h[r][n] = relu(xs[r] . up_e[n])^2                    w [X][N][K]
//   mode 0 (down): y[perm[r]][n] = h[r] . down_e[n]                       w [X][N][K]
// for the sorted rows r of expert e (found from the device-side offsets: no host synchronisation).
//
// The products are turned round: the WEIGHTS are the operand of 256 rows (a pair of CTAs, tcgen05 cta_group::2, 128 rows and accumulator lanes
// each) and an expert's tokens are the columns, 32 to 256 of them in steps of 32.  An expert's weights always fill whole tiles, and the
// tokens it happens to have are rounded up to 32 instead of 128; an expert of more than 256 tokens gets equal tiles.  The pair shares the
// tokens (each CTA brings half of them).  GLU: a CTA's 128 rows are eight of gate and eight of up in turn (one box of a five-dimensional map),
// so that a thread finds both numbers of an output in one load from tensor memory.
// One pair per two SMs walks the tiles t = pair, + pairs, ... (an expert's token tiles innermost: they read the same weights):
//   warp 0   : TMA producer (128 rows of w, half of the tokens, 64 k each, 128-byte swizzle) into a six-stage ring that runs on across tiles
//   warp 1   : TMEM allocation; in rank 0 one elected thread issues tcgen05.mma 256 x n x 16 (bf16 in, fp32 accumulate)
//   warps 2-9: epilogue, 32 tokens at a time: 16x256b loads from tensor memory, the unit, a transposing store into the warp's staging
//              place (tokens of 32 or 64 bytes), whole sectors from there
// Two accumulators of 256 TMEM columns alternate, so the epilogue of a tile runs under the main loop of the next.
// What bounds it: with few tokens the weights' way from HBM (64 tokens, 32 experts of 2048 x 1024: 5.7 TB/s while all pairs have a tile, and
// 3.6 rounds of tiles dealt out in four); with many the shared memory's 128 bytes a clock, which a stage of 64 k passes through twice
// (written and read: about 256 + n clocks where the products take 2 n).  8192 rows of 32 experts, width 2048, ff 1024: first projections 97 us
// with 128-row tiles of one CTA, 72 so; second ones 57 and 45.
// ll_moe_prompt chains the whole layer by programmatic launches; the shared expert's tiles stand before the experts' in the same launch, which
// fills rounds and starts while the router and the sort still run.  Rows brought by gather4 copies instead of a gathering kernel: 301 us a layer
// where it takes 188 (2048 tokens; 128-byte pieces are too many copies).
// Every wait on an mbarrier is bounded; a wait that runs out records a code in g_moe_tc_error, the roles of both CTAs
// stop, copies and products in flight end, TMEM is freed.
#include <algorithm>

#include "tcgen05.cuh"

namespace llb {

// moe_ops.cu: the router alone, and the combination, as parts of a chain of launches
int moe_route_only(const void* x, const float* w_router, const float* bias, int M, int dim, int n_experts, int top, int score, const float* correction,
                   float out_scale, int n_groups, int keep_groups, int group_top, int32_t* expert_idx, float* expert_w, const void* gate_row, float* gate,
                   cudaStream_t st);
int moe_combine_rows(const void* y, const float* expert_w, int top, const void* shared_y, const float* gate, void* out, int M, int dim, cudaStream_t st);

namespace {

constexpr int MT_STAGES = 6, MT_NMAX = 256, MT_NSTEP = 32;
constexpr int MT_A_BYTES = 128 * BK * 2, MT_B_BYTES = MT_NMAX / 2 * BK * 2;
constexpr int MT_EPI_WARPS = 8, MT_THREADS = 64 + 32 * MT_EPI_WARPS, MT_OUT = 32 * 64;      // staging of a warp: 32 tokens of 64 bytes
constexpr size_t MT_SMEM = (size_t)MT_STAGES * (MT_A_BYTES + MT_B_BYTES) + MT_EPI_WARPS * MT_OUT + (2 * MT_STAGES + 4) * 8 + 32 + 1024;
constexpr uint32_t MT_WAIT_LIMIT = 1u << 22;

__device__ int g_moe_tc_error = 0;

struct MtPart {                     // the experts' products, or the shared expert's
  __nv_bfloat16* c;
  int N, nkb, ldc, vec;             // vec: rows of c are whole 16-byte pieces
  int boxes;                        // GLU with N no multiple of 8: gate and up rows come in boxes of eight from a flat map
  float limit;
};
struct MtParams {
  MtPart part[2];                   // experts, shared expert
  const int32_t* offsets;
  const int32_t* perm;
  const int32_t* order;             // experts by falling size of their tiles, or null: as they stand
  int X, M;                         // M: rows of the shared expert (0: there is none)
  int early;                        // the shared expert's operands are there before the kernels that this one waits for have ended
  float alpha, shift;
  int* word;
};
struct MtFail {
  volatile int* here;
  uint32_t there;
  int* word;
};

// A wait that ends: on its phase, when another role has given up, or after the limit.
__device__ __forceinline__ bool mt_wait(uint64_t* bar, uint32_t parity, const MtFail& f, int code) {
  for (uint32_t i = 0; i < MT_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *f.here) return false;
  }
  *f.here = 1;
  store_cluster_u32(f.there, 1u);
  atomicCAS(&g_moe_tc_error, 0, code);
  wait_ran_out(f.word, 400 + code);
  return false;
}

// Walk over the tiles: the shared expert's, then the experts'; every role keeps its own.  Tile: 256 weight rows (column tile `ct`) x `cnt`
// rows from `r0` on, `n` columns of the product.
struct MtWalk {
  int k = -2, e = -1, first = 0, next = 0;      // place in the order, expert (-1: shared), its first tile, the one after its last
  int row = 0, count = 0, tiles = 1, step = 0;
  int ct = 0, r0 = 0, cnt = 0, n = 0;
  static __device__ __forceinline__ int columns(int count, int tiles) { return ((count + tiles - 1) / tiles + MT_NSTEP - 1) / MT_NSTEP * MT_NSTEP; }
  template <int OUTS>
  __device__ __forceinline__ bool seek(const MtParams& p, int t) {
    while (t >= next) {
      if (++k >= p.X) return false;
      if (k < 0) {
        e = -1, row = 0, count = p.M;
      } else {
        if (k == 0 && p.early) pdl_wait();      // (offsets, order, perm: the first look at what the kernels before have left)
        e = p.order != nullptr ? p.order[k] : k;
        row = p.offsets[e];
        count = p.offsets[e + 1] - row;
      }
      tiles = (count + MT_NMAX - 1) / MT_NMAX;
      first = next;
      next += tiles * ((p.part[k < 0].N + 2 * OUTS - 1) / (2 * OUTS));
      if (count > 0) step = columns(count, tiles);
    }
    const int q = t - first;
    ct = q / tiles;
    const int at = (q - ct * tiles) * step;
    r0 = row + at;
    cnt = min(step, count - at);
    n = (cnt + MT_NSTEP - 1) / MT_NSTEP * MT_NSTEP;
    return true;
  }
};
// the i-th tile of a pair: to and fro, so that with tiles of falling size the pairs' sums are alike
__device__ __forceinline__ int mt_tile(int i, int pair, int pairs) { return i * pairs + ((i & 1) ? pairs - 1 - pair : pair); }

__device__ __forceinline__ void pair_box3(void* dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void pair_box5(void* dst, const CUtensorMap* map, int x, int chunk, int e, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(x), "r"(0), "r"(0), "r"(chunk), "r"(e), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void mt_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 16 lanes x 32 columns: v[4 i + j] is lane (lane / 4) + 8 * (j / 2), column 8 i + 2 (lane % 4) + j % 2
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
        "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// four 8 x 8 blocks of packed pairs, transposed: the lane's address is the place of eight numbers of token `lane`
__device__ __forceinline__ void store_tokens(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

struct MtMaps {      // weights; tokens in boxes of 64 and of 16 rows
  CUtensorMap w, t64, t16;
};

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(MT_THREADS, 1)
    moe_gemm_pair_kernel(const __grid_constant__ MtMaps experts, const __grid_constant__ MtMaps shared, const __grid_constant__ MtParams p) {
  constexpr int OUTS = MODE == 1 ? 64 : 128;             // outputs of a CTA's 128 rows
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* sa = base;                              // [STAGES][128][64] bf16, swizzled
  uint8_t* sb = sa + MT_STAGES * MT_A_BYTES;       // [STAGES][up to 128][64]
  uint8_t* so = sb + MT_STAGES * MT_B_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(so + MT_EPI_WARPS * MT_OUT);      // used in rank 0
  uint64_t* empty = full + MT_STAGES;
  uint64_t* acc_full = empty + MT_STAGES;          // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2], used in rank 0: both CTAs' warps arrive
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&experts.w);
    prefetch_tensormap(&experts.t64);
    prefetch_tensormap(&experts.t16);
    prefetch_tensormap(&shared.w);
    prefetch_tensormap(&shared.t64);
    prefetch_tensormap(&shared.t16);
    for (int i = 0; i < MT_STAGES; ++i) mbar_init(&full[i], 1), mbar_init(&empty[i], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&acc_full[i], 1), mbar_init(&acc_empty[i], 2 * MT_EPI_WARPS);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) pair_tmem_alloc(tmem_ptr, 2 * MT_NMAX);
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const MtFail fail{s_fail, cluster_addr(s_fail, (uint32_t)(rank ^ 1)), p.word};
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (!p.early) pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {
    if (elect_one()) {
      MtWalk walk;
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int i = 0; ok && walk.seek<OUTS>(p, mt_tile(i, pair, pairs)); ++i) {
        const bool dense = walk.e < 0;
        const MtPart& part = p.part[dense];
        const MtMaps& maps = dense ? shared : experts;
        const int half = walk.n / 2, r0 = walk.r0 + rank * half, n0 = (walk.ct * 2 + rank) * OUTS, e = dense ? 0 : walk.e, nkb = part.nkb;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = mt_wait(&empty[s], ph, fail, 1))) break;
          if (rank == 0) mbar_expect_tx(&full[s], (uint32_t)(2 * (MT_A_BYTES + half * BK * 2)));      // both CTAs' operands
          const uint32_t bar = cluster_addr(&full[s], 0);
          uint8_t *da = sa + s * MT_A_BYTES, *db = sb + s * MT_B_BYTES;
          if (MODE != 1) {
            pair_box3(da, &maps.w, kb * BK, n0, e, bar);
          } else if (!part.boxes) {
            pair_box5(da, &maps.w, kb * BK, n0 / 8, e, bar);
          } else {
            const int y = e * 2 * part.N + n0;
            for (int j = 0; j < 8; ++j) {
              pair_box(da + j * 2048, &maps.w, kb * BK, y + 8 * j, bar);
              pair_box(da + j * 2048 + 1024, &maps.w, kb * BK, y + part.N + 8 * j, bar);
            }
          }
          int r = 0;
          for (; r + 64 <= half; r += 64) pair_box(db + r * BK * 2, &maps.t64, kb * BK, r0 + r, bar);
          for (; r < half; r += 16) pair_box(db + r * BK * 2, &maps.t16, kb * BK, r0 + r, bar);
          if (++s == MT_STAGES) s = 0, ph ^= 1u;
        }
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint64_t ad = smem_desc_sw128(smem_u32(sa)), bd = smem_desc_sw128(smem_u32(sb));
      MtWalk walk;
      bool ok = true;
      int s = 0, i = 0;
      uint32_t ph = 0;
      for (; rank == 0 && ok && walk.seek<OUTS>(p, mt_tile(i, pair, pairs)); ++i) {
        const int nkb = p.part[walk.e < 0].nkb;
        const uint32_t d = tmem + (uint32_t)((i & 1) * MT_NMAX), idesc = instr_desc_bf16(256, 0) | ((uint32_t)(walk.n >> 3) << 17);
        if (!(ok = mt_wait(&acc_empty[i & 1], (uint32_t)((i >> 1) & 1) ^ 1u, fail, 4))) break;
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = mt_wait(&full[s], ph, fail, 2))) break;
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            mt_mma(d, ad + (uint64_t)(s * (MT_A_BYTES >> 4) + 2 * k), bd + (uint64_t)(s * (MT_B_BYTES >> 4) + 2 * k), idesc, (kb | k) != 0 ? 1u : 0u);
          pair_commit(&empty[s]);
          if (++s == MT_STAGES) s = 0, ph ^= 1u;
        }
        if (ok) pair_commit(&acc_full[i & 1]);
      }
      if (!ok) let_issued_work_end();
    }
  } else {
    const int quarter = warp & 3, part = (warp - 2) >> 2;   // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
    constexpr int DIMS = OUTS / 4, CHUNKS = DIMS / 8;       // outputs of a quarter, 16-byte pieces of a token
    const uint32_t stage = smem_u32(so + (warp - 2) * MT_OUT);
    // where the lane's token lies; pieces of neighbouring tokens change places so that eight tokens cover all banks
    const int turn = MODE == 1 ? (lane >> 2) & 1 : (lane >> 1) & 3;
    const uint32_t mine = stage + (uint32_t)(lane * DIMS * 2);
    MtWalk walk;
    int i = 0;
    for (; walk.seek<OUTS>(p, mt_tile(i, pair, pairs)); ++i) {
      const MtPart& out = p.part[walk.e < 0];
      const float limit = out.limit;
      const int n0 = (walk.ct * 2 + rank) * OUTS + quarter * DIMS;
      if (!__all_sync(0xffffffffu, mt_wait(&acc_full[i & 1], (uint32_t)(i >> 1) & 1u, fail, 3))) break;
      tc_fence_after();
      const uint32_t td = tmem + (uint32_t)((i & 1) * MT_NMAX) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c0 = part * 32; c0 < walk.cnt; c0 += 64) {
        const int tok = c0 + lane;
        int row = walk.r0 + tok;
        if (MODE == 0 && walk.e >= 0 && tok < walk.cnt) row = p.perm[row];
#pragma unroll
        for (int hl = 0; hl < 2; ++hl) {
          uint32_t v[16];
          tmem_ld_16x32(td + ((uint32_t)(16 * hl) << 16) + (uint32_t)c0, v);
          if (MODE == 1) {
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float f[2];
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const float g = fminf(__uint_as_float(v[4 * j + q]), limit);
                const float up = fminf(fmaxf(__uint_as_float(v[4 * j + 2 + q]), -limit), limit);
                f[q] = g / (1.f + expf(-p.alpha * g)) * (up + p.shift);
              }
              o[j] = pack_bf16(f[0], f[1]);
            }
            store_tokens(mine + (uint32_t)((hl ^ turn) * 16), o[0], o[1], o[2], o[3]);
          } else {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              uint32_t o[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                float f0 = __uint_as_float(v[4 * j + 2 * q]), f1 = __uint_as_float(v[4 * j + 2 * q + 1]);
                if (MODE == 3) f0 = fmaxf(f0, 0.f) * fmaxf(f0, 0.f), f1 = fmaxf(f1, 0.f) * fmaxf(f1, 0.f);
                o[j] = pack_bf16(f0, f1);
              }
              store_tokens(mine + (uint32_t)(((2 * hl + q) ^ turn) * 16), o[0], o[1], o[2], o[3]);
            }
          }
        }
        __syncwarp();
#pragma unroll
        for (int it = 0; it < CHUNKS; ++it) {
          const int at = it * 32 + lane, tk = at / CHUNKS, ch = at % CHUNKS;
          const int dst = __shfl_sync(0xffffffffu, row, tk);
          const uint4 u = lds128(stage + (uint32_t)(tk * DIMS * 2 + ((ch ^ (MODE == 1 ? (tk >> 2) & 1 : (tk >> 1) & 3)) * 16)));
          const int col = n0 + 8 * ch;
          if (c0 + tk < walk.cnt && col < out.N) {
            __nv_bfloat16* at_c = out.c + (size_t)dst * out.ldc + col;
            if (out.vec) {
              *reinterpret_cast<uint4*>(at_c) = u;
            } else {
              const uint32_t w[4] = {u.x, u.y, u.z, u.w};
              for (int j = 0; j < 8 && col + j < out.N; ++j) at_c[j] = __ushort_as_bfloat16((uint16_t)(w[j >> 1] >> (16 * (j & 1))));
            }
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[i & 1], 0));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem, 2 * MT_NMAX);
  }
}

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

int mt_encode(const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box, CUtensorMap* out) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled entry point not available");
    return LL_ERR_CUDA;
  }
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d) base=%p", (int)r, base);
    return LL_ERR_CUDA;
  }
  return LL_OK;
}

// The weights' map: GLU as (k, eight rows, gate or up, groups of eight, expert), boxes of 128 rows; else (k, row, expert).
int mt_weight_map(const void* w, int mode, int X, int N, int K, CUtensorMap* out) {
  const cuuint64_t row = (cuuint64_t)K * 2;
  if (mode == 1 && N % 8 == 0) {
    const cuuint64_t dims[5] = {(cuuint64_t)K, 8, 2, (cuuint64_t)N / 8, (cuuint64_t)X}, strides[4] = {row, row * N, row * 8, row * 2 * N};
    const cuuint32_t box[5] = {(cuuint32_t)BK, 8, 2, 8, 1};
    return mt_encode(w, 5, dims, strides, box, out);
  }
  if (mode == 1) return make_map(w, X * 2 * N, K, 8, out);
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)N, (cuuint64_t)X}, strides[2] = {row, row * N};
  const cuuint32_t box[3] = {(cuuint32_t)BK, 128, 1};
  return mt_encode(w, 3, dims, strides, box, out);
}

template <int MODE>
int launch_moe_pair(const MtMaps& experts, const MtMaps& shared, const MtParams& p, int n_rows, cudaStream_t st) {
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(moe_gemm_pair_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MT_SMEM));
    configured.mark();
  }
  const int cols = MODE == 1 ? 128 : 256;
  const long long most = (long long)((p.part[0].N + cols - 1) / cols) * (n_rows / MT_NMAX + std::min(n_rows, p.X)) +
                         (long long)((p.part[1].N + cols - 1) / cols) * ((p.M + MT_NMAX - 1) / MT_NMAX);
  LL_CHECK_ARG(most < (1ll << 30), "moe_grouped_gemm_tc: too many tiles");
  const int pairs = sm_count() > 1 ? sm_count() / 2 : 1;
  LL_CUDA(launch(moe_gemm_pair_kernel<MODE>, dim3(2 * (unsigned)std::min<long long>(most, pairs)), dim3(MT_THREADS), MT_SMEM, st, true, experts,
                 shared, p));
  LL_LAUNCH_OK("moe_gemm_pair_kernel");
  return LL_OK;
}

MtPart mt_part(void* c, int mode, int N, int K, int ldc, float limit) {
  return MtPart{(__nv_bfloat16*)c, N, (K + BK - 1) / BK, ldc, ldc % 8 == 0 && N % 8 == 0, mode == 1 && N % 8 != 0, limit};
}
int mt_maps(const void* w, int mode, int X, int N, int K, const void* a, int rows, MtMaps* m) {
  if (int r = mt_weight_map(w, mode, X, N, K, &m->w)) return r;
  if (int r = make_map(a, rows, K, 64, &m->t64)) return r;
  return make_map(a, rows, K, 16, &m->t16);
}

// The (token, choice) pairs of a prompt in the order of their experts, and the experts in the order of their tiles' size: one block, counts
// and places in shared memory (8192 pairs of 32 experts: 4 us; the pairs of an expert come in no fixed order, which no result depends on).
constexpr int SORT_THREADS = 1024, SORT_KEPT = 16;
__global__ void __launch_bounds__(SORT_THREADS) moe_sort_kernel(const int32_t* expert_idx, int n_pairs, int X, int32_t* __restrict__ offsets,
                                                                int32_t* __restrict__ order, int32_t* __restrict__ perm) {
  extern __shared__ int32_t sort_smem[];
  int32_t *count = sort_smem, *at = count + X, *size = at + X;      // [X] each
  const int tid = threadIdx.x, lane = tid & 31;
  pdl_launch_dependents();
  for (int e = tid; e < X; e += SORT_THREADS) count[e] = 0;
  __syncthreads();
  pdl_wait();
  expert_idx = after_wait(expert_idx);
  int32_t mine[SORT_KEPT], rank[SORT_KEPT];      // the first pairs of a thread keep their places in registers
#pragma unroll
  for (int j = 0; j < SORT_KEPT; ++j) mine[j] = j * SORT_THREADS + tid < n_pairs ? expert_idx[j * SORT_THREADS + tid] : -1;
#pragma unroll
  for (int j = 0; j < SORT_KEPT; ++j)
    if (mine[j] >= 0) rank[j] = atomicAdd(&count[mine[j]], 1);
  __syncthreads();                               // (theirs are the first places; the rest fill an expert's rows from behind)
  for (int i = SORT_KEPT * SORT_THREADS + tid; i < n_pairs; i += SORT_THREADS) atomicAdd(&count[expert_idx[i]], 1);
  __syncthreads();
  if (tid < 32) {
    int before = 0;
    for (int e0 = 0; e0 < X; e0 += 32) {
      const int e = e0 + lane, c = e < X ? count[e] : 0;
      int incl = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
      }
      if (e < X) {
        at[e] = offsets[e] = before + incl - c;
        count[e] = before + incl;
        const int tiles = (c + MT_NMAX - 1) / MT_NMAX;
        size[e] = c > 0 ? MtWalk::columns(c, tiles) : 0;
      }
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) offsets[X] = before;
  }
  __syncthreads();
  for (int e = tid; e < X; e += SORT_THREADS) {
    int place = 0;
    for (int o = 0; o < X; ++o) place += size[o] > size[e] || (size[o] == size[e] && o < e);
    order[place] = e;
  }
#pragma unroll
  for (int j = 0; j < SORT_KEPT; ++j)
    if (mine[j] >= 0) perm[at[mine[j]] + rank[j]] = j * SORT_THREADS + tid;
  for (int i = SORT_KEPT * SORT_THREADS + tid; i < n_pairs; i += SORT_THREADS) perm[atomicSub(&count[expert_idx[i]], 1) - 1] = i;
}

struct MpScratch {
  int32_t *idx, *offsets, *order, *perm;
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
  return M >= 1 && M < (1 << 24) && width > 0 && width % 8 == 0 && ff > 0 && ff % 8 == 0 && shared_ff >= 0 && shared_ff % 8 == 0 && n_experts <= 4096 &&
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
  if (int r = moe_route_only(x, w_router, bias, M, width, n_experts, top, score, correction, out_scale, n_groups, keep_groups, group_top, s.idx, s.weight,
                             gate_row, s.gate, st))
    return r;
  LL_CUDA(launch(moe_sort_kernel, dim3(1), dim3(SORT_THREADS), 3 * sizeof(int32_t) * n_experts, st, true, (const int32_t*)s.idx, n, n_experts, s.offsets,
                 s.order, s.perm));
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
  p.offsets = s.offsets, p.perm = s.perm, p.order = s.order, p.X = n_experts, p.M = shared_ff ? M : 0, p.early = 1;
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
  if (cudaMemcpyFromSymbol(&v, g_moe_tc_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // extern "C"
