// Products of weight matrices with the rows of a token matrix on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), the products turned
// round: the WEIGHTS are the operand of 256 rows (a pair of CTAs, tcgen05 cta_group::2, 128 rows and accumulator lanes each) and the tokens are
// the columns, 32 to 256 of them in steps of 32.  Weights always fill whole tiles, and tokens are rounded up to 32 instead of 128.  The pair shares
// the tokens (each CTA brings half of them).  Grouped (moe_gemm_tc.cu: an expert's weights for its sorted rows) and dense (dense_rows.cu).
//   mode 0: c[r][n] = x[r] . w[n];  mode 3: its relu, squared;  mode 1 (GLU): c[r][n] = glu(x[r] . gate[n], x[r] . up[n]), w = [gate; up].  GLU: a
//   CTA's 128 rows are eight of gate and eight of up in turn (one box of a five-dimensional map), so that a thread finds both numbers of an
//   output in one load from tensor memory.
// One pair per two SMs walks the tiles t = pair, + pairs, ... (a matrix's token tiles innermost: they read the same weights):
//   warp 0   : TMA producer (128 rows of w, half of the tokens, 64 k each, 128-byte swizzle) into a six-stage ring that runs on across tiles
//   warp 1   : TMEM allocation; in rank 0 one elected thread issues tcgen05.mma 256 x n x 16 (bf16 in, fp32 accumulate)
//   warps 2-9: epilogue, 32 tokens at a time: 16x256b loads from tensor memory, the unit, a transposing store into the warp's staging
//              place (tokens of 32 or 64 bytes), whole sectors from there
// Two accumulators of 256 TMEM columns alternate, so the epilogue of a tile runs under the main loop of the next.
// What bounds it: with few tokens the weights' way from HBM; with many a stage of the ring, 64 k, which by timing takes about 256 + n clocks where its
// products take 2 n.  Counters, 8192 rows of 32 experts of 2048 x 1024, first and second projections: tensor pipe 52 and 47 % of the time, HBM 44 and 44,
// L2 39 and 38, shared memory's banks 16 % of their rate reading and 16 writing, issue slots 22 and 15; 2048 rows through 5120 x 2048: 51, 9, 37, 17 and
// 17, 10.  None is full: what is left are the waits of a stage and the unequal ends.
// Every wait on an mbarrier is bounded; a wait that runs out records a code, the roles of both CTAs stop, copies and products in flight end,
// TMEM is freed.
#pragma once
#include <algorithm>

#include "tcgen05.cuh"

namespace llb {
namespace {

constexpr int MT_STAGES = 6, MT_NMAX = 256, MT_NSTEP = 32;
constexpr int MT_A_BYTES = 128 * BK * 2, MT_B_BYTES = MT_NMAX / 2 * BK * 2;
constexpr int MT_EPI_WARPS = 8, MT_THREADS = 64 + 32 * MT_EPI_WARPS, MT_OUT = 32 * 64;      // staging of a warp: 32 tokens of 64 bytes
constexpr size_t MT_SMEM = (size_t)MT_STAGES * (MT_A_BYTES + MT_B_BYTES) + MT_EPI_WARPS * MT_OUT + (2 * MT_STAGES + 4) * 8 + 32 + 1024;
constexpr int MT_TABLE = 2048;      // entries of a CTA's table of where experts' tiles begin
constexpr size_t MT_TABLE_SMEM = (MT_TABLE + 1 + MT_THREADS / 32) * sizeof(int32_t);
constexpr uint32_t MT_WAIT_LIMIT = 1u << 22;

__device__ int g_pair_rows_error = 0;      // per file that instantiates the kernel

struct MtPart {                     // the experts' products, or the shared expert's
  __nv_bfloat16* c;
  int N, nkb, ldc, vec;             // vec: rows of c are whole 16-byte pieces
  int boxes;                        // GLU with N no multiple of 8: gate and up rows come in boxes of eight from a flat map
  int across;                       // not 0 (mode 0): w is [heads][K][64 * across], outputs side by side in memory
  float limit;
};
struct MtParams {
  MtPart part[2];                   // experts, shared expert
  const int32_t* offsets;
  const int32_t* perm;
  const int32_t* order;             // experts by falling size of their tiles, or null: as they stand
  const int32_t* first;             // [X + 1] in that order: row tiles (of up to MT_NMAX rows) before an expert's, or null: every CTA makes a table
  int X, M;                         // M: rows of the shared expert (0: there is none)
  int group, groups;                // experts of an entry of that table, and entries (launch_moe_pair)
  int cuts;                         // tiles that these rows are cut into
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
  atomicCAS(&g_pair_rows_error, 0, code);
  wait_ran_out(f.word, 400 + code);
  return false;
}

// Walk over the tiles: the shared expert's, then the experts'; every role keeps its own.  Tile: 256 weight rows (column tile `ct`) x `cnt`
// rows from `r0` on, `n` columns of the product.  The expert of a tile is looked up in the table of where experts' row tiles begin, from the last one
// on in steps that double.  (Expert by expert, two dependent loads and two divisions each, every role took half a us an expert: 2048 tokens, 256 experts of
// 256 x 64, 219 us a layer where it takes 92; 700 tokens, 512 experts of 512 x 64 415 and 170.)
struct MtWalk {
  int k = -2, e = -1, base = 0, first = 0, next = 0;      // place in the order, expert (-1: shared), tiles before the experts', its first tile, the one after
  int row = 0, count = 0, tiles = 1, step = 0;
  int ct = 0, r0 = 0, cnt = 0, n = 0;
  static __host__ __device__ __forceinline__ int columns(int count, int tiles) { return ((count + tiles - 1) / tiles + MT_NSTEP - 1) / MT_NSTEP * MT_NSTEP; }
  template <int OUTS>
  static __device__ __forceinline__ int column_tiles(const MtPart& part) { return (part.N + 2 * OUTS - 1) / (2 * OUTS); }
  template <int OUTS>
  __device__ __forceinline__ bool seek(const MtParams& p, const int32_t* table, int t) {
    if (k == -2) {
      k = -1, count = p.M, tiles = p.cuts;
      base = next = tiles * column_tiles<OUTS>(p.part[1]);
      if (count > 0) step = columns(count, tiles);
    }
    if (t >= next) {
      if (p.X == 0) return false;
      if (k < 0 && p.early) pdl_wait();      // (offsets, order, first, perm: the first look at what the kernels before have left)
      const int cols = column_tiles<OUTS>(p.part[0]), q = (t - base) / cols;
      if (q >= table[p.groups]) return false;
      int lo = k < 0 ? 0 : k / p.group, hop = 1;
      for (; lo + hop < p.groups && table[lo + hop] <= q; hop *= 2) lo += hop;
      for (; hop > 0; hop /= 2)
        if (lo + hop < p.groups && table[lo + hop] <= q) lo += hop;
      int f = table[lo];
      for (k = lo * p.group;; ++k, f += tiles) {
        e = p.order != nullptr ? p.order[k] : k;
        row = p.offsets[e];
        count = p.offsets[e + 1] - row;
        tiles = (count + MT_NMAX - 1) / MT_NMAX;
        if (q < f + tiles) break;
      }
      first = base + f * cols;
      next = first + tiles * cols;
      step = columns(count, tiles);
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
// The table of a CTA: row tiles before the experts of every entry, and of all; `sums`: a place per warp.  Ends with a barrier of the CTA.
__device__ __forceinline__ void mt_make_table(const MtParams& p, int32_t* table, int32_t* sums) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, per = (p.groups + MT_THREADS - 1) / MT_THREADS, g0 = min(tid * per, p.groups);
  const int g1 = min(g0 + per, p.groups);
  auto row_tiles = [&](int g) {
    int n = 0;
    for (int e = g * p.group; e < min((g + 1) * p.group, p.X); ++e) n += (p.offsets[e + 1] - p.offsets[e] + MT_NMAX - 1) / MT_NMAX;
    return n;
  };
  int own = 0;
  for (int g = g0; g < g1; ++g) own += row_tiles(g);
  int incl = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  int before = incl - own;
  for (int w = 0; w < MT_THREADS / 32; ++w) before += w < warp ? sums[w] : 0;
  for (int g = g0; g < g1; ++g) {
    table[g] = before;
    before += row_tiles(g);
  }
  if (tid == MT_THREADS - 1) table[p.groups] = before;      // (the last thread: all entries stand before its own end)
  __syncthreads();
}
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
// as pair_commit, for the pair of CTAs 2 j and 2 j + 1 of a larger cluster
__device__ __forceinline__ void mt_commit(uint64_t* bar, int j) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)(3u << (2 * j)))
               : "memory");
}
// weights [2 blocks of 64 rows][64 k][64]: the rows run along memory (MN-major), 128-byte swizzle; LBO = distance of the blocks, SBO = of
// groups of eight k
__device__ __forceinline__ uint64_t mt_desc_across(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3fff);
  d |= (uint64_t)(MT_A_BYTES / 2 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
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
  int32_t* s_table = reinterpret_cast<int32_t*>(s_fail + 1);      // [MT_TABLE + 1], then a place per warp

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
  const int32_t* table = p.first;
  if (p.X > 0 && p.first == nullptr) {
    mt_make_table(p, s_table, s_table + MT_TABLE + 1);
    table = s_table;
  }

  if (warp == 0) {
    if (elect_one()) {
      MtWalk walk;
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int i = 0; ok && walk.seek<OUTS>(p, table, mt_tile(i, pair, pairs)); ++i) {
        const bool dense = walk.e < 0;
        const MtPart& part = p.part[dense];
        const MtMaps& maps = dense ? shared : experts;
        const int half = walk.n / 2, r0 = walk.r0 + rank * half, n0 = (walk.ct * 2 + rank) * OUTS, e = dense ? 0 : walk.e, nkb = part.nkb;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = mt_wait(&empty[s], ph, fail, 1))) break;
          if (rank == 0) mbar_expect_tx(&full[s], (uint32_t)(2 * (MT_A_BYTES + half * BK * 2)));      // both CTAs' operands
          const uint32_t bar = cluster_addr(&full[s], 0);
          uint8_t *da = sa + s * MT_A_BYTES, *db = sb + s * MT_B_BYTES;
          if (MODE == 0 && part.across) {
            for (int j = 0; j < 2; ++j) {
              const int blk = (n0 >> 6) + j, head = blk / part.across;
              pair_box3(da + j * (MT_A_BYTES / 2), &maps.w, (blk - head * part.across) * 64, kb * BK, head, bar);
            }
          } else if (MODE != 1) {
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
      const uint64_t bd = smem_desc_sw128(smem_u32(sb));
      MtWalk walk;
      bool ok = true;
      int s = 0, i = 0;
      uint32_t ph = 0;
      for (; rank == 0 && ok && walk.seek<OUTS>(p, table, mt_tile(i, pair, pairs)); ++i) {
        const int nkb = p.part[walk.e < 0].nkb;
        const bool across = MODE == 0 && p.part[walk.e < 0].across != 0;      // 16 k are 16 rows of 128 bytes then, not 32 bytes of a row
        const uint64_t ad = across ? mt_desc_across(smem_u32(sa)) : smem_desc_sw128(smem_u32(sa)), astep = across ? 128 : 2;
        const uint32_t d = tmem + (uint32_t)((i & 1) * MT_NMAX), idesc = instr_desc_bf16(256, 0) | ((uint32_t)(walk.n >> 3) << 17) | (across ? 1u << 15 : 0u);
        if (!(ok = mt_wait(&acc_empty[i & 1], (uint32_t)((i >> 1) & 1) ^ 1u, fail, 4))) break;
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = mt_wait(&full[s], ph, fail, 2))) break;
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            mt_mma(d, ad + (uint64_t)(s * (MT_A_BYTES >> 4)) + astep * (uint64_t)k, bd + (uint64_t)(s * (MT_B_BYTES >> 4) + 2 * k), idesc, (kb | k) != 0 ? 1u : 0u);
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
    for (; walk.seek<OUTS>(p, table, mt_tile(i, pair, pairs)); ++i) {
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
int launch_moe_pair(const MtMaps& experts, const MtMaps& shared, MtParams p, int n_rows, cudaStream_t st) {
  constexpr size_t smem = MT_SMEM + MT_TABLE_SMEM;
  static_assert(smem <= 227 * 1024, "shared memory of a block");
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(moe_gemm_pair_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured.mark();
  }
  p.group = p.first != nullptr || p.X == 0 ? 1 : (p.X + MT_TABLE - 1) / MT_TABLE;
  p.groups = (p.X + p.group - 1) / p.group;
  const int cols = MODE == 1 ? 128 : 256;
  const long long most = (long long)((p.part[0].N + cols - 1) / cols) * (n_rows / MT_NMAX + std::min(n_rows, p.X)) +
                         (long long)((p.part[1].N + cols - 1) / cols) * p.cuts;
  LL_CHECK_ARG(most < (1ll << 30), "moe_grouped_gemm_tc: too many tiles");
  const int pairs = sm_count() > 1 ? sm_count() / 2 : 1;
  LL_CUDA(launch(moe_gemm_pair_kernel<MODE>, dim3(2 * (unsigned)std::min<long long>(most, pairs)), dim3(MT_THREADS), smem, st, true, experts,
                 shared, p));
  LL_LAUNCH_OK("moe_gemm_pair_kernel");
  return LL_OK;
}

MtPart mt_part(void* c, int mode, int N, int K, int ldc, float limit) {
  return MtPart{(__nv_bfloat16*)c, N, (K + BK - 1) / BK, ldc, ldc % 8 == 0 && N % 8 == 0 && ((uintptr_t)c & 15) == 0, mode == 1 && N % 8 != 0, 0, limit};
}
int mt_maps(const void* w, int mode, int X, int N, int K, const void* a, int rows, MtMaps* m) {
  if (int r = mt_weight_map(w, mode, X, N, K, &m->w)) return r;
  if (int r = make_map(a, rows, K, 64, &m->t64)) return r;
  return make_map(a, rows, K, 16, &m->t16);
}

}  // namespace
}  // namespace llb
