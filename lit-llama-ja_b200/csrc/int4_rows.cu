// Many rows through int4 layers on tcgen05 (prompts): y[M][N] = x[M][K] . dequant(W)^T, the weights read in their packed checkpoint form
// (bytes [K/2][N], even k in the low half) and de-quantised inside the main loop with the reference's two bf16 roundings
// (ref: lit_llama/quantization.py:399-408), so that no bf16 copy of W is written and read back.  A second form takes the two layers of a
// gated feed-forward that read the same x: h = silu(x W1^T) * (x W2^T), each step rounded as the separate kernels round it.
//
// Operand roles are swapped: the weights are the A operand and live in tensor memory, where the threads that de-quantise them put them; the
// activations are the B operand, tiles of bn rows x 128 k loaded by TMA.  A pair of CTAs forms one product of 256 weight columns (128 = the
// TMEM lanes of each) x bn rows, and each CTA brings half of the rows: of a CTA of its own x takes 72 KB a step of 128 k at 256 rows from L2,
// 46 bytes a clock and SM; the pair needs 40 KB.  Unpacking reads the bytes by transposing loads (64 single-byte loads a thread before) and
// the scales from shared memory; the loop's registers may not spill or miss in what is left of L1 (that doubled a step's time; of the gated form
// ptxas spills three registers, stored and loaded once each).
// us, one CTA a tile / pairs: 11008 x 4096 at 150, 512, 1100 rows 28 / 24, 51 / 46, 82 / 69; 4096 x 11008 at 150, 512 rows 53 / 48, 87 / 54;
// 32000 x 4096 at 512 rows 140 / 103.  Bound by products at 256 rows a tile (0.84 us a step with all SMs busy, 0.76 at the rate of a large
// dense product), below that by unpacking.  Counters, 512 rows of the gated 11008 x 4096 and of 4096 x 11008 cut along k: tensor pipe 53 and 46 % of the
// time, issue slots 36 and 33, L2 16, HBM 8 and 9.
//   warps 0, 2 : TMA producers: 128 k of bn / 2 rows of x; 64 x 128 packed bytes
//   warp 1     : in the CTA of rank 0, one thread issues 256 x bn x 16 MMAs (A from tensor memory) for both
//   warp 3     : scales and zeros, several steps ahead
//   warps 4-19 : de-quantise in four groups of four warps (a warp per TMEM lane quarter); group g makes every fourth step of 128 k into
//                A buffer g, so that four steps are in the making at a time (one step's chain of waits, loads and stores is 1500 clocks
//                long however many warps share it); then the epilogue, every fourth 16 rows per group
// Gated form: a CTA's 128 columns are 64 of W1 and the same 64 of W2; the warps of the first hand their sums, rounded, to those of the
// second through shared memory.  (13824 x 5120, 1100 rows: 241 us; two layers and their product 274 before.)
// The tiles of a last wave that would leave pairs idle are cut along k (r4_plan); a second small kernel adds their parts, in fp32 and in the order of
// k.  (A prompt of 512 tokens has 32 tiles of its 4096 x 11008 layer for 74 pairs, and 24 in the third wave of the gated one.)
// Persistent: a pair walks tiles with a stride of the grid; a group drains a tile after its first step of the next one, and gives the
// accumulator back as soon as it is in registers, so that the tensor cores wait for the drain alone.
// Every wait is bounded; one that runs out records a code, all roles of both CTAs stop, copies in flight are waited for, tensor memory is
// freed.
#include "int4_unpack.cuh"

namespace llb {
namespace {

constexpr int R4_GROUPS = 4, R4_THREADS = (4 + 4 * R4_GROUPS) * 32;
constexpr int R4_WST = 6;                                              // stages of packed bytes
constexpr int R4_XBYTES = 128 * 1024, R4_XST = 8;                      // the ring of x: as many stages of two halves [bn / 2 rows][64 k] as fit
constexpr int R4_BOX = 16 * 64, R4_OUT = 2 * R4_BOX;                   // a warp stores 16 rows of 32 columns at a time, from two places in turn
constexpr int R4_SWAP = 64 * 16 * 4;                                   // gated form: what a group hands over at a time, 64 columns x 32 rows of bf16
constexpr uint32_t R4_WAIT_LIMIT = 1u << 20;
constexpr int R4_SMEM = R4_XBYTES + R4_WST * (R4_WBYTES + R4_SZ) + 4 * R4_GROUPS * R4_OUT + 512 + 1024;   // (gated: half the warps store, the rest is for the swap)
static_assert(8 * R4_OUT >= R4_GROUPS * R4_SWAP, "the gated form's second half of the staging space");

__device__ int g_r4_error = 0;

struct R4Params {
  const __nv_bfloat16* scales[2];   // [N][G]; the second set: the gated form's W2
  const __nv_bfloat16* zeros[2];
  const __nv_bfloat16* bias[2];
  __nv_bfloat16* y;
  float* part;                   // [(tiles - full) * parts][2 CTAs][bn][128]: sums of parts of tiles
  int M, N, steps, G, steps_per_group, wide, bn, xst, mtiles, tiles, full, parts;      // the tiles from `full` on are cut along k into `parts`
  int* word;                     // wait_word()
};

// What a pair takes: of the tiles before p.full every `pairs`th, whole, then of the parts of the others every `pairs`th, two at most.
struct R4Unit {
  int tile, k0, len;             // `len` steps of a tile from step k0 on (none: 0)
};
struct R4Share {
  int whole, part[2];            // how many whole tiles; which parts
  R4Unit unit[2];
};
__device__ __forceinline__ R4Share r4_share(const R4Params& p, int pair, int pairs) {
  R4Share q{p.full > pair ? (p.full - pair + pairs - 1) / pairs : 0, {pair, pair + pairs}, {{0, 0, 0}, {0, 0, 0}}};
  for (int i = 0; i < 2; ++i) {
    const int t = p.parts > 0 ? q.part[i] / p.parts : 0, c = q.part[i] - t * p.parts;
    if (p.parts == 0 || p.full + t >= p.tiles) continue;
    const int k0 = (int)((long long)p.steps * c / p.parts);
    q.unit[i] = {p.full + t, k0, (int)((long long)p.steps * (c + 1) / p.parts) - k0};
  }
  return q;
}
// its nth unit
__device__ __forceinline__ R4Unit r4_unit(const volatile R4Share* q, int steps, int pair, int pairs, int nth) {
  const int o = nth - q->whole;
  if (o < 0) return {pair + nth * pairs, 0, steps};
  if (o > 1) return {0, 0, 0};
  return {q->unit[o].tile, q->unit[o].k0, q->unit[o].len};
}

struct R4Fail {                  // the flag that stops all roles, here and in the other CTA
  volatile int* here;
  uint32_t there;
  int* word;
};
__device__ __forceinline__ void r4_give_up(const R4Fail& f, int code) {
  *f.here = 1;
  store_cluster_u32(f.there, 1u);
  atomicCAS(&g_r4_error, 0, code);
  wait_ran_out(f.word, 200 + code);
}
__device__ __forceinline__ bool r4_wait(uint64_t* bar, uint32_t parity, const R4Fail& f, int code) {
  for (uint32_t i = 0; i < R4_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *f.here) return false;
  }
  r4_give_up(f, code);
  return false;
}
// The same without suspending the thread between looks: for the thread that feeds the tensor cores, whose wake-up would be waited for.
__device__ __forceinline__ bool r4_spin(uint64_t* bar, uint32_t parity, const R4Fail& f, int code) {
  for (uint32_t i = 0; i < 64u * R4_WAIT_LIMIT; ++i) {
    if (mbar_test_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *f.here) return false;
  }
  r4_give_up(f, code);
  return false;
}
__device__ __forceinline__ void r4_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
template <bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(R4_THREADS, 1)
    int4_rows_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_x,
                     const __grid_constant__ CUtensorMap map_y, const R4Params p) {
  constexpr uint32_t TM_A = 256;                       // D: columns [0, bn); A buffers of 64 columns from 256 on
  constexpr int TILE_N = GATED ? 128 : 256;            // outputs of a pair
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* sx = base;                                  // [xst][2][bn / 2][64] bf16, swizzled
  uint8_t* sw = base + R4_XBYTES;                      // [WST][64][128] packed bytes (gated: [2][64][64]), swizzled
  uint8_t* so = sw + R4_WST * R4_WBYTES;               // [16 warps][2][16 rows][32 columns] bf16, swizzled
  uint8_t* swap = so + 8 * R4_OUT;                     // gated form: [GROUPS][16 pairs of rows][64 columns]
  uint8_t* sz = so + 4 * R4_GROUPS * R4_OUT;           // [WST][128] scale | zero << 16
  uint64_t* x_full = reinterpret_cast<uint64_t*>(sz + R4_WST * R4_SZ);               // used in rank 0
  uint64_t* x_empty = x_full + R4_XST;
  uint64_t* w_full = x_empty + R4_XST;
  uint64_t* w_empty = w_full + R4_WST;
  uint64_t* a_ready = w_empty + R4_WST;                // used in rank 0: both CTAs' warps arrive
  uint64_t* a_free = a_ready + R4_GROUPS;
  uint64_t* d_full = a_free + R4_GROUPS;
  uint64_t* d_empty = d_full + 1;                      // used in rank 0: both CTAs' warps arrive
  uint64_t* g_full = d_empty + 1;                      // gated form: a group's first sums are there
  uint64_t* g_empty = g_full + R4_GROUPS;              // and have been taken
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(g_empty + R4_GROUPS);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  R4Share* share = reinterpret_cast<R4Share*>(s_fail + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_w0);
    prefetch_tensormap(&map_w1);
    prefetch_tensormap(&map_x);
    prefetch_tensormap(&map_y);
    for (int i = 0; i < R4_XST; ++i) mbar_init(&x_full[i], 1), mbar_init(&x_empty[i], 1);
    for (int i = 0; i < R4_WST; ++i) mbar_init(&w_full[i], 2), mbar_init(&w_empty[i], 4);
    for (int i = 0; i < R4_GROUPS; ++i) mbar_init(&a_ready[i], 8), mbar_init(&a_free[i], 1), mbar_init(&g_full[i], 2), mbar_init(&g_empty[i], 2);
    mbar_init(d_full, 1);
    mbar_init(d_empty, 2 * 4 * R4_GROUPS);
    *s_fail = 0;
    *share = r4_share(p, blockIdx.x >> 1, gridDim.x >> 1);
    fence_barrier_init();
  }
  if (warp == 1) pair_tmem_alloc(tmem_ptr, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const R4Fail fail{s_fail, cluster_addr(s_fail, (uint32_t)(rank ^ 1)), p.word};
  const int steps = p.steps, bn = p.bn, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int xb = bn * 128, xst = p.xst;                // bytes of a stage of x in a CTA, stages
  pdl_wait();                                          // (what comes before it runs under the kernel before)
  pdl_launch_dependents();

  if (warp == 0 || warp == 2) {
    if (elect_one()) {
      bool ok = true;
      int s = 0;
      uint32_t ph = 1;
      for (int nth = 0; ok; ++nth) {
        const R4Unit u = r4_unit(share, steps, pair, pairs, nth);
        if (u.len == 0) break;
        const int n0 = (u.tile / p.mtiles) * TILE_N, m0 = (u.tile % p.mtiles) * bn + rank * (bn >> 1);
        if (warp == 0) {
          for (int kb = u.k0; kb < u.k0 + u.len; ++kb) {
            if (!(ok = r4_wait(&x_empty[s], ph, fail, 1))) break;
            if (rank == 0) mbar_expect_tx(&x_full[s], 2u * (uint32_t)xb);      // both CTAs' rows
            const uint32_t bar = cluster_addr(&x_full[s], 0);
            pair_box(sx + s * xb, &map_x, kb * R4_K, m0, bar);
            pair_box(sx + s * xb + (xb >> 1), &map_x, kb * R4_K + 64, m0, bar);
            if (++s == xst) s = 0, ph ^= 1u;
          }
        } else {
          const int c0 = n0 + rank * (TILE_N / 2);
          for (int kb = u.k0; kb < u.k0 + u.len; ++kb) {
            if (!(ok = r4_wait(&w_empty[s], ph, fail, 2))) break;
            mbar_expect_tx(&w_full[s], R4_WBYTES);
            r4_box(sw + s * R4_WBYTES, &map_w0, c0, kb * (R4_K / 2), &w_full[s]);
            if (GATED) r4_box(sw + s * R4_WBYTES + R4_WBYTES / 2, &map_w1, c0, kb * (R4_K / 2), &w_full[s]);
            if (++s == R4_WST) s = 0, ph ^= 1u;
          }
        }
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = instr_desc_bf16(256, bn);
      const uint64_t xd = smem_desc_sw128(smem_u32(sx));
      bool ok = true;
      int s = 0, tl = 0;
      uint32_t ph = 0, blk = 0;
      for (; rank == 0 && ok; ++tl) {
        const int len = r4_unit(share, steps, pair, pairs, tl).len;
        if (len == 0) break;
        if (tl > 0 && !(ok = r4_wait(d_empty, (uint32_t)(tl - 1) & 1u, fail, 3))) break;
        for (int kb = 0; ok && kb < len; ++kb, ++blk) {
          const uint32_t buf = blk % R4_GROUPS;
          if (!(ok = r4_spin(&x_full[s], ph, fail, 5) && r4_spin(&a_ready[buf], (blk / R4_GROUPS) & 1u, fail, 4))) break;
          tc_fence_after();
          const uint64_t bd = xd + (uint64_t)(s * (xb >> 4));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            r4_mma(tmem, tmem + TM_A + 64u * buf + 8u * k, bd + (uint64_t)((k >> 2) * (xb >> 5) + 2 * (k & 3)), idesc, (kb | k) != 0 ? 1u : 0u);
          pair_commit(&a_free[buf]);
          pair_commit(&x_empty[s]);
          if (++s == xst) s = 0, ph ^= 1u;
        }
        if (ok) pair_commit(d_full);
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 3) {
    // scales and zeros, four steps ahead of their use at least: the groups of four steps lie side by side.  (Loaded by the unpacking threads one
    // step ahead, 64 lines a warp and no L1 to speak of, they were half of a step's time.)
    bool ok = true;
    int s = 0;
    uint32_t ph = 1;
    auto fetch = [&](int tile, int kb, uint2 (&sv)[4], uint2 (&zv)[4]) {
      const int n0 = (tile / p.mtiles) * TILE_N;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool second = GATED && q >= 2;
        const int n = n0 + (GATED ? rank * 64 + (q & 1) * 32 : rank * 128 + q * 32) + lane;
        const size_t row = (size_t)min(n, p.N - 1) * p.G;
        sv[q] = r4_four(second ? p.scales[1] : p.scales[0], row, kb, steps, p.G, p.steps_per_group, p.wide);
        zv[q] = r4_four(second ? p.zeros[1] : p.zeros[0], row, kb, steps, p.G, p.steps_per_group, p.wide);
      }
    };
    uint2 sv[4], zv[4];
    R4Unit u = r4_unit(share, steps, pair, pairs, 0);
    if (u.len > 0) fetch(u.tile, u.k0 & ~3, sv, zv);
    for (int nth = 1; ok && u.len > 0; ++nth) {
      const R4Unit next = r4_unit(share, steps, pair, pairs, nth);
      const int end = u.k0 + u.len;
      for (int kb = u.k0 & ~3; ok && kb < end; kb += 4) {
        uint2 sn[4], zn[4];
        const bool last = kb + 4 >= end;
        if (!last || next.len > 0) fetch(last ? next.tile : u.tile, last ? next.k0 & ~3 : kb + 4, sn, zn);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (kb + j < u.k0 || kb + j >= end) continue;
          ok = __all_sync(0xffffffffu, r4_wait(&w_empty[s], ph, fail, 11));
          if (!ok) break;
#pragma unroll
          for (int q = 0; q < 4; ++q) reinterpret_cast<uint32_t*>(sz + s * R4_SZ)[q * 32 + lane] = r4_word(j, sv[q], zv[q]);
          __syncwarp();
          if (lane == 0) mbar_arrive(&w_full[s]);
          if (++s == R4_WST) s = 0, ph ^= 1u;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) sv[q] = sn[q], zv[q] = zn[q];
      }
      u = next;
    }
  } else {
    const int quarter = warp & 3, grp = (warp - 4) >> 2, half = quarter >> 1;        // half: the CTA's first or last 64 columns
    const int col = (GATED ? rank * 64 : rank * 128 + half * 64) + (quarter & 1) * 32 + lane;      // within the pair's outputs
    const bool second = GATED && half == 1;             // columns of W2
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const uint32_t a_ready0 = cluster_addr(&a_ready[grp], 0), d_empty0 = cluster_addr(d_empty, 0);
    bool ok = true;
    uint32_t boxes = 0, swaps = 0;
    // a finished unit: its sums leave tensor memory, then the accumulator is given back, then they are stored
    auto drain = [&](uint32_t nth) {
      const R4Unit u = r4_unit(share, steps, pair, pairs, (int)nth);
      ok = __all_sync(0xffffffffu, r4_wait(d_full, nth & 1u, fail, 6));
      if (!ok) return;
      tc_fence_after();
      const int n = (u.tile / p.mtiles) * TILE_N + col, m0 = (u.tile % p.mtiles) * bn;
      const __nv_bfloat16* b = second ? p.bias[1] : p.bias[0];
      const float bias = b != nullptr && n < p.N ? __bfloat162float(b[n]) : 0.f;
      if (u.tile >= p.full) {                // a part of a tile: its sums go to L2 as they are
        float* const dst = p.part + ((size_t)share->part[(int)nth - share->whole] * 2 + rank) * (size_t)(bn * 128) + quarter * 32 + lane;
#pragma unroll 1
        for (int r = grp * 16; r < bn; r += 16 * R4_GROUPS) {
          uint32_t v[16];
          r4_ld16(tmem + lanes + (uint32_t)r, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 16; ++e) asm volatile("" : "+r"(v[e]));
#pragma unroll
          for (int e = 0; e < 16; ++e) __stcg(dst + (r + e) * 128, __uint_as_float(v[e]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(d_empty0);
        return;
      }
      uint32_t w[4][8];
#pragma unroll
      for (int c = 0; c < 4; c += 2) {       // (bn is a multiple of 32 above 64: pairs of chunks, and only the last chunk of a group can be missing)
        if ((grp + 4 * c) * 16 >= bn) break;
        const bool two = (grp + 4 * (c + 1)) * 16 < bn;
        uint32_t v[32];
        r4_ld16(tmem + lanes + (uint32_t)((grp + 4 * c) * 16), v);
        if (two) r4_ld16(tmem + lanes + (uint32_t)((grp + 4 * c + 4) * 16), v + 16);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 16; ++e) asm volatile("" : "+r"(v[e]), "+r"(v[e + 16]));       // (the loads' results are there from here on)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          w[c][e] = pack_bf16(__uint_as_float(v[2 * e]) + bias, __uint_as_float(v[2 * e + 1]) + bias);
          w[c + 1][e] = pack_bf16(__uint_as_float(v[16 + 2 * e]) + bias, __uint_as_float(v[17 + 2 * e]) + bias);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(d_empty0);
      const bool odd = (lane & 1) != 0;
      uint8_t* const out = so + (GATED ? grp * 2 + (quarter & 1) : grp * 4 + quarter) * R4_OUT;
#pragma unroll
      for (int c = 0; c < 4; c += 2) {
        if ((grp + 4 * c) * 16 >= bn) break;
        if (GATED) {
          // (each lane of the second half meets the words of the same column in the first)
          uint32_t* sums = reinterpret_cast<uint32_t*>(swap + grp * R4_SWAP) + (quarter & 1) * 32 + lane;
          if (half == 0) {
            if (swaps > 0) ok = __all_sync(0xffffffffu, r4_wait(&g_empty[grp], (swaps - 1u) & 1u, fail, 9));
            if (!ok) return;
#pragma unroll
            for (int e = 0; e < 16; ++e) {   // (the first half forms the silu, the second the product and the boxes)
              const uint32_t g = w[c + (e >> 3)][e & 7];
              sums[e * 64] = pack_bf16(silu_fast(__uint_as_float(g << 16)), silu_fast(__uint_as_float(g & 0xffff0000u)));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&g_full[grp]);
            ++swaps;
            continue;
          }
          ok = __all_sync(0xffffffffu, r4_wait(&g_full[grp], swaps & 1u, fail, 10));
          if (!ok) return;
          ++swaps;
#pragma unroll
          for (int e = 0; e < 16; ++e) w[c + (e >> 3)][e & 7] = r4_mul2(sums[e * 64], w[c + (e >> 3)][e & 7]);
          __syncwarp();
          if (lane == 0) mbar_arrive(&g_empty[grp]);
        }
        // a lane holds two rows of its column in a word; neighbours swap, so that a lane has two columns of one row; 16 rows x 32 columns go
        // out as one box while the warp is back at its next step (rows past M and columns past N stay out)
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int r0 = m0 + (grp + 4 * (c + d)) * 16, nb = n - lane;
          if (r0 >= m0 + bn) break;
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the box before the last has left
          __syncwarp();
          uint8_t* box = out + (boxes & 1u) * R4_BOX;
          ++boxes;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const uint32_t v = w[c + d][e], got = __shfl_xor_sync(0xffffffffu, v, 1);
            const uint32_t o = odd ? (got >> 16) | (v & 0xffff0000u) : (v & 0xffffu) | (got << 16);
            *reinterpret_cast<uint32_t*>(box + (2 * e + (odd ? 1 : 0)) * 64 + ((((lane >> 3) ^ e) & 3) * 16) + ((lane >> 1) & 3) * 4) = o;
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            if (r0 < p.M && nb < p.N)
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&map_y), "r"(nb), "r"(r0), "r"(smem_u32(box))
                           : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
    };
    // the group's steps: every fourth of all steps of all of the pair's units
    int len = r4_unit(share, steps, pair, pairs, 0).len, kb = grp, s = grp;
    uint32_t unit = 0, drained = 0, round = 0, wph = 0;    // unit: of the group's next step; round: its how-many-th step
    while (len > 0 && kb >= len) kb -= len, len = r4_unit(share, steps, pair, pairs, (int)++unit).len;
    constexpr int WIDTH = GATED ? 64 : 128;
    const R4Row<WIDTH> row(lane);
    while (ok && (len > 0 || drained < unit)) {
      bool step = len > 0;
      const uint32_t upto = unit;            // units before this one can be drained
      if (step) {
        ok = r4_wait(&w_full[s], wph, fail, 7);
        if (ok && round > 0) ok = r4_wait(&a_free[grp], (round - 1u) & 1u, fail, 8);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;
        // a unit that is done already (for the group whose step was its last) is drained before the step, others after it
        step = drained >= upto || !__any_sync(0xffffffffu, mbar_test_wait(d_full, drained & 1u));
      }
      if (step) {
        tc_fence_after();
        r4_unpack_step<WIDTH>(smem_u32(sw + s * R4_WBYTES + (GATED ? half * (R4_WBYTES / 2) : 0)), (uint32_t)((GATED ? quarter & 1 : quarter) * 32), row,
                              smem_u32(sz + s * R4_SZ) + (uint32_t)(quarter * 128), tmem + lanes + TM_A + 64u * grp);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_empty[s]), mbar_arrive_cluster(a_ready0);
        kb += R4_GROUPS;
        while (len > 0 && kb >= len) kb -= len, len = r4_unit(share, steps, pair, pairs, (int)++unit).len;
        ++round;
        if ((s += R4_GROUPS) >= R4_WST) s -= R4_WST, wph ^= 1u;
      }
      while (ok && drained < upto) drain(drained++);
    }
    tc_fence_before();
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  __syncthreads();
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem, 512);
  }
}

// the output, boxes of 16 rows x 32 columns
int r4_out_map(const void* y, int M, int N, CUtensorMap* out) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled entry point not available");
    return LL_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M}, strides[1] = {(cuuint64_t)N * 2};
  cuuint32_t box[2] = {32, 16}, estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)y, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): output M=%d N=%d", (int)r, M, N);
    return LL_ERR_CUDA;
  }
  return LL_OK;
}

// Clocks of a launch with tiles of bn rows: waves of the persistent grid, 128 k at a time, plus the drain.  A step costs its products, or, with
// few rows, its unpacking (us a step of 13824 x 5120, 900 rows, tiles of 128 / 160 / 192 / 224 / 256 rows: .54 / .56 / .61 / .66 / .78, the last with
// six pairs idle in its third wave).
int r4_step(int bn) { return 4 * bn > 530 + 7 * bn / 5 ? 4 * bn : 530 + 7 * bn / 5; }
long long r4_cost(int M, int N, int tile_n, int steps, int bn, int pairs) {
  const long long tiles = (long long)((M + bn - 1) / bn) * ((N + tile_n - 1) / tile_n);
  return (tiles + pairs - 1) / pairs * ((long long)steps * r4_step(bn) + 1500);
}
// The same of `tiles` tiles cut into `parts` along k each: their steps, the launch that adds the parts up (5 us) and their way through L2 (6 MB a us).
// us on the device, every tile whole / by this rule: 4096 x 11008 at 130, 300, 512 rows 48 / 24, 50 / 34, 50 / 43, from 700 on all whole (53; in the
// parts nearest to paying 58); the gated 11008 x 4096 at 130, 300, 512, 700 rows 45 / 37, 63 / 56, 80 / 74, 109 / 106.  Short layers (R4_SHORT) stay
// whole: 2048 x 5632 of 130 rows would take 15 instead of 27, but calls of its size are bound by the host, for which a second launch and its scratch
// are 2 us (228 rows through a feed-forward of width 2048, a call 49 whole, 51 cut).  The rule goes by sizes alone: such a layer stays whole in a captured
// step as well, where no host is in the way.  Ranges of one length for all pairs, that cross tile ends, were
// 2 to 4 us slower (two drains a pair, more parts); the last pair to arrive adding up in the kernel itself made the loop spill (whole tiles a fifth
// slower).
constexpr long long R4_SHORT = 40000;
constexpr int R4_PARTS = 8;
long long r4_parts_cost(int steps, int bn, int tiles, int parts, int pairs) {
  return (long long)((tiles * parts + pairs - 1) / pairs) * ((long long)((steps + parts - 1) / parts) * r4_step(bn) + 1500) + 7000 + tiles * parts * bn / 4;
}

// How the work is laid out: whole tiles in whole waves; those of a last wave that would leave pairs idle are cut along k, if that pays.
struct R4Plan {
  int bn, full, parts;           // (parts 0: every tile whole)
};
R4Plan r4_plan(int M, int N, int steps, int tile_n, int pairs, int tile_rows, int parts, bool scratch) {
  R4Plan best{};
  long long least = 0;
  const int most = tile_rows ? tile_rows : 256, fewest = tile_rows ? tile_rows : 128;
  for (int bn = most; bn >= fewest; bn -= 32) {
    const long long whole = r4_cost(M, N, tile_n, steps, bn, pairs);
    if (best.bn == 0 || whole < least) best = {bn, ((M + bn - 1) / bn) * ((N + tile_n - 1) / tile_n), 0}, least = whole;
  }
  if (!scratch || (parts == 0 && least < R4_SHORT)) return best;
  for (int bn = most; bn >= fewest; bn -= 32) {
    const int tiles = ((M + bn - 1) / bn) * ((N + tile_n - 1) / tile_n), full = tiles / pairs * pairs, rest = tiles - full;
    if (rest == 0) continue;
    const long long before = r4_cost(full / pairs * bn, tile_n, tile_n, steps, bn, 1);
    for (int s = parts > 0 ? parts : 2; s <= (parts > 0 ? parts : R4_PARTS) && s <= steps && rest * s <= 2 * pairs; ++s) {
      const long long cost = before + r4_parts_cost(steps, bn, rest, s, pairs);
      if (parts > 0 || cost < least) best = {bn, full, s}, least = cost;
    }
  }
  return best;
}
int r4_pairs(int grid) {
  const int sms = grid > 0 ? grid : sm_count() > 0 ? sm_count() : 148;
  return sms > 1 ? (grid > 0 ? (sms + 1) / 2 : sms / 2) : 1;
}
int r4_tiles(int M, int N, int tile_n, int bn) { return ((M + bn - 1) / bn) * ((N + tile_n - 1) / tile_n); }
size_t r4_scratch_bytes(const R4Plan& q, int tiles) {
  return (size_t)(tiles - q.full) * q.parts * 2 * q.bn * 128 * sizeof(float);
}

bool r4_form_ok(int tile_rows, int grid) { return (tile_rows == 0 || (tile_rows % 32 == 0 && tile_rows >= 128 && tile_rows <= 256)) && grid >= 0; }

// The tiles that were cut: their parts in the order of k, then what the epilogue of a whole tile does.  A block: four rows of a tile; a thread: four
// columns (of both layers) of a row.
template <bool GATED>
__global__ void __launch_bounds__(GATED ? 128 : 256) int4_rows_sum_kernel(const float* part, const __nv_bfloat16* __restrict__ b0,
                                                                          const __nv_bfloat16* __restrict__ b1, __nv_bfloat16* y, int M, int N, int bn,
                                                                          int mtiles, int full, int parts) {
  pdl_wait();
  pdl_launch_dependents();
  part = after_wait(part);
  constexpr int OUT = GATED ? 64 : 128, L = GATED ? 2 : 1;              // outputs of a CTA of the pair, layers
  const int t = blockIdx.x, tile = full + t, col = (threadIdx.x & (OUT / 4 - 1)) * 4, rank = (threadIdx.x / (OUT / 4)) & 1;
  const int n = tile / mtiles * (2 * OUT) + rank * OUT + col, r = blockIdx.y * 4 + threadIdx.x / (OUT / 2), m = tile % mtiles * bn + r;
  if (n >= N || m >= M) return;
  const size_t size = (size_t)bn * 256;
  const float* src = part + (size_t)t * parts * size + ((size_t)rank * bn + r) * 128 + col;
  float4 s[L];
#pragma unroll
  for (int h = 0; h < L; ++h) s[h] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int c = 0; c < parts; c += 4) {
    float4 v[L][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < L; ++h) v[h][i] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)min(c + i, parts - 1) * size + h * 64));
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < L; ++h)
        if (c + i < parts) s[h].x += v[h][i].x, s[h].y += v[h][i].y, s[h].z += v[h][i].z, s[h].w += v[h][i].w;
  }
  uint32_t w[L][2];
#pragma unroll
  for (int h = 0; h < L; ++h) {
    const __nv_bfloat16* b = h ? b1 : b0;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (b != nullptr) a = make_float4(__bfloat162float(b[n]), __bfloat162float(b[n + 1]), __bfloat162float(b[n + 2]), __bfloat162float(b[n + 3]));
    w[h][0] = pack_bf16(s[h].x + a.x, s[h].y + a.y), w[h][1] = pack_bf16(s[h].z + a.z, s[h].w + a.w);
  }
  if (GATED) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
      w[0][e] = r4_mul2(pack_bf16(silu_fast(__uint_as_float(w[0][e] << 16)), silu_fast(__uint_as_float(w[0][e] & 0xffff0000u))), w[L - 1][e]);
  }
  *reinterpret_cast<uint2*>(y + (size_t)m * N + n) = make_uint2(w[0][0], w[0][1]);
}

template <bool GATED>
int r4_launch(const uint8_t* qw0, const uint8_t* qw1, const void* x, R4Params p, int K, void* scratch, size_t scratch_bytes, int tile_rows, int grid,
              int parts, cudaStream_t st) {
  constexpr int TILE_N = GATED ? 128 : 256;
  const int pairs = r4_pairs(grid);
  LL_CHECK_ARG((long long)((p.M + 127) / 128) * ((p.N + TILE_N - 1) / TILE_N) < (1ll << 30), "int4_rows: too many tiles");
  const R4Plan q = r4_plan(p.M, p.N, p.steps, TILE_N, pairs, tile_rows, parts, scratch != nullptr);
  p.bn = q.bn, p.full = q.full, p.parts = q.parts;
  p.mtiles = (p.M + p.bn - 1) / p.bn;
  p.tiles = r4_tiles(p.M, p.N, TILE_N, p.bn);
  LL_CHECK_ARG(scratch == nullptr || scratch_bytes >= r4_scratch_bytes(q, p.tiles), "int4_rows: scratch of %zu bytes, %zu are needed", scratch_bytes,
               r4_scratch_bytes(q, p.tiles));
  p.xst = R4_XBYTES / (p.bn * 128);
  p.wide = r4_wide(p.scales[0], p.zeros[0], p.scales[1], p.zeros[1], p.G, p.steps_per_group);
  CUtensorMap mw0, mw1, mx, my;
  if (int r = r4_weight_map(qw0, p.N, K, GATED ? 64 : 128, &mw0)) return r;
  if (int r = r4_weight_map(qw1, p.N, K, GATED ? 64 : 128, &mw1)) return r;
  if (int r = make_map(x, p.M, K, p.bn / 2, &mx)) return r;
  if (int r = r4_out_map(p.y, p.M, p.N, &my)) return r;
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(int4_rows_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, R4_SMEM));
    configured.mark();
  }
  p.word = wait_word();
  int blocks = p.tiles < pairs ? p.tiles : pairs;
  const int cut = p.tiles - q.full;
  if (cut > 0) p.part = (float*)scratch, blocks = q.full > 0 || cut * q.parts > pairs ? pairs : cut * q.parts;
  LL_CUDA(launch(int4_rows_kernel<GATED>, dim3(2 * blocks), dim3(R4_THREADS), R4_SMEM, st, true, mw0, mw1, mx, my, p));
  LL_LAUNCH_OK("int4_rows_kernel");
  if (cut > 0) {
    LL_CUDA(launch(int4_rows_sum_kernel<GATED>, dim3(cut, p.bn / 4), dim3(GATED ? 128 : 256), 0, st, true, (const float*)p.part, p.bias[0], p.bias[1], p.y,
                   p.M, p.N, p.bn, p.mtiles, p.full, p.parts));
    LL_LAUNCH_OK("int4_rows_sum_kernel");
  }
  return LL_OK;
}

}  // namespace
}  // namespace llb

using namespace llb;

extern "C" {

int ll_int4_rows_supported(int N, int K, int group) { return N > 0 && N % 16 == 0 && group > 0 && K > 0 && K % group == 0 && group % R4_K == 0; }

int ll_int4_rows(const uint8_t* qw, const void* scales, const void* zeros, const void* x, const void* bias, void* y, int M, int N, int K, int group,
                 ll_stream stream) {
  return ll_int4_rows_form(qw, scales, zeros, x, bias, y, M, N, K, group, 0, 0, stream);
}

int ll_int4_rows_form(const uint8_t* qw, const void* scales, const void* zeros, const void* x, const void* bias, void* y, int M, int N, int K,
                      int group, int tile_rows, int grid, ll_stream stream) {
  return ll_int4_rows_split(qw, scales, zeros, x, bias, y, nullptr, M, N, K, group, tile_rows, grid, 0, stream);
}

size_t ll_int4_rows_scratch_bytes(int M, int N, int K, int layers, int tile_rows, int grid, int parts) {
  if (M < 1 || N < 1 || K < R4_K || layers < 1 || layers > 2 || grid < 0 || parts < 0 || !r4_form_ok(tile_rows, grid)) return 0;
  const int tile_n = layers == 2 ? 128 : 256;
  if ((long long)((M + 127) / 128) * ((N + tile_n - 1) / tile_n) >= (1ll << 30)) return 0;
  const R4Plan q = r4_plan(M, N, K / R4_K, tile_n, r4_pairs(grid), tile_rows, parts, true);
  return r4_scratch_bytes(q, r4_tiles(M, N, tile_n, q.bn));
}

int ll_int4_rows_split(const uint8_t* qw, const void* scales, const void* zeros, const void* x, const void* bias, void* y, void* scratch, int M, int N,
                       int K, int group, int tile_rows, int grid, int parts, ll_stream stream) {
  return ll_int4_rows_sized(qw, scales, zeros, x, bias, y, scratch, SIZE_MAX, M, N, K, group, tile_rows, grid, parts, stream);
}

int ll_int4_rows_sized(const uint8_t* qw, const void* scales, const void* zeros, const void* x, const void* bias, void* y, void* scratch,
                       size_t scratch_bytes, int M, int N, int K, int group, int tile_rows, int grid, int parts, ll_stream stream) {
  LL_CHECK_ARG(qw && scales && zeros && x && y && M > 0, "int4_rows: null pointer or no rows");
  if (!ll_int4_rows_supported(N, K, group)) {
    set_error("int4_rows needs N %% 16 == 0 and group %% 128 == 0 (N=%d K=%d group=%d)", N, K, group);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG((((uintptr_t)qw | (uintptr_t)x | (uintptr_t)y | (uintptr_t)scratch) & 15) == 0,
               "int4_rows: packed weights, x, y and scratch must be 16-byte aligned");
  LL_CHECK_ARG(r4_form_ok(tile_rows, grid) && parts >= 0, "int4_rows: tiles of 128 to 256 rows, a multiple of 32");
  R4Params p{};
  p.scales[0] = p.scales[1] = (const __nv_bfloat16*)scales, p.zeros[0] = p.zeros[1] = (const __nv_bfloat16*)zeros;
  p.bias[0] = p.bias[1] = (const __nv_bfloat16*)bias, p.y = (__nv_bfloat16*)y;
  p.M = M, p.N = N, p.steps = K / R4_K, p.G = K / group, p.steps_per_group = group / R4_K;
  return r4_launch<false>(qw, qw, x, p, K, scratch, scratch_bytes, tile_rows, grid, parts, (cudaStream_t)stream);
}

int ll_int4_rows_gated(const uint8_t* qw1, const void* scales1, const void* zeros1, const void* bias1, const uint8_t* qw2, const void* scales2,
                       const void* zeros2, const void* bias2, const void* x, void* h, int M, int N, int K, int group, int tile_rows, int grid,
                       ll_stream stream) {
  return ll_int4_rows_gated_split(qw1, scales1, zeros1, bias1, qw2, scales2, zeros2, bias2, x, h, nullptr, M, N, K, group, tile_rows, grid, 0, stream);
}

int ll_int4_rows_gated_split(const uint8_t* qw1, const void* scales1, const void* zeros1, const void* bias1, const uint8_t* qw2, const void* scales2,
                             const void* zeros2, const void* bias2, const void* x, void* h, void* scratch, int M, int N, int K, int group,
                             int tile_rows, int grid, int parts, ll_stream stream) {
  return ll_int4_rows_gated_sized(qw1, scales1, zeros1, bias1, qw2, scales2, zeros2, bias2, x, h, scratch, SIZE_MAX, M, N, K, group, tile_rows, grid, parts,
                                  stream);
}

int ll_int4_rows_gated_sized(const uint8_t* qw1, const void* scales1, const void* zeros1, const void* bias1, const uint8_t* qw2, const void* scales2,
                             const void* zeros2, const void* bias2, const void* x, void* h, void* scratch, size_t scratch_bytes, int M, int N, int K,
                             int group, int tile_rows, int grid, int parts, ll_stream stream) {
  LL_CHECK_ARG(qw1 && scales1 && zeros1 && qw2 && scales2 && zeros2 && x && h && M > 0, "int4_rows_gated: null pointer or no rows");
  if (!ll_int4_rows_supported(N, K, group)) {
    set_error("int4_rows_gated needs N %% 16 == 0 and group %% 128 == 0 (N=%d K=%d group=%d)", N, K, group);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG((((uintptr_t)qw1 | (uintptr_t)qw2 | (uintptr_t)x | (uintptr_t)h | (uintptr_t)scratch) & 15) == 0,
               "int4_rows_gated: packed weights, x, h and scratch must be 16-byte aligned");
  LL_CHECK_ARG(r4_form_ok(tile_rows, grid) && parts >= 0, "int4_rows_gated: tiles of 128 to 256 rows, a multiple of 32");
  R4Params p{};
  p.scales[0] = (const __nv_bfloat16*)scales1, p.zeros[0] = (const __nv_bfloat16*)zeros1, p.bias[0] = (const __nv_bfloat16*)bias1;
  p.scales[1] = (const __nv_bfloat16*)scales2, p.zeros[1] = (const __nv_bfloat16*)zeros2, p.bias[1] = (const __nv_bfloat16*)bias2;
  p.y = (__nv_bfloat16*)h;
  p.M = M, p.N = N, p.steps = K / R4_K, p.G = K / group, p.steps_per_group = group / R4_K;
  return r4_launch<true>(qw1, qw2, x, p, K, scratch, scratch_bytes, tile_rows, grid, parts, (cudaStream_t)stream);
}

// 0, or the code of the first bounded wait that ran out in this file's kernel.  Synchronises the device.
int ll_int4_rows_error(void) {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, g_r4_error, sizeof(int)) == cudaSuccess ? v : -1;
}

}  // extern "C"
