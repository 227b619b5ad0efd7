// Softmax attention of prompts on tcgen05: S = Q K^T and O += P V with fp32 accumulators in tensor memory.
//
// A block owns two tiles of 128 queries of one head, or one (neighbours, one from each end, alone: at_tiles) and walks the keys they can see 64 at a time:
//   warps 0-7, 8-15 : softmax of tile 0 / tile 1; two threads share a query row, each 32 of its 64 scores: they read them from tensor
//                     memory, scale, cap, mask, exponentiate, write the weights back over their own scores as packed bf16 (one term, or
//                     two: hi and what hi left over) and keep the row's sum; at the end they normalise and store the row
//   warp 16         : TMA producer (queries once, then key and value blocks into rings)
//   warps 17, 18    : one thread each issues the MMAs of a tile: the scores of the next key block first, then P V of this one
//   warp 19         : clears value rows that belong to no key
// Scores have two buffers per tile, so that the tensor cores form the next block's scores while a block's weights are made; the
// weights lie where the scores were (MMAs of one thread run in issue order).  The running maximum only moves when a row's scores
// outgrow it by 2^8: the accumulator is then rescaled in place, which after the first blocks of a row hardly ever happens; the
// result does not depend on it.  Capped scores have a bound of their own: where it is at most 2^80 they need no maximum, and the two threads
// of a row nothing from one another before the end.  Weights are then up to 2^c (c = cap * log2(e)) and not 2^8, which the fp32 sums hold while values are
// below 2^(127 - c) / keys and (what is not lost) above 2^(c - 118): with a cap of 50 and 2048 keys 2^44 and 2^-46, with the largest of 55 2^36 and 2^-38.
// Keys are addressed by position in a ring (slot = position % ring): a block of keys ends where the ring wraps.  Rows past the
// last key of the step may hold anything: their scores are masked and their value rows are cleared in shared memory.
//
// What bounds it is the softmax: a row's chain (load, maximum, exponent, split, store) runs at one instruction in four clocks
// for a warp on its own, so a row has two threads and a scheduler four such warps.  2048 queries, 16 heads of 128, two terms, us: 46 (capped at 50 64, at 80
// 65) with neighbouring tiles, one barrier of a tile's 256 threads a block of keys and a running maximum for all capped scores; 37 (40, 47) now.  Bounded and
// other capped scores are two kernels: one for both was a tenth slower for either.
// Counters, uncapped and capped at 50: issue slots 47 and 45 % while a block runs, ALUs 37 and 33, exponential unit 30 and 28, tensor pipe 31 and 29 % of the
// time; the SM with the longest blocks is busy 1.27 times as long as the average one.
// Blocks of 128 keys with one buffer of scores a tile (no second one fits beside the accumulators): 53 and 60, a tile's chain of weights,
// P V and the next scores being what it waits for.
// Every wait is bounded; one that runs out records a code, all roles stop, copies in flight are waited for, tensor memory is freed.
#pragma once
#include <climits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace llb {
namespace {

// One operand of the scores or of the weighted sum: rows of `dim` bf16 numbers, head `h`, row `r`, sequence `b` at
// base + h * head + r * row + b * batch (strides in numbers; rows and heads on 16-byte boundaries).
struct AttnTcOperand {
  const void* base;
  int dim;
  long long head, row, batch;
};

struct AttnTcArgs {
  AttnTcOperand q, q2;         // queries; q2 / k2: a second part of every head's dimensions (base null: none), up to 64 of them
  AttnTcOperand k, k2, v;      // key and value rows by slot; k2 has one head that all share
  const int32_t* pos_ids;      // [T]
  const float* sink;           // [H] or null
  const float* slopes;         // [H] or null: scores fall by slope * (i - j)
  const void* gate;            // bf16 [B * T] rows or null; element-wise, or (gate_per_head) one number per head
  int gate_ld, gate_per_head;
  float scale, softcap;
  int B, T, H, G, window, chunk, ring;
  int terms;                   // bf16 terms of a softmax weight: 1 or 2
  void* y;                     // bf16 [B * T] rows, head h at column h * v.dim
  int y_ld;
};

constexpr int AT_Q = 128, AT_K = 64, AT_C = AT_K / 2, AT_WARPS = 16, AT_THREADS = (AT_WARPS + 4) * 32;
constexpr int AT_QBOX = AT_Q * 64 * 2, AT_KBOX = AT_K * 64 * 2;      // TMA boxes: rows of 64 bf16
constexpr uint32_t AT_WAIT_LIMIT = 1u << 20;
constexpr float AT_LOG2E = 1.4426950408889634f;
constexpr float AT_SLACK = 8.f;                       // a row's scores may outgrow its reference by 2^8 before it moves
constexpr float AT_BOUND = 80.f;                      // scores that a cap keeps within 2^-80 .. 2^80 need no reference (what that leaves to values: above)

__device__ int g_attn_tc_error = 0;     // per file that instantiates the kernel: its entry asks for it (attn_tc_error)

enum AtTiles { AT_NEIGHBOURS, AT_APART, AT_ALONE };     // two next to one another, one from the end and one from the start, one
struct AtParams {
  const int32_t* pos_ids;
  const float* sink;
  const float* slopes;
  const __nv_bfloat16* gate;
  __nv_bfloat16* y;
  float scale, softcap;
  int T, H, group, vdim, window, chunk, ring, gate_ld, gate_per_head, gate_vec, y_ld;
  int tiles;                   // a block's tiles: AtTiles
  int* word;                   // wait_word()
};

__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// value block [blocks of 64 dimensions][64 keys][64]: N runs along a row (MN-major), 128-byte swizzle; LBO = distance of the
// 64-dimension blocks, SBO = distance of groups of eight keys
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3fff);
  d |= (uint64_t)(AT_KBOX >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// the registers of an asynchronous load are what they should be only after the wait: uses stay behind this
__device__ __forceinline__ void tie32(uint32_t* v) {
  asm volatile(""
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                 "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]),
                 "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]),
                 "+r"(v[28]), "+r"(v[29]));
  asm volatile("" : "+r"(v[30]), "+r"(v[31]));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float at_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float at_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// 1 / (1 + e^-x), relative error about 1e-6: the products it enters are rounded to bf16
__device__ __forceinline__ float at_sigmoid(float x) { return at_rcp(1.f + at_exp2(-AT_LOG2E * x)); }
__device__ __forceinline__ uint4 at_load8(const __nv_bfloat16* p, int vec) {
  if (vec) return *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void tma_box4(void* dst, const CUtensorMap* map, int x, int h, int row, int b, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(h), "r"(row), "r"(b), "r"(smem_u32(bar))
      : "memory");
}

// Two fp32 operations per instruction (sm_100): multiply-add, add and multiply of pairs.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_of(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_split(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// A wait that ends: on its phase, when another role has given up, or after the limit.
__device__ __forceinline__ bool at_wait(uint64_t* bar, uint32_t parity, volatile int* fail, int* word, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  for (uint32_t i = 0; i < AT_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  atomicCAS(&g_attn_tc_error, 0, code);
  wait_ran_out(word, 100 + code);
  return false;
}

// Barrier `id` of the 64 threads that share 32 rows; whether any of them says yes.
__device__ __forceinline__ bool at_any(int id, bool yes) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, 64, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"((uint32_t)yes)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ float at_max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

__device__ __forceinline__ int at_first_visible(int i, int window, int chunk) {
  int lo = 0;
  if (window > 0) lo = max(lo, i - window + 1);
  if (chunk > 0) lo = max(lo, (i / chunk) * chunk);
  return lo;
}

// The key block that starts at position kt, slot kt % ring: up to 64 rows, ending at the last key and where the ring wraps.
struct AtBlock {
  int kt, slot, rows, last, ring;
  __device__ __forceinline__ AtBlock(int first, int last_, int ring_) : kt(first), slot(first % ring_), last(last_), ring(ring_) { size(); }
  __device__ __forceinline__ void size() { rows = min(min(AT_K, last - kt + 1), ring - slot); }
  __device__ __forceinline__ bool any() const { return kt <= last; }
  __device__ __forceinline__ bool meets(int lo, int hi) const { return kt + rows - 1 >= lo && kt <= hi; }
  __device__ __forceinline__ void next() {      // (no division: this stands in every role's loop)
    kt += rows;
    slot += rows;
    if (slot == ring) slot = 0;
    size();
  }
};

// tanh(x) = 1 - 2 / (1 + e^(2x)); for |x| < 1/4 as x P(x^2), P the parabola through tanh(sqrt(u)) / sqrt(u) at the three Chebyshev
// points of [0, 1/16] (largest relative error 4e-7, as the exponential form's), which leaves the exponential unit to the softmax
constexpr float AT_T0 = 0.999999603463f, AT_T1 = -0.33321896989f, AT_T2 = 0.128414339271f;
constexpr float AT_TANH_SMALL = 0.25f;

// NB1 / NB2: blocks of 64 dimensions of the two parts of a key row; NBV: of a value row.  KS / VS: stages of key / value blocks.
template <int NB1, int NB2, int NBV>
struct AtShape {
  static constexpr int NB = NB1 + NB2, KS = NB > 2 ? 3 : 4, VS = NB > 2 ? 3 : 4;
  static constexpr int SMEM = 2 * NB * AT_QBOX + KS * NB * AT_KBOX + VS * NBV * AT_KBOX + 512 + 4 * AT_Q * 4 + 1024;
};

// TERMS: bf16 terms of a weight.  CAP: scores are capped, and the cap bounds their weights (AT_BOUNDED) or does not; BIAS: distance bias.
enum AtCap { AT_UNCAPPED, AT_BOUNDED, AT_CAPPED };
template <int NB1, int NB2, int NBV, int TERMS, AtCap CAP, bool BIAS>
__global__ void __launch_bounds__(AT_THREADS, 1) attn_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_q2,
                                                               const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_k2,
                                                               const __grid_constant__ CUtensorMap map_v, const AtParams p) {
  using Shape = AtShape<NB1, NB2, NBV>;
  constexpr int NB = Shape::NB, KS = Shape::KS, VS = Shape::VS, DV = NBV * 64;
  constexpr uint32_t TM_S = 0, TM_O = 256;            // per tile: two score buffers of 64 columns; 128 accumulator columns
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* sq = base;                                 // [2 tiles][NB][128][64]
  uint8_t* sk = sq + 2 * NB * AT_QBOX;                // [KS][NB][64][64]
  uint8_t* sv = sk + KS * NB * AT_KBOX;               // [VS][NBV][64][64]
  uint64_t* q_full = reinterpret_cast<uint64_t*>(sv + VS * NBV * AT_KBOX);
  uint64_t* k_full = q_full + 1;
  uint64_t* k_empty = k_full + KS;
  uint64_t* v_full = k_empty + KS;
  uint64_t* v_empty = v_full + VS;
  uint64_t* s_full = v_empty + VS;                    // [tile][buffer] scores are there
  uint64_t* p_full = s_full + 4;                      // [tile][buffer] weights are there
  uint64_t* o_full = p_full + 4;                      // [tile][buffer] P V is done
  uint64_t* v_clear = o_full + 4;                     // [VS] value rows of no key are zero: at most two blocks of a walk have such
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(v_clear + VS);  // rows (the last one, and one that the wrap cut off before it)
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  int* s_range = s_fail + 1;                          // per tile: smallest and largest position
  float* s_x = reinterpret_cast<float*>(s_range + 4); // [tile][half][row]: what the two threads of a row tell one another

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // neighbours: the last queries see the most keys, so they go first, and the long blocks do not end up as the tail
  const int q_tiles = (p.T + AT_Q - 1) / AT_Q, pair = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int tile0 = p.tiles != AT_NEIGHBOURS ? q_tiles - 1 - (int)blockIdx.x : 2 * pair;
  const int tile1 = p.tiles == AT_ALONE ? tile0 : p.tiles == AT_APART ? (int)blockIdx.x : 2 * pair + 1;
  const int tq0 = tile0 * AT_Q, tq1 = tile1 != tile0 ? tile1 * AT_Q : p.T;      // (the middle one of an odd number stands alone)
  const int h = blockIdx.y, b = blockIdx.z, g = h / p.group;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    mbar_init(q_full, 1);
    for (int i = 0; i < KS; ++i) mbar_init(&k_full[i], 1), mbar_init(&k_empty[i], 2);
    for (int i = 0; i < VS; ++i) mbar_init(&v_full[i], 1), mbar_init(&v_empty[i], 3), mbar_init(&v_clear[i], 1);
    for (int i = 0; i < 4; ++i) mbar_init(&s_full[i], 1), mbar_init(&p_full[i], AT_WARPS / 2), mbar_init(&o_full[i], 1);
    for (int i = 0; i < 2; ++i) {
      s_range[2 * i] = INT_MAX;
      s_range[2 * i + 1] = -1;
    }
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == AT_WARPS + 1) tmem_alloc(tmem_ptr, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  // (Not before the block has its tensor memory: a kernel let in that fits beside it could take that first, and then waits for this one's end.)
  pdl_launch_dependents();
  if (warp == AT_WARPS && elect_one()) {                // the queries do not depend on the positions
    const int tiles = tq1 < p.T ? 2 : 1;
    mbar_expect_tx(q_full, (uint32_t)(tiles * NB * AT_QBOX));
    for (int i = 0; i < tiles; ++i) {
      for (int c = 0; c < NB1; ++c) tma_box4(sq + (i * NB + c) * AT_QBOX, &map_q, c * 64, h, i ? tq1 : tq0, b, q_full);
      for (int c = 0; c < NB2; ++c) tma_box4(sq + (i * NB + NB1 + c) * AT_QBOX, &map_q2, c * 64, h, i ? tq1 : tq0, b, q_full);
    }
  }
  __syncwarp();
  // positions of the tiles' queries
  const int tile = warp >> 3, half = (warp >> 2) & 1, row = (int)(threadIdx.x & (AT_Q - 1)), t = (tile ? tq1 : tq0) + row;
  int qp = 0;
  if (warp < AT_WARPS) {
    if (t < p.T) qp = p.pos_ids[t];
    const int lo = __reduce_min_sync(0xffffffffu, t < p.T ? qp : INT_MAX), hi = __reduce_max_sync(0xffffffffu, t < p.T ? qp : -1);
    if (lane == 0) atomicMin(&s_range[2 * tile], lo), atomicMax(&s_range[2 * tile + 1], hi);
  }
  __syncthreads();
  // what every role walks: key blocks from kt0 to the last visible key; per tile the part of it that its rows see
  int lo[2], hi[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int first = __shfl_sync(0xffffffffu, s_range[2 * i], 0), end = __shfl_sync(0xffffffffu, s_range[2 * i + 1], 0);
    lo[i] = end >= 0 ? at_first_visible(first, p.window, p.chunk) : INT_MAX;
    hi[i] = end;
  }
  const int kt0 = min(lo[0], lo[1]), last = max(hi[0], hi[1]);
  // rows after this key hold nothing of this step, or (positions that do not rise) nothing that a row of this block sees: a block of keys
  // starts at or before it
  const int step_last = max(__shfl_sync(0xffffffffu, p.pos_ids[p.T - 1], 0), last);

  if (warp == AT_WARPS) {
    // ===================== TMA producer =====================
    if (elect_one()) {
      int n = 0;
      bool ok = true;
      for (AtBlock blk(kt0, last, p.ring); blk.any(); blk.next(), ++n) {
        const int ks = n % KS, vs = n % VS;
        if (!(ok = at_wait(&k_empty[ks], ((n / KS) & 1) ^ 1, s_fail, p.word, 1))) break;
        mbar_expect_tx(&k_full[ks], (uint32_t)(NB * AT_KBOX));
        for (int c = 0; c < NB1; ++c) tma_box4(sk + (ks * NB + c) * AT_KBOX, &map_k, c * 64, g, blk.slot, b, &k_full[ks]);
        for (int c = 0; c < NB2; ++c) tma_box4(sk + (ks * NB + NB1 + c) * AT_KBOX, &map_k2, c * 64, 0, blk.slot, b, &k_full[ks]);
        if (!(ok = at_wait(&v_empty[vs], ((n / VS) & 1) ^ 1, s_fail, p.word, 2))) break;
        mbar_expect_tx(&v_full[vs], (uint32_t)(NBV * AT_KBOX));
        for (int c = 0; c < NBV; ++c) tma_box4(sv + (vs * NBV + c) * AT_KBOX, &map_v, c * 64, g, blk.slot, b, &v_full[vs]);
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == AT_WARPS + 1 || warp == AT_WARPS + 2) {
    // ===================== MMA issuers, one thread per tile =====================
    // (one branch of one elected thread around the whole role: an MMA then takes its thread 40 clocks to issue, and 75 from branches
    // inside the loop or from `lane == 0`, which is more than the 50 to 64 clocks it runs)
    if (elect_one()) {
      constexpr uint32_t idesc_s = instr_desc_bf16(AT_Q, AT_K);
      constexpr uint32_t idesc_o = instr_desc_bf16(AT_Q, DV) | (1u << 16);      // V is MN-major
      const int i = warp - AT_WARPS - 1;
      const int mylo = i == 0 ? lo[0] : lo[1], myhi = i == 0 ? hi[0] : hi[1];
      const uint32_t tm_s = tmem + TM_S + 128u * i, tm_o = tmem + TM_O + 128u * i;
      const uint64_t qdesc = smem_desc_sw128(smem_u32(sq + i * NB * AT_QBOX));
      const uint64_t kdesc0 = smem_desc_sw128(smem_u32(sk)), vdesc0 = smem_desc_mn_sw128(smem_u32(sv));
      uint32_t ns = 0u, np = 0u;      // key blocks whose scores / weighted sum the tile has been given
      // S = Q K^T of the n-th key block: the tile's score buffer is free, its weights two blocks back are in use by an MMA issued before
      auto scores = [&](int n, const AtBlock& blk) {
        const int ks = n % KS;
        if (!at_wait(&k_full[ks], (n / KS) & 1, s_fail, p.word, 4)) return false;
        tc_fence_after();
        if (blk.meets(mylo, myhi)) {
          const uint32_t d = tm_s + 64u * (ns & 1u);
          const uint64_t kdesc = kdesc0 + (uint64_t)(ks * NB * (AT_KBOX >> 4));
#pragma unroll
          for (int c = 0; c < NB; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_bf16(d, qdesc + (uint64_t)(c * (AT_QBOX >> 4) + 2 * k), kdesc + (uint64_t)(c * (AT_KBOX >> 4) + 2 * k), idesc_s,
                        (c | k) != 0 ? 1u : 0u);
          umma_commit(&s_full[2 * i + (int)(ns & 1u)]);
          umma_commit(&k_empty[ks]);
          ++ns;
        } else {
          mbar_arrive(&k_empty[ks]);
        }
        return true;
      };
      bool ok = at_wait(q_full, 0, s_fail, p.word, 3);
      AtBlock blk(kt0, last, p.ring), nxt = blk;
      if (ok) ok = scores(0, blk);
      for (int n = 0; ok && blk.any(); blk = nxt, ++n) {
        nxt.next();
        if (nxt.any() && !(ok = scores(n + 1, nxt))) break;
        const int vs = n % VS;
        if (!(ok = at_wait(&v_full[vs], (n / VS) & 1, s_fail, p.word, 5))) break;
        if (step_last - blk.kt + 1 < AT_K && !(ok = at_wait(&v_clear[vs], 0, s_fail, p.word, 10))) break;
        if (blk.meets(mylo, myhi)) {
          const uint32_t buf = np & 1u;
          if (!(ok = at_wait(&p_full[2 * i + (int)buf], (np >> 1) & 1u, s_fail, p.word, 6))) break;
          tc_fence_after();
          const uint64_t vdesc = vdesc0 + (uint64_t)(vs * NBV * (AT_KBOX >> 4));
#pragma unroll
          for (int term = 0; term < TERMS; ++term)
#pragma unroll
            for (int k = 0; k < AT_K / UMMA_K; ++k)            // 16 keys: 8 columns of packed weights, two groups of eight rows
              umma_ts(tm_o, tm_s + 64u * buf + 32u * (k >> 1) + 16u * term + 8u * (k & 1), vdesc + (uint64_t)(128 * k), idesc_o,
                      (np != 0u || (term | k) != 0) ? 1u : 0u);
          umma_commit(&o_full[2 * i + (int)buf]);
          umma_commit(&v_empty[vs]);
          ++np;
        } else {
          mbar_arrive(&v_empty[vs]);
        }
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == AT_WARPS + 3) {
    // ===================== value rows of no key =====================
    // a block that reaches past the step's last key holds rows that may hold anything: their weights are 0, and 0 * NaN is not
    int n = 0;
    bool ok = true;
    for (AtBlock blk(kt0, last, p.ring); ok && blk.any(); blk.next(), ++n) {
      const int keep = step_last - blk.kt + 1, vs = n % VS;
      ok = __all_sync(0xffffffffu, at_wait(&v_full[vs], (n / VS) & 1, s_fail, p.word, 11));
      if (ok && keep < AT_K) {
        const int pieces = (AT_K - keep) * 8;
        for (int e = lane; e < pieces * NBV; e += 32) {
          const int c = e / pieces, r = e - c * pieces;
          *reinterpret_cast<uint4*>(sv + (vs * NBV + c) * AT_KBOX + keep * 128 + r * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&v_clear[vs]);
      }
      if (lane == 0) mbar_arrive(&v_empty[vs]);      // (every block: a wait may not fall two phases behind)
    }
  } else {
    // ===================== softmax, then the epilogue =====================
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t ts0 = tmem + lanes + TM_S + 128u * tile, to = tmem + lanes + TM_O + 128u * tile;
    const int mylo = tile == 0 ? lo[0] : lo[1], myhi = tile == 0 ? hi[0] : hi[1];
    const int qlo = at_first_visible(qp, p.window, p.chunk);
    const float cap2 = CAP ? p.softcap * AT_LOG2E : 0.f;
    // what a raw score is multiplied by: to the argument of tanh, or to units of log2 (a biased score has been brought there)
    const float mul = BIAS ? 1.f : CAP ? p.scale / p.softcap : p.scale * AT_LOG2E;
    const float bias_unit = CAP ? 1.f / p.softcap : AT_LOG2E;
    const float slope = BIAS ? p.slopes[h] * bias_unit : 0.f;
    float* const mine = s_x + (tile * 2 + half) * AT_Q + row;
    const float* const other = s_x + (tile * 2 + (half ^ 1)) * AT_Q + row;
    const int bar = 1 + tile * 4 + (warp & 3);
    constexpr bool bounded = CAP == AT_BOUNDED;
    float ref = bounded ? 0.f : -INFINITY;
    f2 sum2[2] = {f2_of(0.f, 0.f), f2_of(0.f, 0.f)};
    uint32_t n = 0;
    bool ok = true;
    for (AtBlock blk(kt0, last, p.ring); ok && blk.any(); blk.next()) {
      if (blk.meets(mylo, myhi)) {
        const uint32_t ts = ts0 + 64u * (n & 1u);
        ok = at_wait(&s_full[2 * tile + (int)(n & 1u)], (n >> 1) & 1u, s_fail, p.word, 7);
        __syncwarp();
        tc_fence_after();
        uint32_t sr[AT_C];
        tmem_ld32_async(ts + (uint32_t)(AT_C * half), sr);
        tmem_wait_ld();
        tie32(sr);
        const int c0 = blk.kt + AT_C * half;                                    // position of the thread's first column
        if (BIAS) {
          const float d0 = (float)(c0 - qp), k = p.scale * bias_unit;
#pragma unroll
          for (int e = 0; e < AT_C; ++e) sr[e] = __float_as_uint(fmaf(slope, d0 + (float)e, __uint_as_float(sr[e]) * k));
        }
        const int cmin = qlo - c0, cmax = min(blk.rows - 1 - AT_C * half, qp - c0);          // visible columns of this row
        const bool masked = __any_sync(0xffffffffu, cmin > 0 || cmax < AT_C - 1);
        if (masked) {
#pragma unroll
          for (int e = 0; e < AT_C; ++e)
            if (e < cmin || e > cmax) sr[e] = bounded ? 0u : __float_as_uint(-INFINITY);
        }
        float mx = 0.f;
        bool poly = bounded;
        if (!bounded) {
          float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int e = 0; e < AT_C; e += 2) m4[(e >> 1) & 3] = at_max3(m4[(e >> 1) & 3], __uint_as_float(sr[e]), __uint_as_float(sr[e + 1]));
          mx = at_max3(m4[0], m4[1], fmaxf(m4[2], m4[3]));
          if (CAP && !masked) {
            float a4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < AT_C; e += 2)
              a4[(e >> 1) & 3] = at_max3(a4[(e >> 1) & 3], fabsf(__uint_as_float(sr[e])), fabsf(__uint_as_float(sr[e + 1])));
            poly = __all_sync(0xffffffffu, at_max3(a4[0], a4[1], fmaxf(a4[2], a4[3])) * mul < AT_TANH_SMALL);
          }
          if (mx != -INFINITY) {                                              // the row's largest score in units of log2
            mx *= mul;
            if (CAP) mx = cap2 * (1.f - 2.f * at_rcp(1.f + at_exp2(mx * (2.f * AT_LOG2E))));
          }
        }
        __syncwarp();      // the stores to tensor memory below are the whole warp's: lanes part above this line and not between it and them
        if (bounded) {
          if (!__all_sync(0xffffffffu, ok)) break;
        } else if (at_any(bar, !ok || mx > ref + AT_SLACK || (ref == -INFINITY && mx > -INFINITY))) {
          // (one barrier of the rows' two warps per block: does any row's reference have to move, has any wait run out?)
          *mine = mx;
          ok = !at_any(bar, !ok);
          if (!ok) break;
          const float mo = *other;
          const float nref = fmaxf(ref, fmaxf(mx, mo));
          const float f = ref == -INFINITY ? 0.f : at_exp2(ref - nref);
          ref = nref;
          sum2[0] = f2_mul(sum2[0], f2_of(f, f));
          sum2[1] = f2_mul(sum2[1], f2_of(f, f));
          if (n > 0) ok = at_wait(&o_full[2 * tile + (int)((n - 1u) & 1u)], ((n - 1u) >> 1) & 1u, s_fail, p.word, 8);
          __syncwarp();
          tc_fence_after();
          if (at_any(bar, !ok)) {                                      // (also: both threads of a row have read the other's)
            ok = false;
            break;
          }
          if (n > 0) {                                                      // what the blocks before have added up
#pragma unroll 1
            for (int c = 32 * half; c < DV; c += 64) {
              uint32_t o[32];
              tmem_ld32_async(to + (uint32_t)c, o);
              tmem_wait_ld();
              tie32(o);
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
              tmem_st16(to + (uint32_t)c, o);
              tmem_st16(to + (uint32_t)c + 16u, o + 16);
            }
          }
        }
        const float sub = ref == -INFINITY ? 0.f : -ref;
        // exponents
        const f2 sub2 = f2_of(sub, sub), mul2 = f2_of(mul, mul);
        if (!CAP) {
#pragma unroll
          for (int e = 0; e < AT_C; e += 2) {
            const f2 a = f2_fma(f2_of(__uint_as_float(sr[e]), __uint_as_float(sr[e + 1])), mul2, sub2);
            float a0, a1;
            f2_split(a, a0, a1);
            sr[e] = __float_as_uint(a0), sr[e + 1] = __float_as_uint(a1);
          }
        } else {
          // tanh by its polynomial while all scores are small.  Of bounded ones that is seen on the way: where some row's are too large the raw scores,
          // taken from tensor memory again, go through the exponential form.  (A NaN is passed over; NaN * P(NaN) stays NaN.)
          const float m3 = mul * mul * mul, c0p = cap2 * AT_T0 * mul, c1p = cap2 * AT_T1 * m3, c2p = cap2 * AT_T2 * (m3 * mul * mul);
          const f2 p0c = f2_of(c0p, c0p), p1c = f2_of(c1p, c1p), p2c = f2_of(c2p, c2p);
          float u4[4] = {0.f, 0.f, 0.f, 0.f};
          if (poly) {
#pragma unroll
            for (int e = 0; e < AT_C; e += 2) {
              const f2 x = f2_of(__uint_as_float(sr[e]), __uint_as_float(sr[e + 1])), u = f2_mul(x, x);
              const f2 a = f2_fma(x, f2_fma(f2_fma(p2c, u, p1c), u, p0c), sub2);
              float a0, a1, u0, u1;
              f2_split(a, a0, a1);
              f2_split(u, u0, u1);
              if (bounded) u4[(e >> 1) & 3] = at_max3(u4[(e >> 1) & 3], u0, u1);
              sr[e] = __float_as_uint(a0), sr[e + 1] = __float_as_uint(a1);
            }
          }
          if (bounded) {
            poly = __all_sync(0xffffffffu, at_max3(u4[0], u4[1], fmaxf(u4[2], u4[3])) * (mul * mul) < AT_TANH_SMALL * AT_TANH_SMALL);
            if (!poly) {
              tmem_ld32_async(ts + (uint32_t)(AT_C * half), sr);
              tmem_wait_ld();
              tie32(sr);
              if (BIAS) {
#pragma unroll
                for (int e = 0; e < AT_C; ++e) sr[e] = __float_as_uint(fmaf(slope, (float)(c0 + e - qp), __uint_as_float(sr[e]) * (p.scale * bias_unit)));
              }
            }
          }
          if (!poly) {
            const float k2 = mul * (2.f * AT_LOG2E), top = cap2 + sub, two = -2.f * cap2;
#pragma unroll
            for (int e = 0; e < AT_C; ++e) {
              const float a = fmaf(two, at_rcp(1.f + at_exp2(__uint_as_float(sr[e]) * k2)), top);
              sr[e] = __float_as_uint(!bounded && masked && (e < cmin || e > cmax) ? -INFINITY : a);
            }
          }
          if (bounded && masked) {
#pragma unroll
            for (int e = 0; e < AT_C; ++e)
              if (e < cmin || e > cmax) sr[e] = __float_as_uint(-INFINITY);
          }
        }
        // weights
        uint32_t ph[16], pl[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float p0 = at_exp2(__uint_as_float(sr[2 * e])), p1 = at_exp2(__uint_as_float(sr[2 * e + 1]));
          const f2 pp = f2_of(p0, p1);
          ph[e] = pack_bf16(p0, p1);
          const f2 hi = f2_of(__uint_as_float(ph[e] << 16), __uint_as_float(ph[e] & 0xffff0000u));
          // the sum is of the weights as the product sees them: with one term (8 bits) their rounding would not cancel in the quotient
          sum2[e & 1] = f2_add(sum2[e & 1], TERMS == 1 ? hi : pp);
          if (TERMS == 2) {
            float l0, l1;
            f2_split(f2_fma(hi, f2_of(-1.f, -1.f), pp), l0, l1);
            pl[e] = pack_bf16(l0, l1);
          }
        }
        // the weights go over the thread's own scores: 16 columns of the first term, 16 of the second
        tmem_st16(ts + (uint32_t)(AT_C * half), ph);
        if (TERMS == 2) tmem_st16(ts + (uint32_t)(AT_C * half) + 16u, pl);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[2 * tile + (int)(n & 1u)]);
        ++n;
      }
    }
    const bool store = n > 0 && (tile ? tq1 : tq0) < p.T, live = t < p.T;
    const size_t m = (size_t)b * p.T + t;
    const __nv_bfloat16* gt = p.gate && !p.gate_per_head ? p.gate + m * p.gate_ld + (size_t)h * p.vdim : nullptr;
    // the row's gate numbers are asked for before the accumulator is waited for, 16 bytes at a time
    uint4 gu[NBV][4];
#pragma unroll
    for (int z = 0; z < NBV; ++z)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 64 * z + 32 * half + 8 * e;
        gu[z][e] = make_uint4(0u, 0u, 0u, 0u);
        if (gt && live && c < p.vdim) gu[z][e] = at_load8(gt + c, p.gate_vec);
      }
    if (ok && store) ok = at_wait(&o_full[2 * tile + (int)((n - 1u) & 1u)], ((n - 1u) >> 1) & 1u, s_fail, p.word, 9);
    __syncwarp();
    tc_fence_after();
    float s0, s1;
    f2_split(f2_add(sum2[0], sum2[1]), s0, s1);
    *mine = s0 + s1;
    if (!at_any(bar, !ok) && store) {
      float den = half == 0 ? *mine + *other : *other + *mine;            // the halves' sums in the order of the columns
      float num = 1.f;
      if (p.sink) {                                     // (scaled by whichever is larger, the reference or the sink)
        const float sk = p.sink[h] * AT_LOG2E - ref, up = fmaxf(sk, 0.f);
        num = at_exp2(-up);
        den = den * num + at_exp2(sk - up);
      }
      float fin = den > 0.f ? num / den : 0.f;
      if (live && p.gate && p.gate_per_head) fin *= at_sigmoid(__bfloat162float(p.gate[m * p.gate_ld + h]));
      __nv_bfloat16* dst = p.y + m * p.y_ld + (size_t)h * p.vdim;
#pragma unroll
      for (int z = 0; z < NBV; ++z) {
        const int c = 64 * z + 32 * half;
        __syncwarp();
        uint32_t o[32];
        tmem_ld32_async(to + (uint32_t)c, o);
        tmem_wait_ld();
        tie32(o);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (!live || c + 8 * e >= p.vdim) continue;           // (vdim is a multiple of 8)
          const uint32_t gw[4] = {gu[z][e].x, gu[z][e].y, gu[z][e].z, gu[z][e].w};
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float a = __uint_as_float(o[8 * e + 2 * j]) * fin, q = __uint_as_float(o[8 * e + 2 * j + 1]) * fin;
            if (gt) a *= at_sigmoid(bf16_bits_to_f32(gw[j] & 0xffffu)), q *= at_sigmoid(bf16_bits_to_f32(gw[j] >> 16));
            w[j] = pack_bf16(a, q);
          }
          *reinterpret_cast<uint4*>(dst + c + 8 * e) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        __syncwarp();
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == AT_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// rows of one operand as a 4-D map (dimension, head, row, sequence), boxes of 64 dimensions
int at_map(const AttnTcOperand& o, int heads, int rows, int B, int box_rows, CUtensorMap* out) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled entry point not available");
    return LL_ERR_CUDA;
  }
  cuuint64_t dims[4] = {(cuuint64_t)o.dim, (cuuint64_t)heads, (cuuint64_t)rows, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)o.head * 2, (cuuint64_t)o.row * 2, (cuuint64_t)o.batch * 2};
  cuuint32_t box[4] = {64, 1, (cuuint32_t)box_rows, 1}, estr[4] = {1, 1, 1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)o.base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): %d numbers, %d heads, %d rows", (int)r, o.dim, heads, rows);
    return LL_ERR_CUDA;
  }
  return LL_OK;
}

bool at_operand_ok(const AttnTcOperand& o) {
  return o.dim > 0 && o.dim % 8 == 0 && ((uintptr_t)o.base & 15) == 0 && o.head > 0 && o.row > 0 && o.batch > 0 && o.head % 8 == 0 &&
         o.row % 8 == 0 && o.batch % 8 == 0;
}

template <int NB1, int NB2, int NBV, int TERMS, AtCap CAP, bool BIAS>
int at_launch(const AttnTcArgs& a, const AtParams& p, cudaStream_t st) {
  constexpr int smem = AtShape<NB1, NB2, NBV>::SMEM;
  static_assert(smem <= 227 * 1024, "shared memory of a block");
  auto* kernel = attn_tc_kernel<NB1, NB2, NBV, TERMS, CAP, BIAS>;
  LL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  CUtensorMap mq, mq2, mk, mk2, mv;
  if (int r = at_map(a.q, a.H, a.T, a.B, AT_Q, &mq)) return r;
  if (int r = at_map(a.k, a.G, a.ring, a.B, AT_K, &mk)) return r;
  if (int r = at_map(a.v, a.G, a.ring, a.B, AT_K, &mv)) return r;
  mq2 = mq, mk2 = mk;
  if (NB2 > 0) {
    if (int r = at_map(a.q2, a.H, a.T, a.B, AT_Q, &mq2)) return r;
    if (int r = at_map(a.k2, 1, a.ring, a.B, AT_K, &mk2)) return r;
  }
  const int tiles = (a.T + AT_Q - 1) / AT_Q;
  const dim3 grid(p.tiles == AT_ALONE ? tiles : (tiles + 1) / 2, a.H, a.B);
  kernel<<<grid, AT_THREADS, smem, st>>>(mq, mq2, mk, mk2, mv, p);
  LL_LAUNCH_OK("attn_tc_kernel");
  return LL_OK;
}

// Whether the form takes these arguments (sizes, alignment, strides).
bool attn_tc_supported(const AttnTcArgs& a) {
  const bool two = a.q2.base != nullptr;
  if (!at_operand_ok(a.q) || !at_operand_ok(a.k) || !at_operand_ok(a.v) || a.q.dim != a.k.dim || a.q.dim > 128 || a.v.dim > 128) return false;
  if (two && (!at_operand_ok(a.q2) || !at_operand_ok(a.k2) || a.q2.dim != a.k2.dim || a.q2.dim > 64 || a.softcap > 0.f || a.slopes)) return false;
  if (a.gate && !a.gate_per_head && (a.gate_ld % 2 != 0 || ((uintptr_t)a.gate & 3) != 0)) return false;
  return a.B > 0 && a.B <= 65535 && a.H > 0 && a.H <= 65535 && a.T > 0 && a.ring > 0 && a.G > 0 && a.H % a.G == 0 && a.scale > 0.f &&
         a.y_ld % 8 == 0 && ((uintptr_t)a.y & 15) == 0 && (a.terms == 1 || a.terms == 2);
}

// Which tiles a block takes.  With no more tiles than SMs one (us, two a block / one: 32 heads, 300 and 512 queries 15.4 / 13.6, 18.6 / 16.3; 16 heads, 130,
// 512, 1024, 1152 queries 13.3 / 11.0, 17.8 / 14.4, 24.4 / 21.8, 26.8 / 23.7, with a window of 200 of 1024 19.7 / 14.8; 8 heads, 2048 queries 37.8 / 35.1).
// Two neighbours share most of their keys, and with blocks for several rounds of the SMs the long ones, which come first, even out by themselves.  Queries
// that see all keys before them have very unequal walks, though: while the blocks fit the SMs at once, or their second round is more than half full, one tile
// from the end and one from the start make all blocks alike.  neighbours / apart, of heads of 128, by tiles and blocks per SM: 4, 8, 16, 32 tiles at up to
// one 1.10, 1.21, 1.27, 1.28, three 0.90; eight to 64 tiles at 1.08 and 1.3 0.81 - 1.01, at 1.5 - 2 1.02 - 1.15, at 2.2 - 3 0.91 - 1.06, at 3.5 - 7
// 0.87 - 1.00.  Under a window of two thirds, a half and a third of the queries at up to one 1.05 - 1.20 (three tiles 0.87), 0.99 - 1.11, 0.81 - 1.05, at 1.7
// 0.98 - 1.12, 0.94 - 1.07, 0.78 - 1.01.  Chunks stay neighbours (512 of 2048: 21.7, apart 24.7 us).
int at_tiles(const AttnTcArgs& a) {
  const long long tiles = (a.T + AT_Q - 1) / AT_Q, blocks = (tiles + 1) / 2 * a.H * a.B, sms = sm_count() > 0 ? sm_count() : 148;
  if (tiles * a.H * a.B <= sms) return AT_ALONE;
  if (a.chunk > 0 || tiles < 4) return AT_NEIGHBOURS;
  if (blocks <= sms) return a.window <= 0 || 2ll * a.window >= a.T ? AT_APART : AT_NEIGHBOURS;
  return 2 * blocks >= 3 * sms && blocks <= 2 * sms && (a.window <= 0 || a.window >= a.T) ? AT_APART : AT_NEIGHBOURS;
}

enum AttnTcKind { AT_ROTARY, AT_LATENT };     // which forms a file instantiates

template <AttnTcKind KIND>
int attn_tc_launch(const AttnTcArgs& a, cudaStream_t st) {
  const AtParams p{a.pos_ids, a.sink, a.slopes, (const __nv_bfloat16*)a.gate, (__nv_bfloat16*)a.y, a.scale, a.softcap, a.T, a.H, a.H / a.G,
                   a.v.dim, a.window, a.chunk, a.ring, a.gate_ld, a.gate_per_head,
                   a.gate_ld % 8 == 0 && ((uintptr_t)a.gate & 15) == 0, a.y_ld, at_tiles(a), wait_word()};
  const int nb = (a.q.dim + 63) / 64, nbv = (a.v.dim + 63) / 64;
  const AtCap cap = a.softcap <= 0.f ? AT_UNCAPPED : a.softcap * AT_LOG2E <= AT_BOUND ? AT_BOUNDED : AT_CAPPED;
  const bool bias = a.slopes != nullptr, two = a.q2.base != nullptr;
#define LL_AT(N1, N2, NV, TERMS, CC, BB) \
  if (nb == N1 && two == (N2 > 0) && nbv == NV && a.terms == TERMS && cap == CC && bias == BB) return at_launch<N1, N2, NV, TERMS, CC, BB>(a, p, st);
#define LL_AT_SIZES(N2, TERMS, CC, BB) LL_AT(1, N2, 1, TERMS, CC, BB) LL_AT(1, N2, 2, TERMS, CC, BB) LL_AT(2, N2, 1, TERMS, CC, BB) LL_AT(2, N2, 2, TERMS, CC, BB)
  if constexpr (KIND == AT_ROTARY) {
    LL_AT_SIZES(0, 2, AT_UNCAPPED, false) LL_AT_SIZES(0, 2, AT_BOUNDED, false) LL_AT_SIZES(0, 2, AT_CAPPED, false)
    LL_AT_SIZES(0, 2, AT_UNCAPPED, true) LL_AT_SIZES(0, 2, AT_BOUNDED, true) LL_AT_SIZES(0, 2, AT_CAPPED, true)
  } else {
    LL_AT_SIZES(1, 1, AT_UNCAPPED, false) LL_AT_SIZES(1, 2, AT_UNCAPPED, false)
  }
#undef LL_AT_SIZES
#undef LL_AT
  set_error("attn_tc: no form for these arguments");
  return LL_ERR_UNSUPPORTED;
}

// 0, or the code of the first bounded wait that ran out.  Synchronises the device.
int attn_tc_error() {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, g_attn_tc_error, sizeof(int)) == cudaSuccess ? v : -1;
}

}  // namespace
}  // namespace llb
