// Many rows through an int4 layer on tcgen05 (prompts): y[M][N] = x[M][K] . dequant(W)^T, the weights read in their packed checkpoint form
// (bytes [K/2][N], even k in the low half) and de-quantised inside the main loop with the reference's two bf16 roundings
// (ref: lit_llama/quantization.py:399-408), so that no bf16 copy of W is written and read back.
//
// Operand roles are swapped: the weights are the A operand (128 output columns = the 128 TMEM lanes) and live in tensor memory, where the
// threads that de-quantise them put them; the activations are the B operand, tiles of BN rows x 64 k loaded by TMA.
//   warps 0, 2 : TMA producers: 128 k of BN rows of x; 64 x 128 packed bytes
//   warp 1     : one thread issues 128 x BN x 16 MMAs (A from tensor memory)
//   warps 4-19 : de-quantise in four groups of four warps (a warp per TMEM lane quarter); group g makes every fourth step of 128 k into
//                A buffer g, so that four steps are in the making at a time (one step's chain of waits, loads and stores is 1500 clocks
//                long however many warps share it); then the epilogue, a quarter of the rows per group
// Persistent: a CTA walks tiles with a stride of the grid; a group drains a tile after its first step of the next one, and gives the
// accumulator back as soon as it is in registers, so that the tensor cores wait for the drain alone.
// Every wait is bounded; one that runs out records a code, all roles stop, copies in flight are waited for, tensor memory is freed.
#include "tcgen05.cuh"

namespace llb {
namespace {

constexpr int R4_N = 128, R4_K = 128, R4_GROUPS = 4, R4_THREADS = (4 + 4 * R4_GROUPS) * 32;
constexpr int R4_WBYTES = R4_N * R4_K / 2, R4_WST = R4_GROUPS;         // a stage of packed bytes per group
constexpr uint32_t R4_WAIT_LIMIT = 1u << 20;
__host__ __device__ constexpr int r4_xbytes(int bn) { return bn * R4_K * 2; }
__host__ __device__ constexpr int r4_xst(int bn) { return bn >= 256 ? 3 : bn >= 192 ? 4 : 6; }
constexpr int r4_smem(int bn) { return r4_xst(bn) * r4_xbytes(bn) + R4_WST * R4_WBYTES + 512 + 1024; }

__device__ int g_r4_error = 0;

struct R4Params {
  const __nv_bfloat16* scales;   // [N][G]
  const __nv_bfloat16* zeros;
  const __nv_bfloat16* bias;
  __nv_bfloat16* y;
  int M, N, steps, G, steps_per_group, mtiles, tiles;
  int* word;                     // wait_word()
};

__device__ __forceinline__ bool r4_wait(uint64_t* bar, uint32_t parity, volatile int* fail, int* word, int code) {
  for (uint32_t i = 0; i < R4_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  atomicCAS(&g_r4_error, 0, code);
  wait_ran_out(word, 200 + code);
  return false;
}
// The same without suspending the thread between looks: for the thread that feeds the tensor cores, whose wake-up would be waited for.
__device__ __forceinline__ bool r4_spin(uint64_t* bar, uint32_t parity, volatile int* fail, int* word, int code) {
  for (uint32_t i = 0; i < 64u * R4_WAIT_LIMIT; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  atomicCAS(&g_r4_error, 0, code);
  wait_ran_out(word, 200 + code);
  return false;
}
__device__ __forceinline__ void r4_box(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
               "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void r4_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void r4_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ uint32_t r4_sub2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t r4_mul2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

template <int BN>
__global__ void __launch_bounds__(R4_THREADS, 1) int4_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                  const R4Params p) {
  constexpr int XST = r4_xst(BN), XB = r4_xbytes(BN), PART = BN / R4_GROUPS;      // PART: rows a group drains
  constexpr uint32_t TM_A = 256;                       // D: columns [0, BN); A buffers of 64 columns from 256 on
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* sx = base;                                  // [XST][2][BN][64] bf16, swizzled
  uint8_t* sw = base + XST * XB;                       // [WST][64][128] packed bytes
  uint64_t* x_full = reinterpret_cast<uint64_t*>(sw + R4_WST * R4_WBYTES);
  uint64_t* x_empty = x_full + XST;
  uint64_t* w_full = x_empty + XST;
  uint64_t* w_empty = w_full + R4_WST;
  uint64_t* a_ready = w_empty + R4_WST;
  uint64_t* a_free = a_ready + R4_GROUPS;
  uint64_t* d_full = a_free + R4_GROUPS;
  uint64_t* d_empty = d_full + 1;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(d_empty + 1);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_x);
    for (int i = 0; i < XST; ++i) mbar_init(&x_full[i], 1), mbar_init(&x_empty[i], 1);
    for (int i = 0; i < R4_WST; ++i) mbar_init(&w_full[i], 1), mbar_init(&w_empty[i], 4);
    for (int i = 0; i < R4_GROUPS; ++i) mbar_init(&a_ready[i], 4), mbar_init(&a_free[i], 1);
    mbar_init(d_full, 1);
    mbar_init(d_empty, 4 * R4_GROUPS);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_ptr, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const int steps = p.steps;

  if (warp == 0 || warp == 2) {
    if (elect_one()) {
      bool ok = true;
      int s = 0;
      uint32_t ph = 1;
      for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
        const int n0 = (tile / p.mtiles) * R4_N, m0 = (tile % p.mtiles) * BN;
        if (warp == 0) {
          for (int kb = 0; kb < steps; ++kb) {
            if (!(ok = r4_wait(&x_empty[s], ph, s_fail, p.word, 1))) break;
            mbar_expect_tx(&x_full[s], XB);
            r4_box(sx + s * XB, &map_x, kb * R4_K, m0, &x_full[s]);
            r4_box(sx + s * XB + XB / 2, &map_x, kb * R4_K + 64, m0, &x_full[s]);
            if (++s == XST) s = 0, ph ^= 1u;
          }
        } else {
          for (int kb = 0; kb < steps; ++kb) {
            if (!(ok = r4_wait(&w_empty[s], ph, s_fail, p.word, 2))) break;
            mbar_expect_tx(&w_full[s], R4_WBYTES);
            r4_box(sw + s * R4_WBYTES, &map_w, n0, kb * (R4_K / 2), &w_full[s]);
            if (++s == R4_WST) s = 0, ph ^= 1u;
          }
        }
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc_bf16(R4_N, BN);
      const uint64_t xd = smem_desc_sw128(smem_u32(sx));
      bool ok = true;
      int s = 0, tl = 0;
      uint32_t ph = 0, blk = 0;
      for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x, ++tl) {
        if (tl > 0 && !(ok = r4_wait(d_empty, (uint32_t)(tl - 1) & 1u, s_fail, p.word, 3))) break;
        for (int kb = 0; ok && kb < steps; ++kb, ++blk) {
          const uint32_t buf = blk % R4_GROUPS;
          if (!(ok = r4_spin(&x_full[s], ph, s_fail, p.word, 5) && r4_spin(&a_ready[buf], (blk / R4_GROUPS) & 1u, s_fail, p.word, 4))) break;
          tc_fence_after();
          const uint64_t bd = xd + (uint64_t)(s * (XB >> 4));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            r4_mma(tmem, tmem + TM_A + 64u * buf + 8u * k, bd + (uint64_t)((k >> 2) * (XB >> 5) + 2 * (k & 3)), idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit(&a_free[buf]);
          umma_commit(&x_empty[s]);
          if (++s == XST) s = 0, ph ^= 1u;
        }
        if (ok) umma_commit(d_full);
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp >= 4) {
    const int quarter = warp & 3, grp = (warp >> 2) - 1, col = quarter * 32 + lane;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    bool ok = true;
    // a finished tile: its sums leave tensor memory, then the accumulator is given back, then they are stored
    auto drain = [&](int tile, uint32_t nth) {
      ok = __all_sync(0xffffffffu, r4_wait(d_full, nth & 1u, s_fail, p.word, 6));
      if (!ok) return;
      tc_fence_after();
      const int n = (tile / p.mtiles) * R4_N + col, m0 = (tile % p.mtiles) * BN + grp * PART;
      const float bias = p.bias != nullptr && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
      uint32_t w[PART / 2];
#pragma unroll
      for (int c = 0; c < PART; c += 16) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(tmem + lanes + (uint32_t)(grp * PART + c))
            : "memory");
#pragma unroll
        for (int e = 0; e < 16; e += 2) w[(c + e) / 2] = pack_bf16(__uint_as_float(v[e]) + bias, __uint_as_float(v[e + 1]) + bias);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(d_empty);
      // a lane holds two rows of its column in a word; neighbours swap, so that a lane stores two columns of one row
      const bool odd = (lane & 1) != 0;
      __nv_bfloat16* dst = p.y + (size_t)(m0 + (odd ? 1 : 0)) * p.N + (n & ~1);
      const int left = p.M - m0 - (odd ? 1 : 0);
#pragma unroll
      for (int e = 0; e < PART / 2; ++e) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, w[e], 1);
        const uint32_t o = odd ? (got >> 16) | (w[e] & 0xffff0000u) : (w[e] & 0xffffu) | (got << 16);
        if (2 * e < left && n < p.N) *reinterpret_cast<uint32_t*>(dst + (size_t)(2 * e) * p.N) = o;
      }
      __syncwarp();
    };
    // the group's steps: every fourth of all steps of all of the CTA's tiles
    int tile = blockIdx.x, kb = grp, drained = blockIdx.x;
    uint32_t nth = 0;
    auto normal = [&]() {
      while (kb >= steps && tile < p.tiles) kb -= steps, tile += gridDim.x;
    };
    auto params = [&](uint32_t& sv, uint32_t& zv) {
      if (tile >= p.tiles) return;
      const size_t at = (size_t)min((tile / p.mtiles) * R4_N + col, p.N - 1) * p.G + kb / p.steps_per_group;
      sv = *reinterpret_cast<const uint16_t*>(p.scales + at);
      zv = *reinterpret_cast<const uint16_t*>(p.zeros + at);
    };
    uint32_t sn = 0, zn = 0, round = 0;      // round: the group's how-many-th step
    normal();
    params(sn, zn);
    while (ok && tile < p.tiles) {
      const int cur = tile;
      const uint32_t s2 = sn * 0x00010001u, z2 = zn * 0x00010001u;
      // an integer zero (every RTN / GPTQ checkpoint): (128 + q) - (128 + zero) in ONE exact subtraction
      const float zf = __uint_as_float(zn << 16);
      const bool zint = zf == floorf(zf) && zf >= 0.f && zf <= 64.f;
      const uint32_t zc2 = zint ? (uint32_t)(0x4300u + (uint32_t)zf) * 0x00010001u : 0x43004300u;
      // a column's zero may be whole and its neighbour's not: the warp goes one way (the store below is the whole warp's), a whole zero
      // then subtracts 0
      const bool one_step = __all_sync(0xffffffffu, zint);
      const uint32_t zr2 = zint ? 0u : z2;
      kb += R4_GROUPS;
      normal();
      params(sn, zn);                        // of the next step, under this one's work
      const int s = grp;
      ok = r4_wait(&w_full[s], round & 1u, s_fail, p.word, 7);
      if (ok && round > 0) ok = r4_wait(&a_free[grp], (round - 1u) & 1u, s_fail, p.word, 8);
      if (!(ok = __all_sync(0xffffffffu, ok))) break;
      tc_fence_after();
      const uint8_t* src = sw + s * R4_WBYTES + col;
      const uint32_t ta = tmem + lanes + TM_A + 64u * grp;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t b = src[(c * 16 + j) * R4_N];
          uint32_t a = r4_sub2(((b * 0x1001u) & 0x000f000fu) | 0x43004300u, zc2);      // bf16 (128 + q) of both halves, minus 128 (+ zero)
          if (!one_step) a = r4_sub2(a, zr2);
          r[j] = r4_mul2(a, s2);
        }
        r4_st16(ta + 16u * c, r);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_empty[s]), mbar_arrive(&a_ready[grp]);
      ++round;
      while (ok && drained < cur) {
        drain(drained, nth++);
        drained += gridDim.x;
      }
    }
    while (ok && drained < p.tiles) {
      drain(drained, nth++);
      drained += gridDim.x;
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// packed bytes [K/2][N] as a 2-D map, boxes of 128 columns x 64 rows
int r4_weight_map(const void* qw, int N, int K, CUtensorMap* out) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled entry point not available");
    return LL_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)(K / 2)}, strides[1] = {(cuuint64_t)N};
  cuuint32_t box[2] = {R4_N, R4_K / 2}, estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)qw, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): packed weights N=%d K=%d", (int)r, N, K);
    return LL_ERR_CUDA;
  }
  return LL_OK;
}

template <int BN>
int r4_launch(const CUtensorMap& mw, const void* x, R4Params p, int K, int grid, cudaStream_t st) {
  CUtensorMap mx;
  if (int r = make_map(x, p.M, K, BN, &mx)) return r;
  LL_CUDA(cudaFuncSetAttribute(int4_rows_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, r4_smem(BN)));
  p.mtiles = (p.M + BN - 1) / BN;
  p.tiles = p.mtiles * ((p.N + R4_N - 1) / R4_N);
  int4_rows_kernel<BN><<<p.tiles < grid ? p.tiles : grid, R4_THREADS, r4_smem(BN), st>>>(mw, mx, p);
  LL_LAUNCH_OK("int4_rows_kernel");
  return LL_OK;
}

// Clocks of a launch with tiles of bn rows: waves of the persistent grid, 128 k at a time (see the head of the file), plus the drain.  (A
// step takes 600 clocks at least, however few the rows: tiles of 64 never cost less than tiles of 128.)
long long r4_cost(int M, int N, int steps, int bn, int sms) {
  const long long tiles = (long long)((M + bn - 1) / bn) * ((N + R4_N - 1) / R4_N);
  return (tiles + sms - 1) / sms * ((long long)steps * (4 * bn > 600 ? 4 * bn : 600) + 1200);
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
  LL_CHECK_ARG(qw && scales && zeros && x && y && M > 0, "int4_rows: null pointer or no rows");
  if (!ll_int4_rows_supported(N, K, group)) {
    set_error("int4_rows needs N %% 16 == 0 and group %% 128 == 0 (N=%d K=%d group=%d)", N, K, group);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG((((uintptr_t)qw | (uintptr_t)x | (uintptr_t)y) & 15) == 0, "int4_rows: packed weights, x and y must be 16-byte aligned");
  R4Params p{};
  p.scales = (const __nv_bfloat16*)scales, p.zeros = (const __nv_bfloat16*)zeros, p.bias = (const __nv_bfloat16*)bias, p.y = (__nv_bfloat16*)y;
  p.M = M, p.N = N, p.steps = K / R4_K, p.G = K / group, p.steps_per_group = group / R4_K;
  p.word = wait_word();
  LL_CHECK_ARG((tile_rows == 0 || tile_rows == 128 || tile_rows == 192 || tile_rows == 256) && grid >= 0, "int4_rows: tiles of 128, 192 or 256 rows");
  if (grid == 0) grid = sm_count();
  CUtensorMap mw;
  if (int r = r4_weight_map(qw, N, K, &mw)) return r;
  if (tile_rows == 0) {
    tile_rows = 256;
    for (int bn = 192; bn >= 128; bn -= 64)
      if (r4_cost(M, N, p.steps, bn, grid) < r4_cost(M, N, p.steps, tile_rows, grid)) tile_rows = bn;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (tile_rows == 256) return r4_launch<256>(mw, x, p, K, grid, st);
  if (tile_rows == 192) return r4_launch<192>(mw, x, p, K, grid, st);
  return r4_launch<128>(mw, x, p, K, grid, st);
}

// 0, or the code of the first bounded wait that ran out in this file's kernel.  Synchronises the device.
int ll_int4_rows_error(void) {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, g_r4_error, sizeof(int)) == cudaSuccess ? v : -1;
}

}  // extern "C"
