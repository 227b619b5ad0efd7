// Batches of up to 128 rows through int4 layers on tcgen05: y[M][N] = x[M][K] . dequant(W)^T from the checkpoint bytes, and the gated pair
// h = silu(x W1^T) * (x W2^T) of two layers that read the same x, rounded as the separate kernels round it.
//
// What counts is unpacking: a weight is used for few rows.  All steps (128 columns x 128 k) of all column tiles, of both layers in the gated
// form, are laid end to end and cut into one equal range per SM, so that no SM waits for a last wave and no split has to divide K; a range
// crosses tile ends and leaves partial sums of every tile that it touches, in fp32, which a second small kernel adds in the order of k.
// Roles are those of int4_rows.cu, with one CTA a range:
//   warps 0, 2 : TMA producers: 128 k of the rows of x; 64 x 128 packed bytes, 8 to 12 steps ahead
//   warp 1     : one thread issues 128 x MP x 16 MMAs (A from tensor memory), two accumulators in turn
//   warp 3     : scales and zeros
//   warps 4-19 : unpack in four groups, every fourth step, into 4 or 6 A buffers; then a quarter of the rows of a finished tile each
// us on the device, a split of K that fills whole waves and a sum / this kernel and its sum: 11008 x 4096 at 32 and 128 rows 25 / 18 and 40 / 22,
// 4096 x 11008 21 / 17 and 31 / 22, 5632 x 2048 13 / 10 and 17 / 13; the gated pair 11008 x 4096 of 32 rows 54 / 28.  Bound by 0.4 us a step of
// bytes on their way and unpacking (2.5 TB/s of packed weights) and 8 us around it: first bytes, last tile, partial sums.
// Every wait is bounded; one that runs out records a code, all roles stop, copies in flight are waited for, tensor memory is freed.
#include "int4_unpack.cuh"

namespace llb {
namespace {

constexpr int B4_GROUPS = 4, B4_THREADS = (4 + 4 * B4_GROUPS) * 32;
constexpr uint32_t B4_WAIT_LIMIT = 1u << 20;
constexpr int b4_xst(int mp) { return mp > 64 ? 4 : mp > 32 ? 6 : 8; }
constexpr int b4_wst(int mp) { return mp > 64 ? 8 : 12; }
constexpr int b4_abufs(int mp) { return mp > 64 ? 4 : 6; }
constexpr int b4_smem(int mp) { return b4_xst(mp) * mp * 256 + b4_wst(mp) * (R4_WBYTES + R4_SZ) + 1024 + 1024; }

__device__ int g_b4_error = 0;

struct B4Params {
  const __nv_bfloat16* scales[2];   // [N][G]; the second set: the gated form's W2
  const __nv_bfloat16* zeros[2];
  float* part;                      // [ranges][slots][MP][128]
  int M, N, steps, G, steps_per_group, wide, ntiles, total, slots;      // ntiles: column tiles of a layer; total: steps of all tiles
  int* word;                        // wait_word()
};

__device__ __forceinline__ bool b4_wait(uint64_t* bar, uint32_t parity, volatile int* fail, int* word, int code) {
  for (uint32_t i = 0; i < B4_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  atomicCAS(&g_b4_error, 0, code);
  wait_ran_out(word, 220 + code);
  return false;
}
// the same without suspending the thread between looks
__device__ __forceinline__ bool b4_spin(uint64_t* bar, uint32_t parity, volatile int* fail, int* word, int code) {
  for (uint32_t i = 0; i < 64u * B4_WAIT_LIMIT; ++i) {
    if (mbar_test_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  atomicCAS(&g_b4_error, 0, code);
  wait_ran_out(word, 220 + code);
  return false;
}
__device__ __forceinline__ void b4_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void b4_ld4(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
}
// range `c` of `n`: its first step
__host__ __device__ __forceinline__ int b4_first(int c, int total, int n) { return (int)((long long)c * total / n); }

template <int MP>
__global__ void __launch_bounds__(B4_THREADS, 1) int4_batch_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                                                                   const __grid_constant__ CUtensorMap map_x, const B4Params p) {
  constexpr int XST = b4_xst(MP), WST = b4_wst(MP), NA = b4_abufs(MP), XB = MP * 256;
  constexpr uint32_t TM_A = NA == 4 ? 256 : 128;       // D: columns [0, MP) and [MP, 2 MP)
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* sx = base;                                  // [XST][2][MP][64] bf16, swizzled
  uint8_t* sw = base + XST * XB;                       // [WST][64][128] packed bytes, swizzled
  uint8_t* sz = sw + WST * R4_WBYTES;                  // [WST] scales and zeros
  uint64_t* x_full = reinterpret_cast<uint64_t*>(sz + WST * R4_SZ);
  uint64_t* x_empty = x_full + XST;
  uint64_t* w_full = x_empty + XST;
  uint64_t* w_empty = w_full + WST;
  uint64_t* a_ready = w_empty + WST;
  uint64_t* a_free = a_ready + NA;
  uint64_t* d_full = a_free + NA;                      // [2]
  uint64_t* d_empty = d_full + 2;                      // [2]
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(d_empty + 2);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_w0);
    prefetch_tensormap(&map_w1);
    prefetch_tensormap(&map_x);
    for (int i = 0; i < XST; ++i) mbar_init(&x_full[i], 1), mbar_init(&x_empty[i], 1);
    for (int i = 0; i < WST; ++i) mbar_init(&w_full[i], 2), mbar_init(&w_empty[i], 4);
    for (int i = 0; i < NA; ++i) mbar_init(&a_ready[i], 4), mbar_init(&a_free[i], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&d_full[i], 1), mbar_init(&d_empty[i], 4 * B4_GROUPS);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_ptr, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const int steps = p.steps, first = b4_first(blockIdx.x, p.total, gridDim.x), n = b4_first(blockIdx.x + 1, p.total, gridDim.x) - first;
  const int tile0 = first / steps, kb0 = first - tile0 * steps;
  pdl_wait();                                          // (what comes before it runs under the kernel before)
  pdl_launch_dependents();

  if (warp == 0 || warp == 2) {
    if (elect_one()) {
      bool ok = true;
      int s = 0, tile = tile0, kb = kb0;
      uint32_t ph = 1;
      for (int i = 0; i < n; ++i) {
        if (warp == 0) {
          if (!(ok = b4_wait(&x_empty[s], ph, s_fail, p.word, 1))) break;
          mbar_expect_tx(&x_full[s], XB);
          r4_box(sx + s * XB, &map_x, kb * R4_K, 0, &x_full[s]);
          r4_box(sx + s * XB + XB / 2, &map_x, kb * R4_K + 64, 0, &x_full[s]);
          if (++s == XST) s = 0, ph ^= 1u;
        } else {
          if (!(ok = b4_wait(&w_empty[s], ph, s_fail, p.word, 2))) break;
          const bool second = tile >= p.ntiles;
          const int n0 = (second ? tile - p.ntiles : tile) * 128;
          mbar_expect_tx(&w_full[s], R4_WBYTES);
          r4_box(sw + s * R4_WBYTES, second ? &map_w1 : &map_w0, n0, kb * (R4_K / 2), &w_full[s]);
          if (++s == WST) s = 0, ph ^= 1u;
        }
        if (++kb == steps) kb = 0, ++tile;
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc_bf16(128, MP);
      const uint64_t xd = smem_desc_sw128(smem_u32(sx));
      bool ok = true;
      int s = 0, buf = 0, kb = kb0, seg = 0;
      uint32_t ph = 0, aph = 0;
      for (int i = 0; i < n; ++i) {
        const bool begin = i == 0 || kb == 0;
        if (begin && !(ok = b4_wait(&d_empty[seg & 1], (uint32_t)((seg >> 1) & 1) ^ 1u, s_fail, p.word, 3))) break;
        if (!(ok = b4_spin(&x_full[s], ph, s_fail, p.word, 5) && b4_spin(&a_ready[buf], aph, s_fail, p.word, 4))) break;
        tc_fence_after();
        const uint64_t bd = xd + (uint64_t)(s * (XB >> 4));
        const uint32_t d = tmem + (uint32_t)((seg & 1) * MP);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          b4_mma(d, tmem + TM_A + 64u * buf + 8u * k, bd + (uint64_t)((k >> 2) * (XB >> 5) + 2 * (k & 3)), idesc, !begin || k != 0 ? 1u : 0u);
        umma_commit(&a_free[buf]);
        umma_commit(&x_empty[s]);
        if (++s == XST) s = 0, ph ^= 1u;
        if (++buf == NA) buf = 0, aph ^= 1u;
        if (++kb == steps || i == n - 1) {
          umma_commit(&d_full[seg & 1]);
          kb = 0;
          ++seg;
        }
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 3) {
    // windows of four steps of a tile: their numbers lie side by side; the next window's are on their way while these are handed over
    bool ok = true;
    int s = 0;
    uint32_t ph = 1;
    auto fetch = [&](int tile, int kb, uint2 (&sv)[4], uint2 (&zv)[4]) {
      const bool second = tile >= p.ntiles;
      const int n0 = (second ? tile - p.ntiles : tile) * 128;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const size_t row = (size_t)min(n0 + q * 32 + lane, p.N - 1) * p.G;
        sv[q] = r4_four(second ? p.scales[1] : p.scales[0], row, kb, steps, p.G, p.steps_per_group, p.wide);
        zv[q] = r4_four(second ? p.zeros[1] : p.zeros[0], row, kb, steps, p.G, p.steps_per_group, p.wide);
      }
    };
    uint2 sv[4], zv[4];
    int tile = tile0, kb = kb0 & ~3, skip = kb0 & 3, i = 0;
    if (n > 0) fetch(tile, kb, sv, zv);
    while (ok && i < n) {
      uint2 sn[4], zn[4];
      int nt = tile, nk = kb + 4;
      if (nk >= steps) nk = 0, ++nt;
      if (i + min(4, steps - kb) - skip < n) fetch(nt, nk, sn, zn);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j < skip || kb + j >= steps || i >= n) continue;
        ok = __all_sync(0xffffffffu, b4_wait(&w_empty[s], ph, s_fail, p.word, 11));
        if (!ok) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) reinterpret_cast<uint32_t*>(sz + s * R4_SZ)[q * 32 + lane] = r4_word(j, sv[q], zv[q]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_full[s]);
        if (++s == WST) s = 0, ph ^= 1u;
        ++i;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) sv[q] = sn[q], zv[q] = zn[q];
      tile = nt, kb = nk, skip = 0;
    }
  } else {
    constexpr int ROWS = MP / B4_GROUPS;
    const int quarter = warp & 3, grp = (warp - 4) >> 2;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const R4Row<128> row(lane);
    bool ok = true;
    // a finished tile: a quarter of the rows of the warp's 32 columns
    auto drain = [&](int seg) {
      ok = __all_sync(0xffffffffu, b4_wait(&d_full[seg & 1], (uint32_t)(seg >> 1) & 1u, s_fail, p.word, 6));
      if (!ok) return;
      tc_fence_after();
      uint32_t v[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; r += 4) b4_ld4(tmem + lanes + (uint32_t)((seg & 1) * MP + grp * ROWS + r), v + r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int r = 0; r < ROWS; ++r) asm volatile("" : "+r"(v[r]));          // (the loads' results are there from here on)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&d_empty[seg & 1]);
      float* dst = p.part + (((size_t)blockIdx.x * p.slots + seg) * MP + grp * ROWS) * 128 + quarter * 32 + lane;
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (grp * ROWS + r < p.M) dst[(size_t)r * 128] = __uint_as_float(v[r]);
    };
    // the group's steps: every fourth of the range
    const int segs = n > 0 ? (kb0 + n - 1) / steps + 1 : 0;
    int i = grp, kb = kb0 + grp, seg = 0, drained = 0, s = grp, buf = grp;
    uint32_t wph = 0, aph = 1;
    while (kb >= steps) kb -= steps, ++seg;
    while (ok && drained < segs) {
      int upto = segs;                       // segments before this one can be drained
      if (i < n) {
        upto = seg;
        ok = b4_wait(&w_full[s], wph, s_fail, p.word, 7);
        if (ok) ok = b4_wait(&a_free[buf], aph, s_fail, p.word, 8);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;
        tc_fence_after();
        r4_unpack_step<128>(smem_u32(sw + s * R4_WBYTES), (uint32_t)(quarter * 32), row, smem_u32(sz + s * R4_SZ) + (uint32_t)(quarter * 128),
                            tmem + lanes + TM_A + 64u * buf);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_empty[s]), mbar_arrive(&a_ready[buf]);
        i += B4_GROUPS;
        kb += B4_GROUPS;
        while (kb >= steps) kb -= steps, ++seg;
        if ((s += B4_GROUPS) >= WST) s -= WST, wph ^= 1u;
        if ((buf += B4_GROUPS) >= NA) buf -= NA, aph ^= 1u;
      }
      while (ok && drained < upto) drain(drained++);
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// A tile's partial sums, in the order of k: eight rows x 128 columns a block, a row per warp, four columns per thread.
template <bool GATED>
__global__ void __launch_bounds__(256) int4_batch_sum_kernel(const float* __restrict__ part, const __nv_bfloat16* __restrict__ b0,
                                                             const __nv_bfloat16* __restrict__ b1, __nv_bfloat16* __restrict__ y, int M, int N,
                                                             int steps, int ntiles, int total, int ranges, int slots, int mp) {
  pdl_wait();
  pdl_launch_dependents();
  part = after_wait(part);
  const int m = blockIdx.y * 8 + (threadIdx.x >> 5), col = (threadIdx.x & 31) * 4, n = blockIdx.x * 128 + col;
  if (m >= M || n >= N) return;
  auto sum = [&](int tile) {
    // the ranges that hold steps tile * steps .. + steps - 1; all but the first begin inside the tile, which is then their first
    const int a = tile * steps, c0 = (int)(((long long)(a + 1) * ranges - 1) / total), c1 = (int)(((long long)(a + steps) * ranges - 1) / total);
    const int slot = tile - b4_first(c0, total, ranges) / steps;
    const float* src = part + (size_t)m * 128 + col;
    const size_t tile_size = (size_t)mp * 128;
    float4 acc = __ldcg(reinterpret_cast<const float4*>(src + ((size_t)c0 * slots + slot) * tile_size));
    for (int c = c0 + 1; c <= c1; c += 4) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)min(c + u, c1) * slots * tile_size));
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + u <= c1) acc.x += v[u].x, acc.y += v[u].y, acc.z += v[u].z, acc.w += v[u].w;
    }
    return acc;
  };
  auto biased = [&](float4 v, const __nv_bfloat16* b) {
    if (b != nullptr)
      v.x += __bfloat162float(b[n]), v.y += __bfloat162float(b[n + 1]), v.z += __bfloat162float(b[n + 2]), v.w += __bfloat162float(b[n + 3]);
    return v;
  };
  float4 o = biased(sum(blockIdx.x), b0);
  if (GATED) {
    const float4 u = biased(sum(ntiles + blockIdx.x), b1);
    o.x = __fmul_rn(silu_act<__nv_bfloat16>(bf16r(o.x)), bf16r(u.x)), o.y = __fmul_rn(silu_act<__nv_bfloat16>(bf16r(o.y)), bf16r(u.y));
    o.z = __fmul_rn(silu_act<__nv_bfloat16>(bf16r(o.z)), bf16r(u.z)), o.w = __fmul_rn(silu_act<__nv_bfloat16>(bf16r(o.w)), bf16r(u.w));
  }
  *reinterpret_cast<uint2*>(y + (size_t)m * N + n) = make_uint2(pack_bf16(o.x, o.y), pack_bf16(o.z, o.w));
}

int b4_mp(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128; }
// steps of all tiles, ranges they are cut into (at least four steps each), partial tiles a range can touch
struct B4Plan {
  int ntiles, steps, total, ranges, slots;
};
B4Plan b4_plan(int N, int K, int layers, int grid) {
  B4Plan q;
  q.ntiles = (N + 127) / 128, q.steps = K / R4_K, q.total = layers * q.ntiles * q.steps;
  const int sms = grid > 0 ? grid : sm_count() > 0 ? sm_count() : 148, most = (q.total + 3) / 4;
  q.ranges = sms < most ? sms : most;
  q.slots = ((q.total + q.ranges - 1) / q.ranges + q.steps - 2) / q.steps + 1;
  return q;
}

template <int MP>
int b4_launch(const uint8_t* qw0, const uint8_t* qw1, const void* x, const B4Params& p, int K, const B4Plan& q, cudaStream_t st) {
  CUtensorMap m0, m1, mx;
  if (int r = r4_weight_map(qw0, p.N, K, 128, &m0)) return r;
  if (int r = r4_weight_map(qw1, p.N, K, 128, &m1)) return r;
  if (int r = make_map(x, p.M, K, MP, &mx)) return r;
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(int4_batch_kernel<MP>, cudaFuncAttributeMaxDynamicSharedMemorySize, b4_smem(MP)));
    configured.mark();
  }
  LL_CUDA(launch(int4_batch_kernel<MP>, dim3(q.ranges), dim3(B4_THREADS), b4_smem(MP), st, true, m0, m1, mx, p));
  LL_LAUNCH_OK("int4_batch_kernel");
  return LL_OK;
}

int b4_run(const uint8_t* qw0, const uint8_t* qw1, const void* x, const void* b0, const void* b1, void* y, B4Params p, int K, int group, bool gated,
           int grid, cudaStream_t st) {
  if (!ll_int4_rows_supported(p.N, K, group)) {
    set_error("int4_batch needs N %% 16 == 0 and group %% 128 == 0 (N=%d K=%d group=%d)", p.N, K, group);
    return LL_ERR_UNSUPPORTED;
  }
  LL_CHECK_ARG(p.M >= 1 && p.M <= 128, "int4_batch: 1 to 128 rows (got %d)", p.M);
  LL_CHECK_ARG((((uintptr_t)qw0 | (uintptr_t)qw1 | (uintptr_t)x | (uintptr_t)y | (uintptr_t)p.part) & 15) == 0,
               "int4_batch: packed weights, x, y and scratch must be 16-byte aligned");
  LL_CHECK_ARG((long long)(gated ? 2 : 1) * ((p.N + 127) / 128) * (K / R4_K) < (1ll << 30) && grid >= 0, "int4_batch: too many steps");
  const B4Plan q = b4_plan(p.N, K, gated ? 2 : 1, grid);
  p.steps = q.steps, p.G = K / group, p.steps_per_group = group / R4_K, p.ntiles = q.ntiles, p.total = q.total, p.slots = q.slots;
  p.wide = r4_wide(p.scales[0], p.zeros[0], p.scales[1], p.zeros[1], p.G, p.steps_per_group);
  p.word = wait_word();
  const int mp = b4_mp(p.M);
  int r;
  if (mp == 16) r = b4_launch<16>(qw0, qw1, x, p, K, q, st);
  else if (mp == 32) r = b4_launch<32>(qw0, qw1, x, p, K, q, st);
  else if (mp == 64) r = b4_launch<64>(qw0, qw1, x, p, K, q, st);
  else r = b4_launch<128>(qw0, qw1, x, p, K, q, st);
  if (r) return r;
  LL_CUDA(launch(gated ? int4_batch_sum_kernel<true> : int4_batch_sum_kernel<false>, dim3(q.ntiles, (p.M + 7) / 8), dim3(256), 0, st, true,
                 (const float*)p.part, (const __nv_bfloat16*)b0, (const __nv_bfloat16*)b1, (__nv_bfloat16*)y, p.M, p.N, q.steps, q.ntiles, q.total, q.ranges,
                 q.slots, mp));
  LL_LAUNCH_OK("int4_batch_sum_kernel");
  return LL_OK;
}

}  // namespace
}  // namespace llb

using namespace llb;

extern "C" {

size_t ll_int4_batch_scratch_bytes(int M, int N, int K, int layers, int grid) {
  if (M < 1 || M > 128 || N <= 0 || K < R4_K || layers < 1 || layers > 2 || grid < 0) return 0;
  const B4Plan q = b4_plan(N, K, layers, grid);
  return (size_t)q.ranges * q.slots * b4_mp(M) * 128 * sizeof(float);
}

int ll_int4_batch(const uint8_t* qw, const void* scales, const void* zeros, const void* x, const void* bias, void* y, void* scratch, int M, int N, int K,
                  int group, int grid, ll_stream stream) {
  LL_CHECK_ARG(qw && scales && zeros && x && y && scratch, "int4_batch: null pointer");
  B4Params p{};
  p.scales[0] = p.scales[1] = (const __nv_bfloat16*)scales, p.zeros[0] = p.zeros[1] = (const __nv_bfloat16*)zeros;
  p.part = (float*)scratch, p.M = M, p.N = N;
  return b4_run(qw, qw, x, bias, nullptr, y, p, K, group, false, grid, (cudaStream_t)stream);
}

int ll_int4_batch_gated(const uint8_t* qw1, const void* scales1, const void* zeros1, const void* bias1, const uint8_t* qw2, const void* scales2,
                        const void* zeros2, const void* bias2, const void* x, void* h, void* scratch, int M, int N, int K, int group, int grid,
                        ll_stream stream) {
  LL_CHECK_ARG(qw1 && scales1 && zeros1 && qw2 && scales2 && zeros2 && x && h && scratch, "int4_batch_gated: null pointer");
  B4Params p{};
  p.scales[0] = (const __nv_bfloat16*)scales1, p.zeros[0] = (const __nv_bfloat16*)zeros1;
  p.scales[1] = (const __nv_bfloat16*)scales2, p.zeros[1] = (const __nv_bfloat16*)zeros2;
  p.part = (float*)scratch, p.M = M, p.N = N;
  return b4_run(qw1, qw2, x, bias1, bias2, h, p, K, group, true, grid, (cudaStream_t)stream);
}

// 0, or the code of the first bounded wait that ran out in this file's kernel.  Synchronises the device.
int ll_int4_batch_error(void) {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, g_b4_error, sizeof(int)) == cudaSuccess ? v : -1;
}

}  // extern "C"
