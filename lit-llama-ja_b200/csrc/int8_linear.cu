// llm.int8 (LLM.int8(), arXiv:2208.07339) Linear for sm_100a: row-wise int8 weight quantisation and the
// outlier-decomposed int8 x int8 -> int32 matmul.
// ref: lit_llama/quantization.py:36-75 (Linear8bitLt over bitsandbytes, has_fp16_weights=False,
// threshold=6.0).  bitsandbytes itself is un-vendored and unpinned in the reference, so the arithmetic follows
// the published algorithm as restated in oracle/quant.py (int8_quantize_weight, int8_linear_forward):
//   A = x.half(); outlier columns = features with any |A| >= threshold;
//   SCA[m] = absmax over the entries of row m below the threshold; CA = rint(127 A / SCA), outlier columns 0;
//   C32 = CA . CB^T (int32, exact); out = fp16(C32 * SCA * SCB / 127^2 (+ bias));
//   out = fp16(out + fp16(A[:, idx] . fp16(CB[:, idx] * SCB / 127)^T)); cast to the input dtype.
// Up to 64 rows: HBM-bound on the int8 weight read (N*K bytes per layer).  One kernel prepares the activations (row maxima, outlier list,
// quantised rows), one streams the weights as the A operand of tcgen05 kind::i8 MMAs (128 output columns = the 128 TMEM lanes, int32
// accumulators) with K cut into ranges whose partial sums are stored, one adds them up (integers: exact in any order) and finishes.
// Prompts (M > 64): the same arithmetic per block of 64 rows (a feature is an outlier for a block of 64 rows), all blocks at once: row
// statistics, quantised rows, outlier lists, then one 128 x 128-tiled product and one finishing kernel.  See int8_gemm_tc_kernel.
#include "tcgen05.cuh"

namespace llb {
namespace {

template <typename T> __device__ __forceinline__ float to_half_f32(T v);
template <> __device__ __forceinline__ float to_half_f32<float>(float v) { return __half2float(__float2half_rn(v)); }
template <> __device__ __forceinline__ float to_half_f32<__nv_bfloat16>(__nv_bfloat16 v) {
  return __half2float(__float2half_rn(__bfloat162float(v)));
}
template <> __device__ __forceinline__ float to_half_f32<__half>(__half v) { return __half2float(v); }

// ---------------------------------------------------------------- weight quantisation (load time)
template <typename T>
__global__ void int8_quant_weight_kernel(const T* __restrict__ w, int8_t* __restrict__ cb, float* __restrict__ scb, int K) {
  __shared__ float red[32];
  const T* row = w + (size_t)blockIdx.x * K;
  float mx = 0.f;
  for (int k = threadIdx.x; k < K; k += blockDim.x) mx = fmaxf(mx, fabsf(to_half_f32<T>(row[k])));
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    v = warp_max(v);
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  mx = red[0];
  if (threadIdx.x == 0) scb[blockIdx.x] = mx;
  const float inv = __fdiv_rn(127.f, mx == 0.f ? 1.f : mx);
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const float q = rintf(__fmul_rn(to_half_f32<T>(row[k]), inv));
    cb[(size_t)blockIdx.x * K + k] = (int8_t)fminf(fmaxf(q, -127.f), 127.f);
  }
}

// eight neighbouring activations as x.half() values in fp32; vec: on a 16-byte boundary
template <typename T> __device__ __forceinline__ void int8_load8(const T* p, float (&v)[8], int vec) {
  constexpr int P = 16 / sizeof(T);
  if (!vec) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_half_f32<T>(p[i]);
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; i += P) {
    const uint4 u = *reinterpret_cast<const uint4*>(p + i);
    const T* t = reinterpret_cast<const T*>(&u);
#pragma unroll
    for (int e = 0; e < P; ++e) v[i + e] = to_half_f32<T>(t[e]);
  }
}

// ================================================================================================== prompts: M > 64
// x.half() without storing it: sca[m] = absmax over the entries of row m below thr; flag[block of 64 rows][k] = 1 where any
// |entry| >= thr.  One CTA per row.
template <typename T>
__global__ void __launch_bounds__(256) int8_row_stats_kernel(const T* __restrict__ x, uint8_t* __restrict__ flag, float* __restrict__ sca, int K,
                                                            float thr, int vec) {
  __shared__ float red[8];
  const int m = blockIdx.x;
  const T* row = x + (size_t)m * K;
  uint8_t* fl = flag + (size_t)(m / 64) * K;
  float mx = 0.f;
  for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {      // (K is a multiple of 128)
    float v[8];
    int8_load8<T>(row + k, v, vec);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float a = fabsf(v[e]);
      if (a >= thr) fl[k + e] = 1;
      else mx = fmaxf(mx, a);
    }
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) mx = fmaxf(mx, red[w]);
    sca[m] = mx;
  }
}

// CA[m][k], eight entries per thread
template <typename T>
__global__ void __launch_bounds__(256) int8_row_quant_kernel(const T* __restrict__ x, const uint8_t* __restrict__ flag, const float* __restrict__ sca,
                                                            int8_t* __restrict__ ca, int K, float thr, long long pieces, int vec) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= pieces) return;
  const int per = K / 8, m = (int)(i / per), k = (int)(i - (long long)m * per) * 8;
  float v[8];
  int8_load8<T>(x + (size_t)m * K + k, v, vec);
  const uint2 f = *reinterpret_cast<const uint2*>(flag + (size_t)(m / 64) * K + k);
  const float s = sca[m], inv = __fdiv_rn(127.f, s == 0.f ? 1.f : s);
  uint32_t o[2] = {0u, 0u};
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const uint32_t out = ((e < 4 ? f.x : f.y) >> (8 * (e & 3))) & 0xffu;
    float q = 0.f;
    if (out == 0u && fabsf(v[e]) < thr) q = fminf(fmaxf(rintf(__fmul_rn(v[e], inv)), -127.f), 127.f);
    o[e >> 2] |= ((uint32_t)(int)q & 0xffu) << (8 * (e & 3));
  }
  *reinterpret_cast<uint2*>(ca + (size_t)m * K + k) = make_uint2(o[0], o[1]);
}

// ascending outlier list of every block of 64 rows; one CTA per block
__global__ void __launch_bounds__(1024) int8_lists_kernel(const uint8_t* __restrict__ flag, int32_t* __restrict__ idx, int32_t* __restrict__ count, int K) {
  __shared__ int s_warp[32];
  const uint8_t* fl = flag + (size_t)blockIdx.x * K;
  int32_t* list = idx + (size_t)blockIdx.x * K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  for (int k0 = 0; k0 < K; k0 += 4096) {             // a thread looks at four neighbouring columns
    const int k = k0 + threadIdx.x * 4;
    const uint32_t f = k < K ? *reinterpret_cast<const uint32_t*>(fl + k) : 0u;
    const int n = __popc(f);
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int at = base + incl - n, total = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) at += s_warp[w];
      total += s_warp[w];
    }
    for (int e = 0; e < 4; ++e)
      if ((f >> (8 * e)) & 1u) list[at++] = k + e;
    base += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) count[blockIdx.x] = base;
}

// C32[M][N] = CA[M][K] . CB[N][K]^T on tcgen05 (kind::i8, K = 32 an instruction).  A CTA owns 128 x 128 outputs: TMA producer, one issuing
// thread, four epilogue warps; tiles of 128 x 128 bytes in a ring of three, so that two CTAs share an SM (one's first loads and epilogue run
// under the other's products).  A 7B feed-forward of 512 rows: 24 passes of 64 rows through mma.sync, four kernels each, took 1435 us on the
// device (the weights read eight times, the accumulator added up by atomics); three products of 40 us and 28 us around each make 211 us.
// Every wait is bounded; one that runs out records a code, the roles stop and tensor memory is freed.
constexpr int I8_BN = 128, I8_STAGES = 3, I8_BOX = 128 * 128;
constexpr uint32_t I8_WAIT_LIMIT = 1u << 20;
__device__ int g_int8_tc_error = 0;

__device__ __forceinline__ bool i8_wait(uint64_t* bar, uint32_t parity, volatile int* fail, int* word, int code) {
  for (uint32_t i = 0; i < I8_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *fail) return false;
  }
  *fail = 1;
  atomicCAS(&g_int8_tc_error, 0, code);
  wait_ran_out(word, 300 + code);
  return false;
}
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void i8_box(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
               "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}

__global__ void __launch_bounds__(192, 2) int8_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                                                             int32_t* __restrict__ c, int M, int N, int K, int* word) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t *sa = base, *sb = base + I8_STAGES * I8_BOX;
  uint64_t* full = reinterpret_cast<uint64_t*>(sb + I8_STAGES * I8_BOX);
  uint64_t* empty = full + I8_STAGES;
  uint64_t* done = empty + I8_STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done + 1);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * I8_BN, nkb = K / 128;      // (x runs over the rows: CTAs side by side share weights)
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_b);
    for (int i = 0; i < I8_STAGES; ++i) mbar_init(&full[i], 1), mbar_init(&empty[i], 1);
    mbar_init(done, 1);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_ptr, I8_BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % I8_STAGES;
        if (!(ok = i8_wait(&empty[s], ((kb / I8_STAGES) & 1) ^ 1, s_fail, word, 1))) break;
        mbar_expect_tx(&full[s], 2 * I8_BOX);
        i8_box(sa + s * I8_BOX, &map_a, kb * 128, m0, &full[s]);
        i8_box(sb + s * I8_BOX, &map_b, kb * 128, n0, &full[s]);
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // D = int32 (2 at bit 4), A = B = signed int8 (1 at bits 7 and 10), both K-major
      constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(I8_BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint64_t ad = smem_desc_sw128(smem_u32(sa)), bd = smem_desc_sw128(smem_u32(sb));
      bool ok = true;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % I8_STAGES;
        if (!(ok = i8_wait(&full[s], (kb / I8_STAGES) & 1, s_fail, word, 2))) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_i8(tmem, ad + (uint64_t)(s * (I8_BOX >> 4) + 2 * k), bd + (uint64_t)(s * (I8_BOX >> 4) + 2 * k), idesc, (kb | k) != 0 ? 1u : 0u);
        umma_commit(&empty[s]);
      }
      umma_commit(done);             // also after a failure: the epilogue's wait ends
      if (!ok) let_issued_work_end();
    }
  } else {
    const int quarter = warp & 3, m = m0 + quarter * 32 + lane;
    const bool ok = __all_sync(0xffffffffu, i8_wait(done, 0, s_fail, word, 3) && *(volatile int*)s_fail == 0);
    tc_fence_after();
    if (ok) {
#pragma unroll 1
      for (int c0 = 0; c0 < I8_BN; c0 += 32) {
        if (n0 + c0 >= N) break;
        uint32_t v[32];
        tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
        if (m < M) {
          int32_t* dst = c + (size_t)m * N + n0 + c0;
          if (n0 + c0 + 32 <= N && (N & 3) == 0) {
#pragma unroll
            for (int e = 0; e < 32; e += 4)
              *reinterpret_cast<int4*>(dst + e) = make_int4((int)v[e], (int)v[e + 1], (int)v[e + 2], (int)v[e + 3]);
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (n0 + c0 + e < N) dst[e] = (int)v[e];
          }
        }
        __syncwarp();                // the next load from tensor memory is the whole warp's
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, I8_BN);
  }
}

// out = fp16(C32 SCA SCB / 127^2 (+ bias)), plus fp16 of the outlier part, for 64 columns x ROWS rows (of one outlier list) per CTA.  C32 is
// the sum of `parts` partial sums, `part` numbers apart.
// Outlier part: the weights and activations of L outliers at a time stand in shared memory as fp32, already rounded; the next L are asked
// for (all list entries, then all they point to) before these are added.  64 rows: a thread owns four columns of four rows, two 16-byte
// reads for 16 multiply-adds.  16 rows: a list of up to L is added by a thread per row and four columns; a longer one is shared among the
// quarters of the threads, four columns of four rows each, a quarter of every L, whose sums are added in order.  Four CTAs an SM:
// a batch of 64 rows has 688 of them for 11008 columns.
// Three layers of a 4096-wide feed-forward, 32 rows whose inputs have 6 / 30 / 100 / 200 outlier features (their products up to thousands):
// 78 / 121 / 424 / 519 us a call on the device.  32 outliers at a time, each weight behind its own list entry: 78 / 259 / 1725 / 2131; the
// kernel beside the mma.sync product: 123 / 181 / 536 / 647.  (A stage of 128 leaves three CTAs an SM: 87 with 12 outliers, 84 with 64.)
template <typename T, int ROWS>
__global__ void __launch_bounds__(256, 4) int8_finish_rows_kernel(const int32_t* __restrict__ c32, int parts, size_t part, const float* __restrict__ sca,
                                                              const float* __restrict__ scb, const T* __restrict__ bias, const T* __restrict__ x,
                                                              const int8_t* __restrict__ cb, const int8_t* __restrict__ cbt,
                                                              const int32_t* __restrict__ idx, const int32_t* __restrict__ count,
                                                              T* __restrict__ y, int M, int N, int K) {
  static_assert(ROWS == 16 || ROWS == 64, "rows of a CTA");
  constexpr int SL = 64 / ROWS, L = SL == 1 ? 32 : 64, NW = L * 16 / 256, NA = L * ROWS / 256, AS = 256 / ROWS;   // SL: shares of the list
  __shared__ __align__(16) float w_s[L][64], a_s[L][ROWS];
  const int tid = threadIdx.x, n0 = blockIdx.x * 64, m0 = blockIdx.y * ROWS, blk = m0 / 64, col = (tid & 15) * 4;
  const int cnt = count[blk];
  float acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
  if (cnt > 0) {
    const int32_t* list = idx + (size_t)blk * K;
    // what a thread brings: four columns of NW outliers' weights, one row of NA outliers' activations.  Entries past the list's end, columns
    // past N and rows past M repeat the last one: they are never added, or added to what nobody stores.  Steps that lie past the end for the
    // whole CTA are left out (a gather from every row each: 512 rows with six outliers, three layers: 264 us a call with them, 244 without).
    const int wi = tid >> 4, ai = tid / ROWS;
    const T* xr = x + (size_t)min(m0 + (tid & (ROWS - 1)), M - 1) * K;
    const bool words = cbt != nullptr && (N & 3) == 0 && ((uintptr_t)cbt & 3) == 0;
    float sb127[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) sb127[j] = __fdiv_rn(scb[min(n0 + col + j, N - 1)], 127.f);
    uint32_t q[NW];
    float av[NA];
    auto fetch = [&](int b) {
      int kw[NW], ka[NA];
#pragma unroll
      for (int u = 0; u < NW; ++u) q[u] = 0u, kw[u] = b + 16 * u < cnt ? __ldg(list + min(b + wi + 16 * u, cnt - 1)) : 0;
#pragma unroll
      for (int u = 0; u < NA; ++u) av[u] = 0.f, ka[u] = b + AS * u < cnt ? __ldg(list + min(b + ai + AS * u, cnt - 1)) : 0;
      if (words) {
        const int8_t* src = cbt + min(n0 + col, N - 4);
#pragma unroll
        for (int u = 0; u < NW; ++u)
          if (b + 16 * u < cnt) q[u] = __ldg(reinterpret_cast<const uint32_t*>(src + (size_t)kw[u] * N));
      } else {
#pragma unroll
        for (int u = 0; u < NW; ++u) {
          if (b + 16 * u >= cnt) continue;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int n = min(n0 + col + j, N - 1);
            const int8_t v = cbt != nullptr ? __ldg(cbt + (size_t)kw[u] * N + n) : __ldg(cb + (size_t)n * K + kw[u]);
            q[u] |= (uint32_t)(uint8_t)v << (8 * j);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < NA; ++u)
        if (b + AS * u < cnt) av[u] = to_half_f32<T>(xr[ka[u]]);
    };
    auto stage = [&]() {
#pragma unroll
      for (int u = 0; u < NW; ++u) {
        float w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = __half2float(__float2half_rn(__fmul_rn((float)(int8_t)(q[u] >> (8 * j)), sb127[j])));
        *reinterpret_cast<float4*>(&w_s[wi + 16 * u][col]) = make_float4(w[0], w[1], w[2], w[3]);
      }
#pragma unroll
      for (int u = 0; u < NA; ++u) a_s[ai + AS * u][tid & (ROWS - 1)] = av[u];
    };
    fetch(0);
    if (SL > 1 && cnt <= L) {
      stage();
      __syncthreads();
      const int row = tid >> 4;
#pragma unroll 4
      for (int i = 0; i < cnt; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(&w_s[i][col]);
        const float a = a_s[i][row];
        acc[0][0] = fmaf(a, w.x, acc[0][0]);
        acc[0][1] = fmaf(a, w.y, acc[0][1]);
        acc[0][2] = fmaf(a, w.z, acc[0][2]);
        acc[0][3] = fmaf(a, w.w, acc[0][3]);
      }
    } else {
      const int r0 = ((tid >> 4) & (ROWS / 4 - 1)) * 4, sl = tid / (256 / SL);
      for (int b = 0; b < cnt; b += L) {
        if (b > 0) __syncthreads();                        // the outliers before have been added
        stage();
        __syncthreads();
        if (b + L < cnt) fetch(b + L);
        const int i0 = sl * (L / SL), i1 = min(min(L, cnt - b), i0 + L / SL);
#pragma unroll 4
        for (int i = i0; i < i1; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(&w_s[i][col]), a4 = *reinterpret_cast<const float4*>(&a_s[i][r0]);
          const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            acc[r][0] = fmaf(a[r], w.x, acc[r][0]);
            acc[r][1] = fmaf(a[r], w.y, acc[r][1]);
            acc[r][2] = fmaf(a[r], w.z, acc[r][2]);
            acc[r][3] = fmaf(a[r], w.w, acc[r][3]);
          }
        }
      }
      if (SL > 1) {                                        // every thread finishes one row: its sums come through shared memory
        __syncthreads();
        float* sums = &w_s[0][0];                          // [SL][ROWS][64]
#pragma unroll
        for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(sums + (sl * ROWS + r0 + r) * 64 + col) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        __syncthreads();
        const int row = tid >> 4;
        float4 o = *reinterpret_cast<const float4*>(sums + row * 64 + col);
#pragma unroll
        for (int z = 1; z < SL; ++z) {
          const float4 v = *reinterpret_cast<const float4*>(sums + (z * ROWS + row) * 64 + col);
          o.x += v.x, o.y += v.y, o.z += v.z, o.w += v.w;
        }
        acc[0][0] = o.x, acc[0][1] = o.y, acc[0][2] = o.z, acc[0][3] = o.w;
      }
    }
  }
  constexpr int R = ROWS / 16;                             // rows a thread finishes
  const int n = n0 + col, fr = (tid >> 4) * R;
  if (n >= N) return;
  float sb[4], bv[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    sb[j] = n + j < N ? scb[n + j] : 0.f;
    bv[j] = n + j < N && bias != nullptr ? to_half_f32<T>(bias[n + j]) : 0.f;
  }
  const bool vec = n + 4 <= N && (N & 3) == 0;             // (then a partial sum starts on a 16-byte boundary too)
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int m = m0 + fr + r;
    if (m >= M) break;
    const float sa = sca[m];
    const size_t at = (size_t)m * N + n;
    int cv[4] = {0, 0, 0, 0};
    for (int z = 0; z < parts; ++z) {
      const int32_t* src = c32 + (size_t)z * part + at;
      if (vec) {
        const int4 v = __ldcs(reinterpret_cast<const int4*>(src));
        cv[0] += v.x, cv[1] += v.y, cv[2] += v.z, cv[3] += v.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) cv[j] += n + j < N ? src[j] : 0;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (n + j >= N) break;
      float out = __fmul_rn(__fmul_rn(__fmul_rn((float)cv[j], sa), sb[j]), 1.0f / (127.0f * 127.0f));
      if (bias != nullptr) out = __fadd_rn(out, bv[j]);
      out = __half2float(__float2half_rn(out));
      if (cnt > 0) out = __half2float(__float2half_rn(__fadd_rn(out, __half2float(__float2half_rn(acc[r][j])))));
      dt<T>::st(y, at + j, out);
    }
  }
}

constexpr int I8_PASS = 1024;        // rows of one pass: bounds the int32 product (57 MB at 13824 columns)
struct WsRows {
  int8_t* ca; int32_t* c32; uint8_t* flag; int32_t* idx; float* sca; int32_t* count;
  size_t flag_bytes, total;
};
WsRows carve_rows(void* base, int M, int N, int K) {
  WsRows w;
  const int rows = M < I8_PASS ? M : I8_PASS, blocks = (rows + 63) / 64;
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o += (b + 255) & ~(size_t)255; return r; };
  uint8_t* p = (uint8_t*)base;
  w.ca = (int8_t*)(p + take((size_t)rows * K));
  w.c32 = (int32_t*)(p + take((size_t)rows * N * 4));
  w.flag_bytes = (size_t)blocks * K;
  w.flag = (uint8_t*)(p + take(w.flag_bytes));
  w.idx = (int32_t*)(p + take((size_t)blocks * K * 4));
  w.sca = (float*)(p + take((size_t)rows * 4));
  w.count = (int32_t*)(p + take((size_t)blocks * 4));
  w.total = o;
  return w;
}

// [rows][K] int8 row-major -> 2-D map, boxes of box_rows x 128 bytes, 128-byte swizzle, rows past the end zero
int make_map_i8(const void* base, int rows, int K, int box_rows, CUtensorMap* out) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled entry point not available");
    return LL_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K};
  cuuint32_t box[2] = {128, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): int8 rows=%d K=%d", (int)r, rows, K);
    return LL_ERR_CUDA;
  }
  return LL_OK;
}

template <typename T>
int int8_rows_t(const T* x, const int8_t* cb, const int8_t* cbt, const float* scb, const T* bias, T* y, int M, int N, int K, float thr,
                void* ws_base, cudaStream_t st) {
  constexpr int smem = 2 * I8_STAGES * I8_BOX + (2 * I8_STAGES + 1) * 8 + 16 + 1024;
  LL_CUDA(cudaFuncSetAttribute(int8_gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const WsRows w = carve_rows(ws_base, M, N, K);
  const int vec = ((uintptr_t)x & 15) == 0;
  CUtensorMap ma, mb;
  if (int r = make_map_i8(cb, N, K, 128, &mb)) return r;
  for (int r0 = 0; r0 < M; r0 += I8_PASS) {
    const int rows = min(I8_PASS, M - r0), blocks = (rows + 63) / 64;
    const T* xp = x + (size_t)r0 * K;
    LL_CUDA(cudaMemsetAsync(w.flag, 0, w.flag_bytes, st));
    int8_row_stats_kernel<T><<<rows, 256, 0, st>>>(xp, w.flag, w.sca, K, thr, vec);
    const long long pieces = (long long)rows * (K / 8);
    int8_row_quant_kernel<T><<<(unsigned)((pieces + 255) / 256), 256, 0, st>>>(xp, w.flag, w.sca, w.ca, K, thr, pieces, vec);
    int8_lists_kernel<<<blocks, 1024, 0, st>>>(w.flag, w.idx, w.count, K);
    if (int r = make_map_i8(w.ca, rows, K, 128, &ma)) return r;
    int8_gemm_tc_kernel<<<dim3((rows + BM - 1) / BM, (N + I8_BN - 1) / I8_BN), 192, smem, st>>>(ma, mb, w.c32, rows, N, K, wait_word());
    int8_finish_rows_kernel<T, 64><<<dim3((N + 63) / 64, blocks), 256, 0, st>>>(w.c32, 1, 0, w.sca, scb, bias, xp, cb, cbt, w.idx, w.count,
                                                                           y + (size_t)r0 * N, rows, N, K);
    LL_LAUNCH_OK("int8 linear kernels (prompts)");
  }
  return LL_OK;
}

// ================================================================================================== up to 64 rows
// One kernel: x.half(), row maxima of the entries below thr, quantised rows, outlier columns as an ascending list.  A CTA owns a row and
// holds it in registers between its maximum and its codes (up to I8P_HELD * 4096 features; a longer row is read again).  Whether a column
// stands out in some row is known when every row is done, so the CTA that finishes last makes the list and clears the listed columns'
// codes.  No CTA waits for another: nothing says that all of them run at the same time.  (A CTA per 64 columns and one wait of the whole
// grid in the middle took 2 us less a layer, and stood still, or went on with counts that were not there, when other streams held the SMs.)
// 32 rows through a 7B feed-forward, three layers: 78 us on the device; 123 before the product ran on tcgen05.
constexpr int I8P_THREADS = 512, I8P_HELD = 4;
template <typename T>
__global__ void __launch_bounds__(I8P_THREADS) int8_prep_kernel(const T* __restrict__ x, int8_t* __restrict__ ca, float* __restrict__ sca,
                                                               uint8_t* __restrict__ flag, int32_t* __restrict__ idx, int32_t* __restrict__ count,
                                                               int32_t* __restrict__ arrive, int K, float thr, int vec) {
  constexpr int WARPS = I8P_THREADS / 32, STEP = I8P_THREADS * 8;
  __shared__ float s_max[WARPS];
  __shared__ int s_warp[WARPS], s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, M = gridDim.x;
  const T* row = x + (size_t)blockIdx.x * K;
  float held[I8P_HELD][8], mx = 0.f;
#pragma unroll
  for (int i = 0; i < I8P_HELD; ++i)
    if (i * STEP + tid * 8 < K) int8_load8<T>(row + i * STEP + tid * 8, held[i], vec);      // (K is a multiple of 128)
  auto look = [&](const float (&v)[8], int k) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float a = fabsf(v[e]);
      if (a >= thr) flag[k + e] = 1;                         // (several rows may store the same 1)
      else mx = fmaxf(mx, a);
    }
  };
#pragma unroll
  for (int i = 0; i < I8P_HELD; ++i)
    if (i * STEP + tid * 8 < K) look(held[i], i * STEP + tid * 8);
  for (int k = I8P_HELD * STEP + tid * 8; k < K; k += STEP) {
    float v[8];
    int8_load8<T>(row + k, v, vec);
    look(v, k);
  }
  mx = warp_max(mx);
  if (lane == 0) s_max[warp] = mx;
  __syncthreads();
  mx = s_max[0];
#pragma unroll
  for (int w = 1; w < WARPS; ++w) mx = fmaxf(mx, s_max[w]);
  if (tid == 0) sca[blockIdx.x] = mx;
  const float inv = __fdiv_rn(127.f, mx == 0.f ? 1.f : mx);
  auto codes = [&](const float (&v)[8], int k) {
    uint32_t o[2] = {0u, 0u};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float q = 0.f;
      if (fabsf(v[e]) < thr) q = fminf(fmaxf(rintf(__fmul_rn(v[e], inv)), -127.f), 127.f);
      o[e >> 2] |= ((uint32_t)(int)q & 0xffu) << (8 * (e & 3));
    }
    *reinterpret_cast<uint2*>(ca + (size_t)blockIdx.x * K + k) = make_uint2(o[0], o[1]);
  };
#pragma unroll
  for (int i = 0; i < I8P_HELD; ++i)
    if (i * STEP + tid * 8 < K) codes(held[i], i * STEP + tid * 8);
  for (int k = I8P_HELD * STEP + tid * 8; k < K; k += STEP) {
    float v[8];
    int8_load8<T>(row + k, v, vec);
    codes(v, k);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(arrive, 1) == M - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  int base = 0;
  for (int k0 = 0; k0 < K; k0 += I8P_THREADS * 32) {         // a thread looks at 32 neighbouring columns
    const int k = k0 + tid * 32;
    uint32_t f[8];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint4 u = k < K ? __ldcg(reinterpret_cast<const uint4*>(flag + k) + j) : make_uint4(0u, 0u, 0u, 0u);
      f[4 * j] = u.x, f[4 * j + 1] = u.y, f[4 * j + 2] = u.z, f[4 * j + 3] = u.w;
    }
    int n = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) n += __popc(f[j]);
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int at = base + incl - n, total = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const int c = s_warp[w];
      if (w < warp) at += c;
      total += c;
    }
    if (n > 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        for (int e = 0; e < 4; ++e)
          if ((f[j] >> (8 * e)) & 1u) idx[at++] = k + 4 * j + e;
    }
    base += total;
    __syncthreads();
  }
  if (tid == 0) *count = base;
  // (the list is complete: a barrier of this CTA, which wrote it, lies behind the last entry)
  for (int i = tid; i < base * M; i += I8P_THREADS) {
    const int m = i / base;
    ca[(size_t)m * K + idx[i - m * base]] = 0;
  }
}

// part[range][m][n] = the sum over the range's k of CA[m][k] CB[n][k]: the weights are the A operand (128 output columns a CTA), streamed
// through a ring of 16 KB boxes; two CTAs share an SM.  MP: rows rounded up to 16, 32, 48 or 64.
// A batch of 32 through a 7B feed-forward: mma.sync straight from global memory, two loads in flight a thread and int32 atomics, took 17.5 us
// a layer (2.6 TB/s of weights) and the preparation beside it 9.4 us, the finish 10 us.
constexpr int i8c_stages(int mp) { return mp > 32 ? 4 : 5; }
constexpr int i8c_smem(int mp) { return i8c_stages(mp) * (I8_BOX + mp * 128) + 256 + 1024; }
template <int MP>
__global__ void __launch_bounds__(192, 2) int8_columns_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                int32_t* __restrict__ part, int M, int N, int nkb, int per, int* word) {
  constexpr int STAGES = i8c_stages(MP), XB = MP * 128, COLS = MP <= 32 ? 32 : 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t *sw = base, *sx = base + STAGES * I8_BOX;
  uint64_t* full = reinterpret_cast<uint64_t*>(sx + STAGES * XB);
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(done + 1);
  int* s_fail = reinterpret_cast<int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * 128, kb0 = blockIdx.y * per, kb1 = min(kb0 + per, nkb);
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_x);
    for (int i = 0; i < STAGES; ++i) mbar_init(&full[i], 1), mbar_init(&empty[i], 1);
    mbar_init(done, 1);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_ptr, COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      int s = 0;
      uint32_t ph = 1;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = i8_wait(&empty[s], ph, s_fail, word, 5))) break;
        mbar_expect_tx(&full[s], I8_BOX + XB);
        i8_box(sw + s * I8_BOX, &map_w, kb * 128, n0, &full[s]);
        i8_box(sx + s * XB, &map_x, kb * 128, 0, &full[s]);
        if (++s == STAGES) s = 0, ph ^= 1u;
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MP >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint64_t wd = smem_desc_sw128(smem_u32(sw)), xd = smem_desc_sw128(smem_u32(sx));
      bool ok = true;
      int s = 0;
      uint32_t ph = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = i8_wait(&full[s], ph, s_fail, word, 6))) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_i8(tmem, wd + (uint64_t)(s * (I8_BOX >> 4) + 2 * k), xd + (uint64_t)(s * (XB >> 4) + 2 * k), idesc, kb != kb0 || k != 0 ? 1u : 0u);
        umma_commit(&empty[s]);
        if (++s == STAGES) s = 0, ph ^= 1u;
      }
      umma_commit(done);             // also after a failure: the epilogue's wait ends
      if (!ok) let_issued_work_end();
    }
  } else {
    const int quarter = warp & 3, n = n0 + quarter * 32 + lane;
    const bool ok = __all_sync(0xffffffffu, i8_wait(done, 0, s_fail, word, 7) && *(volatile int*)s_fail == 0);
    tc_fence_after();
    if (ok) {
      int32_t* dst = part + (size_t)blockIdx.y * M * N + n;
#pragma unroll
      for (int c0 = 0; c0 < COLS; c0 += 32) {
        uint32_t v[32];
        tmem_ld_32x32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
        for (int e = 0; e < 32; ++e)
          if (c0 + e < M && n < N) dst[(size_t)(c0 + e) * N] = (int)v[e];
        __syncwarp();                // the next load from tensor memory is the whole warp's
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, COLS);
  }
}

// ranges of k (per: blocks of 128 in each): every CTA of the grid resident at two an SM, if the columns alone do not fill the device
int i8c_ranges(int N, int K, int sms, int* per) {
  const int tiles = (N + 127) / 128, nkb = K / 128;
  int ranges = 2 * (sms > 0 ? sms : 148) / tiles;
  ranges = ranges < 1 ? 1 : ranges > nkb ? nkb : ranges;
  *per = (nkb + ranges - 1) / ranges;
  return (nkb + *per - 1) / *per;
}

struct Ws {
  int8_t* ca; int32_t* part; float* sca; int32_t* idx; uint8_t* flag; int32_t* count; int32_t* arrive;
  size_t zero_off, zero_bytes, total;
};
Ws carve(void* base, int M, int N, int K) {
  Ws w;
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o += (b + 255) & ~(size_t)255; return r; };
  uint8_t* p = (uint8_t*)base;
  int per;
  w.ca = (int8_t*)(p + take((size_t)M * K));
  w.part = (int32_t*)(p + take((size_t)i8c_ranges(N, K, sm_count(), &per) * M * N * 4));
  w.idx = (int32_t*)(p + take((size_t)K * 4));
  w.sca = (float*)(p + take(64 * 4));
  w.zero_off = o;  // cleared at the start of every call
  w.flag = p + take((size_t)K);
  w.count = (int32_t*)(p + take(4));
  w.arrive = (int32_t*)(p + take(4));
  w.zero_bytes = o - w.zero_off;
  w.total = o;
  return w;
}

template <int MP>
int i8c_launch(const CUtensorMap& mw, const Ws& w, int M, int N, int K, int sms, cudaStream_t st) {
  CUtensorMap mx;
  if (int r = make_map_i8(w.ca, M, K, MP, &mx)) return r;
  LL_CUDA(cudaFuncSetAttribute(int8_columns_tc_kernel<MP>, cudaFuncAttributeMaxDynamicSharedMemorySize, i8c_smem(MP)));
  int per;
  const int ranges = i8c_ranges(N, K, sms, &per);
  int8_columns_tc_kernel<MP><<<dim3((N + 127) / 128, ranges), 192, i8c_smem(MP), st>>>(mw, mx, w.part, M, N, K / 128, per, wait_word());
  LL_LAUNCH_OK("int8_columns_tc_kernel");
  return LL_OK;
}

template <typename T>
int int8_linear_t(const T* x, const int8_t* cb, const int8_t* cbt, const float* scb, const T* bias, T* y, int M, int N, int K, float thr,
                  void* ws_base, cudaStream_t st) {
  const int sms = sm_count();
  const int vec = ((uintptr_t)x & 15) == 0;
  CUtensorMap mw;
  if (int r = make_map_i8(cb, N, K, 128, &mw)) return r;
  for (int m0 = 0; m0 < M; m0 += 64) {
    const int Mp = min(64, M - m0);
    const Ws w = carve(ws_base, Mp, N, K);
    const T* xp = x + (size_t)m0 * K;
    LL_CUDA(cudaMemsetAsync((uint8_t*)ws_base + w.zero_off, 0, w.zero_bytes, st));
    int8_prep_kernel<T><<<Mp, I8P_THREADS, 0, st>>>(xp, w.ca, w.sca, w.flag, w.idx, w.count, w.arrive, K, thr, vec);
    LL_LAUNCH_OK("int8_prep_kernel");
    int r;
    if (Mp <= 16) r = i8c_launch<16>(mw, w, Mp, N, K, sms, st);
    else if (Mp <= 32) r = i8c_launch<32>(mw, w, Mp, N, K, sms, st);
    else if (Mp <= 48) r = i8c_launch<48>(mw, w, Mp, N, K, sms, st);
    else r = i8c_launch<64>(mw, w, Mp, N, K, sms, st);
    if (r) return r;
    int per;
    int8_finish_rows_kernel<T, 16><<<dim3((N + 63) / 64, (Mp + 15) / 16), 256, 0, st>>>(
        w.part, i8c_ranges(N, K, sms, &per), (size_t)Mp * N, w.sca, scb, bias, xp, cb, cbt, w.idx, w.count, y + (size_t)m0 * N, Mp, N, K);
    LL_LAUNCH_OK("int8_finish_rows_kernel");
  }
  return LL_OK;
}

}  // namespace
}  // namespace llb

using namespace llb;

extern "C" {

size_t ll_int8_workspace_bytes(int M, int N, int K) {
  const size_t pass = carve(nullptr, M < 64 ? M : 64, N, K).total;
  if (M <= 64) return pass;
  const size_t rows = carve_rows(nullptr, M, N, K).total;
  return rows > pass ? rows : pass;
}

int ll_int8_tc_error(void) {
  int v = 0;
  return cudaMemcpyFromSymbol(&v, g_int8_tc_error, sizeof(int)) == cudaSuccess ? v : -1;
}

int ll_int8_quantize_weight(const void* w, int w_dtype, int8_t* cb, float* scb, int N, int K, ll_stream stream) {
  LL_CHECK_ARG(w && cb && scb && N > 0 && K > 0, "bad int8_quantize_weight arguments");
  cudaStream_t st = (cudaStream_t)stream;
  if (w_dtype == LL_F32) int8_quant_weight_kernel<float><<<N, 256, 0, st>>>((const float*)w, cb, scb, K);
  else if (w_dtype == LL_BF16) int8_quant_weight_kernel<__nv_bfloat16><<<N, 256, 0, st>>>((const __nv_bfloat16*)w, cb, scb, K);
  else if (w_dtype == LL_F16) int8_quant_weight_kernel<__half><<<N, 256, 0, st>>>((const __half*)w, cb, scb, K);
  else {
    set_error("int8_quantize_weight: unsupported dtype %d", w_dtype);
    return LL_ERR_UNSUPPORTED;
  }
  LL_LAUNCH_OK("int8_quant_weight_kernel");
  return LL_OK;
}

int ll_int8_linear(const void* x, int act_dtype, const int8_t* cb, const int8_t* cbt, const float* scb, const void* bias, void* y,
                   int M, int N, int K, float threshold, void* workspace, size_t workspace_bytes, ll_stream stream) {
  LL_CHECK_ARG(x && cb && scb && y && workspace, "null pointer");
  LL_CHECK_ARG(M > 0 && N > 0 && K > 0 && K % 128 == 0, "int8 linear needs K %% 128 == 0 (M=%d N=%d K=%d)", M, N, K);
  LL_CHECK_ARG(((uintptr_t)cb & 15) == 0 && ((uintptr_t)workspace & 255) == 0, "cb must be 16-byte, workspace 256-byte aligned");
  LL_CHECK_ARG(workspace_bytes >= ll_int8_workspace_bytes(M < 64 ? M : 64, N, K), "workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  // prompts go through one product; with a workspace that only holds a pass of 64 rows, through passes
  if (M > 64 && workspace_bytes >= ll_int8_workspace_bytes(M, N, K)) {
    if (act_dtype == LL_BF16)
      return int8_rows_t<__nv_bfloat16>((const __nv_bfloat16*)x, cb, cbt, scb, (const __nv_bfloat16*)bias, (__nv_bfloat16*)y, M, N, K, threshold, workspace, st);
    if (act_dtype == LL_F16)
      return int8_rows_t<__half>((const __half*)x, cb, cbt, scb, (const __half*)bias, (__half*)y, M, N, K, threshold, workspace, st);
    if (act_dtype == LL_F32)
      return int8_rows_t<float>((const float*)x, cb, cbt, scb, (const float*)bias, (float*)y, M, N, K, threshold, workspace, st);
  }
  if (act_dtype == LL_BF16)
    return int8_linear_t<__nv_bfloat16>((const __nv_bfloat16*)x, cb, cbt, scb, (const __nv_bfloat16*)bias, (__nv_bfloat16*)y, M, N, K, threshold, workspace, st);
  if (act_dtype == LL_F16)
    return int8_linear_t<__half>((const __half*)x, cb, cbt, scb, (const __half*)bias, (__half*)y, M, N, K, threshold, workspace, st);
  if (act_dtype == LL_F32)
    return int8_linear_t<float>((const float*)x, cb, cbt, scb, (const float*)bias, (float*)y, M, N, K, threshold, workspace, st);
  set_error("int8_linear: unsupported activation dtype %d", act_dtype);
  return LL_ERR_UNSUPPORTED;
}

}  // extern "C"
