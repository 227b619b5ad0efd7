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
// Prompts (M > 64): the same arithmetic per block of 64 rows (a feature is an outlier for a block of 64 rows), all blocks at once: the same
// preparation, a kernel for the outlier parts of long lists, then one for the product and its finish (int8_pair_kernel).
// Either way the two layers of a gated feed-forward that read the same x go together: x is prepared once, one product over both, one finish.
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

constexpr int I8_BOX = 128 * 128;
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

// fp16(c SCA SCB / 127^2 (+ bias)), plus fp16 of the outlier part where the list is not empty, rounded to fp16
__device__ __forceinline__ float int8_finish(float c, float sa, float sb, bool has_bias, float bias, int cnt, float odd) {
  float out = __fmul_rn(__fmul_rn(__fmul_rn(c, sa), sb), 1.0f / (127.0f * 127.0f));
  if (has_bias) out = __fadd_rn(out, bias);
  out = __half2float(__float2half_rn(out));
  if (cnt > 0) out = __half2float(__float2half_rn(__fadd_rn(out, __half2float(__float2half_rn(odd)))));
  return out;
}

// One layer's weights, scales and bias as the finishing code reads them (cbt: CB transposed, or null).
template <typename T>
struct I8Layer {
  const int8_t* cb;
  const int8_t* cbt;
  const float* scb;
  const T* bias;
};

// out = fp16(C32 SCA SCB / 127^2 (+ bias)), plus fp16 of the outlier part, for 64 columns x 16 rows (of one outlier list) per CTA.  C32 is
// the sum of `parts` partial sums, `part` numbers apart.  GATED: of both layers (the second's partial sums lie `layer` numbers further), and
// y = silu(out1) * out2, rounded as ll_silu_mul rounds it.
// Outlier part: the weights and activations of 64 outliers at a time stand in shared memory as fp32, already rounded; the next 64 are asked
// for (all list entries, then all they point to) before these are added.  A list of up to 64 is added by a thread per row and four columns; a
// longer one is shared among the quarters of the threads, four columns of four rows each, a quarter of every 64, whose sums are added in
// order.  Four CTAs an SM: a batch of 64 rows has 688 of them for 11008 columns.
// Three layers of a 4096-wide feed-forward, 32 rows whose inputs have 6 / 30 / 100 / 200 outlier features (their products up to thousands):
// 78 / 121 / 424 / 519 us a call on the device.  32 outliers at a time, each weight behind its own list entry: 78 / 259 / 1725 / 2131; the
// kernel beside the mma.sync product: 123 / 181 / 536 / 647.  (A stage of 128 leaves three CTAs an SM: 87 with 12 outliers, 84 with 64.)
template <typename T, bool GATED>
__global__ void __launch_bounds__(256, 4) int8_finish_rows_kernel(const int32_t* __restrict__ c32, int parts, size_t part, size_t layer,
                                                              const float* __restrict__ sca, const I8Layer<T> l0, const I8Layer<T> l1,
                                                              const T* __restrict__ x, const int32_t* __restrict__ idx, const int32_t* __restrict__ count,
                                                              T* __restrict__ y, int M, int N, int K) {
  constexpr int ROWS = 16, SL = 4, L = 64, NW = L * 16 / 256, NA = L * ROWS / 256, AS = 256 / ROWS;   // SL: shares of the list
  __shared__ __align__(16) float w_s[L][64], a_s[L][ROWS];
  const int tid = threadIdx.x, n0 = blockIdx.x * 64, m0 = blockIdx.y * ROWS, blk = m0 / 64, col = (tid & 15) * 4;
  pdl_launch_dependents();
  const int cnt = count[blk];
  float first[4];                                          // GATED: the first layer's outputs
#pragma unroll 1
  for (int which = 0; which < (GATED ? 2 : 1); ++which) {
    const int8_t *cb = which ? l1.cb : l0.cb, *cbt = which ? l1.cbt : l0.cbt;
    const float* scb = which ? l1.scb : l0.scb;
    const T* bias = which ? l1.bias : l0.bias;
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
    if (cnt > 0) {
      if (which) __syncthreads();                          // the first layer's outliers have been added
      const int32_t* list = idx + (size_t)blk * K;
      // what a thread brings: four columns of NW outliers' weights, one row of NA outliers' activations.  Entries past the list's end, columns
      // past N and rows past M repeat the last one: they are never added, or added to what nobody stores.  Steps that lie past the end for the
      // whole CTA are left out.
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
              const int c = min(n0 + col + j, N - 1);
              const int8_t v = cbt != nullptr ? __ldg(cbt + (size_t)kw[u] * N + c) : __ldg(cb + (size_t)c * K + kw[u]);
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
      const int row = tid >> 4;
      if (cnt <= L) {
        stage();
        __syncthreads();
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
        const int r0 = (row & (ROWS / 4 - 1)) * 4, sl = tid / (256 / SL);
        for (int b = 0; b < cnt; b += L) {
          if (b > 0) __syncthreads();                      // the outliers before have been added
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
        __syncthreads();                                   // every thread finishes one row: its sums come through shared memory
        float* sums = &w_s[0][0];                          // [SL][ROWS][64]
#pragma unroll
        for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(sums + (sl * ROWS + r0 + r) * 64 + col) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        __syncthreads();
        float4 o = *reinterpret_cast<const float4*>(sums + row * 64 + col);
#pragma unroll
        for (int z = 1; z < SL; ++z) {
          const float4 v = *reinterpret_cast<const float4*>(sums + (z * ROWS + row) * 64 + col);
          o.x += v.x, o.y += v.y, o.z += v.z, o.w += v.w;
        }
        acc[0][0] = o.x, acc[0][1] = o.y, acc[0][2] = o.z, acc[0][3] = o.w;
      }
    }
    const int n = n0 + col, m = m0 + (tid >> 4);
    const bool vec = n + 4 <= N && (N & 3) == 0;           // (then a partial sum starts on a 16-byte boundary too)
    if (n >= N || m >= M) continue;                        // (which takes part in the barriers of the second layer's list)
    const float sa = sca[m];
    const size_t at = (size_t)m * N + n;
    float sb[4], bv[4];                                    // (asked for before the sums are there)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sb[j] = n + j < N ? scb[n + j] : 0.f;
      bv[j] = n + j < N && bias != nullptr ? to_half_f32<T>(bias[n + j]) : 0.f;
    }
    int cv[4] = {0, 0, 0, 0};
    for (int z = 0; z < parts; ++z) {
      const int32_t* src = c32 + (which ? layer : 0) + (size_t)z * part + at;
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
      const float out = int8_finish((float)cv[j], sa, sb[j], bias != nullptr, bv[j], cnt, acc[0][j]);
      if constexpr (!GATED) dt<T>::st(y, at + j, out);
      else if (which == 0) first[j] = dt<T>::rd(out);
      else dt<T>::st(y, at + j, __fmul_rn(silu_act<T>(first[j]), dt<T>::rd(out)));
    }
  }
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

// ================================================================================================== preparation
// One kernel: x.half(), row maxima of the entries below thr, quantised rows, and for every block of 64 rows the outlier columns as an ascending
// list.  A CTA owns a row and
// holds it in registers between its maximum and its codes (up to I8P_HELD * 4096 features; a longer row is read again).  Whether a column
// stands out in some row is known when the block's rows are done, so the CTA that finishes last of them makes the list and clears the listed
// columns' codes.  No CTA waits for another: nothing says that all of them run at the same time.  (A CTA per 64 columns and one wait of the whole
// grid in the middle took 2 us less a layer, and stood still, or went on with counts that were not there, when other streams held the SMs.)
// 32 rows through a 7B feed-forward, three layers: 78 us on the device; 123 before the product ran on tcgen05.
constexpr int I8P_THREADS = 512, I8P_HELD = 4;
// Codes of eight entries: rint(v * inv), 0 for those from thr on and those of `out`.  An entry below thr is at most its row's maximum, so the product
// is within 127 and a rounding, and 1.5 * 2^23 added to it leaves the nearest whole number (ties to even) in the low bits.  (By rintf,
// bounds and a conversion, all but the bounds at a quarter of the rate: 512 rows through a 7B feed-forward 112 us a call instead of 108, 32 rows 65
// instead of 63.)
__device__ __forceinline__ uint2 int8_codes(const float (&v)[8], float inv, float thr, uint32_t out) {
  uint32_t q[8];
#pragma unroll
  for (int e = 0; e < 8; ++e)
    q[e] = __float_as_uint(__fadd_rn(fabsf(v[e]) < thr && !((out >> e) & 1u) ? __fmul_rn(v[e], inv) : 0.f, 12582912.f));
  uint32_t o[2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
    o[h] = __byte_perm(__byte_perm(q[4 * h], q[4 * h + 1], 0x0040), __byte_perm(q[4 * h + 2], q[4 * h + 3], 0x0040), 0x5410);
  return make_uint2(o[0], o[1]);
}
template <typename T>
__global__ void __launch_bounds__(I8P_THREADS) int8_prep_kernel(const T* __restrict__ x, int8_t* __restrict__ ca, float* __restrict__ sca,
                                                               uint8_t* __restrict__ flag, int32_t* __restrict__ idx, int32_t* __restrict__ count,
                                                               int32_t* __restrict__ arrive, int K, float thr, int vec, int early) {
  constexpr int WARPS = I8P_THREADS / 32, STEP = I8P_THREADS * 8;
  __shared__ float s_max[WARPS];
  __shared__ int s_warp[WARPS], s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blk = blockIdx.x / 64, m0 = blk * 64, M = min(64, (int)gridDim.x - m0);
  flag += (size_t)blk * K, idx += (size_t)blk * K;
  if (early) pdl_launch_dependents();
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
    *reinterpret_cast<uint2*>(ca + (size_t)blockIdx.x * K + k) = int8_codes(v, inv, thr, 0u);
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
  if (tid == 0) s_last = atomicAdd(arrive + blk, 1) == M - 1;
  __syncthreads();
  // Of prompts the next kernel's CTAs come while the lists are made.  (Let in from the start on they pile up on the SMs that have no row: 130 rows
  // with long lists 2300 us instead of 1280.)
  pdl_launch_dependents();
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
  if (tid == 0) count[blk] = base;
  // (the list is complete: a barrier of this CTA, which wrote it, lies behind the last entry)
  for (int i = tid; i < base * M; i += I8P_THREADS) {
    const int m = i / base;
    ca[(size_t)(m0 + m) * K + idx[i - m * base]] = 0;
  }
}

// The same for few rows in one cluster of eight CTAs, every eighth row a CTA: the columns that stand out are bits in shared memory, each CTA marks
// those of its rows, and past one cluster barrier ORs all eight CTAs' (CTAs of a cluster run at the same time).  Codes are written once, nothing has
// to be cleared before, and the kernel starts under the one before it.  Bound by the arithmetic of eight SMs, 2 us a row of 11008.  us a layer of
// 11008 x 4096 and of 4096 x 11008, clearing and a CTA per row / here: 1 row 17 / 12 and 18 / 14, 8 rows 17 / 13 and 18 / 15; 24 rows of 4096 features
// 17 / 15.  Against a CTA per row with the weights ahead of it, without and with 30 outliers, 32 rows of 4096 features 14.9 / 15.8 and 21.1 / 19.5,
// 48 rows 16.9 / 18.7 and 23.5 / 23.8, 16 rows of 11008 16.3 / 16.8 and 19.6 / 19.1.
constexpr int I8F_THREADS = 1024, I8F_CTAS = 8, I8F_MOST = 16384;          // features a CTA takes
__device__ __forceinline__ uint32_t int8_peer_word(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
template <typename T>
__global__ void __cluster_dims__(I8F_CTAS, 1, 1) __launch_bounds__(I8F_THREADS, 1)
    int8_prep_few_kernel(const T* x, int8_t* __restrict__ ca, float* __restrict__ sca, int32_t* __restrict__ idx, int32_t* __restrict__ count,
                         int M, int K, float thr, int vec) {
  constexpr int WARPS = I8F_THREADS / 32;
  extern __shared__ __align__(16) uint32_t i8p_smem[];
  __shared__ float s_max[WARPS];
  __shared__ int s_warp[WARPS];
  const int words = K / 32;
  uint32_t *own = i8p_smem, *all = own + words;        // a bit per column: of this CTA's rows, of the block's
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)cluster_rank();
  const int held = (M + I8F_CTAS - 1) / I8F_CTAS;        // rows of a CTA at most
  const int per = held <= 1 ? 32 : held <= 2 ? 16 : held <= 4 ? 8 : 4, m = rank + warp / per * I8F_CTAS, step = per * 256;   // warps of a row
  const int k0 = (tid - warp / per * per * 32) * 8;
  const bool mine = m < M;
  const size_t at = (size_t)m * K;
  for (int i = tid; i < words; i += I8F_THREADS) own[i] = 0u;
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();
  const T* row = after_wait(x) + at;
  float mx = 0.f;
  if (mine) {
#pragma unroll 4
    for (int k = k0; k < K; k += step) {                 // (K is a multiple of 128)
      float v[8];
      int8_load8<T>(row + k, v, vec);
      uint32_t bits = 0u;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float a = fabsf(v[e]);
        if (a >= thr) bits |= 1u << e;
        else mx = fmaxf(mx, a);
      }
      if (bits) atomicOr(&own[k >> 5], bits << (k & 31));
    }
  }
  mx = warp_max(mx);
  if (lane == 0) s_max[warp] = mx;
  cluster_sync();                                        // (of this CTA's threads too)
  for (int i = tid; i < words; i += I8F_THREADS) {
    uint32_t w = 0u;
#pragma unroll
    for (int r = 0; r < I8F_CTAS; ++r) w |= int8_peer_word(cluster_addr(own + i, (uint32_t)r));
    all[i] = w;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // waited for at the end: no CTA leaves while its bits are read
  __syncthreads();
  if (mine) {
    mx = s_max[warp / per * per];
    for (int w = 1; w < per; ++w) mx = fmaxf(mx, s_max[warp / per * per + w]);
    if (k0 == 0) sca[m] = mx;
    const float inv = __fdiv_rn(127.f, mx == 0.f ? 1.f : mx);
#pragma unroll 4
    for (int k = k0; k < K; k += step) {
      float v[8];
      int8_load8<T>(row + k, v, vec);
      const uint32_t bits = all[k >> 5] >> (k & 31);
      *reinterpret_cast<uint2*>(ca + at + k) = int8_codes(v, inv, thr, bits);
    }
  }
  if (rank == I8F_CTAS - 1) {                            // (the CTA with the fewest rows)
    int base = 0;
    for (int i0 = 0; i0 < words; i0 += I8F_THREADS) {
      const uint32_t w = i0 + tid < words ? all[i0 + tid] : 0u;
      const int n = __popc(w);
      int incl = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += u;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      int to = base + incl - n, total = 0;
      for (int u = 0; u < WARPS; ++u) {
        const int c = s_warp[u];
        if (u < warp) to += c;
        total += c;
      }
      for (uint32_t left = w; left; left &= left - 1u) idx[to++] = (i0 + tid) * 32 + __ffs((int)left) - 1;
      base += total;
      __syncthreads();
    }
    if (tid == 0) *count = base;
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ================================================================================================== up to 64 rows
// part[range][m][n] = the sum over the range's k of CA[m][k] CB[n][k]: the weights are the A operand (128 output columns a CTA), streamed
// through a ring of 16 KB boxes; two CTAs share an SM.  MP: rows rounded up to 16, 32, 48 or 64.
// A batch of 32 through a 7B feed-forward: mma.sync straight from global memory, two loads in flight a thread and int32 atomics, took 17.5 us
// a layer (2.6 TB/s of weights) and the preparation beside it 9.4 us, the finish 10 us.
constexpr int i8c_stages(int mp) { return mp > 32 ? 4 : 5; }
constexpr int i8c_smem(int mp) { return i8c_stages(mp) * (I8_BOX + mp * 128) + 256 + 1024; }
template <int MP>
__global__ void __launch_bounds__(192, 2) int8_columns_tc_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                                                                const __grid_constant__ CUtensorMap map_x, int32_t* __restrict__ part, int M, int N, int nkb,
                                                                int per, int tiles, size_t layer, int* word) {
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
  const bool second = (int)blockIdx.x >= tiles;              // column tiles of the second layer
  const int n0 = ((int)blockIdx.x - (second ? tiles : 0)) * 128, kb0 = blockIdx.y * per, kb1 = min(kb0 + per, nkb);
  const CUtensorMap* map_w = second ? &map_w1 : &map_w0;
  if (threadIdx.x == 0) {
    prefetch_tensormap(map_w);
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
      // the weights of the first stages come while the rows are prepared (the preparation waits for all before it and only then lets this kernel in:
      // whoever made the weights is done).  us a layer of 4096 x 11008 that a CTA per row prepares, 32 and 64 rows: 19 / 17, 21 / 19.
      const int ahead = min(STAGES, kb1 - kb0);
      for (int i = 0; i < ahead; ++i) {
        mbar_expect_tx(&full[i], I8_BOX + XB);
        i8_box(sw + i * I8_BOX, map_w, (kb0 + i) * 128, n0, &full[i]);
      }
      pdl_wait();
      for (int kb = kb0; kb < kb1; ++kb) {
        if (kb - kb0 >= ahead) {
          if (!(ok = i8_wait(&empty[s], ph, s_fail, word, 5))) break;
          mbar_expect_tx(&full[s], I8_BOX + XB);
          i8_box(sw + s * I8_BOX, map_w, kb * 128, n0, &full[s]);
        }
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
    pdl_wait();                      // (the partial sums' place may be the kernel's before)
    const bool ok = __all_sync(0xffffffffu, i8_wait(done, 0, s_fail, word, 7) && *(volatile int*)s_fail == 0);
    tc_fence_after();
    if (ok) {
      int32_t* dst = part + (second ? layer : 0) + (size_t)blockIdx.y * M * N + n;
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
int i8c_ranges(int N, int K, int layers, int sms, int* per) {
  const int tiles = layers * ((N + 127) / 128), nkb = K / 128;
  int ranges = 2 * (sms > 0 ? sms : 148) / tiles;
  ranges = ranges < 1 ? 1 : ranges > nkb ? nkb : ranges;
  *per = (nkb + ranges - 1) / ranges;
  return (nkb + *per - 1) / *per;
}

// What the preparation leaves for a step of M rows, the partial sums of a step of up to 64 (partial) and the outlier parts of a longer one.
int i8r_pitch(int N) { return (N + 255) & ~255; }      // of an outlier part's rows: whole tiles
struct Ws {
  int8_t* ca; int32_t* part; __half* odd; float* sca; int32_t* idx; uint8_t* flag; int32_t* count; int32_t* arrive;
  int32_t* next;                 // of int8_outlier_rows_kernel's tiles
  size_t zero_off, zero_bytes, total;
};
Ws carve(void* base, int M, int N, int K, int layers, bool partial) {
  Ws w;
  const size_t blocks = (size_t)(M + 63) / 64;
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o += (b + 255) & ~(size_t)255; return r; };
  uint8_t* p = (uint8_t*)base;
  int per;
  w.ca = (int8_t*)(p + take((size_t)M * K));
  w.part = (int32_t*)(p + take(partial ? (size_t)layers * i8c_ranges(N, K, layers, sm_count(), &per) * M * N * 4 : 0));
  w.odd = (__half*)(p + take(partial ? 0 : (size_t)layers * M * i8r_pitch(N) * 2));
  w.idx = (int32_t*)(p + take(blocks * K * 4));
  w.sca = (float*)(p + take((size_t)M * 4));
  w.zero_off = o;  // cleared at the start of every call
  w.flag = p + take(blocks * K);
  w.arrive = (int32_t*)(p + take(blocks * 4));
  w.next = (int32_t*)(p + take(4));
  w.zero_bytes = o - w.zero_off;
  w.count = (int32_t*)(p + take(blocks * 4));
  w.total = o;
  return w;
}

template <typename T>
int int8_prepare(const T* x, const Ws& w, void* base, int M, int K, float thr, cudaStream_t st) {
  const int vec = ((uintptr_t)x & 15) == 0 ? 1 : 0;
  if (M <= 64 && (long long)((M + I8F_CTAS - 1) / I8F_CTAS) * K <= I8F_MOST) {
    LL_CUDA(launch(int8_prep_few_kernel<T>, dim3(I8F_CTAS), dim3(I8F_THREADS), K / 32 * 8, st, true, x, w.ca, w.sca, w.idx, w.count, M, K, thr, vec));
    LL_LAUNCH_OK("int8_prep_few_kernel");
    return LL_OK;
  }
  LL_CUDA(cudaMemsetAsync((uint8_t*)base + w.zero_off, 0, w.zero_bytes, st));
  int8_prep_kernel<T><<<M, I8P_THREADS, 0, st>>>(x, w.ca, w.sca, w.flag, w.idx, w.count, w.arrive, K, thr, vec, M <= 64 ? 1 : 0);
  LL_LAUNCH_OK("int8_prep_kernel");
  return LL_OK;
}

template <int MP>
int i8c_launch(const CUtensorMap& m0, const CUtensorMap& m1, const Ws& w, int M, int N, int K, int layers, int per, int ranges, cudaStream_t st) {
  CUtensorMap mx;
  if (int r = make_map_i8(w.ca, M, K, MP, &mx)) return r;
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(int8_columns_tc_kernel<MP>, cudaFuncAttributeMaxDynamicSharedMemorySize, i8c_smem(MP)));
    configured.mark();
  }
  const int tiles = (N + 127) / 128;
  LL_CUDA(launch(int8_columns_tc_kernel<MP>, dim3(layers * tiles, ranges), dim3(192), i8c_smem(MP), st, true, m0, m1, mx, w.part, M, N, K / 128, per, tiles,
                 (size_t)ranges * M * N, wait_word()));
  LL_LAUNCH_OK("int8_columns_tc_kernel");
  return LL_OK;
}

// up to 64 rows of one layer, or of two whose gated product is wanted
template <typename T, bool GATED>
int int8_pass(const T* x, const I8Layer<T>& l0, const I8Layer<T>& l1, T* y, int M, int N, int K, float thr, void* base, cudaStream_t st) {
  constexpr int layers = GATED ? 2 : 1;
  const Ws w = carve(base, M, N, K, layers, true);
  if (int r = int8_prepare<T>(x, w, base, M, K, thr, st)) return r;
  CUtensorMap m0, m1;
  if (int r = make_map_i8(l0.cb, N, K, 128, &m0)) return r;
  if (int r = make_map_i8(l1.cb, N, K, 128, &m1)) return r;
  int per, r;
  const int ranges = i8c_ranges(N, K, layers, sm_count(), &per);
  if (M <= 16) r = i8c_launch<16>(m0, m1, w, M, N, K, layers, per, ranges, st);
  else if (M <= 32) r = i8c_launch<32>(m0, m1, w, M, N, K, layers, per, ranges, st);
  else if (M <= 48) r = i8c_launch<48>(m0, m1, w, M, N, K, layers, per, ranges, st);
  else r = i8c_launch<64>(m0, m1, w, M, N, K, layers, per, ranges, st);
  if (r) return r;
  // (Not under the product: its CTAs would pile up on the SMs that are done first, 24 rows with long lists 43 us instead of 33.)
  int8_finish_rows_kernel<T, GATED><<<dim3((N + 63) / 64, (M + 15) / 16), 256, 0, st>>>(w.part, ranges, (size_t)M * N, (size_t)ranges * M * N, w.sca, l0, l1, x,
                                                                                     w.idx, w.count, y, M, N, K);
  LL_LAUNCH_OK("int8_finish_rows_kernel");
  return LL_OK;
}

// ================================================================================================== prompts: M > 64
// The product and its finish in one kernel, by pairs of CTAs (tcgen05 cta_group::2, kind::i8, K = 32 an instruction): tiles of 256 rows x BN
// columns a pair, persistent, two int32 accumulators in tensor memory, so that a tile is finished (scales, bias, outlier part, rounding,
// stores by TMA) under the next one's products.  GATED: the tile's columns are BN / 2 of the first layer (rank 0 brings them) and the same of
// the second, and y = silu(out1) * out2.
//   warp 0: TMA producer; warp 1: in rank 0, one thread issues the products; warps 2-9: finish, 32 rows and half of the columns per warp,
//   32 columns at a time (GATED: 16 of either layer), read from tensor memory so that a thread has four rows of eight columns
// Outlier part: a warp's 32 rows belong to one block of 64 rows, so to one list.  Of a short list (i8r_limit) its activations are gathered before
// the tile's sums are there, and so are the scales and the first eight outliers' weights of its columns; the weights of four outliers x 32
// columns pass through shared memory as fp32, already rounded.  The parts of longer lists a kernel before this one has left as fp16
// (int8_outlier_rows_kernel: a warp has no other warp's rows to share a list's weights with).  us a call, a feed-forward of 4096 x 11008 whose
// input has 6 and 30 outlier features, and its hidden state more of them: a warp reading its lists to the end / three products with their finish by 64 rows / here:
// 512 rows 582 / 326 / 234, 1900 / 725 / 667 and, of one layer alone with 64, 300, 1000 outliers, 175 / 105 / 87, 773 / 263 / 258, 2265 / 729 / 732;
// 2048 rows 2043 / 1061 / 690 and 7235 / 2432 / 2116, alone 522 / 357 / 266, 2543 / 950 / 887, 7377 / 2691 / 2620.
// (Four finishing warps, one a scheduler, took 35 us a tile of the gated form, four times as long as its products.)
// 512 rows through a 7B feed-forward with six outlier features: 53 us for both gated layers and 27 for the third, preparation 24; 127 for three
// products of 128 x 128 tiles a CTA, 55 for their finish and 45 for preparation and the gated product before.  2048 rows: 305 us a call (701).
// Bound by the weights' way from memory and, with outliers, by the finish (weights asked for one by one: 10 us a tile instead of 3).
constexpr int I8R_PASS = 8192;                           // rows of one pass: bounds the workspace (outlier parts of a gated pair: 453 MB at 13824 columns)
constexpr int I8R_WARPS = 8, I8R_THREADS = (2 + I8R_WARPS) * 32;                           // finishing warps: two per 32 rows, half of the columns each
constexpr int I8R_LIST = 32, I8R_OUT = 32 * 64, I8R_W = 6 * 32 * 4;
constexpr int i8r_stages(int bn) { return bn > 128 ? 5 : 6; }
constexpr int i8r_smem(int bn) {
  return i8r_stages(bn) * (I8_BOX + bn * 64) + I8R_WARPS * (2 * I8R_OUT + I8R_LIST * 64 + I8R_LIST * 4 + I8R_W) + 512 + 1024;
}

// The outlier part of blocks of 64 rows whose lists are longer than `limit`, rounded to fp16 as the finish adds it: 64 rows x 64 columns of a
// layer at a time.  The weights and activations of 32 outliers stand in shared memory as fp32, already rounded, and the next 32 are asked for
// (all list entries, then all they point to) before these are added; a thread owns four columns of four rows, two 16-byte reads for 16
// multiply-adds, and adds in the order of the list.  WORDS: CB transposed is there, on 4-byte boundaries.
template <typename T, bool WORDS>
__global__ void __launch_bounds__(256, 4) int8_outlier_rows_kernel(const I8Layer<T> l0, const I8Layer<T> l1, const T* __restrict__ x, const int32_t* __restrict__ idx,
                                                              const int32_t* __restrict__ count, int32_t* __restrict__ next, __half* __restrict__ odd,
                                                              int M, int N, int K, int layers, int pitch, int limit) {
  constexpr int L = 32, NW = L * 16 / 256, NA = L * 64 / 256;
  __shared__ __align__(16) float w_s[L][64], a_s[L][64];
  __shared__ int s_item, s_blk[I8R_PASS / 64];
  pdl_launch_dependents();                                 // (what follows waits for this kernel's end, and this one for the preparation's)
  pdl_wait();
  const int tid = threadIdx.x, col = (tid & 15) * 4;
  const int tiles = (N + 63) / 64, per = layers * tiles, blocks = (M + 63) / 64;
  const bool single = (int)gridDim.x >= blocks * per;      // a CTA per tile of every block
  if (!single) {                                           // the blocks with long lists, in order
    if (tid < 32) {
      int n = 0;
      for (int b0 = 0; b0 < blocks; b0 += 32) {
        const uint32_t any = __ballot_sync(0xffffffffu, b0 + tid < blocks && count[b0 + tid] > limit);
        if ((any >> tid) & 1u) s_blk[n + __popc(any & ((1u << tid) - 1u))] = b0 + tid;
        n += __popc(any);
      }
      if (tid == 0) s_item = n;
    }
    __syncthreads();
  }
  const int items = single ? blocks * per : s_item * per;
  for (int item = blockIdx.x; item < items;) {
    const int m0 = (single ? item / per : s_blk[item / per]) * 64, cnt = count[m0 / 64];
    if (cnt <= limit) break;                               // (single)
    const bool second = item % per >= tiles;
    const int n = item % per % tiles * 64 + col;
    const int32_t* list = idx + (size_t)(m0 / 64) * K;
    // what a thread brings: four columns of NW outliers' weights, one row of NA outliers' activations.  Entries past the list's end, columns
    // past N and rows past M repeat the last one: they are never added, or added to what nobody stores or reads.
    const T* xr = x + (size_t)min(m0 + (tid & 63), M - 1) * K;
    const int8_t* src = WORDS ? (second ? l1.cbt : l0.cbt) + min(n, N - 4) : nullptr;
    uint32_t q[NW];
    float av[NA], acc[4][4], sb127[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) sb127[j] = __fdiv_rn((second ? l1.scb : l0.scb)[min(n + j, N - 1)], 127.f);
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
    auto fetch = [&](int b) {
      int kw[NW], ka[NA];
#pragma unroll
      for (int u = 0; u < NW; ++u) kw[u] = __ldg(list + min(b + (tid >> 4) + 16 * u, cnt - 1));
#pragma unroll
      for (int u = 0; u < NA; ++u) ka[u] = __ldg(list + min(b + (tid >> 6) + 4 * u, cnt - 1));
#pragma unroll
      for (int u = 0; u < NW; ++u) {
        if (WORDS) {
          q[u] = __ldg(reinterpret_cast<const uint32_t*>(src + (size_t)kw[u] * N));
        } else {
          const I8Layer<T>& l = second ? l1 : l0;
          q[u] = 0u;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = min(n + j, N - 1);
            const int8_t v = l.cbt != nullptr ? __ldg(l.cbt + (size_t)kw[u] * N + c) : __ldg(l.cb + (size_t)c * K + kw[u]);
            q[u] |= (uint32_t)(uint8_t)v << (8 * j);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < NA; ++u) av[u] = to_half_f32<T>(xr[ka[u]]);
    };
    fetch(0);
    const int r0 = (tid >> 4) * 4;
    for (int b = 0; b < cnt; b += L) {
      __syncthreads();                                     // the outliers before have been added
#pragma unroll
      for (int u = 0; u < NW; ++u) {
        float w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = __half2float(__float2half_rn(__fmul_rn((float)(int8_t)(q[u] >> (8 * j)), sb127[j])));
        *reinterpret_cast<float4*>(&w_s[(tid >> 4) + 16 * u][col]) = make_float4(w[0], w[1], w[2], w[3]);
      }
#pragma unroll
      for (int u = 0; u < NA; ++u) a_s[(tid >> 6) + 4 * u][tid & 63] = av[u];
      __syncthreads();
      if (b + L < cnt) fetch(b + L);
      const int end = min(L, cnt - b);
#pragma unroll 4
      for (int i = 0; i < end; ++i) {
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
    __half* dst = odd + (size_t)(second ? M : 0) * pitch + n;          // (n < pitch: a row is whole tiles)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (m0 + r0 + r >= M) break;
      const __half2 lo = __floats2half2_rn(acc[r][0], acc[r][1]), hi = __floats2half2_rn(acc[r][2], acc[r][3]);
      *reinterpret_cast<uint2*>(dst + (size_t)(m0 + r0 + r) * pitch) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
    if (single) break;
    __syncthreads();                                       // the item has been read by all
    if (tid == 0) s_item = (int)gridDim.x + atomicAdd(next, 1);
    __syncthreads();
    item = s_item;
  }
}

template <typename T>
struct I8RParams {
  I8Layer<T> layer[2];
  const T* x;
  const float* sca;
  const int32_t* idx;
  const int32_t* count;
  const __half* odd;                                 // [layer][M][pitch] outlier parts of blocks with longer lists than a warp holds
  T* y;
  int M, N, K, pitch, limit, mtiles, ntiles, boxes;  // limit: of what a warp adds itself; boxes: TMA stores y
  int* word;
};
struct I8Fail {
  volatile int* here;
  uint32_t there;
  int* word;
};
__device__ __forceinline__ bool i8r_wait(uint64_t* bar, uint32_t parity, const I8Fail& f, int code) {
  for (uint32_t i = 0; i < I8_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *f.here) return false;
  }
  *f.here = 1;
  store_cluster_u32(f.there, 1u);
  atomicCAS(&g_int8_tc_error, 0, code);
  wait_ran_out(f.word, 300 + code);
  return false;
}
__device__ __forceinline__ void i8r_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 16 lanes x 16 columns: of every 8 columns a thread gets columns 2 (lane % 4), + 1 of lanes lane / 4 and lane / 4 + 8
__device__ __forceinline__ void i8r_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
// two outputs in the activation dtype, packed (16-bit dtypes)
template <typename T> __device__ __forceinline__ uint32_t i8r_pack(float a, float b);
template <> __device__ __forceinline__ uint32_t i8r_pack<__nv_bfloat16>(float a, float b) { return pack_bf16(a, b); }
template <> __device__ __forceinline__ uint32_t i8r_pack<__half>(float a, float b) {
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t i8r_pack<float>(float, float) { return 0u; }

template <typename T, int BN, bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(I8R_THREADS, 1)
    int8_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                     const __grid_constant__ CUtensorMap map_y, const I8RParams<T> p) {
  constexpr int STAGES = i8r_stages(BN), B_BYTES = BN * 64, COLS = GATED ? BN / 2 : BN, CH = GATED ? 16 : 32, NCH = COLS / 2 / CH;
  // COLS: outputs of a tile, CH: outputs a thread forms at a time, NCH: how many times
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);
  uint8_t *sa = base, *sb = base + STAGES * I8_BOX, *so = sb + STAGES * B_BYTES;
  uint8_t* s_list = so + I8R_WARPS * 2 * I8R_OUT;      // per warp: [LIST][32] fp16 activations
  uint8_t* s_idx = s_list + I8R_WARPS * I8R_LIST * 64; //           [LIST] columns
  uint8_t* s_w = s_idx + I8R_WARPS * I8R_LIST * 4;     //           [4][32] fp32 weights, [32] scales, [32] biases
  uint64_t* full = reinterpret_cast<uint64_t*>(s_w + I8R_WARPS * I8R_W);      // used in rank 0
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
    for (int i = 0; i < 2; ++i) mbar_init(&acc_full[i], 1), mbar_init(&acc_empty[i], 2 * I8R_WARPS);
    *s_fail = 0;
    fence_barrier_init();
  }
  if (warp == 1) pair_tmem_alloc(tmem_ptr, 2 * BN);
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const I8Fail fail{s_fail, cluster_addr(s_fail, (uint32_t)(rank ^ 1)), p.word};
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, tiles = p.mtiles * p.ntiles, nkb = p.K / 128;
  pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      int s = 0;
      uint32_t ph = 1;
      for (int t = pair; ok && t < tiles; t += pairs) {
        const int m0 = (t % p.mtiles) * 256 + rank * 128, n0 = (t / p.mtiles) * COLS + (GATED ? 0 : rank * (BN / 2));
        const CUtensorMap* mw = GATED && rank == 1 ? &map_w1 : &map_w0;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = i8r_wait(&empty[s], ph, fail, 1))) break;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * (I8_BOX + B_BYTES));      // both CTAs' operands
          const uint32_t bar = cluster_addr(&full[s], 0);
          pair_box(sa + s * I8_BOX, &map_x, kb * 128, m0, bar);
          pair_box(sb + s * B_BYTES, mw, kb * 128, n0, bar);
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
      }
      if (!ok) let_issued_work_end();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // D = int32 (2 at bit 4), A = B = signed int8 (1 at bits 7 and 10), both K-major
      constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint64_t ad = smem_desc_sw128(smem_u32(sa)), bd = smem_desc_sw128(smem_u32(sb));
      bool ok = true;
      int s = 0, i = 0;
      uint32_t ph = 0;
      for (int t = pair; rank == 0 && ok && t < tiles; t += pairs, ++i) {
        if (!(ok = i8r_wait(&acc_empty[i & 1], (uint32_t)((i >> 1) & 1) ^ 1u, fail, 4))) break;
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = i8r_wait(&full[s], ph, fail, 2))) break;
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 4; ++k)
            i8r_mma(tmem + (uint32_t)((i & 1) * BN), ad + (uint64_t)(s * (I8_BOX >> 4) + 2 * k), bd + (uint64_t)(s * (B_BYTES >> 4) + 2 * k), idesc,
                    (kb | k) != 0 ? 1u : 0u);
          pair_commit(&empty[s]);
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
        if (ok) pair_commit(&acc_full[i & 1]);
      }
      if (!ok) let_issued_work_end();
    }
  } else {
    const int quarter = warp & 3, ew = warp - 2, part = ew >> 2;
    uint8_t* out = so + ew * 2 * I8R_OUT;
    __half* a_s = reinterpret_cast<__half*>(s_list + ew * I8R_LIST * 64);      // [LIST][8][4]: rows g, g + 8, g + 16, g + 24 side by side
    int* k_s = reinterpret_cast<int*>(s_idx + ew * I8R_LIST * 4);
    float* w_s = reinterpret_cast<float*>(s_w + ew * I8R_W);
    // what a thread finishes: rows g, g + 8, .. of the warp's 32, columns 2 t4, + 1 of every 8 (as tensor memory is read in 16 x 256-bit pieces)
    const int g = lane >> 2, t4 = lane & 3;
    // the weight column a lane brings, and its place among those that the threads of one t4 read
    const int place = ((lane & 7) >> 1) * 8 + (lane >> 3) * 2 + (lane & 1);
    const bool second = GATED && lane >= 16;
    const int lcol = GATED ? lane & 15 : lane;
    const int8_t *cb = second ? p.layer[1].cb : p.layer[0].cb, *cbt = second ? p.layer[1].cbt : p.layer[0].cbt;
    const float* scb = second ? p.layer[1].scb : p.layer[0].scb;
    const T* bias = second ? p.layer[1].bias : p.layer[0].bias;
    const bool any_bias = p.layer[0].bias != nullptr || (GATED && p.layer[1].bias != nullptr);
    int i = 0;
    uint32_t boxes = 0;
    for (int t = pair; t < tiles; t += pairs, ++i) {
      const int r0 = (t % p.mtiles) * 256 + rank * 128 + quarter * 32, n0 = (t / p.mtiles) * COLS, m = min(r0 + lane, p.M - 1);
      // the block's list and this row's activations of its entries; the outlier part of a longer list is there already
      const int all = r0 < p.M ? p.count[r0 / 64] : 0, cnt = all <= p.limit ? all : 0;
      const int32_t* list = p.idx + (size_t)(r0 / 64) * p.K;
      const T* xr = p.x + (size_t)m * p.K;
      __syncwarp();
      if (lane < cnt) k_s[lane] = __ldg(list + lane);
      __syncwarp();
      for (int l = 0; l < cnt; l += 4) {
        T v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = xr[k_s[min(l + j, cnt - 1)]];
#pragma unroll
        for (int j = 0; j < 4; ++j) a_s[(l + j) * 32 + (lane & 7) * 4 + (lane >> 3)] = __float2half_rn(to_half_f32<T>(v[j]));
      }
      float sca[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) sca[r] = p.sca[min(r0 + g + 8 * r, p.M - 1)];
      // the weights of outliers l .. l + 3 in the lane's column of the chunk at cc, all loads in flight together (past the list's end the last
      // one again: never added)
      auto fetch = [&](int cc, int l) {
        const int n = min(n0 + cc + lcol, p.N - 1);
        const int8_t* src = cbt != nullptr ? cbt + n : cb + (size_t)n * p.K;
        const size_t step = cbt != nullptr ? (size_t)p.N : 1;
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = (uint8_t)__ldg(src + (size_t)k_s[min(l + j, cnt - 1)] * step);
        return v[0] | (v[1] << 8) | (v[2] << 16) | (v[3] << 24);
      };
      // what the tile's chunks want of their columns, asked for before the sums are there: scales, weights of the first eight outliers
      const int c_end = (part + 1) * (COLS / 2);
      float scale[NCH];
      uint32_t q0[NCH], q1[NCH];
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int cc = part * (COLS / 2) + c * CH;
        scale[c] = __ldg(scb + min(n0 + cc + lcol, p.N - 1));
        q0[c] = q1[c] = 0u;
      }
      if (cnt > 0) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) q0[c] = fetch(part * (COLS / 2) + c * CH, 0);
      }
      if (cnt > 4) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) q1[c] = fetch(part * (COLS / 2) + c * CH, 4);
      }
      if (!__all_sync(0xffffffffu, i8r_wait(&acc_full[i & 1], (uint32_t)(i >> 1) & 1u, fail, 3))) break;
      tc_fence_after();
      const uint32_t td = tmem + (uint32_t)((i & 1) * BN) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int cc = part * (COLS / 2); cc < c_end; cc += CH) {
        // scales and biases of the chunk's columns for every lane to read
        const int n = min(n0 + cc + lcol, p.N - 1);
        const float sb = scale[0], sb127 = __fdiv_rn(sb, 127.f);
        __syncwarp();
        w_s[4 * 32 + place] = sb;
        w_s[5 * 32 + place] = bias != nullptr ? to_half_f32<T>(bias[n]) : 0.f;
        float odd[32];                       // [row half of 16][8 columns][g, g + 8][2 t4, + 1]
#pragma unroll
        for (int e = 0; e < 32; ++e) odd[e] = 0.f;
        uint32_t q = q0[0], qn = q1[0];
#pragma unroll 1
        for (int l = 0; l < cnt; l += 4) {
          const uint32_t w4 = q;
          q = qn;
          if (l + 8 < cnt) qn = fetch(cc, l + 8);
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 4; ++j) w_s[j * 32 + place] = __half2float(__float2half_rn(__fmul_rn((float)(int8_t)(w4 >> (8 * j)), sb127)));
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (l + j >= cnt) break;
            const uint2 h = *reinterpret_cast<const uint2*>(a_s + (l + j) * 32 + g * 4);
            const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&h.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&h.y));
            const float a[4] = {lo.x, lo.y, hi.x, hi.y};
            const float4 w0 = *reinterpret_cast<const float4*>(w_s + j * 32 + t4 * 8), w1 = *reinterpret_cast<const float4*>(w_s + j * 32 + t4 * 8 + 4);
            const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int e = 0; e < 32; ++e) odd[e] = fmaf(a[(e >> 4) * 2 + ((e >> 1) & 1)], w[((e >> 2) & 3) * 2 + (e & 1)], odd[e]);
          }
        }
        if (all > p.limit) {
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const int b = (e >> 2) & 3, row = min(r0 + (e >> 4) * 16 + ((e >> 1) & 1) * 8 + g, p.M - 1);
            const __half* src = p.odd + (size_t)((GATED && b >= 2 ? p.M : 0) + row) * p.pitch + n0 + cc + (GATED ? b & 1 : b) * 8 + 2 * t4;
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(src));
            odd[e] = f.x, odd[e + 1] = f.y;
          }
        }
        __syncwarp();
        uint32_t v[32];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          i8r_ld16(td + ((uint32_t)(16 * h) << 16) + (uint32_t)cc, v + 16 * h);
          i8r_ld16(td + ((uint32_t)(16 * h) << 16) + (uint32_t)(GATED ? BN / 2 + cc : cc + 16), v + 16 * h + 8);
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 32; ++e) asm volatile("" : "+r"(v[e]));          // (the loads' results are there from here on)
        if (cc + CH >= c_end) {              // the warp's sums have left tensor memory
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[i & 1], 0));
        }
        const float4 s0 = *reinterpret_cast<const float4*>(w_s + 4 * 32 + t4 * 8), s1 = *reinterpret_cast<const float4*>(w_s + 4 * 32 + t4 * 8 + 4);
        const float sv[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        float o[32];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {    // int8_finish, two columns at a time (the sum of two fp16 numbers rounds to fp16 the same from fp32)
          const int b = (e >> 2) & 3;
          const float sa = sca[(e >> 4) * 2 + ((e >> 1) & 1)];
          float f0 = __fmul_rn(__fmul_rn(__fmul_rn((float)(int)v[e], sa), sv[b * 2]), 1.0f / (127.0f * 127.0f));
          float f1 = __fmul_rn(__fmul_rn(__fmul_rn((float)(int)v[e + 1], sa), sv[b * 2 + 1]), 1.0f / (127.0f * 127.0f));
          if (any_bias) {
            const float2 bv = *reinterpret_cast<const float2*>(w_s + 5 * 32 + t4 * 8 + b * 2);
            f0 = __fadd_rn(f0, bv.x), f1 = __fadd_rn(f1, bv.y);
          }
          __half2 h = __floats2half2_rn(f0, f1);
          if (all > 0) h = __hadd2_rn(h, __floats2half2_rn(odd[e], odd[e + 1]));
          const float2 r = __half22float2(h);
          o[e] = r.x, o[e + 1] = r.y;
        }
        if constexpr (GATED) {               // columns b of the first layer and b + 2 of the second: the product takes the first's place
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if ((e & 8) == 0) o[e] = __fmul_rn(silu_act<T>(dt<T>::rd(o[e])), dt<T>::rd(o[e + 8]));
        }
        if (p.boxes) {                       // boxes of 32 rows x 32 columns (GATED: in two halves)
          const int half = GATED ? (cc >> 4) & 1 : 0;
          const bool last = !GATED || half == 1;
          uint8_t* box = out + (boxes & 1u) * I8R_OUT;
          if (half == 0) {
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the box before the last has left
            __syncwarp();
          }
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            if (GATED && (e & 8) != 0) continue;
            const int row = (e >> 4) * 16 + ((e >> 1) & 1) * 8 + g, piece = half * 2 + ((e >> 2) & 3);
            *reinterpret_cast<uint32_t*>(box + row * 64 + ((piece ^ ((row >> 1) & 3)) * 16) + t4 * 4) = i8r_pack<T>(o[e], o[e + 1]);
          }
          if (last) {
            fence_proxy_async();
            __syncwarp();
            const int c0 = n0 + (cc & ~31);
            if (lane == 0) {
              if (r0 < p.M && c0 < p.N)
                asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&map_y), "r"(c0), "r"(r0),
                             "r"(smem_u32(box))
                             : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            ++boxes;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            if (GATED && (e & 8) != 0) continue;
            const int row = r0 + (e >> 4) * 16 + ((e >> 1) & 1) * 8 + g, c = n0 + cc + ((e >> 2) & 3) * 8 + 2 * t4 + (e & 1);
            if (row < p.M && c < p.N) dt<T>::st(p.y, (size_t)row * p.N + c, o[e]);
          }
        }
#pragma unroll
        for (int c = 0; c + 1 < NCH; ++c) scale[c] = scale[c + 1], q0[c] = q0[c + 1], q1[c] = q1[c + 1];
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

// the output as a map of boxes of 32 rows x 32 numbers of two bytes (their type does not matter to a copy)
int i8r_out_map(const void* y, int M, int N, CUtensorMap* out) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled entry point not available");
    return LL_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M}, strides[1] = {(cuuint64_t)N * 2};
  cuuint32_t box[2] = {32, 32}, estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)y, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): output M=%d N=%d", (int)r, M, N);
    return LL_ERR_CUDA;
  }
  return LL_OK;
}

template <typename T, int BN, bool GATED>
int i8r_launch(const I8RParams<T>& q, cudaStream_t st, const int8_t* ca) {
  constexpr int COLS = GATED ? BN / 2 : BN;
  I8RParams<T> p = q;
  p.mtiles = (p.M + 255) / 256, p.ntiles = (p.N + COLS - 1) / COLS;
  p.boxes = sizeof(T) == 2 && p.N % 8 == 0 && ((uintptr_t)p.y & 15) == 0;
  p.word = wait_word();
  const long long tiles = (long long)p.mtiles * p.ntiles;
  LL_CHECK_ARG(tiles < (1ll << 30), "int8 linear: too many tiles");
  CUtensorMap mx, m0, m1, my;
  if (int r = make_map_i8(ca, p.M, p.K, 128, &mx)) return r;
  if (int r = make_map_i8(p.layer[0].cb, p.N, p.K, BN / 2, &m0)) return r;
  if (int r = make_map_i8(p.layer[GATED ? 1 : 0].cb, p.N, p.K, BN / 2, &m1)) return r;
  my = mx;
  if (p.boxes) {
    if (int r = i8r_out_map(p.y, p.M, p.N, &my)) return r;
  }
  static PerDevice configured;
  if (!configured) {
    LL_CUDA(cudaFuncSetAttribute(int8_pair_kernel<T, BN, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, i8r_smem(BN)));
    configured.mark();
  }
  const int pairs = sm_count() > 1 ? sm_count() / 2 : 1;
  LL_CUDA(launch(int8_pair_kernel<T, BN, GATED>, dim3(2 * (unsigned)(tiles < pairs ? tiles : pairs)), dim3(I8R_THREADS), i8r_smem(BN), st, true, mx, m0, m1, my, p));
  LL_LAUNCH_OK("int8_pair_kernel");
  return LL_OK;
}

// Entries of a list up to which the finishing warps add the outlier part themselves.  us, here / in the kernel before, one layer of 11008 x 4096
// with 18, 26, 30 outliers: 65 rows 36 / 32, 41 / 33, 43 / 33; 512 rows 55 / 60, 67 / 64, 73 / 65; 2048 rows 143 / 175, 175 / 183, 191 / 187.
int i8r_limit(int rows) { return rows <= 384 ? 16 : 28; }
template <typename T, bool GATED>
int int8_rows(const T* x, const I8Layer<T>& l0, const I8Layer<T>& l1, T* y, int M, int N, int K, float thr, void* base, cudaStream_t st) {
  for (int r0 = 0; r0 < M; r0 += I8R_PASS) {
    const int rows = min(I8R_PASS, M - r0);
    const Ws w = carve(base, rows, N, K, GATED ? 2 : 1, false);
    const T* xp = x + (size_t)r0 * K;
    if (int r = int8_prepare<T>(xp, w, base, rows, K, thr, st)) return r;
    // a CTA per tile where that is a few rounds of four an SM; more tiles are taken one by one by that many CTAs, so that passing over blocks with
    // short lists stays cheap (2048 x 11008: 1.5 us instead of 6.5).
    const int items = (rows + 63) / 64 * ((N + 63) / 64) * (GATED ? 2 : 1), ctas = 4 * (sm_count() > 0 ? sm_count() : 148), limit = i8r_limit(rows);
    const bool words = l0.cbt != nullptr && l1.cbt != nullptr && (N & 3) == 0 && (((uintptr_t)l0.cbt | (uintptr_t)l1.cbt) & 3) == 0;
    LL_CUDA(launch(words ? int8_outlier_rows_kernel<T, true> : int8_outlier_rows_kernel<T, false>, dim3(items <= 4 * ctas ? items : ctas), dim3(256), 0, st,
                   true, l0, l1, xp, (const int32_t*)w.idx, (const int32_t*)w.count, w.next, w.odd, rows, N, K, GATED ? 2 : 1, i8r_pitch(N), limit));
    LL_LAUNCH_OK("int8_outlier_rows_kernel");
    I8RParams<T> p{};
    p.layer[0] = l0, p.layer[1] = l1, p.x = xp, p.sca = w.sca, p.idx = w.idx, p.count = w.count, p.y = y + (size_t)r0 * N;
    p.odd = w.odd, p.pitch = i8r_pitch(N), p.limit = limit;
    p.M = rows, p.N = N, p.K = K;
    // tiles of half the columns take 0.6 of the time: what the waves cost (as the dense products' rule)
    const long long pairs = sm_count() > 1 ? sm_count() / 2 : 1, mt = (rows + 255) / 256, wide = GATED ? 128 : 256;
    const long long w256 = (mt * ((N + wide - 1) / wide) + pairs - 1) / pairs, w128 = (mt * ((2 * N + wide - 1) / wide) + pairs - 1) / pairs;
    const int r = 3 * w128 < 5 * w256 ? i8r_launch<T, 128, GATED>(p, st, w.ca) : i8r_launch<T, 256, GATED>(p, st, w.ca);
    if (r) return r;
  }
  return LL_OK;
}

size_t i8_workspace_bytes(int M, int N, int K, int layers) {
  const size_t pass = carve(nullptr, M < 64 ? M : 64, N, K, layers, true).total;
  if (M <= 64) return pass;
  const size_t rows = carve(nullptr, M < I8R_PASS ? M : I8R_PASS, N, K, layers, false).total;
  return rows > pass ? rows : pass;
}

// prompts go through one product; with a workspace that only holds a pass of 64 rows, through passes
template <typename T, bool GATED>
int int8_run(const void* x, const I8Layer<T>& l0, const I8Layer<T>& l1, void* y, int M, int N, int K, float thr, void* base, size_t bytes, cudaStream_t st) {
  if (M > 64 && bytes >= i8_workspace_bytes(M, N, K, GATED ? 2 : 1)) return int8_rows<T, GATED>((const T*)x, l0, l1, (T*)y, M, N, K, thr, base, st);
  for (int m0 = 0; m0 < M; m0 += 64) {
    const int r = int8_pass<T, GATED>((const T*)x + (size_t)m0 * K, l0, l1, (T*)y + (size_t)m0 * N, min(64, M - m0), N, K, thr, base, st);
    if (r) return r;
  }
  return LL_OK;
}

}  // namespace
}  // namespace llb

using namespace llb;

extern "C" {

size_t ll_int8_workspace_bytes(int M, int N, int K) { return i8_workspace_bytes(M, N, K, 1); }
size_t ll_int8_gated_workspace_bytes(int M, int N, int K) { return i8_workspace_bytes(M, N, K, 2); }

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
#define LL_I8(T)                                                        \
  do {                                                                  \
    const I8Layer<T> l{cb, cbt, scb, (const T*)bias};                   \
    return int8_run<T, false>(x, l, l, y, M, N, K, threshold, workspace, workspace_bytes, st); \
  } while (0)
  if (act_dtype == LL_BF16) LL_I8(__nv_bfloat16);
  if (act_dtype == LL_F16) LL_I8(__half);
  if (act_dtype == LL_F32) LL_I8(float);
#undef LL_I8
  set_error("int8_linear: unsupported activation dtype %d", act_dtype);
  return LL_ERR_UNSUPPORTED;
}

int ll_int8_gated(const void* x, const int8_t* cb1, const int8_t* cbt1, const float* scb1, const void* bias1, const int8_t* cb2, const int8_t* cbt2,
                  const float* scb2, const void* bias2, void* h, int M, int N, int K, float threshold, void* workspace, size_t workspace_bytes,
                  ll_stream stream) {
  LL_CHECK_ARG(x && cb1 && scb1 && cb2 && scb2 && h && workspace, "null pointer");
  LL_CHECK_ARG(M > 0 && N > 0 && K > 0 && K % 128 == 0, "int8 linear needs K %% 128 == 0 (M=%d N=%d K=%d)", M, N, K);
  LL_CHECK_ARG((((uintptr_t)cb1 | (uintptr_t)cb2) & 15) == 0 && ((uintptr_t)workspace & 255) == 0, "cb must be 16-byte, workspace 256-byte aligned");
  LL_CHECK_ARG(workspace_bytes >= ll_int8_gated_workspace_bytes(M < 64 ? M : 64, N, K), "workspace too small");
  typedef __nv_bfloat16 T;
  const I8Layer<T> l0{cb1, cbt1, scb1, (const T*)bias1}, l1{cb2, cbt2, scb2, (const T*)bias2};
  return int8_run<T, true>(x, l0, l1, h, M, N, K, threshold, workspace, workspace_bytes, (cudaStream_t)stream);
}

}  // extern "C"
