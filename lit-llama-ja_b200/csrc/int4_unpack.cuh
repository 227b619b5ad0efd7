// Packed int4 weights (checkpoint bytes [K/2][N], even k in the low half) on their way into tensor memory: the map of the bytes, the loads that
// transpose them, the arithmetic that unpacks them with the reference's two bf16 roundings (ref: lit_llama/quantization.py:399-408) and the
// stores that leave them as the A operand.  Shared by the kernels for many rows and for batches.
#pragma once
#include "tcgen05.cuh"

namespace llb {
namespace {

constexpr int R4_K = 128, R4_WBYTES = 128 * R4_K / 2;      // k of a step; its packed bytes: 128 columns (one box, or two of 64)
constexpr int R4_SZ = 128 * 4;                             // a step's scales and zeros: a word per column

__device__ __forceinline__ void r4_box(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
               "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void r4_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                 "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr)
               : "memory");
}
// 32 k-pairs x 16 columns of packed bytes, four bytes of a column's k-pairs in a word: r[0], r[1] (r[2], r[3]: the next 16 k-pairs) hold
// columns lane / 4 and lane / 4 + 8 and the k-pairs whose rows the lanes 4 (lane % 4) .. + 3 point at
__device__ __forceinline__ void r4_ldt(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// 16 lanes x 32 columns of tensor memory: of every 8 columns a thread writes columns 2 (lane % 4), + 1 of lanes lane / 4 and lane / 4 + 8
__device__ __forceinline__ void r4_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ uint32_t r4_prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ uint32_t r4_sub2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t r4_add2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t r4_mul2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// four bytes of a column -> the bf16 pairs of their k: (128 + q) - z, where z is 128 + zero if that is a bf16 number (then the difference is
// rounded once, as the reference's q - zero is); FRACTION: (128 + q) - 128, exact, minus the zero z; times the scale
template <bool FRACTION>
__device__ __forceinline__ void r4_unpack(uint32_t w, uint32_t s2, uint32_t z2, uint32_t& o0, uint32_t& o1, uint32_t& o2, uint32_t& o3) {
  const uint32_t lo = w & 0x0f0f0f0fu, hi = (w >> 4) & 0x0f0f0f0fu;
  const uint32_t p = r4_prmt(lo, hi, 0x5140), q = r4_prmt(lo, hi, 0x7362);
  uint32_t v[4] = {r4_prmt(p, 0x43u, 0x4140), r4_prmt(p, 0x43u, 0x4342), r4_prmt(q, 0x43u, 0x4140), r4_prmt(q, 0x43u, 0x4342)};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (FRACTION) v[i] = r4_sub2(v[i], 0x43004300u);
    v[i] = r4_mul2(r4_sub2(v[i], z2), s2);
  }
  o0 = v[0], o1 = v[1], o2 = v[2], o3 = v[3];
}
// what r4_ldt brought, as r4_st16 stores it; s2, z2: the scales and zeros of columns lane / 4 and lane / 4 + 8
template <bool FRACTION>
__device__ __forceinline__ void r4_unpack16(const uint32_t (&w)[4], const uint32_t* s2, const uint32_t* z2, uint32_t (&r)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int o = (i >> 1) * 8 + (i & 1) * 2;
    r4_unpack<FRACTION>(w[i], s2[i & 1], z2[i & 1], r[o], r[o + 1], r[o + 4], r[o + 5]);
  }
}

// Where a lane points r4_ldt at in a box of 64 rows of WIDTH columns of packed bytes (16-byte pieces swizzled over the box's width): of 16
// k-pairs, four lanes name those of which the threads of one lane % 4 write two and two tensor-memory columns.
template <int WIDTH>
struct R4Row {
  uint32_t at, turn;
  __device__ __forceinline__ explicit R4Row(int lane) {
    const int li = lane & 15, krow = (lane >> 4) * 16 + (li >> 2) * 2 + (li & 1) + (li & 2) * 4;
    at = (uint32_t)(krow * WIDTH), turn = (uint32_t)((WIDTH == 128 ? krow & 7 : (krow >> 1) & 3) * 16);
  }
};
// A warp's 32 columns of a step (64 k-pairs; `src`: their box, `col`: the first's place in it, `nums`: shared-memory address of their scales and
// zeros) into 64 columns of its lanes of tensor memory.  Where 128 + zero is a bf16 number (any whole zero of an RTN / GPTQ checkpoint) one
// subtraction does; a column's zero may be so and its neighbour's not: the warp goes one way.
template <int WIDTH>
__device__ __forceinline__ void r4_unpack_step(uint32_t src, uint32_t col, const R4Row<WIDTH>& row, uint32_t nums, uint32_t ta) {
  uint32_t s2[4], z2[4], m2[4];
  bool whole = true;
#pragma unroll
  for (int i = 0; i < 4; ++i) {              // columns lane / 4 + 8 i
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(nums + (uint32_t)(((threadIdx.x & 31) >> 2) * 4 + i * 32)));
    s2[i] = r4_prmt(v, 0u, 0x1010), z2[i] = r4_prmt(v, 0u, 0x3232);
    m2[i] = r4_add2(z2[i], 0x43004300u);
    whole = whole && r4_sub2(m2[i], 0x43004300u) == z2[i];
  }
  whole = __all_sync(0xffffffffu, whole);
#pragma unroll
  for (int h = 0; h < 2; ++h) {              // 16 of the columns
#pragma unroll
    for (int c = 0; c < 2; ++c) {            // 32 of the k-pairs
      uint32_t w[4], r[16];
      r4_ldt(src + row.at + ((col + (uint32_t)(h * 16)) ^ row.turn) + (uint32_t)(c * 32 * WIDTH), w);
      if (whole) r4_unpack16<false>(w, s2 + 2 * h, m2 + 2 * h, r);
      else r4_unpack16<true>(w, s2 + 2 * h, z2 + 2 * h, r);
      r4_st16(ta + ((uint32_t)(16 * h) << 16) + 32u * c, r);
    }
  }
}

// The numbers of steps kb .. kb + 3 of a column (a row of scales or zeros, [G] in groups of `per` steps), in one load where rows allow it:
// wide 4: one of 8 bytes, 2: two of 4, 1: one by one.
__device__ __forceinline__ uint2 r4_four(const __nv_bfloat16* src, size_t row, int kb, int steps, int G, int per, int wide) {
  const uint16_t* at = reinterpret_cast<const uint16_t*>(src) + row;
  if (wide == 4) return *reinterpret_cast<const uint2*>(at + kb);
  if (wide == 2) return make_uint2(*reinterpret_cast<const uint32_t*>(at + kb), *reinterpret_cast<const uint32_t*>(at + min(kb + 2, G - 2)));
  uint32_t v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = at[min(kb + j, steps - 1) / per];
  return make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
}
inline int r4_wide(const void* s0, const void* z0, const void* s1, const void* z1, int G, int per) {
  const uintptr_t at = (uintptr_t)s0 | (uintptr_t)z0 | (uintptr_t)s1 | (uintptr_t)z1;
  return per != 1 ? 1 : G % 4 == 0 && at % 8 == 0 ? 4 : G % 2 == 0 && at % 4 == 0 ? 2 : 1;
}
// step kb + j's scale (low half) and zero of a column, from what r4_four brought
__device__ __forceinline__ uint32_t r4_word(int j, const uint2& sv, const uint2& zv) {
  return r4_prmt(j < 2 ? sv.x : sv.y, j < 2 ? zv.x : zv.y, j & 1 ? 0x7632 : 0x5410);
}

// packed bytes [K/2][N] as a 2-D map, boxes of `width` (64 or 128) columns x 64 rows: 128 where a CTA's columns lie side by side (half as many
// pieces for the copy engine)
int r4_weight_map(const void* qw, int N, int K, int width, CUtensorMap* out) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled entry point not available");
    return LL_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)(K / 2)}, strides[1] = {(cuuint64_t)N};
  cuuint32_t box[2] = {(cuuint32_t)width, R4_K / 2}, estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)qw, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        width == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): packed weights N=%d K=%d", (int)r, N, K);
    return LL_ERR_CUDA;
  }
  return LL_OK;
}

}  // namespace
}  // namespace llb
