// Weights of a few rows on their way through CUDA cores: 16-byte loads, their eight numbers as floats, the sums.
#pragma once
#include "common.cuh"

namespace llb {
namespace {

// 16 bytes of weights, read once (asm volatile: the loads stay together ahead of the sums; left to the compiler they went one by one)
__device__ __forceinline__ uint4 sr_ld(const __nv_bfloat16* row, int piece) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(reinterpret_cast<const uint4*>(row) + piece));
  return v;
}
// 16 bytes of a row that many warps read (asm volatile: it stays behind the wait for the kernel that made it)
__device__ __forceinline__ uint4 sr_ldx(const __nv_bfloat16* row, int piece) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(reinterpret_cast<const uint4*>(row) + piece));
  return v;
}
__device__ __forceinline__ void sr_floats(const uint4& u, float (&x)[8]) {
  x[0] = __uint_as_float(u.x << 16), x[1] = __uint_as_float(u.x & 0xffff0000u), x[2] = __uint_as_float(u.y << 16), x[3] = __uint_as_float(u.y & 0xffff0000u);
  x[4] = __uint_as_float(u.z << 16), x[5] = __uint_as_float(u.z & 0xffff0000u), x[6] = __uint_as_float(u.w << 16), x[7] = __uint_as_float(u.w & 0xffff0000u);
}
// acc += the products of eight bf16 numbers with eight of x
__device__ __forceinline__ void sr_dot(float& acc, const float (&w)[8], const float (&x)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) acc = fmaf(w[i], x[i], acc);
}

}  // namespace
}  // namespace llb
