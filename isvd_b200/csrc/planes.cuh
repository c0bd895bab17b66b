// Device helpers of the bf16 plane representation x = x0 + x1 + x2 (+ O(2^-24 |x|)), shared by
// the kernels that write planes (splits, GEMM epilogues).
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace isvdb {

// Piece q of x: x0 = bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1) (round to nearest).
template <class T>
__device__ __forceinline__ void split3(T x, __nv_bfloat16 *o, int np) {
  double r = (double)x;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q >= np) break;
    const __nv_bfloat16 h = __double2bfloat16(r);
    o[q] = h;
    r -= (double)__bfloat162float(h);
  }
}

// Pieces of an FP32 value in FP32 arithmetic: x - bf16(x) is exact in FP32 (the rounding error of
// an 8-bit rounding of a 24-bit significand), and so is the next remainder.  Infinities and NaN stay
// whole in the first piece; a value that would round up to infinity is truncated there instead.
__device__ __forceinline__ void split3f(float x, __nv_bfloat16 *o) {
  __nv_bfloat16 h0 = __float2bfloat16_rn(x);
  float f0 = __bfloat162float(h0), r1 = x - f0;
  if (!(fabsf(f0) <= 3.4028235e38f)) {
    const bool finite = fabsf(x) <= 3.4028235e38f;
    f0 = finite ? __uint_as_float(__float_as_uint(x) & 0xffff0000u) : x;
    h0 = __float2bfloat16_rn(f0);
    r1 = finite ? x - f0 : 0.f;
  }
  const __nv_bfloat16 h1 = __float2bfloat16_rn(r1);
  o[0] = h0;
  o[1] = h1;
  o[2] = __float2bfloat16_rn(r1 - __bfloat162float(h1));
}

__device__ __forceinline__ uint4 pack8(const __nv_bfloat16 *v) {
  uint4 u;
  u.x = (uint32_t)__bfloat16_as_ushort(v[0]) | ((uint32_t)__bfloat16_as_ushort(v[1]) << 16);
  u.y = (uint32_t)__bfloat16_as_ushort(v[2]) | ((uint32_t)__bfloat16_as_ushort(v[3]) << 16);
  u.z = (uint32_t)__bfloat16_as_ushort(v[4]) | ((uint32_t)__bfloat16_as_ushort(v[5]) << 16);
  u.w = (uint32_t)__bfloat16_as_ushort(v[6]) | ((uint32_t)__bfloat16_as_ushort(v[7]) << 16);
  return u;
}

}  // namespace isvdb
