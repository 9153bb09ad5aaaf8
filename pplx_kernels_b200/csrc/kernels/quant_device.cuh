// Block quantisation bf16 -> e4m3 inside a warp: 16 values per lane, 8 lanes per 128-column
// block.  Shared by the sends that convert tokens on their way (dispatch.cu, single_rank.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp8.h>

namespace pplx {

// `lo`, `hi`: this lane's 16 bf16 values (read only when `live`).  Returns the 16 e4m3 values
// in `q` and the scale of the lane's block: max(amax, 1e-4) / 448, or with `pow2` the smallest
// power of two that is not below it.  All 32 lanes call it (shuffles).
__device__ __forceinline__ void warp_quantize16(const int4& lo, const int4& hi, bool live, bool pow2,
                                                int4& q, float& scale) {
  float f[16];
  float amax = 0.f;
  if (live) {
    const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&lo);
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&hi);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = __bfloat1622float2(a[j]);
      const float2 y = __bfloat1622float2(b[j]);
      f[2 * j] = x.x;
      f[2 * j + 1] = x.y;
      f[8 + 2 * j] = y.x;
      f[8 + 2 * j + 1] = y.y;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
  }
  // 8 consecutive lanes hold one 128-column block.
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
  if (!live) return;
  amax = fmaxf(amax, 1e-4f);
  float inv = 448.0f / amax;
  scale = amax / 448.0f;
  if (pow2) {
    // The smallest power of two that is not below amax / 448: hardware block scaling.
    const uint32_t bits = __float_as_uint(scale);
    scale = __uint_as_float(((bits >> 23) + ((bits & 0x7fffffu) != 0u ? 1u : 0u)) << 23);
    inv = 1.0f / scale;
  }
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t p0 = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j] * inv, f[4 * j + 1] * inv),
                                                 __NV_SATFINITE, __NV_E4M3);
    const uint32_t p1 = __nv_cvt_float2_to_fp8x2(
        make_float2(f[4 * j + 2] * inv, f[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    w[j] = p0 | (p1 << 16);
  }
  q = make_int4(w[0], w[1], w[2], w[3]);
}

}  // namespace pplx
