// Eight-element vectors of the expert outputs and of the combined tokens, and the choice of an
// instantiation by their dtypes.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../core/ptx.cuh"
#include "a2a_kernels.h"

namespace pplx {

template <typename T>
struct Vec8;

template <>
struct Vec8<float> {
  int4 a, b;
  __device__ __forceinline__ void load_cg(const void* p) {
    a = ptx::ld_cg_v4(p);
    b = ptx::ld_cg_v4(static_cast<const uint8_t*>(p) + 16);
  }
  __device__ __forceinline__ void load_nc(const void* p) {
    a = ptx::ld_nc_v4(p);
    b = ptx::ld_nc_v4(static_cast<const uint8_t*>(p) + 16);
  }
  __device__ __forceinline__ void fma_into(float (&acc)[8], float w) const {
    acc[0] = fmaf(w, __int_as_float(a.x), acc[0]);
    acc[1] = fmaf(w, __int_as_float(a.y), acc[1]);
    acc[2] = fmaf(w, __int_as_float(a.z), acc[2]);
    acc[3] = fmaf(w, __int_as_float(a.w), acc[3]);
    acc[4] = fmaf(w, __int_as_float(b.x), acc[4]);
    acc[5] = fmaf(w, __int_as_float(b.y), acc[5]);
    acc[6] = fmaf(w, __int_as_float(b.z), acc[6]);
    acc[7] = fmaf(w, __int_as_float(b.w), acc[7]);
  }
};

__device__ __forceinline__ float2 unpack2(__half2 h) { return __half22float2(h); }
__device__ __forceinline__ float2 unpack2(__nv_bfloat162 h) { return __bfloat1622float2(h); }

template <typename T2>
struct Vec8Half {
  int4 a;
  __device__ __forceinline__ void load_cg(const void* p) { a = ptx::ld_cg_v4(p); }
  __device__ __forceinline__ void load_nc(const void* p) { a = ptx::ld_nc_v4(p); }
  __device__ __forceinline__ void fma_into(float (&acc)[8], float w) const {
    const T2* h = reinterpret_cast<const T2*>(&a);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack2(h[j]);
      acc[2 * j] = fmaf(w, f.x, acc[2 * j]);
      acc[2 * j + 1] = fmaf(w, f.y, acc[2 * j + 1]);
    }
  }
};
template <>
struct Vec8<__half> : Vec8Half<__half2> {};
template <>
struct Vec8<__nv_bfloat16> : Vec8Half<__nv_bfloat162> {};

__device__ __forceinline__ int4 pack8(const float (&acc)[8], __half*) {
  int4 r;
  __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2half2_rn(acc[2 * j], acc[2 * j + 1]);
  return r;
}
__device__ __forceinline__ int4 pack8(const float (&acc)[8], __nv_bfloat16*) {
  int4 r;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
  return r;
}

// Calls fn.template operator()<T, U>() for the (in, out) dtype pair.
template <typename F>
cudaError_t dispatch_types(DType in, DType out, F&& fn) {
  const bool out_bf16 = out == DType::kBF16;
  if (out != DType::kBF16 && out != DType::kF16) return cudaErrorInvalidValue;
  switch (in) {
    case DType::kF32:
      return out_bf16 ? fn.template operator()<float, __nv_bfloat16>()
                      : fn.template operator()<float, __half>();
    case DType::kF16:
      return out_bf16 ? fn.template operator()<__half, __nv_bfloat16>()
                      : fn.template operator()<__half, __half>();
    case DType::kBF16:
      return out_bf16 ? fn.template operator()<__nv_bfloat16, __nv_bfloat16>()
                      : fn.template operator()<__nv_bfloat16, __half>();
  }
  return cudaErrorInvalidValue;
}

}  // namespace pplx
