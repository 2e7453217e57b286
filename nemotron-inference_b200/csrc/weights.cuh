// Weights of the dense and scaled-FP8 linears as the FP32 values that the reference multiplies with.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"

namespace nmoe {

// The activation the linear multiplies with: the row itself, or for the scaled-FP8 family its
// round trip through E4M3 (scaled_fp8_linear.cu:94-106).
__device__ __forceinline__ float input_value(float v, float fp8_scale) {
  if (fp8_scale == 0.0f) return v;
  return __fmul_rn(decode_e4m3(encode_e4m3(__fdiv_rn(v, fp8_scale))), fp8_scale);
}

template <int KIND>
struct WeightVector;  // 16 bytes of W as FP32 values
template <>
struct WeightVector<kWeightFp8> {
  static constexpr int kCount = 16;
  static __device__ __forceinline__ void unpack(const uint4& raw, float scale, float (&v)[16]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __half2_raw two = __nv_cvt_fp8x2_to_halfraw2(
          static_cast<__nv_fp8x2_storage_t>(w[i >> 1] >> (16 * (i & 1))), __NV_E4M3);
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
      v[2 * i] = __fmul_rn(f.x, scale);
      v[2 * i + 1] = __fmul_rn(f.y, scale);
    }
  }
};
// Half of such a vector of sixteen.
template <int KIND>
__device__ __forceinline__ void unpack_half(const uint4& raw, int half, float scale, float (&v)[8]) {
  static_assert(KIND == kWeightFp8, "sixteen codes");
  const uint32_t w[2] = {half != 0 ? raw.z : raw.x, half != 0 ? raw.w : raw.y};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2_raw two = __nv_cvt_fp8x2_to_halfraw2(
        static_cast<__nv_fp8x2_storage_t>(w[i >> 1] >> (16 * (i & 1))), __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
    v[2 * i] = __fmul_rn(f.x, scale);
    v[2 * i + 1] = __fmul_rn(f.y, scale);
  }
}
template <>
struct WeightVector<kWeightBf16> {
  static constexpr int kCount = 8;
  static __device__ __forceinline__ void unpack(const uint4& raw, float, float (&v)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};
template <>
struct WeightVector<kWeightF32> {
  static constexpr int kCount = 4;
  static __device__ __forceinline__ void unpack(const uint4& raw, float, float (&v)[4]) {
    v[0] = __uint_as_float(raw.x);
    v[1] = __uint_as_float(raw.y);
    v[2] = __uint_as_float(raw.z);
    v[3] = __uint_as_float(raw.w);
  }
};

}  // namespace nmoe
