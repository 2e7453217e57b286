// One row by one block: RMSNorm, then the dynamic NVFP4 quantiser (csrc/quant.cu describes both; the
// small-batch front end in csrc/front.cu runs the same steps).
#pragma once

#include "common.cuh"

namespace nmoe {

constexpr int kWarpsPerBlock = 8;

__device__ __forceinline__ float (&eight_of(float (&v)[16], int i))[8] {
  return *reinterpret_cast<float(*)[8]>(&v[i]);
}

template <bool BF16>
__device__ __forceinline__ void load8(const void* base, size_t index, float (&v)[8]) {
  if constexpr (BF16) {
    const uint4 raw = *reinterpret_cast<const uint4*>(
        reinterpret_cast<const __nv_bfloat16*>(base) + index);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  } else {
    const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + index);
    const float4 b =
        *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + index + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}

// tensor scale rule of nvfp4_packing.cpp:119-126
__device__ __forceinline__ float tensor_scale_from_amax(float amax) {
  return amax > kFp4Max * kFp8Max ? clamp_scale(__fdiv_rn(amax, kFp4Max * kFp8Max)) : 1.0f;
}

// Codes of half a 16-element block (nvfp4_packing.cpp:140-153): x / divisor, IEEE-rounded, then
// E2M1.  One reciprocal per block and a residual correction per value give the correctly rounded
// quotient unless the divisor's significand is all ones (div_by_reciprocal), where the division
// itself is used.
__device__ __forceinline__ uint32_t quantize_half_block(const float (&v)[8], float divisor,
                                                        float reciprocal) {
  uint32_t word = 0;
  if ((__float_as_uint(divisor) & 0x007fffffu) != 0x007fffffu) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const uint32_t byte = encode_e2m1x2(div_by_reciprocal(v[i], divisor, reciprocal),
                                          div_by_reciprocal(v[i + 1], divisor, reciprocal));
      word |= (byte & 0xffu) << (4 * i);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const uint32_t byte = encode_e2m1x2(__fdiv_rn(v[i], divisor), __fdiv_rn(v[i + 1], divisor));
      word |= (byte & 0xffu) << (4 * i);
    }
  }
  return word;
}

template <int CHUNKS>
struct NormShared {
  float4 row_values[CHUNKS * kWarpsPerBlock * 32 * 2];
  float partial_sums[kWarpsPerBlock * 32];
  float warp_max[kWarpsPerBlock];
};

// By all kWarpsPerBlock * 32 threads.  Thread c owns the 8-element chunks c, c + 256, ...: it loads them
// at once, and hands the values over through shared memory for the sum of squares, in which thread t
// adds up columns t, t + 256, ... in order.  `inv_rms_known()` runs once inv_rms_out[row] is written
// (by thread 0); it may hand that on to blocks that are running, so the pointer is not __restrict__: the
// store must not move behind what the callback does.
template <bool BF16, int CHUNKS, typename Known>
__device__ __forceinline__ void norm_quant_by_block(
    const void* in, int row, int cols, const float* __restrict__ norm_weight, float eps,
    float* __restrict__ normalized, uint8_t* __restrict__ packed, uint8_t* __restrict__ sf_row_major,
    uint8_t* __restrict__ sf_tiled, int k_tiles, float* __restrict__ tensor_scale,
    float* inv_rms_out, bool word_scales, NormShared<CHUNKS>& shared,
    Known&& inv_rms_known) {
  constexpr int kThreads = kWarpsPerBlock * 32;
  auto& row_values = shared.row_values;
  auto& partial_sums = shared.partial_sums;
  auto& warp_max = shared.warp_max;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunks = cols / 8;
  const size_t row_base = static_cast<size_t>(row) * cols;
  float w[CHUNKS][8];
  if (norm_weight != nullptr) {
#pragma unroll
    for (int j = 0; j < CHUNKS; ++j) {
      if (j * kThreads + tid < chunks) load8<false>(norm_weight, (j * kThreads + tid) * 8, w[j]);
    }
  }
  wait_for_predecessor();

  float v[CHUNKS][8];
#pragma unroll
  for (int j = 0; j < CHUNKS; ++j) {
    const int ch = j * kThreads + tid;
    if (ch < chunks) {
      load8<BF16>(in, row_base + static_cast<size_t>(ch) * 8, v[j]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[j][i] = 0.0f;
    }
  }

  if (norm_weight != nullptr) {
    // the association of norm_quant_kernel
#pragma unroll
    for (int j = 0; j < CHUNKS; ++j) {
      row_values[(j * kThreads + tid) * 2] = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
      row_values[(j * kThreads + tid) * 2 + 1] = make_float4(v[j][4], v[j][5], v[j][6], v[j][7]);
    }
    __syncthreads();
    const float* values = reinterpret_cast<const float*>(row_values);
    float partial = 0.0f;
#pragma unroll 8
    for (int it = 0; it < CHUNKS * 8; ++it) {
      const float x = values[it * 256 + tid];
      partial = __fmaf_rn(x, x, partial);
    }
    partial_sums[tid] = partial;
    __syncthreads();
    // strides 128, 64 and 32 of the halving tree, by every warp; then inside the warp
    const float* p = partial_sums + lane;
    const float a = __fadd_rn(__fadd_rn(p[0], p[128]), __fadd_rn(p[64], p[192]));
    const float b = __fadd_rn(__fadd_rn(p[32], p[160]), __fadd_rn(p[96], p[224]));
    float sum = __fadd_rn(a, b);
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
      sum = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, stride));
    }
    sum = __shfl_sync(0xffffffffu, sum, 0);
    const float mean = __fdiv_rn(sum, static_cast<float>(cols));
    const float inv_rms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
    if (tid == 0 && inv_rms_out != nullptr) inv_rms_out[row] = inv_rms;
    inv_rms_known();
#pragma unroll
    for (int j = 0; j < CHUNKS; ++j) {
      if (j * kThreads + tid < chunks) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[j][i] = __fmul_rn(__fmul_rn(v[j][i], inv_rms), w[j][i]);
      }
    }
  }

  float half_max[CHUNKS];  // of this thread's half blocks
  float amax = 0.0f;
#pragma unroll
  for (int j = 0; j < CHUNKS; ++j) {
    half_max[j] = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) half_max[j] = fmaxf(half_max[j], fabsf(v[j][i]));
    amax = fmaxf(amax, half_max[j]);
  }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, stride));
  }
  if (lane == 0) warp_max[warp] = amax;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kWarpsPerBlock; ++i) amax = fmaxf(amax, warp_max[i]);
  const float ts = tensor_scale_from_amax(amax);
  if (tid == 0 && tensor_scale != nullptr) tensor_scale[row] = ts;

  const int blocks_per_row = cols / 16;
  const float scale_divisor = __fmul_rn(kFp4Max, ts);
  const float scale_reciprocal = __frcp_rn(scale_divisor);
#pragma unroll
  for (int j = 0; j < CHUNKS; ++j) {
    const int ch = j * kThreads + tid;
    if (normalized != nullptr && ch < chunks) {
      float* dst = normalized + row_base + static_cast<size_t>(ch) * 8;
      *reinterpret_cast<float4*>(dst) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(v[j][4], v[j][5], v[j][6], v[j][7]);
    }
    if (packed == nullptr) continue;
    // lanes 2i and 2i + 1 hold the two halves of a 16-element block
    const float block_max = fmaxf(half_max[j], __shfl_xor_sync(0xffffffffu, half_max[j], 1));
    const float bs = block_scale(block_max, scale_divisor, scale_reciprocal);
    const float divisor = __fmul_rn(ts, bs);
    const uint32_t word = quantize_half_block(v[j], divisor, __frcp_rn(divisor));
    const uint32_t sf = encode_e4m3(bs);
    // four consecutive blocks (eight lanes) are one aligned word in both layouts
    uint32_t sf_word = sf | (__shfl_down_sync(0xffffffffu, sf, 2) << 8);
    sf_word |= __shfl_down_sync(0xffffffffu, sf_word, 4) << 16;
    if (ch >= chunks) continue;
    *reinterpret_cast<uint32_t*>(packed + row_base / 2 + static_cast<size_t>(ch) * 4) = word;
    const int block = ch >> 1;
    uint8_t* row_major =
        sf_row_major != nullptr ? sf_row_major + static_cast<size_t>(row) * blocks_per_row + block
                                : nullptr;
    uint8_t* tiled =
        sf_tiled != nullptr ? sf_tiled + swizzled_scale_offset(row, block, k_tiles) : nullptr;
    if (word_scales) {
      if ((lane & 7) == 0) {
        if (row_major != nullptr) *reinterpret_cast<uint32_t*>(row_major) = sf_word;
        if (tiled != nullptr) *reinterpret_cast<uint32_t*>(tiled) = sf_word;
      }
    } else if ((lane & 1) == 0) {
      if (row_major != nullptr) *row_major = static_cast<uint8_t>(sf);
      if (tiled != nullptr) *tiled = static_cast<uint8_t>(sf);
    }
  }
}

}  // namespace nmoe
