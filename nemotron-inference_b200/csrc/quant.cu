// RMSNorm + dynamic NVFP4 activation quantiser, dequantiser and scale re-tiling.
//
// Replaces RmsNormKernel (runtime/src/backend/primitive_ops.cu:26-59), the host
// packer PackRowMajorFp32ToNvfp4 (runtime/src/backend/nvfp4_packing.cpp:90-157),
// its device mirror (runtime/src/backend/device_nvfp4_matrix.cu:64-171: amax,
// tensor scale, pack, swizzle -- four kernels and four synchronisations) and
// SwizzleRowMajorNvfp4ScalesForExecution
// (runtime/src/backend/nvfp4_scale_layout.cpp:68-87) with one pass per row.
//
// A warp or a block owns a row.  The sum of squares reproduces the reference kernel's
// association exactly (256 strided FMA partials, halving tree), so that the
// normalised activations -- and therefore every FP4 code derived from them --
// are a pure function of the input bits.  inv_rms is 1/sqrt(mean+eps) with two
// correctly rounded operations (the reference kernel's rsqrtf is within 2 ulp
// of it).
#include "common.cuh"
#include "kernels.h"
#include "quant_row.cuh"

namespace nmoe {
namespace {

__device__ __forceinline__ void zero_words(int32_t* words, int count) {
  if (blockIdx.x != 0) return;
  for (int i = threadIdx.x; i < count; i += blockDim.x) words[i] = 0;
}

// Rows of any length, and one tensor scale for a whole matrix (PER_ROW_SCALE false).
template <bool BF16, bool PER_ROW_SCALE>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
norm_quant_kernel(const void* in, int rows, int cols,
                  const float* __restrict__ norm_weight, float eps,
                  float* __restrict__ normalized, uint8_t* __restrict__ packed,
                  uint8_t* __restrict__ sf_row_major, uint8_t* __restrict__ sf_tiled, int k_tiles,
                  float* __restrict__ tensor_scale, const float* __restrict__ global_amax,
                  float* __restrict__ inv_rms_out, int32_t* __restrict__ zero, int zero_count) {
  release_successor();
  wait_for_predecessor();
  zero_words(zero, zero_count);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * kWarpsPerBlock + warp;
  if (row >= rows) return;
  const size_t row_base = static_cast<size_t>(row) * cols;

  float inv_rms = 1.0f;
  if (norm_weight != nullptr) {
    // The reference kernel keeps 256 partial sums, partial[t] accumulating columns
    // t, t+256, ... in order, and folds them with a halving tree.  Lane L owns
    // t = 8L .. 8L+7: its it-th 8-element chunk (columns 8(L+32 it) ..) is exactly
    // columns t + 256 it, so 16-byte loads reproduce the same partial sums.
    float partial[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int row_chunks = cols / 8;
#pragma unroll 4
    for (int ch = lane; ch < row_chunks; ch += 32) {
      float x[8];
      load8<BF16>(in, row_base + static_cast<size_t>(ch) * 8, x);
#pragma unroll
      for (int i = 0; i < 8; ++i) partial[i] = __fmaf_rn(x[i], x[i], partial[i]);
    }
    // halving tree: strides 128, 64, 32, 16, 8 pair lane L with L+16, +8, +4, +2, +1
    // (same i); strides 4, 2, 1 stay inside the lane
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        partial[i] = __fadd_rn(partial[i], __shfl_down_sync(0xffffffffu, partial[i], stride));
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) partial[i] = __fadd_rn(partial[i], partial[i + 4]);
    partial[0] = __fadd_rn(partial[0], partial[2]);
    partial[1] = __fadd_rn(partial[1], partial[3]);
    float sum = __fadd_rn(partial[0], partial[1]);
    sum = __shfl_sync(0xffffffffu, sum, 0);
    const float mean = __fdiv_rn(sum, static_cast<float>(cols));
    inv_rms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
    if (lane == 0 && inv_rms_out != nullptr) inv_rms_out[row] = inv_rms;
  }

  const int chunks = cols / 8;
  float ts = 1.0f;
  if constexpr (PER_ROW_SCALE) {
    float amax = 0.0f;
#pragma unroll 4
    for (int ch = lane; ch < chunks; ch += 32) {
      float v[8];
      load8<BF16>(in, row_base + static_cast<size_t>(ch) * 8, v);
      if (norm_weight != nullptr) {
        const float4 w0 = *reinterpret_cast<const float4*>(norm_weight + ch * 8);
        const float4 w1 = *reinterpret_cast<const float4*>(norm_weight + ch * 8 + 4);
        const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], inv_rms), w[i]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    }
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, stride));
    }
    ts = tensor_scale_from_amax(amax);
    if (lane == 0 && tensor_scale != nullptr) tensor_scale[row] = ts;
  } else {
    ts = tensor_scale_from_amax(*global_amax);
    if (row == 0 && lane == 0 && tensor_scale != nullptr) tensor_scale[0] = ts;
  }

  const int blocks_per_row = cols / 16;
  const int iterations = (chunks + 31) / 32;
  for (int it = 0; it < iterations; ++it) {
    const int ch = it * 32 + lane;
    const bool active = ch < chunks;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (active) {
      load8<BF16>(in, row_base + static_cast<size_t>(ch) * 8, v);
      if (norm_weight != nullptr) {
        const float4 w0 = *reinterpret_cast<const float4*>(norm_weight + ch * 8);
        const float4 w1 = *reinterpret_cast<const float4*>(norm_weight + ch * 8 + 4);
        const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], inv_rms), w[i]);
      }
      if (normalized != nullptr) {
        float* dst = normalized + row_base + static_cast<size_t>(ch) * 8;
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
    // a 16-block is shared by lanes (2i, 2i+1)
    float half_max = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) half_max = fmaxf(half_max, fabsf(v[i]));
    const float block_max = fmaxf(half_max, __shfl_xor_sync(0xffffffffu, half_max, 1));
    const float scale_divisor = __fmul_rn(kFp4Max, ts);
    const float bs = block_scale(block_max, scale_divisor, __frcp_rn(scale_divisor));
    const float divisor = __fmul_rn(ts, bs);
    const uint32_t word = quantize_half_block(v, divisor, __frcp_rn(divisor));
    if (active && packed != nullptr) {
      *reinterpret_cast<uint32_t*>(packed + row_base / 2 + static_cast<size_t>(ch) * 4) = word;
      if ((lane & 1) == 0) {
        const uint8_t sf = static_cast<uint8_t>(encode_e4m3(bs));
        const int block = ch >> 1;
        if (sf_row_major != nullptr) {
          sf_row_major[static_cast<size_t>(row) * blocks_per_row + block] = sf;
        }
        if (sf_tiled != nullptr) sf_tiled[swizzled_scale_offset(row, block, k_tiles)] = sf;
      }
    }
  }
}

// norm_quant_kernel for rows of up to ITERS * 256 elements, one tensor scale per row: the row
// is read once and stays in registers (as FP32) through the three phases -- sum of squares,
// maximum, codes -- which the general kernel above re-reads it for.  Issue-bound; 4096 rows of 2688
// 23.5 us with the general kernel, 18.4 so, 16384 rows 63 and 59.
template <bool BF16, int ITERS>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
norm_quant_row_kernel(const void* in, int rows, int cols,
                      const float* __restrict__ norm_weight, float eps,
                      float* __restrict__ normalized, uint8_t* __restrict__ packed,
                      uint8_t* __restrict__ sf_row_major, uint8_t* __restrict__ sf_tiled,
                      int k_tiles, float* __restrict__ tensor_scale,
                      float* __restrict__ inv_rms_out, bool word_scales,
                      int32_t* __restrict__ zero, int zero_count) {
  release_successor();
  wait_for_predecessor();
  zero_words(zero, zero_count);
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= rows) return;
  const size_t row_base = static_cast<size_t>(row) * cols;
  const int chunks = cols / 8;

  float v[ITERS][8];
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int ch = it * 32 + lane;
    if (ch < chunks) {
      load8<BF16>(in, row_base + static_cast<size_t>(ch) * 8, v[it]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[it][i] = 0.0f;
    }
  }

  if (norm_weight != nullptr) {
    // the association of norm_quant_kernel (zeros past the end leave the partial sums as
    // they are)
    float partial[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
#pragma unroll
      for (int i = 0; i < 8; ++i) partial[i] = __fmaf_rn(v[it][i], v[it][i], partial[i]);
    }
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        partial[i] = __fadd_rn(partial[i], __shfl_down_sync(0xffffffffu, partial[i], stride));
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) partial[i] = __fadd_rn(partial[i], partial[i + 4]);
    partial[0] = __fadd_rn(partial[0], partial[2]);
    partial[1] = __fadd_rn(partial[1], partial[3]);
    float sum = __fadd_rn(partial[0], partial[1]);
    sum = __shfl_sync(0xffffffffu, sum, 0);
    const float mean = __fdiv_rn(sum, static_cast<float>(cols));
    const float inv_rms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
    if (lane == 0 && inv_rms_out != nullptr) inv_rms_out[row] = inv_rms;
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
      const int ch = it * 32 + lane;
      if (ch < chunks) {
        const float4 w0 = *reinterpret_cast<const float4*>(norm_weight + ch * 8);
        const float4 w1 = *reinterpret_cast<const float4*>(norm_weight + ch * 8 + 4);
        const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) v[it][i] = __fmul_rn(__fmul_rn(v[it][i], inv_rms), w[i]);
      }
    }
  }

  float half_max[ITERS + 1];  // of this lane's half block, per step
  float amax = 0.0f;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    half_max[it] = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) half_max[it] = fmaxf(half_max[it], fabsf(v[it][i]));
    amax = fmaxf(amax, half_max[it]);
  }
  half_max[ITERS] = 0.0f;
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, stride));
  }
  const float ts = tensor_scale_from_amax(amax);
  if (lane == 0 && tensor_scale != nullptr) tensor_scale[row] = ts;

  if (normalized != nullptr) {
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
      const int ch = it * 32 + lane;
      if (ch < chunks) {
        float* dst = normalized + row_base + static_cast<size_t>(ch) * 8;
        *reinterpret_cast<float4*>(dst) = make_float4(v[it][0], v[it][1], v[it][2], v[it][3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(v[it][4], v[it][5], v[it][6], v[it][7]);
      }
    }
  }
  if (packed == nullptr) return;

  // Two steps at a time: a 16-element block is shared by lanes (2i, 2i+1), so the even lane of
  // a pair works out the scale of its block in the first step and the odd lane that of its
  // block in the second, and they exchange what the codes need.
  const int blocks_per_row = cols / 16;
  const float scale_divisor = __fmul_rn(kFp4Max, ts);
  const float scale_reciprocal = __frcp_rn(scale_divisor);
  const bool odd = (lane & 1) != 0;
#pragma unroll
  for (int it = 0; it < ITERS; it += 2) {
    const float first_max = fmaxf(half_max[it], __shfl_xor_sync(0xffffffffu, half_max[it], 1));
    const float second_max =
        fmaxf(half_max[it + 1], __shfl_xor_sync(0xffffffffu, half_max[it + 1], 1));
    const float block_max = odd ? second_max : first_max;
    const float bs = block_scale(block_max, scale_divisor, scale_reciprocal);
    const float divisor = __fmul_rn(ts, bs);
    const float reciprocal = __frcp_rn(divisor);
    const float other_divisor = __shfl_xor_sync(0xffffffffu, divisor, 1);
    const float other_reciprocal = __shfl_xor_sync(0xffffffffu, reciprocal, 1);
    const uint32_t sf = encode_e4m3(bs);
    // four consecutive blocks (eight lanes) are one aligned word in both layouts
    uint32_t sf_word = sf | (__shfl_down_sync(0xffffffffu, sf, 2) << 8);
    sf_word |= __shfl_down_sync(0xffffffffu, sf_word, 4) << 16;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (it + j < ITERS) {
        const int ch = (it + j) * 32 + lane;
        const bool own = odd == (j == 1);
        const uint32_t word = quantize_half_block(v[it + j], own ? divisor : other_divisor,
                                                  own ? reciprocal : other_reciprocal);
        if (ch < chunks) {
          *reinterpret_cast<uint32_t*>(packed + row_base / 2 + static_cast<size_t>(ch) * 4) = word;
        }
      }
    }
    const int ch = (it + (odd ? 1 : 0)) * 32 + lane;  // the step whose scale this lane holds
    const int block = ch >> 1;
    if (ch < chunks) {
      if (word_scales) {
        if ((lane & 7) < 2) {
          if (sf_row_major != nullptr) {
            *reinterpret_cast<uint32_t*>(
                sf_row_major + static_cast<size_t>(row) * blocks_per_row + block) = sf_word;
          }
          if (sf_tiled != nullptr) {
            *reinterpret_cast<uint32_t*>(sf_tiled + swizzled_scale_offset(row, block, k_tiles)) =
                sf_word;
          }
        }
      } else {
        if (sf_row_major != nullptr) {
          sf_row_major[static_cast<size_t>(row) * blocks_per_row + block] =
              static_cast<uint8_t>(sf);
        }
        if (sf_tiled != nullptr) {
          sf_tiled[swizzled_scale_offset(row, block, k_tiles)] = static_cast<uint8_t>(sf);
        }
      }
    }
  }
}

// The same for few rows, a block per row (norm_quant_by_block).
//
// Bound by latency, and by fetching its own instructions: the row kernel unrolls ITERS steps of
// codes, which made one row of 4096 take 17.9 us alone with cold caches (this one 4.3) and one of
// 2688 7.1 (4.2).
template <bool BF16, int CHUNKS>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
norm_quant_block_kernel(const void* in, int cols, const float* __restrict__ norm_weight, float eps,
                        float* __restrict__ normalized, uint8_t* __restrict__ packed,
                        uint8_t* __restrict__ sf_row_major, uint8_t* __restrict__ sf_tiled,
                        int k_tiles, float* __restrict__ tensor_scale,
                        float* __restrict__ inv_rms_out, bool word_scales,
                        int32_t* __restrict__ zero, int zero_count) {
  __shared__ NormShared<CHUNKS> shared;
  release_successor();
  norm_quant_by_block<BF16, CHUNKS>(in, blockIdx.x, cols, norm_weight, eps, normalized, packed,
                                    sf_row_major, sf_tiled, k_tiles, tensor_scale, inv_rms_out,
                                    word_scales, shared, [] {});
  // (after the wait for the predecessor, which may still count in them)
  zero_words(zero, zero_count);
}

// ComputeGlobalMaxAbsKernel, device_nvfp4_matrix.cu:64-75
__global__ void global_amax_kernel(const float* __restrict__ in, size_t count,
                                   float* __restrict__ amax) {
  float local = 0.0f;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    local = fmaxf(local, fabsf(in[i]));
  }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    local = fmaxf(local, __shfl_xor_sync(0xffffffffu, local, stride));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(reinterpret_cast<int*>(amax), __float_as_int(local));  // non-negative floats
  }
}

// DequantizeNvfp4Matrix, expert_layer.cpp:154-186: scale product first.
__global__ void dequant_kernel(const uint8_t* __restrict__ packed,
                               const uint8_t* __restrict__ sf_row_major,
                               const float* __restrict__ tensor_scale, bool per_row, int rows,
                               int cols, float* __restrict__ out) {
  const size_t bytes = static_cast<size_t>(rows) * cols / 2;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < bytes;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t element = i * 2;
    const size_t row = element / cols;
    const size_t col = element - row * cols;
    const float ts = tensor_scale[per_row ? row : 0];
    const float s = __fmul_rn(decode_e4m3(sf_row_major[row * (cols / 16) + col / 16]), ts);
    const uint32_t byte = packed[i];
    out[element] = __fmul_rn(decode_e2m1(byte & 15u), s);
    out[element + 1] = __fmul_rn(decode_e2m1(byte >> 4), s);
  }
}

__global__ void swizzle_kernel(const uint8_t* __restrict__ row_major, int rows, int blocks,
                               int k_tiles, uint8_t* __restrict__ tiled) {
  const size_t count = static_cast<size_t>(rows) * blocks;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t row = i / blocks;
    const size_t block = i - row * blocks;
    tiled[swizzled_scale_offset(row, block, k_tiles)] = row_major[i];
  }
}

}  // namespace

namespace {

// Which kernel takes a batch, by measurement (between events, bf16 rows with RMSNorm unless it says
// otherwise, us).
//
// Rows of up to kRegisterCols columns: a block each for few rows, the register kernel for more, which
// is the one that reads a row once and needs no shared memory.  2688 columns: 300 FP32 rows 8.3 by
// blocks and 11.2 in registers, 600 bf16 rows 10.3 and 10.5, 1184 rows 13.1 and 11.3.  Its steps are
// unrolled, so a row pays for all of them: it comes in four lengths, each of which is faster than the
// general kernel or level with it where it is used (16384 rows of 1280 columns: 6 steps 28.7,
// 11 steps 45, general 32.8; of 2048: 8 steps 49, general 48; of 2688: 11 steps 59, general 63).
//
// Longer rows do not fit the registers (16384 rows of 4096: 16 steps 131, blocks 96, general 89; of
// 5376: 21 steps 179, blocks 137, general 114).  FP32 rows always get blocks (of 4096: 103 against
// 147; of 5376 without RMSNorm 97 against 134), bf16 rows up to 24 per SM (2048 rows of 4096: 18.4
// against 20.5, 4096 rows 30.3 against 30.8; 4096 rows of 5376: 40.2 against 38.1).
constexpr int kRegisterCols = 11 * 256;
constexpr int kBlockCols = 6144;
constexpr int kBlockRowsPerSm = 6;
constexpr int kLongBlockRowsPerSm = 24;

bool block_per_row(bool bf16, int rows, int cols, int num_sms) {
  if (cols > kBlockCols) return false;
  if (cols <= kRegisterCols) return rows <= kBlockRowsPerSm * num_sms;
  return !bf16 || rows <= kLongBlockRowsPerSm * num_sms;
}

template <bool BF16>
void launch_norm_quant_t(int rows, int num_sms, LaunchStream stream, const void* in, int cols,
                         const float* norm_weight, float eps, float* normalized, uint8_t* packed,
                         uint8_t* sf_row_major, uint8_t* sf_tiled, int k_tiles,
                         float* tensor_scale, float* inv_rms, int32_t* zero, int zero_count) {
  const int grid = (rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const bool word_scales =
      cols % 64 == 0 && ((reinterpret_cast<uintptr_t>(sf_row_major) |
                          reinterpret_cast<uintptr_t>(sf_tiled)) & 3u) == 0;
  auto run_block = [&](auto kernel) {
    launch_kernel(kernel, rows, kWarpsPerBlock * 32, 0, stream, in, cols, norm_weight, eps,
                  normalized, packed, sf_row_major, sf_tiled, k_tiles, tensor_scale, inv_rms,
                  word_scales, zero, zero_count);
  };
  auto run_row = [&](auto kernel) {
    launch_kernel(kernel, grid, kWarpsPerBlock * 32, 0, stream, in, rows, cols, norm_weight, eps,
                  normalized, packed, sf_row_major, sf_tiled, k_tiles, tensor_scale, inv_rms,
                  word_scales, zero, zero_count);
  };
  if (block_per_row(BF16, rows, cols, num_sms)) {
    if (cols <= 2048) {
      run_block(norm_quant_block_kernel<BF16, 1>);
    } else if (cols <= 4096) {
      run_block(norm_quant_block_kernel<BF16, 2>);
    } else {
      run_block(norm_quant_block_kernel<BF16, 3>);
    }
  } else if (cols <= 4 * 256) {
    run_row(norm_quant_row_kernel<BF16, 4>);
  } else if (cols <= 6 * 256) {
    run_row(norm_quant_row_kernel<BF16, 6>);
  } else if (cols <= 8 * 256) {
    run_row(norm_quant_row_kernel<BF16, 8>);
  } else if (cols <= kRegisterCols) {
    run_row(norm_quant_row_kernel<BF16, 11>);
  } else {
    launch_kernel(norm_quant_kernel<BF16, true>, grid, kWarpsPerBlock * 32, 0, stream, in, rows,
                  cols, norm_weight, eps, normalized, packed, sf_row_major, sf_tiled, k_tiles,
                  tensor_scale, nullptr, inv_rms, zero, zero_count);
  }
}

}  // namespace

cudaError_t launch_norm_quant(const void* in, bool in_bf16, int rows, int cols,
                              const float* norm_weight, float eps, float* normalized,
                              uint8_t* packed, uint8_t* sf_row_major, uint8_t* sf_tiled,
                              int k_blocks, float* tensor_scale, int num_sms, LaunchStream stream,
                              float* inv_rms, int32_t* zero, int zero_count) {
  if (rows <= 0 || cols <= 0 || cols % 16 != 0) return cudaErrorInvalidValue;
  if (in_bf16) {
    launch_norm_quant_t<true>(rows, num_sms, stream, in, cols, norm_weight, eps, normalized, packed,
                              sf_row_major, sf_tiled, k_blocks * 4, tensor_scale, inv_rms, zero,
                              zero_count);
  } else {
    launch_norm_quant_t<false>(rows, num_sms, stream, in, cols, norm_weight, eps, normalized, packed,
                               sf_row_major, sf_tiled, k_blocks * 4, tensor_scale, inv_rms, zero,
                              zero_count);
  }
  return cudaGetLastError();
}

cudaError_t launch_quant_matrix(const float* in, int rows, int cols, uint8_t* packed,
                                uint8_t* sf_row_major, float* tensor_scale, float* amax_scratch,
                                cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || cols % 16 != 0) return cudaErrorInvalidValue;
  cudaError_t err = cudaMemsetAsync(amax_scratch, 0, sizeof(float), stream);
  if (err != cudaSuccess) return err;
  const size_t count = static_cast<size_t>(rows) * cols;
  global_amax_kernel<<<stride_blocks(count, 256), 256, 0, stream>>>(in, count, amax_scratch);
  const int grid = (rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
  norm_quant_kernel<false, false><<<grid, kWarpsPerBlock * 32, 0, stream>>>(
      in, rows, cols, nullptr, 0.0f, nullptr, packed, sf_row_major, nullptr, 0, tensor_scale,
      amax_scratch, nullptr, nullptr, 0);
  return cudaGetLastError();
}

cudaError_t launch_dequant(const uint8_t* packed, const uint8_t* sf_row_major,
                           const float* tensor_scale, bool per_row_scale, int rows, int cols,
                           float* out, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || cols % 16 != 0) return cudaErrorInvalidValue;
  const size_t bytes = static_cast<size_t>(rows) * cols / 2;
  dequant_kernel<<<stride_blocks(bytes, 256), 256, 0, stream>>>(packed, sf_row_major, tensor_scale,
                                                           per_row_scale, rows, cols, out);
  return cudaGetLastError();
}

cudaError_t launch_swizzle_scales(const uint8_t* row_major, int rows, int cols, uint8_t* tiled,
                                  cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || cols % 16 != 0) return cudaErrorInvalidValue;
  const int blocks = cols / 16;
  const int k_tiles = (blocks + 3) / 4;
  const size_t padded = static_cast<size_t>((rows + 127) / 128) * 128 * k_tiles * 4;
  cudaError_t err = cudaMemsetAsync(tiled, 0, padded, stream);
  if (err != cudaSuccess) return err;
  swizzle_kernel<<<stride_blocks(static_cast<size_t>(rows) * blocks, 256), 256, 0, stream>>>(
      row_major, rows, blocks, k_tiles, tiled);
  return cudaGetLastError();
}

}  // namespace nmoe
