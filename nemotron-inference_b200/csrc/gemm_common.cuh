// What the expert GEMM kernels share: the row tile a CTA works on, and the two epilogues that take
// a 128-row accumulator out of TMEM.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"

namespace nmoe {

__device__ __forceinline__ void report_timeout(int32_t* error) {
  if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
}

// BATCH 16-column chunks of this warp's TMEM lane quarter, all in flight before one wait: a chunk's
// arithmetic is one long dependent chain, several of them fill each other's gaps.
template <int BATCH>
__device__ __forceinline__ void load_chunks(uint32_t t_addr, int count, uint32_t (&raw)[BATCH][16]) {
#pragma unroll
  for (int j = 0; j < BATCH; ++j) {
    if (j < count) tmem_ld_x16_async(t_addr + j * 16, raw[j]);
  }
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < BATCH; ++j) tmem_ld_fence(raw[j]);
}

// relu^2 and NVFP4 quantisation of 16 columns from `n` of row `grow`; returns the largest value.
__device__ __forceinline__ float quantise_chunk(const GemmArgs& args, float (&v)[16], int n, int grow,
                                                float scale, bool store) {
  const uint64_t scale2 = pack2(scale, scale);
  uint64_t squares[8];
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {  // Relu2: x > 0 ? x*x : 0
    float a, b;
    unpack2(mul2(pack2(v[2 * i], v[2 * i + 1]), scale2), a, b);
    const uint64_t x = pack2(fmaxf(a, 0.0f), fmaxf(b, 0.0f));
    squares[i] = mul2(x, x);
    unpack2(squares[i], a, b);
    amax = fmaxf(fmaxf(a, b), amax);
  }
  uint32_t lo, hi;
  const uint32_t sf = quantize_block16_unit_scale(squares, amax, lo, hi);
  if (!store) return 0.0f;
  *reinterpret_cast<uint2*>(args.out_packed + static_cast<size_t>(grow) * (args.N / 2) + n / 2) =
      make_uint2(lo, hi);
  args.out_sf[swizzled_scale_offset(grow, n / 16, args.out_k_blocks * 4)] = static_cast<uint8_t>(sf);
  return amax;
}

__device__ __forceinline__ void report_range(const GemmArgs& args, float largest) {
  if (largest > kFp4Max * kFp8Max && args.error != nullptr) {
    atomicCAS(args.error, kDevOk, kDevActivationRange);
  }
}

// Sixteen values as bf16 or binary16 (a value beyond 65504 becomes an infinity here; the combine
// kernel reports it).
__device__ __forceinline__ void pack_rows16(int kind, const float (&v)[16], uint32_t (&w)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (kind == kRowBf16) {
      const __nv_bfloat162 two = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&two);
    } else {
      const __half2 two = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&two);
    }
  }
}

// Scale [x routing weight] [-> relu^2] of 16 columns from `n`, stored in the output row at `dest`.
__device__ __forceinline__ void store_chunk(const GemmArgs& args, float (&v)[16], int n,
                                            unsigned long long dest, float scale, float wt) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = __fmul_rn(v[i], scale);
    if (args.row_weight != nullptr) v[i] = __fmul_rn(v[i], wt);
    if (args.relu2) {  // Relu2 (expert_layer.cpp:138-140): x > 0 ? x * x : 0
      const float p = fmaxf(v[i], 0.0f);
      v[i] = __fmul_rn(p, p);
    }
  }
  if (args.out_kind == kRowF32) {
    float4* d = reinterpret_cast<float4*>(dest + static_cast<size_t>(n) * 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
    return;
  }
  uint32_t w[8];
  pack_rows16(args.out_kind, v, w);
  uint4* d = reinterpret_cast<uint4*>(dest + static_cast<size_t>(n) * 2);
  d[0] = make_uint4(w[0], w[1], w[2], w[3]);
  d[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// Up projection: relu^2 and NVFP4 quantisation of columns [n0 + 16 * chunk_begin,
// n0 + 16 * chunk_end) of the accumulator at `t_addr` (this warp's lane quarter); the thread owns
// row `grow` of the hidden activations.
template <int BATCH>
__device__ __forceinline__ void epilogue_quantise(const GemmArgs& args, uint32_t t_addr, int n0,
                                                  int chunk_begin, int chunk_end, int grow,
                                                  bool row_valid, float scale) {
  float row_max = 0.0f;
  chunk_end = min(chunk_end, (args.N - n0) / 16);
  for (int first = chunk_begin; first < chunk_end; first += BATCH) {
    uint32_t raw[BATCH][16];
    load_chunks<BATCH>(t_addr + first * 16, chunk_end - first, raw);
#pragma unroll
    for (int j = 0; j < BATCH; ++j) {
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(raw[j][i]);
      row_max = fmaxf(row_max, quantise_chunk(args, v, n0 + (first + j) * 16, grow, scale,
                                              row_valid && first + j < chunk_end));
    }
  }
  report_range(args, row_max);
}

// Byte address of the output row of activation row `grow` (0 = nothing to store); with
// out_segments it lies in the memory of the rank the row returns to.
__device__ __forceinline__ unsigned long long output_row_address(const GemmArgs& args, int grow) {
  const int d = args.dest_row != nullptr ? args.dest_row[grow]
                                         : grow * args.dest_mul + args.dest_add;
  if (d < 0) return 0;
  const size_t row_bytes = static_cast<size_t>(args.N) * (args.out_kind == kRowF32 ? 4 : 2);
  if (args.out_segments != nullptr) {
    const int slot = d + args.segment_slot0;
    const int segment = slot / args.segment_rows;
    return args.out_segments[segment] +
           static_cast<size_t>(slot - segment * args.segment_rows) * row_bytes;
  }
  return reinterpret_cast<unsigned long long>(args.out_rows) + d * row_bytes;
}

// Row-storing epilogue without staging: every thread stores its own row, 16 columns (32 or 64
// bytes, whole sectors) at a time.
template <int BATCH>
__device__ __forceinline__ void epilogue_rows_direct(const GemmArgs& args, uint32_t t_addr, int n0,
                                                     int chunk_begin, int chunk_end,
                                                     unsigned long long dest, float scale,
                                                     float wt) {
  chunk_end = min(chunk_end, (args.N - n0) / 16);
  for (int first = chunk_begin; first < chunk_end; first += BATCH) {
    uint32_t raw[BATCH][16];
    load_chunks<BATCH>(t_addr + first * 16, chunk_end - first, raw);
    if (dest == 0) continue;
#pragma unroll
    for (int j = 0; j < BATCH; ++j) {
      if (first + j >= chunk_end) break;
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(raw[j][i]);
      store_chunk(args, v, n0 + (first + j) * 16, dest, scale, wt);
    }
  }
}

// Row-storing epilogue through shared memory: each thread owns one row of the tile, but a store
// instruction should write few lines.  64 bytes of 32 rows are staged at a time (`stage`:
// kStageBytes of this warp's own; a row's pitch of five 16-byte units keeps both directions free
// of bank conflicts), then every four lanes write one row's 64 bytes.
constexpr int kStagePitch = 80;
constexpr int kStageBytes = 32 * kStagePitch;

__device__ __forceinline__ void epilogue_rows(const GemmArgs& args, uint32_t t_addr, int n0,
                                              int chunk_begin, int chunk_end,
                                              unsigned long long dest, float scale, float wt,
                                              uint8_t* stage) {
  const int lane = threadIdx.x & 31;
  uint8_t* own = stage + lane * kStagePitch;
  const uint8_t* part = stage + (lane >> 2) * kStagePitch + (lane & 3) * 16;
  const bool f32 = args.out_kind == kRowF32;
  const float factor = args.row_weight != nullptr ? wt : 1.0f;
  chunk_end = min(chunk_end, (args.N - n0) / 16);
  const int step = f32 ? 1 : 2;
  for (int ch = chunk_begin; ch < chunk_end; ch += step) {
    const bool wide = !f32 && ch + 1 < chunk_end;
    uint32_t raw[2][16];
    load_chunks<2>(t_addr + ch * 16, wide ? 2 : 1, raw);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (j == 1 && !wide) break;
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        // (a factor of one leaves every value as it is)
        v[i] = __fmul_rn(__fmul_rn(__uint_as_float(raw[j][i]), scale), factor);
        if (args.relu2) {  // Relu2 (expert_layer.cpp:138-140): x > 0 ? x * x : 0
          const float p = fmaxf(v[i], 0.0f);
          v[i] = __fmul_rn(p, p);
        }
      }
      if (f32) {
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          *reinterpret_cast<float4*>(own + i * 4) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
      } else {
        uint32_t w[8];
        pack_rows16(args.out_kind, v, w);
        *reinterpret_cast<uint4*>(own + j * 32) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(own + j * 32 + 16) = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
    __syncwarp();
    const bool mine = f32 || wide || (lane & 3) < 2;
    const size_t at = static_cast<size_t>(n0 + ch * 16) * (f32 ? 4 : 2) + (lane & 3) * 16;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const unsigned long long d = __shfl_sync(0xffffffffu, dest, it * 8 + (lane >> 2));
      if (d != 0 && mine) {
        *reinterpret_cast<uint4*>(d + at) =
            *reinterpret_cast<const uint4*>(part + it * 8 * kStagePitch);
      }
    }
  }
}

}  // namespace nmoe
