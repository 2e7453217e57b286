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

// 32 bytes from a 32-byte boundary: a whole sector by one thread.
__device__ __forceinline__ void store_sector(void* to, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to), "r"(w[0]),
               "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// relu^2 and NVFP4 quantisation of 16 columns: eight bytes of codes and the block's E4M3 scale;
// returns the largest value.
__device__ __forceinline__ float quantise_chunk(const float (&v)[16], float scale, uint32_t& lo,
                                                uint32_t& hi, uint32_t& sf) {
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
  sf = quantize_block16_unit_scale(squares, amax, lo, hi);
  return amax;
}

// Where the codes and the scale of block `block` (16 columns) of row `grow` go.
__device__ __forceinline__ uint8_t* hidden_codes(const GemmArgs& args, int grow, int block) {
  return args.out_packed + static_cast<size_t>(grow) * (args.N / 2) + block * 8;
}
__device__ __forceinline__ uint8_t* hidden_scale(const GemmArgs& args, int grow, int block) {
  return args.out_sf + swizzled_scale_offset(grow, block, args.out_k_blocks * 4);
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
    if (args.out_aligned) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t w[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) w[h] = __float_as_uint(v[8 * i + h]);
        store_sector(d + 2 * i, w);
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
    return;
  }
  uint32_t w[8];
  pack_rows16(args.out_kind, v, w);
  if (args.out_aligned) {
    store_sector(reinterpret_cast<void*>(dest + static_cast<size_t>(n) * 2), w);
    return;
  }
  uint4* d = reinterpret_cast<uint4*>(dest + static_cast<size_t>(n) * 2);
  d[0] = make_uint4(w[0], w[1], w[2], w[3]);
  d[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// Up projection: relu^2 and NVFP4 quantisation of columns [n0 + 16 * chunk_begin,
// n0 + 16 * chunk_end) of the accumulator at `t_addr` (this warp's lane quarter); the thread owns
// row `grow` of the hidden activations.
//
// Four blocks from a multiple of four are one sector of codes and one word of scales.  Stored block by
// block (8 bytes and 1 byte, each a sector's transaction) they held up the loads of the tiles behind:
// 98304 rows of 1856 took 250 us, 213 without the stores.
template <int BATCH>
__device__ __forceinline__ void epilogue_quantise(const GemmArgs& args, uint32_t t_addr, int n0,
                                                  int chunk_begin, int chunk_end, int grow,
                                                  bool row_valid, float scale) {
  float row_max = 0.0f;
  chunk_end = min(chunk_end, (args.N - n0) / 16);
  for (int c = chunk_begin; c < chunk_end;) {
    const int block = n0 / 16 + c;
    const int count = min(4 - (block & 3), chunk_end - c);
    uint32_t codes[8], scales[4];
#pragma unroll
    for (int first = 0; first < 4; first += BATCH) {
      if (first >= count) break;
      uint32_t raw[BATCH][16];
      load_chunks<BATCH>(t_addr + (c + first) * 16, count - first, raw);
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        if (first + j >= count) break;
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(raw[j][i]);
        const int k = first + j;
        const float largest = quantise_chunk(v, scale, codes[2 * k], codes[2 * k + 1], scales[k]);
        if (row_valid) row_max = fmaxf(row_max, largest);
      }
    }
    if (row_valid && count == 4) {
      store_sector(hidden_codes(args, grow, block), codes);
      *reinterpret_cast<uint32_t*>(hidden_scale(args, grow, block)) =
          scales[0] | (scales[1] << 8) | (scales[2] << 16) | (scales[3] << 24);
    } else if (row_valid) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (j >= count) break;
        *reinterpret_cast<uint2*>(hidden_codes(args, grow, block + j)) =
            make_uint2(codes[2 * j], codes[2 * j + 1]);
        *hidden_scale(args, grow, block + j) = static_cast<uint8_t>(scales[j]);
      }
    }
    c += count;
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

// Row-storing epilogue: every thread stores its own row, 16 columns (32 or 64 bytes, whole sectors) at
// a time.  In the CTA-pair kernel, lines of 128 bytes put together in shared memory first took 300 us
// for 98304 rows of 2688, this 289: the room it leaves is a sixth pipeline stage.
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

}  // namespace nmoe
