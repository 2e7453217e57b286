// Route plan, token permute and the weighted combine.
//
// The reference walks tokens one by one and, inside, the token's selected
// experts (runtime/src/backend/expert_layer.cpp:871-954), accumulating
// routed_row += down * weight in selection order (:951-953) and finishing with
// mixer = routed + shared, out = input + mixer (:1064-1069).  Here the
// (token, slot) pairs are bucketed by expert so that each expert's rows form
// 128-row aligned slots for the grouped GEMM, and the combine kernel adds the
// per-slot results back in the reference's order.
#include <algorithm>

#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"

namespace nmoe {
namespace {

constexpr int kMaxPlanExperts = 512;

// Rows per tile of an expert with `count` rows in `tiles` tiles.  Two CTAs that share a weight tile wait
// for the one with more rows to load, so a pair's tiles get equal shares (in steps of the GEMM's boxes;
// 96 and 96 rows in the place of 128 and 64).  Single tiles are filled one after the other.
__device__ __forceinline__ int rows_per_tile(int count, int tiles, int tile_multiple) {
  if (tile_multiple == 1 || tiles <= 1) return 128;
  return ((count + tiles - 1) / tiles + kPairBoxRows - 1) / kPairBoxRows * kPairBoxRows;
}

// By all THREADS threads of a block: tiles_of[e] = row tiles of expert e, first_tile[e] = tiles of
// the experts before it; returns the number of all tiles.  Ends with a barrier.
template <int THREADS>
__device__ __forceinline__ int scan_expert_tiles(const int32_t* counts, int experts,
                                                 int tile_multiple, int* first_tile,
                                                 int* tiles_of) {
  constexpr int kPer = kMaxPlanExperts / THREADS < 1 ? 1 : kMaxPlanExperts / THREADS;
  constexpr int kWarps = THREADS / 32;
  __shared__ int warp_total[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int tiles[kPer];
  int mine = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = static_cast<int>(threadIdx.x) * kPer + i;
    tiles[i] = 0;
    if (e < experts) {
      const int t = (counts[e] + 127) / 128;
      tiles[i] = (t + tile_multiple - 1) / tile_multiple * tile_multiple;
    }
    mine += tiles[i];
  }
  int inclusive = mine;
#pragma unroll
  for (int stride = 1; stride < 32; stride <<= 1) {
    const int other = __shfl_up_sync(0xffffffffu, inclusive, stride);
    if (lane >= stride) inclusive += other;
  }
  if (lane == 31) warp_total[warp] = inclusive;
  __syncthreads();
  int before = inclusive - mine, total = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) before += warp_total[w];
    total += warp_total[w];
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = static_cast<int>(threadIdx.x) * kPer + i;
    if (e < experts) {
      first_tile[e] = before;
      tiles_of[e] = tiles[i];
      before += tiles[i];
    }
  }
  __syncthreads();
  return total;
}

// The tile list of the grouped GEMM, by all threads of one block.
template <int THREADS>
__device__ __forceinline__ void write_row_tiles(const PlanBuffers& plan, int experts,
                                                int tile_multiple, int max_row_tiles, int total,
                                                const int* first_tile, const int* tiles_of,
                                                int32_t* error) {
  if (threadIdx.x == 0) {
    if (total > max_row_tiles && error != nullptr) atomicCAS(error, kDevOk, kDevPlanOverflow);
    *plan.num_row_tiles = min(total, max_row_tiles);
  }
  for (int e = threadIdx.x; e < experts; e += THREADS) {
    const int count = plan.expert_counts[e];
    const int per_tile = rows_per_tile(count, tiles_of[e], tile_multiple);
    for (int i = 0; i < tiles_of[e] && first_tile[e] + i < max_row_tiles; ++i) {
      RowTile tile;
      tile.row0 = (first_tile[e] + i) * 128;
      tile.rows = max(0, min(per_tile, count - i * per_tile));
      tile.expert = e;
      tile.reserved = 0;
      plan.row_tiles[first_tile[e] + i] = tile;
    }
  }
}

struct PlacedRows {
  uint8_t* packed;
  uint8_t* sf_tiled;
  float* tensor_scale;
  float* weight;
  int32_t* dest;
  int32_t* pair_row;  // nullable
};

constexpr int kPlaceThreads = 256;

// Plan and permute in one kernel.  Every block works out for itself where each expert's row slots
// start (a scan over the histogram: cheaper than a launch that tells it) and block 0 writes the tile
// list; then a warp reads a source row once and writes it to the slots of `pairs_per_row / share`
// of its pairs.  A pair's position inside its expert was handed out when the histogram was counted,
// so a warp waits for one round of loads, not for an atomic after them; records of other ranks
// bring no position and take theirs from a cursor.
//
// Small batches are bound by launches and the chain of loads: a histogram memset, the plan and the
// permute were three launches, a pass over 1 token took 49.2 us with them and 45.0 now, 7 tokens
// 75.8 and 69.6, 64 tokens 155 and 149.  Large ones are bound by the writes: 98304 pairs of 1512
// bytes took 76 us, now 62 (between events, hidden 2688).
__global__ void __launch_bounds__(kPlaceThreads)
place_rows_kernel(PlanBuffers plan, PermuteSource src, int pairs, int share, int experts,
                  int tile_multiple, int max_row_tiles, int cols, int k_tiles, PlacedRows out,
                  int dest_stride, int32_t* error) {
  __shared__ int first_tile[kMaxPlanExperts];
  __shared__ int tiles_of[kMaxPlanExperts];
  release_successor();
  wait_for_predecessor();
  const int lane = threadIdx.x & 31;
  const int units = pairs / src.pairs_per_row * share;
  const int warps = gridDim.x * (kPlaceThreads / 32);
  const int row_bytes = cols / 2, blocks = cols / 16;
  const int first_unit = blockIdx.x * (kPlaceThreads / 32) + (threadIdx.x >> 5);
  const int total = scan_expert_tiles<kPlaceThreads>(plan.expert_counts, experts, tile_multiple,
                                                     first_tile, tiles_of);
  if (blockIdx.x == 0) {
    write_row_tiles<kPlaceThreads>(plan, experts, tile_multiple, max_row_tiles, total, first_tile, tiles_of, error);
  }
  for (int unit = first_unit; unit < units; unit += warps) {
    const int source_row = unit / share, part = unit - source_row * share;
    // Lane l looks up the l-th of this warp's pairs: its row in the sorted buffers, or -1.
    int row = -1;
    const int slot = part + lane * share;
    if (slot < src.pairs_per_row) {
      const int pair = source_row * src.pairs_per_row + slot;
      // (an unused slot of a fixed-capacity segment names nothing)
      const bool used = src.valid_counts == nullptr ||
                        (pair % src.capacity) < min(src.valid_counts[pair / src.capacity],
                                                    src.capacity);
      const int expert = used ? *reinterpret_cast<const int32_t*>(
                                    reinterpret_cast<const uint8_t*>(src.expert) +
                                    static_cast<size_t>(pair) * src.expert_stride)
                              : -1;
      // a record that arrived corrupt or half written (a peer that timed out) names no
      // expert of this stack: the histogram kernel has reported it, nothing is indexed by it
      if (expert >= 0 && expert < experts) {
        const int position = src.position != nullptr ? src.position[pair]
                                                     : atomicAdd(&plan.expert_cursor[expert], 1);
        // an expert's rows stay inside the tiles the plan gave it, whatever the histogram said,
        // and plan overflow was already reported
        const int per_tile =
            rows_per_tile(plan.expert_counts[expert], tiles_of[expert], tile_multiple);
        const int of_expert = position / per_tile, tile = first_tile[expert] + of_expert;
        if (position >= 0 && of_expert < tiles_of[expert] && tile < max_row_tiles) {
          row = tile * 128 + position - of_expert * per_tile;
          out.tensor_scale[row] = *reinterpret_cast<const float*>(
              reinterpret_cast<const uint8_t*>(src.tensor_scale) +
              static_cast<size_t>(source_row) * src.tensor_scale_stride);
          out.weight[row] = *reinterpret_cast<const float*>(
              reinterpret_cast<const uint8_t*>(src.weight) +
              static_cast<size_t>(pair) * src.weight_stride);
          out.dest[row] = source_row * dest_stride + slot;
          if (out.pair_row != nullptr) out.pair_row[pair] = row;
        }
      }
    }
    const int mine = (src.pairs_per_row - part + share - 1) / share;

    const uint8_t* from_bytes = src.packed + static_cast<size_t>(source_row) * src.packed_stride;
    const bool wide = ((reinterpret_cast<uintptr_t>(from_bytes) |
                        reinterpret_cast<uintptr_t>(out.packed)) & 15u) == 0 && (cols & 31) == 0;
    if (wide) {
      // 16 bytes per lane: a warp moves 512 contiguous bytes per instruction
      constexpr int kAhead = 3;  // pieces per lane held in registers: 1536 B of a row
      const uint4* from = reinterpret_cast<const uint4*>(from_bytes);
      const int pieces = row_bytes / 16;
      for (int q0 = 0; q0 < pieces; q0 += 32 * kAhead) {
        uint4 ahead[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
          const int q = q0 + lane + 32 * j;
          if (q < pieces) ahead[j] = from[q];
        }
        for (int i = 0; i < mine; ++i) {
          const int to = __shfl_sync(0xffffffffu, row, i);
          if (to < 0) continue;
          uint4* dst = reinterpret_cast<uint4*>(out.packed + static_cast<size_t>(to) * row_bytes);
#pragma unroll
          for (int j = 0; j < kAhead; ++j) {
            const int q = q0 + lane + 32 * j;
            if (q < pieces) dst[q] = ahead[j];
          }
        }
      }
    } else {
      const uint32_t* from = reinterpret_cast<const uint32_t*>(from_bytes);
      for (int i = 0; i < mine; ++i) {
        const int to = __shfl_sync(0xffffffffu, row, i);
        if (to < 0) continue;
        uint32_t* dst =
            reinterpret_cast<uint32_t*>(out.packed + static_cast<size_t>(to) * row_bytes);
        for (int w = lane; w < cols / 8; w += 32) dst[w] = from[w];
      }
    }

    const uint8_t* sf_src = src.sf + static_cast<size_t>(source_row) * src.sf_stride;
    if ((blocks & 3) == 0) {
      // four consecutive blocks are one aligned 32-bit word on both sides
      const uint32_t* sf_src_w = reinterpret_cast<const uint32_t*>(sf_src);
      for (int k0 = 0; k0 < blocks / 4; k0 += 64) {
        uint32_t word[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int kt = k0 + lane + 32 * j;
          if (kt < blocks / 4) word[j] = sf_src_w[kt];
        }
        for (int i = 0; i < mine; ++i) {
          const int to = __shfl_sync(0xffffffffu, row, i);
          if (to < 0) continue;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int kt = k0 + lane + 32 * j;
            if (kt < blocks / 4) {
              *reinterpret_cast<uint32_t*>(
                  out.sf_tiled + swizzled_scale_offset(to, kt * 4, k_tiles)) = word[j];
            }
          }
        }
      }
    } else {
      for (int i = 0; i < mine; ++i) {
        const int to = __shfl_sync(0xffffffffu, row, i);
        if (to < 0) continue;
        for (int b = lane; b < blocks; b += 32) {
          out.sf_tiled[swizzled_scale_offset(to, b, k_tiles)] = sf_src[b];
        }
      }
    }
  }
}

__device__ __forceinline__ void unpack_bf16x8(const uint4& raw, float (&v)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ void unpack_f16x8(const uint4& raw, float (&v)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 pair = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    v[2 * i] = pair.x;
    v[2 * i + 1] = pair.y;
  }
}

// Eight consecutive elements of row `row` of a [rows][hidden] matrix of RowKind KIND.
template <int KIND>
__device__ __forceinline__ void load_row8(const void* base, size_t row, int hidden, int c,
                                          float (&v)[8]) {
  if constexpr (KIND == kRowBf16) {
    unpack_bf16x8(*reinterpret_cast<const uint4*>(
                      reinterpret_cast<const __nv_bfloat16*>(base) + row * hidden + c), v);
  } else if constexpr (KIND == kRowF16) {
    unpack_f16x8(*reinterpret_cast<const uint4*>(
                     reinterpret_cast<const __half*>(base) + row * hidden + c), v);
  } else {
    const float* p = reinterpret_cast<const float*>(base) + row * hidden + c;
    const float4 a = *reinterpret_cast<const float4*>(p);
    const float4 b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}

template <bool BF16>
__device__ __forceinline__ void store_row8(void* base, size_t row, int hidden, int c,
                                           const float (&v)[8]) {
  if constexpr (BF16) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&pair);
    }
    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(base) + row * hidden + c) =
        make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    float* p = reinterpret_cast<float*>(base) + row * hidden + c;
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// out[t] = in[t] + ((sum_k parts[t][k]) + parts[t][top_k]): the routed parts are
// added in selection order (expert_layer.cpp:951-953), then the shared expert's
// row and the residual (:1064-1069).  Eight elements per thread, 16- or 32-byte
// accesses; the parts are rows of RowKind PARTS.
template <bool IN_BF16, bool OUT_BF16, int PARTS>
__global__ void combine_kernel(const void* __restrict__ in, const void* parts,
                               int rows, int hidden, int top_k, void* __restrict__ out,
                               int32_t* __restrict__ error) {
  release_successor();
  wait_for_predecessor();
  const int octs = hidden / 8;
  const size_t total = static_cast<size_t>(rows) * octs;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t t = i / octs;
    const int c = static_cast<int>(i - t * octs) * 8;
    const size_t first = t * (top_k + 1);
    float routed[8];
    load_row8<PARTS>(parts, first, hidden, c, routed);
    for (int k = 1; k < top_k; ++k) {
      float p[8];
      load_row8<PARTS>(parts, first + k, hidden, c, p);
#pragma unroll
      for (int j = 0; j < 8; ++j) routed[j] = __fadd_rn(routed[j], p[j]);
    }
    float shared[8], x[8], r[8];
    load_row8<PARTS>(parts, first + top_k, hidden, c, shared);
    load_row8<IN_BF16 ? kRowBf16 : kRowF32>(in, t, hidden, c, x);
    bool finite = true;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float mixer = __fadd_rn(routed[j], shared[j]);
      finite = finite && isfinite(mixer);
      r[j] = __fadd_rn(x[j], mixer);
    }
    if constexpr (PARTS == kRowF16) {
      // a row that left binary16's range on its way here (the GEMM stores an infinity)
      if (!finite && error != nullptr) atomicCAS(error, kDevOk, kDevActivationRange);
    }
    store_row8<OUT_BF16>(out, t, hidden, c, r);
  }
}

template <bool A, bool B>
void launch_combine_t(const void* in, const void* parts, RowKind parts_kind, int rows, int hidden,
                      int top_k, void* out, int32_t* error, int blocks, LaunchStream stream) {
  if (parts_kind == kRowBf16) {
    launch_kernel(combine_kernel<A, B, kRowBf16>, blocks, 256, 0, stream, in, parts, rows, hidden, top_k, out,
                                                               error);
  } else if (parts_kind == kRowF16) {
    launch_kernel(combine_kernel<A, B, kRowF16>, blocks, 256, 0, stream, in, parts, rows, hidden, top_k, out,
                                                              error);
  } else {
    launch_kernel(combine_kernel<A, B, kRowF32>, blocks, 256, 0, stream, in, parts, rows, hidden, top_k, out,
                                                              error);
  }
}

}  // namespace

cudaError_t launch_place_rows(const PlanBuffers& plan, const PermuteSource& src, int pairs,
                              int experts, int tile_multiple, int max_row_tiles, int cols,
                              int k_blocks, uint8_t* sorted_packed, uint8_t* sorted_sf_tiled,
                              float* sorted_tensor_scale, float* sorted_weight,
                              int32_t* sorted_dest, int32_t* pair_row, int dest_stride,
                              int32_t* error, int num_sms, LaunchStream stream) {
  if (pairs <= 0 || src.pairs_per_row <= 0 || src.pairs_per_row > 32 ||
      pairs % src.pairs_per_row != 0 || experts <= 0 || experts > kMaxPlanExperts ||
      tile_multiple < 1) {
    return cudaErrorInvalidValue;
  }
  constexpr int kWarps = kPlaceThreads / 32;
  // While there is little to write each pair gets a warp, then a row's pairs share what was read of
  // it.  The two meet at about 6 MB (between events; six pairs a row of 1512 bytes each: 3072 pairs
  // 9.9 us against 10.3, 4608 10.2 against 10.3, 6144 12.1 against 10.3; 22 pairs of 576 bytes: 5632
  // pairs 10.2 against 12.3, 9856 12.2 against 12.3, 14080 14.3 against 12.3).
  constexpr size_t kPairBytesPerSm = 40 * 1024;
  const size_t bytes = static_cast<size_t>(pairs) * (cols / 2 + cols / 16);
  const int share = bytes <= kPairBytesPerSm * num_sms ? src.pairs_per_row : 1;
  const int units = pairs / src.pairs_per_row * share;
  const int blocks = std::min((units + kWarps - 1) / kWarps, num_sms * 6);  // each pays for the scan
  const PlacedRows out{sorted_packed, sorted_sf_tiled, sorted_tensor_scale, sorted_weight,
                       sorted_dest, pair_row};
  launch_kernel(place_rows_kernel, blocks, kPlaceThreads, 0, stream, plan, src, pairs, share, experts,
                                                          tile_multiple, max_row_tiles, cols,
                                                          k_blocks * 4, out, dest_stride, error);
  return cudaGetLastError();
}

cudaError_t launch_combine(const void* in, bool in_bf16, const void* parts, RowKind parts_kind,
                           int rows, int hidden, int top_k, void* out, bool out_bf16,
                           int32_t* error, LaunchStream stream) {
  if (rows <= 0 || hidden % 8 != 0 || top_k < 1) return cudaErrorInvalidValue;
  const size_t total = static_cast<size_t>(rows) * (hidden / 8);
  const int blocks = stride_blocks(total, 256);
  if (in_bf16 && out_bf16) {
    launch_combine_t<true, true>(in, parts, parts_kind, rows, hidden, top_k, out, error, blocks, stream);
  } else if (in_bf16) {
    launch_combine_t<true, false>(in, parts, parts_kind, rows, hidden, top_k, out, error, blocks, stream);
  } else if (out_bf16) {
    launch_combine_t<false, true>(in, parts, parts_kind, rows, hidden, top_k, out, error, blocks, stream);
  } else {
    launch_combine_t<false, false>(in, parts, parts_kind, rows, hidden, top_k, out, error, blocks, stream);
  }
  return cudaGetLastError();
}

}  // namespace nmoe
