// Grouped NVFP4 GEMM for the routed and shared experts: tcgen05 block-scaled
// FP4 MMA (kind::mxf4nvf4, 16-element UE4M3 blocks) with TMA-fed shared-memory
// stages and double-buffered TMEM accumulators.
//
// Replaces, for all (token, expert) pairs at once, the reference's per-row host
// linear RunNvfp4LinearHost (runtime/src/backend/expert_layer.cpp:231-267:
// dequantise activation, dequantise weight, CpuMatmulRowMajor :212-229) and
// the steps fused behind it:
//   kGemmUp  : ApplyRelu2 (:269-275) and the re-quantisation of the activated
//              row that the next RunNvfp4LinearHost call performs through
//              PackRowMajorFp32ToNvfp4 (runtime/src/backend/nvfp4_packing.cpp:130-153);
//   kGemmDown: the routing-weight multiply of :951-953 (the sum over slots is
//              done by the combine kernel so that it stays in slot order).
//
// Operand roles: A = activations (128 token rows per tile, K-major packed E2M1),
// B = expert weights (BN output features per tile, K-major packed E2M1).  One
// K block is 256 elements = one 128-byte swizzled shared-memory row = four
// K=64 MMAs.  Block scales travel shared memory -> TMEM with tcgen05.cp in the
// 32-lane x 16-byte form; activations use the reference's 128x4 tile order
// (runtime/src/backend/nvfp4_scale_layout.cpp:14-28) unchanged.
//
// This file holds the kernel of the batches that are bound by arithmetic, csrc/expert_stream.cu
// that of the batches bound by reading the weights.  Every mbarrier wait is bounded; on a timeout
// the CTA records kDevWaitTimeout and unwinds.
#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "gemm_common.cuh"
#include "kernels.h"

namespace nmoe {
namespace {

constexpr int kEpilogueWarps = 8;  // two per TMEM lane quarter (sixteen measured no faster)

// The row tile of CTA `cta_rank` in tile unit `rt`, a pair of row tiles.
struct TileRows {
  int row0;      // first row of the 128-row slot
  int rows;      // valid rows in it
  int load_row0; // where the operands are read from (a valid slot even when rows == 0)
  int expert;
};

__device__ __forceinline__ TileRows tile_rows_of(const GemmArgs& args, int rt, int num_row_tiles,
                                                 uint32_t cta_rank) {
  TileRows t;
  const int index = 2 * rt + static_cast<int>(cta_rank);
  if (args.row_tiles != nullptr) {
    // the plan gives every expert an even number of tiles
    const int safe = min(index, num_row_tiles - 1);
    t.row0 = args.row_tiles[safe].row0;
    t.rows = index < num_row_tiles ? args.row_tiles[safe].rows : 0;
    t.expert = args.row_tiles[safe].expert;
    t.load_row0 = t.row0;
  } else {
    t.row0 = index * 128;
    t.rows = max(0, min(128, args.dense_rows - t.row0));
    t.expert = 0;
    t.load_row0 = min(t.row0, ((args.dense_rows - 1) >> 7) << 7);
  }
  return t;
}

// ---------------------------------------------------------------------------
// CTA-pair kernel: one 256 x kPairBN tile per cluster of two CTAs
// (tcgen05.mma.cta_group::2, M = 256).
//
// What bounds a K block is what an SM takes in.  A pair stages each weight tile once for 256 rows (half
// in each CTA), 35 KB per CTA and K block, and with the epilogue left out a K block takes 660 cycles, 54
// bytes each, hardly less with half of the MMAs (98304 rows, up: 193 us and 187).  The rows stored by
// the epilogue come on top of that: 221 us for up, 284 for down.  Experts' rows are therefore spread
// evenly over a pair's CTAs (csrc/plan.cu): 128 and 64 rows cost as much as 128 and 128.  At 4096 tokens
// it is HBM: 436 MB in 79 us, 0.85 of the copy rate.
//
// Roles per CTA: warp 0 loads (the CTA's own 128 activation rows, its half of the weight tile, the
// scales of its rows and of the whole weight tile), warp 1 of cluster rank 0 issues the scale
// copies and the MMAs for both CTAs, warps 2-9 run the epilogue of the CTA's 128 rows.  Copies
// and MMAs of one thread execute in order, so nothing waits between them; the bytes of both CTAs
// complete on rank 0's full barrier, so nothing is handed over inside a K block.  No multicast:
// the loads of the partner name the leader's barrier.
//
// Measured, benchmark layer, up / down projection, against 128 x 208 tiles of single CTAs: 16384
// tokens 334 / 405 -> 221 / 284 us, 8192 tokens 192 / 223 -> 134 / 163.
// ---------------------------------------------------------------------------
constexpr int kPairBN = 208;
constexpr int kPairBRows = kPairBN / 2;        // weight rows staged per CTA
constexpr int kPairSfBufs = 2;
constexpr int kPairThreads = (2 + kEpilogueWarps) * 32;
constexpr int kPairABytes = 128 * 128;
constexpr int kPairBBytes = kPairBRows * 128;
constexpr int kPairSfaBytes = 2048;
constexpr int kPairSfbGroups = 8;              // two groups of 128 weight rows x 4 MMAs
constexpr int kPairSfbBytes = kPairSfbGroups * 512;
constexpr int kPairStageBytes = kPairABytes + kPairBBytes + kPairSfaBytes + kPairSfbBytes;
constexpr int kPairSfCol = 2 * kPairBN;        // TMEM: two accumulators, then the scale buffers
constexpr int kPairSfBufCols = 16 + 4 * kPairSfbGroups;
constexpr int kPairStages = 6;
constexpr int kPairBarBytes = ((2 * kPairStages + 4) * 8 + 16 + 15) / 16 * 16;
constexpr int kPairSmemBytes = kPairStages * kPairStageBytes + kPairBarBytes + 1024;
static_assert(kPairSfCol + kPairSfBufs * kPairSfBufCols <= 512, "TMEM budget");
static_assert(kPairBRows % 8 == 0, "half a weight tile is whole 8-row swizzle groups");
static_assert(kPairBBytes % 1024 == 0, "stage regions keep the 1024-byte swizzle alignment");
static_assert(kPairSmemBytes <= kMaxSharedBytes, "shared memory budget");

// Activation rows are loaded 16 at a time.
__device__ __forceinline__ int boxes_of(int rows) {
  return (rows + kPairBoxRows - 1) / kPairBoxRows;
}
// Bytes that a CTA with `rows` activation rows loads of them per K block, with its slot's scales.
__device__ __forceinline__ uint32_t row_bytes(int rows) {
  return rows > 0 ? boxes_of(rows) * (kPairBoxRows * 128) + kPairSfaBytes : 0u;
}

template <int MODE>
__global__ void __launch_bounds__(kPairThreads, 1)
grouped_gemm_pair_kernel(const __grid_constant__ GemmMaps maps, const GemmArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) &
                                             ~static_cast<uintptr_t>(1023u));
  constexpr int kStages = kPairStages;
  uint8_t* sA = smem;
  uint8_t* sB = sA + kStages * kPairABytes;
  uint8_t* sSFA = sB + kStages * kPairBBytes;
  uint8_t* sSFB = sSFA + kStages * kPairSfaBytes;
  // full_bar (the leader's): the bytes of both CTAs
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sSFB + kStages * kPairSfbBytes);
  uint64_t* empty_bar = full_bar + kStages;  // both CTAs: the MMAs have read the stage
  uint64_t* tmem_full_bar = empty_bar + kStages;
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);

  const int warp = warp_uniform(static_cast<int>(threadIdx.x >> 5));
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0u;
  const int unit = static_cast<int>(blockIdx.x >> 1);
  const int units = static_cast<int>(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full_bar[a], 1);
      mbar_init(&tmem_empty_bar[a], 2 * kEpilogueWarps);
    }
    fence_barrier_init();
    for (int i = 0; i < kPairBoxes; ++i) prefetch_tensormap(&maps.a[i]);
    prefetch_tensormap(&maps.b_tail);
    prefetch_tensormap(&maps.b_full);
    prefetch_tensormap(&maps.sfa);
    prefetch_tensormap(&maps.sfb);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();  // the partner's barriers exist before anything arrives
  tcgen05_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  const int num_row_tiles = warp_uniform(
      args.row_tiles != nullptr ? *args.num_row_tiles : (args.dense_rows + 127) / 128);
  const int row_units = (num_row_tiles + 1) / 2;
  const int total_tiles = row_units * args.n_tiles;
  const int k_blocks = args.k_blocks;
  const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
  const uint32_t leader_full0 = cluster_address_of(&full_bar[0], 0);

  if (warp == 0) {
    // ------------------------------------------------------------- producer
    const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
    const uint32_t sfa0 = smem_u32(sSFA), sfb0 = smem_u32(sSFB);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = unit; t < total_tiles && ok; t += units) {
      const int rt = t / args.n_tiles;
      const int nt = t - rt * args.n_tiles;
      const TileRows rows = tile_rows_of(args, rt, num_row_tiles, cta_rank);
      const int load_row0 = warp_uniform(rows.load_row0);
      const int expert = warp_uniform(rows.expert);
      // Rows that do not exist are not loaded: the MMAs read what an earlier tile left in their place,
      // in rows that are never stored.
      const int own_rows = warp_uniform(rows.rows);
      const int other_rows =
          warp_uniform(tile_rows_of(args, rt, num_row_tiles, cta_rank ^ 1u).rows);
      const int box = max(boxes_of(own_rows) - 1, 0);
      const uint32_t tile_bytes = row_bytes(own_rows) + row_bytes(other_rows) +
                                  2 * (kPairBBytes + kPairSfbBytes);
      // the scale maps' rows are 1024 bytes: two to a K block of activations, four to one of weights
      const int sfa_row = (load_row0 >> 7) * k_blocks * 2;
      const int sfb_row = (expert * args.n_tiles + nt) * k_blocks * 4;
      const int b_row = nt * kPairBN + static_cast<int>(cta_rank) * kPairBRows;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_warp(empty0 + stage * 8, phase ^ 1u)) {
          report_timeout(args.error);
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t bar = leader_full0 + stage * 8;
          if (leader) mbar_arrive_expect_tx_at(full0 + stage * 8, tile_bytes);
          if (own_rows > 0) {
            tma_load_2d_pair_at(a0 + stage * kPairABytes, &maps.a[box], kb * 128, load_row0, bar);
            tma_load_2d_pair_at(sfa0 + stage * kPairSfaBytes, &maps.sfa, 0, sfa_row + kb * 2, bar);
          }
          if (kb < args.kb_full) {
            // the map's rows are eight weight rows' 128 bytes of a K block
            tma_load_2d_pair_at(b0 + stage * kPairBBytes, &maps.b_full, 0,
                                ((expert * args.kb_full + kb) * args.N + b_row) >> 3, bar);
          } else {
            tma_load_2d_pair_at(b0 + stage * kPairBBytes, &maps.b_tail, 0, expert * args.N + b_row,
                                bar);
          }
          tma_load_2d_pair_at(sfb0 + stage * kPairSfbBytes, &maps.sfb, 0, sfb_row + kb * 4, bar);
        }
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------- scale copies and MMAs, for both CTAs
    if (leader) {
      constexpr uint32_t idesc = make_idesc_nvf4_pair(kPairBN);
      const uint64_t a_desc0 = make_smem_desc(smem_u32(sA), 0, 1024, 2);
      const uint64_t b_desc0 = make_smem_desc(smem_u32(sB), 0, 1024, 2);
      const uint64_t sfa_desc0 = make_smem_desc(smem_u32(sSFA), 0, 128, 0);
      const uint64_t sfb_desc0 = make_smem_desc(smem_u32(sSFB), 0, 128, 0);
      const int last_mmas = args.K / 64 - 4 * (k_blocks - 1);
      int stage = 0;
      uint32_t phase = 0;
      int local = 0;
      uint32_t sf_buf = 0;
      bool ok = true;
      for (int t = unit; t < total_tiles && ok; t += units, ++local) {
        const int acc = local & 1;
        const uint32_t acc_phase = (local >> 1) & 1u;
        // both CTAs' epilogues have drained this accumulator
        if (!mbar_wait_warp(smem_u32(&tmem_empty_bar[acc]), acc_phase ^ 1u)) {
          report_timeout(args.error);
          break;
        }
        tcgen05_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kPairBN;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait_warp(full0 + stage * 8, phase)) {
            report_timeout(args.error);
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint64_t a_desc = advance_smem_desc(a_desc0, stage * kPairABytes);
          const uint64_t b_desc = advance_smem_desc(b_desc0, stage * kPairBBytes);
          const uint64_t sfa_desc = advance_smem_desc(sfa_desc0, stage * kPairSfaBytes);
          const uint64_t sfb_desc = advance_smem_desc(sfb_desc0, stage * kPairSfbBytes);
          const uint32_t sf_tmem = tmem_base + kPairSfCol + sf_buf * kPairSfBufCols;
          if (elect_one()) {
            if (kb + 1 < k_blocks || last_mmas == 4) {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                tcgen05_cp_pair_32x128b_warpx4(sf_tmem + 4 * c,
                                               advance_smem_desc(sfa_desc, c * 512));
              }
#pragma unroll
              for (int c = 0; c < kPairSfbGroups; ++c) {
                tcgen05_cp_pair_32x128b_warpx4(sf_tmem + 16 + 4 * c,
                                               advance_smem_desc(sfb_desc, c * 512));
              }
#pragma unroll
              for (int kt = 0; kt < 4; ++kt) {
                tcgen05_mma_pair_nvf4(d_tmem, advance_smem_desc(a_desc, kt * 32),
                                      advance_smem_desc(b_desc, kt * 32), idesc, sf_tmem + 4 * kt,
                                      sf_tmem + 16 + kPairSfbGroups * kt,
                                      kt != 0 ? 1u : kb != 0 ? 1u : 0u);
              }
            } else {
              // the scales of a partial last K block: of the MMAs it issues only
              for (int c = 0; c < last_mmas; ++c) {
                tcgen05_cp_pair_32x128b_warpx4(sf_tmem + 4 * c,
                                               advance_smem_desc(sfa_desc, c * 512));
              }
              for (int c = 0; c < last_mmas * (kPairSfbGroups / 4); ++c) {
                tcgen05_cp_pair_32x128b_warpx4(sf_tmem + 16 + 4 * c,
                                               advance_smem_desc(sfb_desc, c * 512));
              }
              for (int kt = 0; kt < last_mmas; ++kt) {
                tcgen05_mma_pair_nvf4(d_tmem, advance_smem_desc(a_desc, kt * 32),
                                      advance_smem_desc(b_desc, kt * 32), idesc, sf_tmem + 4 * kt,
                                      sf_tmem + 16 + kPairSfbGroups * kt,
                                      (kb | kt) != 0 ? 1u : 0u);
              }
            }
            tcgen05_commit_pair(&empty_bar[stage], 3);  // frees the stage in both CTAs
          }
          if (++sf_buf == kPairSfBufs) sf_buf = 0;
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok && elect_one()) tcgen05_commit_pair(&tmem_full_bar[acc], 3);
      }
    }
  } else {
    // -------------------------------------------------------------- epilogue
    const int quarter = warp & 3;           // TMEM lanes a warp may read: 32 * (warp % 4)
    const int group = (warp - 2) >> 2;      // which share of the tile's 16-column chunks
    const int r = quarter * 32 + lane;      // row inside this CTA's 128 rows == TMEM lane
    constexpr int kChunks = kPairBN / 16;
    static_assert(kEpilogueWarps == 8, "two groups");
    const uint32_t leader_empty0 = cluster_address_of(&tmem_empty_bar[0], 0);
    int local = 0;
    for (int t = unit; t < total_tiles; t += units, ++local) {
      const int acc = local & 1;
      const uint32_t acc_phase = (local >> 1) & 1u;
      const int rt = t / args.n_tiles;
      const int nt = t - rt * args.n_tiles;
      const TileRows tile = tile_rows_of(args, rt, num_row_tiles, cta_rank);
      const bool row_valid = r < tile.rows;
      const int grow = tile.row0 + r;
      float scale = args.w_tensor_scale[tile.expert];
      if (args.a_tensor_scale != nullptr && row_valid) scale *= args.a_tensor_scale[grow];
      unsigned long long dest = 0;
      float wt = 1.0f;
      if (MODE == kGemmDown && row_valid) {
        dest = output_row_address(args, grow);
        if (args.row_weight != nullptr) wt = args.row_weight[grow];
      }
      if (!mbar_wait(&tmem_full_bar[acc], acc_phase)) {
        report_timeout(args.error);
        break;
      }
      if (quarter * 32 < tile.rows) {  // (else none of the warp's rows exist)
        tcgen05_fence_after();
        const uint32_t t_addr =
            tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * kPairBN;
        const int n0 = nt * kPairBN;
        // the two groups part where 64 columns, which are stored together, begin
        const int middle = (n0 / 16 + kChunks / 2 + 2) / 4 * 4 - n0 / 16;
        const int chunk_begin = group == 0 ? 0 : middle;
        const int chunk_end = group == 0 ? middle : kChunks;
        if constexpr (MODE == kGemmUp) {
          epilogue_quantise<2>(args, t_addr, n0, chunk_begin, chunk_end, grow, row_valid, scale);
        } else {
          epilogue_rows_direct<2>(args, t_addr, n0, chunk_begin, chunk_end, dest, scale, wt);
        }
        tcgen05_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_at(leader_empty0 + acc * 8);
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  // neither CTA leaves while the other may still signal its barriers
  cluster_sync_all();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <int MODE>
cudaError_t launch_pair(const GemmMaps& maps, const GemmArgs& args, int num_sms,
                        cudaStream_t stream) {
  auto kernel = grouped_gemm_pair_kernel<MODE>;
  cudaError_t err = allow_shared_memory(kernel);
  if (err != cudaSuccess) return err;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(num_sms & ~1), 1, 1);
  config.blockDim = dim3(kPairThreads, 1, 1);
  config.dynamicSmemBytes = kPairSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = 2;
  attribute.val.clusterDim.y = 1;
  attribute.val.clusterDim.z = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, maps, args);
}

__global__ void relayout_weight_scales_kernel(const uint8_t* __restrict__ src, int experts, int N,
                                              int K, int bn, int gs, int n_tiles, int k_blocks,
                                              uint32_t* __restrict__ out, size_t words) {
  const int blocks_per_row = K / 16;
  for (size_t w = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; w < words;
       w += static_cast<size_t>(gridDim.x) * blockDim.x) {
    // word index = ((((e*n_tiles + nt)*k_blocks + kb)*gs + chunk)*32 + lane)*4 + j
    size_t rest = w;
    const int j = rest & 3;
    rest >>= 2;
    const int lane = rest & 31;
    rest >>= 5;
    const int chunk = rest % gs;
    rest /= gs;
    const int kb = rest % k_blocks;
    rest /= k_blocks;
    const int nt = rest % n_tiles;
    const int e = static_cast<int>(rest / n_tiles);
    const int col = chunk * 4 + j;  // TMEM column inside this K block
    const int kt = col / gs;        // K tile (64 elements) inside the K block
    const int g = col - kt * gs;    // 32-row group inside the N tile
    const int local_row = g * 32 + lane;
    const int n = nt * bn + local_row;
    uint32_t word = 0;
    if (local_row < bn && n < N) {
      const uint8_t* row = src + (static_cast<size_t>(e) * N + n) * blocks_per_row;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int block = (kb * 4 + kt) * 4 + b;
        if (block < blocks_per_row) word |= static_cast<uint32_t>(row[block]) << (8 * b);
      }
    }
    out[w] = word;
  }
}

// [experts][N][K/2] row-major -> K-block-major: full 128-byte K blocks as
// [expert][k block][row][128], the partial last block as [expert][row][tail_pitch].
__global__ void relayout_weight_packed_kernel(const uint4* __restrict__ src, int experts, int N,
                                              int row_chunks, int kb_full, int tail_pitch_chunks,
                                              uint4* __restrict__ dst_full,
                                              uint4* __restrict__ dst_tail, size_t chunks) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < chunks;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % row_chunks);  // 16-byte chunk inside the row
    const size_t row = i / row_chunks;               // expert * N + n
    const int n = static_cast<int>(row % N);
    const size_t e = row / N;
    const int kb = c >> 3;
    if (kb < kb_full) {
      // 16-byte chunk j of row n is stored at position j ^ (n % 8): the 128-byte
      // shared-memory swizzle, applied here once so that a plain bulk copy of a
      // panel slice lands in shared memory exactly as a swizzling tensor copy would
      dst_full[((e * kb_full + kb) * N + n) * 8 + ((c & 7) ^ (n & 7))] = src[i];
    } else {
      dst_tail[row * tail_pitch_chunks + (c - kb_full * 8)] = src[i];
    }
  }
}

}  // namespace

cudaError_t relayout_weight_packed(const uint8_t* row_major, int experts, int N, int K,
                                   int tail_pitch_bytes, uint8_t* full, uint8_t* tail,
                                   cudaStream_t stream) {
  const int row_chunks = K / 32;
  const size_t chunks = static_cast<size_t>(experts) * N * row_chunks;
  const int blocks = stride_blocks(chunks, 256);
  relayout_weight_packed_kernel<<<blocks, 256, 0, stream>>>(
      reinterpret_cast<const uint4*>(row_major), experts, N, row_chunks, K / 256,
      tail_pitch_bytes / 16, reinterpret_cast<uint4*>(full), reinterpret_cast<uint4*>(tail),
      chunks);
  return cudaGetLastError();
}

GemmTileInfo pair_tile_info() {
  return GemmTileInfo{kPairBN, kPairSfbGroups, kPairSfbBytes, kPairBRows};
}

cudaError_t launch_pair_gemm(GemmMode mode, const GemmMaps& maps, const GemmArgs& args, int num_sms,
                             cudaStream_t stream) {
  if (num_sms < 2) return cudaErrorInvalidValue;
  return mode == kGemmUp ? launch_pair<kGemmUp>(maps, args, num_sms, stream)
                         : launch_pair<kGemmDown>(maps, args, num_sms, stream);
}

size_t weight_scale_layout_bytes(int experts, int N, int K, int bn, int sfb_groups) {
  const size_t n_tiles = (N + bn - 1) / bn;
  const size_t k_blocks = (K + 255) / 256;
  return static_cast<size_t>(experts) * n_tiles * k_blocks * sfb_groups * 512;
}

cudaError_t relayout_weight_scales(const uint8_t* row_major, int experts, int N, int K, int bn,
                                   int sfb_groups, uint8_t* out, cudaStream_t stream) {
  const int n_tiles = (N + bn - 1) / bn;
  const int k_blocks = (K + 255) / 256;
  const size_t words = weight_scale_layout_bytes(experts, N, K, bn, sfb_groups) / 4;
  const int threads = 256;
  const int blocks = static_cast<int>(std::min<size_t>((words + threads - 1) / threads, 65535));
  relayout_weight_scales_kernel<<<blocks, threads, 0, stream>>>(
      row_major, experts, N, K, bn, sfb_groups, n_tiles, k_blocks,
      reinterpret_cast<uint32_t*>(out), words);
  return cudaGetLastError();
}

}  // namespace nmoe
