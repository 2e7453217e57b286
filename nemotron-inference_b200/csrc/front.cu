// The front end of a pass over a handful of tokens in one launch: RMSNorm and quantiser, the gate's
// FP64 logits, selection, plan and placing.
//
// As four launches (norm_quant_block_kernel, exact_gemv_block_kernel, router_topk_kernel,
// place_rows_kernel) a pass over one token spent as long in front of its experts as in them: each
// started its own blocks, fetched its own instructions and waited for the one before to drain.  Here a
// block per token normalises and quantises its row, a block per expert forms the expert's logits as soon
// as the tokens' 1/rms is known (its weights and the tokens' rows are in registers by then), and the
// block that finishes last selects, plans and places.  Bound by the latency of that chain.
//
// Whole pass of the benchmark layer, four launches against this: 1 token 36.6 us and 30.7, 4 tokens 46.5
// and 41.7, 7 tokens 57.7 and 55.9, 8 tokens 59.1 and 57.5 (the experts read their weights for the rest).
//
// Blocks wait for others of the launch only where those have a lower index and wait for nothing, so that
// they end whatever the GPU runs beside them; the wait is bounded all the same.
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "quant_row.cuh"
#include "topk.cuh"

namespace nmoe {
namespace {

constexpr int kThreads = 256;
constexpr int kChunks = 2;  // of eight columns per thread: kFrontMaxCols columns
static_assert(kThreads == kWarpsPerBlock * 32 && kFrontMaxCols == kThreads * kChunks * 8, "block shape");

__device__ __forceinline__ int load_acquire_word(const int32_t* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_release_word(int32_t* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Waits (about a second at most) until *word is set.
__device__ __forceinline__ bool wait_word(const int32_t* word) {
  if (load_acquire_word(word) != 0) return true;
  const long long start = clock64();
  while (load_acquire_word(word) == 0) {
    if (clock64() - start > (1ll << 31)) return false;
  }
  return true;
}

// Eight gate values from element `i`.
__device__ __forceinline__ void load_gate8(const FrontArgs& args, size_t i, float (&g)[8]) {
  if (args.gate_bf16) {
    load8<true>(args.gate, i, g);
  } else {
    load8<false>(args.gate, i, g);
  }
}

struct Scratch {
  int32_t row_known[kFrontMaxRows];  // zero between launches, as is the next
  int32_t finished;                  // blocks whose logits are there
  float score[kFrontMaxRows][kFrontMaxExperts];
  float choice[kFrontMaxRows][kFrontMaxExperts];
};
static_assert(sizeof(Scratch) == front_scratch_bytes(), "scratch size");

// The logits and scores of one expert for ROWS tokens from `row0` (the last one repeated where there
// are fewer).
template <int ROWS>
__device__ __forceinline__ void expert_logits(const FrontArgs& args, Scratch* scratch, int expert,
                                              int row0) {
  __shared__ double warp_sum[ROWS][kWarpsPerBlock];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cols = args.cols;
  float g[kChunks][8], w[kChunks][8], x[ROWS][kChunks][8];
#pragma unroll
  for (int j = 0; j < kChunks; ++j) {
    const int k = (j * kThreads + static_cast<int>(threadIdx.x)) * 8;
    if (k >= cols) continue;
    load_gate8(args, static_cast<size_t>(expert) * cols + k, g[j]);
    load8<false>(args.norm_weight, k, w[j]);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const size_t from = static_cast<size_t>(min(row0 + r, args.rows - 1)) * cols + k;
      if (args.in_bf16) {
        load8<true>(args.in, from, x[r][j]);
      } else {
        load8<false>(args.in, from, x[r][j]);
      }
    }
  }
  const int mine = row0 + static_cast<int>(threadIdx.x);  // the row this thread looks after, if any
  const bool has_row = static_cast<int>(threadIdx.x) < ROWS && mine < args.rows;
  if (has_row && !wait_word(scratch->row_known + mine) && args.error != nullptr) {
    atomicCAS(args.error, kDevOk, kDevWaitTimeout);
  }
  __syncthreads();
  double acc[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float inv_rms = __ldcg(args.inv_rms + min(row0 + r, args.rows - 1));
    acc[r] = 0.0;
#pragma unroll
    for (int j = 0; j < kChunks; ++j) {
      if ((j * kThreads + static_cast<int>(threadIdx.x)) * 8 >= cols) continue;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        // (the roundings of the norm itself)
        acc[r] = fma(static_cast<double>(__fmul_rn(__fmul_rn(x[r][j][i], inv_rms), w[j][i])),
                     static_cast<double>(g[j][i]), acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
      acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], stride);
    }
    if (lane == 0) warp_sum[r][warp] = acc[r];
  }
  __syncthreads();
  if (has_row) {
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < kWarpsPerBlock; ++i) sum += warp_sum[threadIdx.x][i];
    float logit = static_cast<float>(sum);
    if (args.logit_offset != nullptr) logit = __fadd_rn(logit, args.logit_offset[expert]);
    const float score = sigmoid_ref(logit);
    args.logits[static_cast<size_t>(mine) * args.experts + expert] = logit;
    scratch->score[mine][expert] = score;
    scratch->choice[mine][expert] = __fadd_rn(score, args.bias[expert]);
  }
}

// Selection of all tokens and the tiles that follow from it, by one block.
template <int PER_LANE>
__device__ __forceinline__ void select_and_plan(const FrontArgs& args, const Scratch* scratch) {
  __shared__ float scores[kFrontMaxRows][PER_LANE * 32];
  __shared__ float choices[kFrontMaxRows][PER_LANE * 32];
  __shared__ int16_t slot_of[kFrontMaxExperts][kFrontMaxRows];  // -1: token did not select expert
  __shared__ int warp_tiles[kWarpsPerBlock];
  static_assert(kFrontMaxExperts == kThreads && kFrontMaxRows == kWarpsPerBlock, "block shape");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int experts = args.experts, top_k = args.top_k, e = threadIdx.x;
  // (all loads are on their way before the first of them is stored)
  float score_of[kFrontMaxRows], choice_of[kFrontMaxRows];
#pragma unroll
  for (int r = 0; r < kFrontMaxRows; ++r) {
    score_of[r] = __ldcg(&scratch->score[min(r, args.rows - 1)][e]);
    choice_of[r] = __ldcg(&scratch->choice[min(r, args.rows - 1)][e]);
  }
#pragma unroll
  for (int r = 0; r < kFrontMaxRows; ++r) {
    slot_of[e][r] = -1;
    if (r < args.rows && e < PER_LANE * 32) {
      scores[r][e] = score_of[r];
      choices[r][e] = choice_of[r];
    }
  }
  __syncthreads();
  int index = 0;
  float weight = 0.0f;
  if (warp < args.rows) {
    float score;
    const float sum = select_experts<PER_LANE>(scores[warp], choices[warp], experts, top_k,
                                               args.n_group, args.topk_group, index, score);
    weight = selected_weight(score, sum, args.norm_topk_prob, args.routed_scaling);
    if (lane < top_k) slot_of[index][warp] = static_cast<int16_t>(lane);
  }
  __syncthreads();
  // thread e: whether expert e has a tile, and how many experts before it do
  int16_t slots[kFrontMaxRows];
  bool selected = false;
#pragma unroll
  for (int r = 0; r < kFrontMaxRows; ++r) {
    slots[r] = slot_of[e][r];
    selected = selected || slots[r] >= 0;
  }
  const uint32_t of_warp = __ballot_sync(0xffffffffu, selected);
  if (lane == 0) warp_tiles[warp] = __popc(of_warp);
  __syncthreads();
  int tile = __popc(of_warp & ((1u << lane) - 1u)), total = 0;
#pragma unroll
  for (int i = 0; i < kWarpsPerBlock; ++i) {
    if (i < warp) tile += warp_tiles[i];
    total += warp_tiles[i];
  }
  int* tile_of = reinterpret_cast<int*>(&scores[0][0]);  // (the scores have been used)
  if (selected) {
    tile_of[e] = tile;
    args.row_tiles[tile] = RowTile{tile * 128, args.rows, e, 0};
#pragma unroll
    for (int r = 0; r < kFrontMaxRows; ++r) {
      if (r < args.rows) {
        args.dest[tile * 128 + r] = slots[r] < 0 ? -1 : r * args.dest_stride + slots[r];
      }
    }
  }
  if (e == 0) *args.num_row_tiles = total;
  __syncthreads();
  if (warp < args.rows && lane < top_k) {
    const int pair = warp * top_k + lane, row = tile_of[index] * 128 + warp;
    args.top_index[pair] = index;
    args.top_weight[pair] = weight;
    args.row_weight[row] = weight;
    args.pair_row[pair] = row;
  }
}

template <int ROWS, int PER_LANE>
__global__ void __launch_bounds__(kThreads)
front_kernel(const __grid_constant__ FrontArgs args) {
  __shared__ bool last;
  __shared__ NormShared<kChunks> norm_shared;
  Scratch* scratch = static_cast<Scratch*>(args.scratch);
  release_successor();
  const int block = blockIdx.x;
  if (block < args.rows) {
    const bool word_scales = args.cols % 64 == 0;
    auto known = [&] {
      if (threadIdx.x == 0) store_release_word(scratch->row_known + block, 1);
    };
    auto run = [&](auto bf16) {
      norm_quant_by_block<decltype(bf16)::value, kChunks>(
          args.in, block, args.cols, args.norm_weight, args.eps, args.normalized, args.packed,
          args.sf_row_major, args.sf_tiled, args.k_tiles, args.tensor_scale, args.inv_rms,
          word_scales, norm_shared, known);
    };
    if (args.in_bf16) run(std::true_type()); else run(std::false_type());
    return;
  }
  const int unit = block - args.rows;
  expert_logits<ROWS>(args, scratch, unit % args.experts, unit / args.experts * ROWS);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // what this block's threads stored, as of the barrier
    last = atomicAdd(&scratch->finished, 1) == static_cast<int>(gridDim.x) - args.rows - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  select_and_plan<PER_LANE>(args, scratch);
  // (every block that waits for a row has seen it)
  if (threadIdx.x == 0) scratch->finished = 0;
  if (static_cast<int>(threadIdx.x) < args.rows) scratch->row_known[threadIdx.x] = 0;
}

}  // namespace

cudaError_t launch_front(const FrontArgs& args, cudaStream_t stream) {
  if (args.rows < 1 || args.rows > kFrontMaxRows || args.cols > kFrontMaxCols || args.cols % 16 != 0 ||
      args.experts < 1 || args.experts > kFrontMaxExperts || args.top_k > 32) {
    return cudaErrorInvalidValue;
  }
  auto run = [&](auto kernel, int rows_per_block) {
    const int units = (args.rows + rows_per_block - 1) / rows_per_block * args.experts;
    launch_kernel(kernel, dim3(args.rows + units), kThreads, 0, stream, args);
  };
  auto run_rows = [&](auto per_lane) {
    constexpr int kPerLane = decltype(per_lane)::value;
    if (args.rows == 1) {
      run(front_kernel<1, kPerLane>, 1);
    } else {
      run(front_kernel<4, kPerLane>, 4);
    }
  };
  if (args.experts <= 128) {
    run_rows(std::integral_constant<int, 4>());
  } else {
    run_rows(std::integral_constant<int, kFrontMaxExperts / 32>());
  }
  return cudaGetLastError();
}

}  // namespace nmoe
