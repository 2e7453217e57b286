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
// Whole pass of the benchmark layer, four launches against this: 1 token 36.6 us and 31.6, 4 tokens 46.5
// and 42.2, 7 tokens 57.3 and 54.7, 8 tokens 58.2 and 57.1 (the experts read their weights for the rest).
// It pays for one token, and for more while all blocks of the gate are resident at once (front_pays).
//
// One token of a latent layer has its linears here too, eight outputs to a block: they were two FP64 gemvs
// and two quantisers on the same chain.  With what follows the experts in one launch as well
// (latent_tail_kernel, csrc/exact.cu) a pass of the checkpoint's layer is three launches instead of
// twelve: 78.6 -> 57.9 us.  Two tokens are faster on three streams (88 us against 94 in this way).
//
// Blocks wait only for blocks of a lower index, which are started before them, so that
// they end whatever the GPU runs beside them; the wait is bounded all the same.
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "quant_row.cuh"
#include "topk.cuh"
#include "weights.cuh"

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
  int32_t row_known[kFrontMaxRows];    // whether 1/rms is; cleared by the launch behind, as is the next
  int32_t row_rounded[kFrontLinears];  // ... the one row as a linear multiplies with it
  int32_t finished;                    // blocks whose logits are there; zero between launches, as is the next
  int32_t linear_finished[kFrontLinears];
  float score[kFrontMaxRows][kFrontMaxExperts];
  float choice[kFrontMaxRows][kFrontMaxExperts];
};
static_assert(sizeof(Scratch) == front_scratch_bytes(), "scratch size");

// The logits and scores of EXPERTS experts (`step` apart) for ROWS tokens from `row0` (the last one
// repeated where there are fewer).
template <int ROWS, int EXPERTS>
__device__ __forceinline__ void expert_logits(const FrontArgs& args, Scratch* scratch, int expert0,
                                              int step, int row0) {
  constexpr int kSums = ROWS * EXPERTS;
  __shared__ double warp_sum[kSums][kWarpsPerBlock];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cols = args.cols;
  float g[EXPERTS][kChunks][8], w[kChunks][8], x[ROWS][kChunks][8];
#pragma unroll
  for (int j = 0; j < kChunks; ++j) {
    const int k = (j * kThreads + static_cast<int>(threadIdx.x)) * 8;
    if (k >= cols) continue;
#pragma unroll
    for (int e = 0; e < EXPERTS; ++e) {
      load_gate8(args, static_cast<size_t>(min(expert0 + e * step, args.experts - 1)) * cols + k,
                 g[e][j]);
    }
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
  // the sum this thread looks after, if any
  const int mine = static_cast<int>(threadIdx.x) / EXPERTS + row0;
  const int expert = expert0 + static_cast<int>(threadIdx.x) % EXPERTS * step;
  const bool has_sum =
      static_cast<int>(threadIdx.x) < kSums && mine < args.rows && expert < args.experts;
  if (has_sum && !wait_word(scratch->row_known + mine) && args.error != nullptr) {
    atomicCAS(args.error, kDevOk, kDevWaitTimeout);
  }
  __syncthreads();
  double acc[kSums];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float inv_rms = __ldcg(args.inv_rms + min(row0 + r, args.rows - 1));
#pragma unroll
    for (int e = 0; e < EXPERTS; ++e) acc[r * EXPERTS + e] = 0.0;
#pragma unroll
    for (int j = 0; j < kChunks; ++j) {
      if ((j * kThreads + static_cast<int>(threadIdx.x)) * 8 >= cols) continue;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        // (the roundings of the norm itself)
        const double y =
            static_cast<double>(__fmul_rn(__fmul_rn(x[r][j][i], inv_rms), w[j][i]));
#pragma unroll
        for (int e = 0; e < EXPERTS; ++e) {
          acc[r * EXPERTS + e] = fma(y, static_cast<double>(g[e][j][i]), acc[r * EXPERTS + e]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kSums; ++i) {
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
      acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], stride);
    }
    if (lane == 0) warp_sum[i][warp] = acc[i];
  }
  __syncthreads();
  if (has_sum) {
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

template <int PER_LANE>
struct SelectShared {
  float scores[kFrontMaxRows][PER_LANE * 32];
  float choices[kFrontMaxRows][PER_LANE * 32];
  int16_t slot_of[PER_LANE * 32][kFrontMaxRows];  // -1: token did not select expert
  uint32_t list[PER_LANE > 4 ? kFrontMaxRows : 1][kSelectList];
  int warp_tiles[kWarpsPerBlock];
};

// Selection of all tokens and the tiles that follow from it, by one block.
template <int PER_LANE>
__device__ __forceinline__ void select_and_plan(const FrontArgs& args, const Scratch* scratch,
                                                SelectShared<PER_LANE>& shared) {
  static_assert(kFrontMaxRows == kWarpsPerBlock, "a warp per token");
  constexpr int kOwn = (PER_LANE * 32 + kThreads - 1) / kThreads;  // experts of a thread
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int experts = args.experts, top_k = args.top_k, e0 = static_cast<int>(threadIdx.x) * kOwn;
  {
    // (the loads of kBatch rows are on their way before the first of them is stored)
    constexpr int kBatch = kFrontMaxRows / kOwn;
#pragma unroll 1
    for (int r0 = 0; r0 < args.rows; r0 += kBatch) {
      float score_of[kBatch][kOwn], choice_of[kBatch][kOwn];
#pragma unroll
      for (int r = 0; r < kBatch; ++r) {
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
          if (r0 + r >= args.rows) continue;
          score_of[r][i] = __ldcg(&scratch->score[r0 + r][e0 + i]);
          choice_of[r][i] = __ldcg(&scratch->choice[r0 + r][e0 + i]);
        }
      }
#pragma unroll
      for (int r = 0; r < kBatch; ++r) {
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
          if (r0 + r >= args.rows || e0 + i >= PER_LANE * 32) continue;
          shared.slot_of[e0 + i][r0 + r] = -1;
          shared.scores[r0 + r][e0 + i] = score_of[r][i];
          shared.choices[r0 + r][e0 + i] = choice_of[r][i];
        }
      }
    }
  }
  __syncthreads();
  int index = 0;
  float weight = 0.0f;
  if (warp < args.rows) {
    float score;
    const float sum = select_experts<PER_LANE>(
        shared.scores[warp], shared.choices[warp], shared.list[PER_LANE > 4 ? warp : 0], experts, top_k,
        args.n_group, args.topk_group, select_narrows(PER_LANE, top_k), index, score);
    weight = selected_weight(score, sum, args.norm_topk_prob, args.routed_scaling);
    if (lane < top_k) shared.slot_of[index][warp] = static_cast<int16_t>(lane);
  }
  __syncthreads();
  // how many experts before this thread's have a tile
  bool selected[kOwn];
  int mine = 0;
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    selected[i] = false;
    if (e0 + i < experts) {
#pragma unroll
      for (int r = 0; r < kFrontMaxRows; ++r) {
        selected[i] = selected[i] || (r < args.rows && shared.slot_of[e0 + i][r] >= 0);
      }
    }
    mine += selected[i] ? 1 : 0;
  }
  int inclusive = mine;
#pragma unroll
  for (int stride = 1; stride < 32; stride <<= 1) {
    const int other = __shfl_up_sync(0xffffffffu, inclusive, stride);
    if (lane >= stride) inclusive += other;
  }
  if (lane == 31) shared.warp_tiles[warp] = inclusive;
  __syncthreads();
  int tile = inclusive - mine, total = 0;
#pragma unroll
  for (int i = 0; i < kWarpsPerBlock; ++i) {
    if (i < warp) tile += shared.warp_tiles[i];
    total += shared.warp_tiles[i];
  }
  int* tile_of = reinterpret_cast<int*>(&shared.scores[0][0]);  // (the scores have been used)
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    if (!selected[i]) continue;
    const int e = e0 + i;
    tile_of[e] = tile;
    args.row_tiles[tile] = RowTile{tile * 128, args.rows, e, 0};
#pragma unroll
    for (int r = 0; r < kFrontMaxRows; ++r) {
      const int slot = shared.slot_of[e][r];
      if (r < args.rows) args.dest[tile * 128 + r] = slot < 0 ? -1 : r * args.dest_stride + slot;
    }
    ++tile;
  }
  if (threadIdx.x == 0) *args.num_row_tiles = total;
  __syncthreads();
  if (warp < args.rows && lane < top_k) {
    const int pair = warp * top_k + lane, row = tile_of[index] * 128 + warp;
    args.top_index[pair] = index;
    args.top_weight[pair] = weight;
    args.row_weight[row] = weight;
    args.pair_row[pair] = row;
  }
}

// The token's row as a linear multiplies with it.
__device__ __forceinline__ void round_row(const FrontArgs& args, Scratch* scratch,
                                          const FrontLinear& linear) {
  const int k = static_cast<int>(threadIdx.x) * 16;
  float x[16], w[16];
  if (k < args.cols) {
#pragma unroll
    for (int i = 0; i < 16; i += 8) {
      load8<false>(args.norm_weight, k + i, eight_of(w, i));
      if (args.in_bf16) {
        load8<true>(args.in, k + i, eight_of(x, i));
      } else {
        load8<false>(args.in, k + i, eight_of(x, i));
      }
    }
  }
  if (threadIdx.x == 0 && !wait_word(scratch->row_known) && args.error != nullptr) {
    atomicCAS(args.error, kDevOk, kDevWaitTimeout);
  }
  __syncthreads();
  const float inv_rms = __ldcg(args.inv_rms);
  if (k >= args.cols) return;
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    float4 v;
    // (the roundings of the norm itself)
    v.x = input_value(__fmul_rn(__fmul_rn(x[i], inv_rms), w[i]), linear.fp8_scale);
    v.y = input_value(__fmul_rn(__fmul_rn(x[i + 1], inv_rms), w[i + 1]), linear.fp8_scale);
    v.z = input_value(__fmul_rn(__fmul_rn(x[i + 2], inv_rms), w[i + 2]), linear.fp8_scale);
    v.w = input_value(__fmul_rn(__fmul_rn(x[i + 3], inv_rms), w[i + 3]), linear.fp8_scale);
    *reinterpret_cast<float4*>(linear.rounded + k + i) = v;
  }
}

// Eight outputs of a linear for the token.  A thread holds sixteen columns of the weight rows; its part of
// the token is widened once for eight products.  Bound by the conversions of the weights.
constexpr int kLinearOutputs = 8;
template <int KIND>
__device__ __forceinline__ void linear_outputs(const FrontArgs& args, const Scratch* scratch,
                                               const FrontLinear& linear, int which, int n0,
                                               double (&warp_sum)[kWarpsPerBlock][kLinearOutputs]) {
  using Vector = WeightVector<KIND>;
  constexpr int kVectors = 16 / Vector::kCount;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cols = args.cols, k = static_cast<int>(threadIdx.x) * 16;
  const bool active = k < cols;
  const size_t row_bytes = static_cast<size_t>(cols) * (16 / Vector::kCount);
  const uint8_t* weight = reinterpret_cast<const uint8_t*>(linear.weight);
  const uint8_t* rows = weight + static_cast<size_t>(k) * (16 / Vector::kCount);
  auto weight_row = [&](int i) {
    return reinterpret_cast<const uint4*>(rows + min(n0 + i, linear.N - 1) * row_bytes);
  };
  uint4 raw[KIND == kWeightFp8 ? kLinearOutputs : 1][kVectors];
  if (KIND == kWeightFp8 && active) {
#pragma unroll
    for (int i = 0; i < kLinearOutputs; ++i) raw[i][0] = weight_row(i)[0];
  }
  // The weights of a block that starts when this one is through: HBM is idle until the row is known.
  const int ahead = n0 + args.resident_blocks * kLinearOutputs;
  if (ahead < linear.N) {
    const size_t bytes = min(kLinearOutputs, linear.N - ahead) * row_bytes;
    const uint8_t* from = weight + ahead * row_bytes;
    for (size_t b = threadIdx.x * 128; b < bytes; b += kThreads * 128) prefetch_l2(from + b);
  }
  if (threadIdx.x == 0 && !wait_word(&scratch->row_rounded[which]) && args.error != nullptr) {
    atomicCAS(args.error, kDevOk, kDevWaitTimeout);
  }
  __syncthreads();
  double acc[kLinearOutputs];
#pragma unroll
  for (int i = 0; i < kLinearOutputs; ++i) acc[i] = 0.0;
  if (active) {
    // (eight columns at a time, in a loop: the first blocks wait for its instructions)
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const float4* x = reinterpret_cast<const float4*>(linear.rounded + k + half * 8);
      const float4 a = __ldcg(x), b = __ldcg(x + 1);
      const double y[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < kLinearOutputs; ++i) {
        float values[8];
        if constexpr (KIND == kWeightFp8) {
          unpack_half<KIND>(raw[i][0], half, linear.scale, values);
        } else if constexpr (KIND == kWeightBf16) {
          Vector::unpack(weight_row(i)[half], linear.scale, values);
        } else {
          const float4* from = reinterpret_cast<const float4*>(weight_row(i)) + 2 * half;
          const float4 c = from[0], d = from[1];
          values[0] = c.x; values[1] = c.y; values[2] = c.z; values[3] = c.w;
          values[4] = d.x; values[5] = d.y; values[6] = d.z; values[7] = d.w;
        }
        // (two sums: a chain of eight is what a warp would wait for)
        double odd = 0.0;
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          acc[i] = fma(y[j], static_cast<double>(values[j]), acc[i]);
          odd = fma(y[j + 1], static_cast<double>(values[j + 1]), odd);
        }
        acc[i] += odd;
      }
    }
  }
  const double sum = warp_sum8(acc, lane);
  if ((lane & 3) == 0) {
    warp_sum[warp][((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = sum;
  }
  __syncthreads();
  const int n = n0 + static_cast<int>(threadIdx.x);
  if (threadIdx.x < kLinearOutputs && n < linear.N) {
    double total = 0.0;
#pragma unroll
    for (int i = 0; i < kWarpsPerBlock; ++i) total += warp_sum[i][threadIdx.x];
    float value = static_cast<float>(total);
    if (linear.relu2) value = value > 0.0f ? __fmul_rn(value, value) : 0.0f;
    linear.out[n] = value;
  }
}

// Counts a block whose results are stored; whether it is the last of `blocks`.
__device__ __forceinline__ bool last_of(int32_t* finished, int blocks) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // what this block's threads stored, as of the barrier
    last = atomicAdd(finished, 1) == blocks - 1;
    __threadfence();
    if (last) *finished = 0;  // for the next launch
  }
  __syncthreads();
  return last;
}

__host__ __device__ constexpr int linear_blocks(int N) {
  return (N + kLinearOutputs - 1) / kLinearOutputs;
}

template <int ROWS, int PER_LANE, bool LINEARS>
__global__ void __launch_bounds__(kThreads, LINEARS     ? kFrontLinearBlocksPerSm
                                            : ROWS == 1 ? 4
                                                        : kFrontBlocksPerSm)
front_kernel(const __grid_constant__ FrontArgs args) {
  // columns that a block quantises: the rows', or those of a linear's outputs
  constexpr int kQuantChunks = LINEARS ? kFrontLinearMaxN / (kThreads * 8) : kChunks;
  union Shared {
    NormShared<kQuantChunks> norm;
    SelectShared<PER_LANE> select;
    double warp_sum[kWarpsPerBlock][kLinearOutputs];
  };
  __shared__ __align__(16) uint8_t room[sizeof(Shared)];
  Shared& shared = *reinterpret_cast<Shared*>(room);
  Scratch* scratch = static_cast<Scratch*>(args.scratch);
  release_successor();
  int block = blockIdx.x;
  if (block < args.rows) {
    auto known = [&] {
      if (threadIdx.x == 0) store_release_word(scratch->row_known + block, 1);
    };
    auto run = [&](auto bf16) {
      norm_quant_by_block<decltype(bf16)::value, kQuantChunks>(
          args.in, block, args.cols, args.norm_weight, args.eps, args.normalized, args.packed,
          args.sf_row_major, args.sf_tiled, args.k_tiles, args.tensor_scale, args.inv_rms,
          args.cols % 64 == 0, shared.norm, known);
    };
    if (args.in_bf16) run(std::true_type()); else run(std::false_type());
    return;
  }
  block -= args.rows;
  if constexpr (LINEARS) {
    if (block < args.linears) {
      round_row(args, scratch, args.linear[block]);
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();  // what this block's threads stored, as of the barrier
        store_release_word(&scratch->row_rounded[block], 1);
      }
      return;
    }
    block -= args.linears;
  }
  // (beside the linears' blocks there is less room)
  constexpr int kExperts = LINEARS ? 2 : 1;
  const int step = (args.experts + kExperts - 1) / kExperts;
  const int gate_blocks = (args.rows + ROWS - 1) / ROWS * step;
  if (!LINEARS || block < gate_blocks) {
    expert_logits<ROWS, kExperts>(args, scratch, block % step, step, block / step * ROWS);
    if (!last_of(&scratch->finished, gate_blocks)) return;
    select_and_plan<PER_LANE>(args, scratch, shared.select);
  } else {
    block -= gate_blocks;
    int which = 0;
    if (args.linears > 1 && block >= linear_blocks(args.linear[0].N)) {
      block -= linear_blocks(args.linear[0].N);
      which = 1;
    }
    const FrontLinear& linear = args.linear[which];
    const int n0 = block * kLinearOutputs;
    if (linear.kind == kWeightFp8) {
      linear_outputs<kWeightFp8>(args, scratch, linear, which, n0, shared.warp_sum);
    } else if (linear.kind == kWeightBf16) {
      linear_outputs<kWeightBf16>(args, scratch, linear, which, n0, shared.warp_sum);
    } else {
      linear_outputs<kWeightF32>(args, scratch, linear, which, n0, shared.warp_sum);
    }
    if (!last_of(&scratch->linear_finished[which], linear_blocks(linear.N))) return;
    norm_quant_by_block<false, kQuantChunks>(
        linear.out, 0, linear.N, nullptr, 0.0f, nullptr, linear.packed, linear.sf_row_major,
        linear.sf_tiled, linear.k_tiles, linear.tensor_scale, nullptr, linear.N % 64 == 0, shared.norm,
        [] {});
  }
}

}  // namespace

// One token: four launches against one, 128 experts of 2688 27.4 us and 26.8, 256 of 4096 33.0 and 29.3, 512
// of 4096 43.5 and 39.6 (small experts, whole pass).  Several: a block of the gate is 124 registers a thread
// and two fit an SM; with more of them than that a second wave computes what the first has long been waited
// for.  128 experts, 4 tokens (128 blocks) 33.2 and 31.4, 8 tokens (256) 37.2 and 36.4; 256 of 2048, 4 tokens
// (256) 33.1 and 33.4, 8 tokens (512) 37.2 and 41.6; 160 of 2048, 8 tokens (320) 35.1 and 36.9; 384 of 2048, 2
// tokens (384) 31.0 and 33.9, 8 tokens (768) 39.3 and 46.4; 512 of 4096, 8 tokens 98.9 and 108.6.
bool front_pays(int rows, int experts, int num_sms) {
  if (rows == 1) return experts <= kFrontMaxExperts;
  if (rows > kFrontMaxRows || experts > kFrontMaxExpertsOfRows) return false;
  const int blocks = (rows + kFrontRowsPerBlock - 1) / kFrontRowsPerBlock * experts;
  return blocks <= kFrontBlocksPerSm * num_sms;
}

cudaError_t launch_front(const FrontArgs& args, cudaStream_t stream) {
  if ((args.rows > 1 && args.experts > kFrontMaxExpertsOfRows) ||
      args.rows < 1 || args.rows > kFrontMaxRows || args.cols > kFrontMaxCols || args.cols % 16 != 0 ||
      args.experts < 1 || args.experts > kFrontMaxExperts || args.top_k > 32 ||
      args.linears > kFrontLinears || (args.linears > 0 && args.rows != 1)) {
    return cudaErrorInvalidValue;
  }
  int blocks = args.rows;
  for (int i = 0; i < args.linears; ++i) {
    if (args.linear[i].N % 16 != 0 || args.linear[i].N > kFrontLinearMaxN) return cudaErrorInvalidValue;
    blocks += linear_blocks(args.linear[i].N);
  }
  auto run = [&](auto kernel, int rows_per_block) {
    const int gate = args.linears > 0 ? (args.experts + 1) / 2 + args.linears
                                      : (args.rows + rows_per_block - 1) / rows_per_block * args.experts;
    launch_kernel(kernel, dim3(blocks + gate), kThreads, 0, stream, args);
  };
  auto run_rows = [&](auto per_lane, auto linears) {
    constexpr int kPerLane = decltype(per_lane)::value;
    constexpr bool kLinears = decltype(linears)::value;
    if constexpr (!kLinears) {
      if constexpr (kPerLane * 32 <= kFrontMaxExpertsOfRows) {
        if (args.rows > 1) {
          return run(front_kernel<kFrontRowsPerBlock, kPerLane, false>, kFrontRowsPerBlock);
        }
      }
    }
    run(front_kernel<1, kPerLane, kLinears>, 1);
  };
  auto run_experts = [&](auto linears) {
    if (args.experts <= 128) {
      run_rows(std::integral_constant<int, 4>(), linears);
    } else if (args.experts <= 256) {
      run_rows(std::integral_constant<int, 8>(), linears);
    } else {
      run_rows(std::integral_constant<int, kFrontMaxExperts / 32>(), linears);
    }
  };
  if (args.linears > 0) run_experts(std::true_type()); else run_experts(std::false_type());
  return cudaGetLastError();
}

}  // namespace nmoe
