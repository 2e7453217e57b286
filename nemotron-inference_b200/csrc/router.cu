// Router: gate logits and sigmoid top-k with correction bias.
//
// Replaces the gate projection (UploadedLinearOp::Run dense fallback,
// runtime/src/backend/linear_op.cpp:97-118: sequential DOUBLE accumulation on the
// host) and SelectTopExperts (runtime/src/backend/expert_layer.cpp:277-367).
//
// Logits are accumulated in FP64 from the FP32 normalised activations and the
// gate weights widened to FP32 (as the reference's upload does): every product
// is exact in double, so the result differs
// from the reference's sequential double sum only by double rounding noise
// (~1e-16 relative) and rounds to the same FP32 logit.  That is what keeps the
// selected expert sets identical to the reference's, not merely close.
#include "common.cuh"
#include "kernels.h"
#include "topk.cuh"

namespace nmoe {
namespace {

constexpr int kWarps = 8;

// One warp computes TPW tokens x EPW experts; lanes split the hidden dimension.
template <int TPW, int EPW>
__global__ void __launch_bounds__(kWarps * 32)
router_logits_kernel(const float* __restrict__ y, const float* __restrict__ gate,
                     const float* __restrict__ logit_offset, int rows, int experts, int hidden,
                     float* __restrict__ logits) {
  const int lane = threadIdx.x & 31;
  const int warp_global = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int expert_tiles = experts / EPW;
  const int token_tile = warp_global / expert_tiles;
  const int expert_tile = warp_global - token_tile * expert_tiles;
  const int t0 = token_tile * TPW;
  const int e0 = expert_tile * EPW;
  if (t0 >= rows) return;

  double acc[TPW][EPW];
#pragma unroll
  for (int i = 0; i < TPW; ++i)
#pragma unroll
    for (int j = 0; j < EPW; ++j) acc[i][j] = 0.0;

  int k_begin = lane;
  if constexpr (TPW == 1) {
    if ((hidden & 127) == 0) {
      // small batches: 16-byte loads, three steps in flight (the loop is a chain of
      // load -> FMA otherwise and costs a memory latency per step)
      const float4* y4 = reinterpret_cast<const float4*>(y + static_cast<size_t>(t0) * hidden);
      const int quads = hidden / 4;
#pragma unroll 3
      for (int q = lane; q < quads; q += 32) {
        const float4 a4 = y4[q];
        const double a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int j = 0; j < EPW; ++j) {
          const float4 w4 =
              reinterpret_cast<const float4*>(gate + static_cast<size_t>(e0 + j) * hidden)[q];
          acc[0][j] = fma(a[0], static_cast<double>(w4.x), acc[0][j]);
          acc[0][j] = fma(a[1], static_cast<double>(w4.y), acc[0][j]);
          acc[0][j] = fma(a[2], static_cast<double>(w4.z), acc[0][j]);
          acc[0][j] = fma(a[3], static_cast<double>(w4.w), acc[0][j]);
        }
      }
      k_begin = hidden;  // nothing left for the scalar loop
    }
  }
  for (int k = k_begin; k < hidden; k += 32) {
    double a[TPW];
#pragma unroll
    for (int i = 0; i < TPW; ++i) {
      const int t = min(t0 + i, rows - 1);
      a[i] = static_cast<double>(y[static_cast<size_t>(t) * hidden + k]);
    }
#pragma unroll
    for (int j = 0; j < EPW; ++j) {
      const double w = static_cast<double>(gate[static_cast<size_t>(e0 + j) * hidden + k]);
#pragma unroll
      for (int i = 0; i < TPW; ++i) acc[i][j] = fma(a[i], w, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TPW; ++i) {
#pragma unroll
    for (int j = 0; j < EPW; ++j) {
      double v = acc[i][j];
#pragma unroll
      for (int stride = 16; stride > 0; stride >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, stride);
      }
      if (lane == 0 && t0 + i < rows) {
        float logit = static_cast<float>(v);
        if (logit_offset != nullptr) logit = __fadd_rn(logit, logit_offset[e0 + j]);
        logits[static_cast<size_t>(t0 + i) * experts + e0 + j] = logit;
      }
    }
  }
}

constexpr int kMaxExperts = 512;

// One block per token.  All threads evaluate sigmoids (the exponential in double is the
// longest single step; one for each expert while blocks are few, else 128), one warp selects:
// expert e lives in lane e % 32, and a round is one warp-wide maximum of order-preserving keys and one
// minimum over the indices that hold it (ties go to the lower expert).  Every lane keeps the best of its
// own at hand, or many experts are narrowed down to some forty first, two to a lane (csrc/topk.cuh).
// Bound by the latency of that chain: 1 token, 128 experts, top-6 14.9 -> 8.2 us between events; 3000
// tokens, 512 experts, top-22 27.4 us with sixteen choices a lane, 19.1 narrowed down.
// NARROWED: select_narrows(); a kernel that held both ways took the registers of the wider one (1003 tokens, 384
// experts, top-8 205.7 us a pass and 214.5).
template <int PER_LANE, bool NARROWED>
__global__ void __launch_bounds__(PER_LANE * 32 < 128 ? 128 : PER_LANE * 32)
router_topk_kernel(const float* logits, const float* __restrict__ bias, int experts,
                   int top_k, int n_group, int topk_group, bool norm_topk_prob,
                   float routed_scaling, int32_t* __restrict__ top_index,
                   float* __restrict__ top_weight, int32_t* __restrict__ expert_counts,
                   int32_t* __restrict__ position) {
  __shared__ float score_smem[PER_LANE * 32];
  __shared__ float choice_smem[PER_LANE * 32];
  __shared__ uint32_t list[kSelectList];
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x;
  release_successor();
  wait_for_predecessor();
  for (int e = threadIdx.x; e < experts; e += blockDim.x) {
    const float score = sigmoid_ref(logits[static_cast<size_t>(row) * experts + e]);
    score_smem[e] = score;
    choice_smem[e] = __fadd_rn(score, bias[e]);
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;

  int my_index;
  float my_score;
  const float weight_sum =
      select_experts<PER_LANE>(score_smem, choice_smem, list, experts, top_k, n_group, topk_group,
                               NARROWED, my_index, my_score);
  if (lane < top_k) {
    top_index[static_cast<size_t>(row) * top_k + lane] = my_index;
    top_weight[static_cast<size_t>(row) * top_k + lane] =
        selected_weight(my_score, weight_sum, norm_topk_prob, routed_scaling);
    if (expert_counts != nullptr) {
      const int place = atomicAdd(&expert_counts[my_index], 1);
      if (position != nullptr) position[static_cast<size_t>(row) * top_k + lane] = place;
    }
  }
}

}  // namespace

cudaError_t launch_router_logits(const float* normalized, const float* gate,
                                 const float* logit_offset, int rows, int experts, int hidden,
                                 float* logits, int num_sms, cudaStream_t stream) {
  if (rows <= 0 || experts <= 0 || hidden <= 0) return cudaErrorInvalidValue;
  if (rows >= 256 && experts % 16 == 0) {
    const int warps = ((rows + 1) / 2) * (experts / 16);
    router_logits_kernel<2, 16><<<(warps + kWarps - 1) / kWarps, kWarps * 32, 0, stream>>>(
        normalized, gate, logit_offset, rows, experts, hidden, logits);
  } else if (experts % 4 == 0 && rows * (experts / 4) >= num_sms * kWarps) {
    // four experts per warp once that still gives every SM a block
    const int warps = rows * (experts / 4);
    router_logits_kernel<1, 4><<<(warps + kWarps - 1) / kWarps, kWarps * 32, 0, stream>>>(
        normalized, gate, logit_offset, rows, experts, hidden, logits);
  } else {
    // a handful of rows: one (row, expert) pair per warp, so that the gate streams
    // through all SMs instead of a few
    const int warps = rows * experts;
    router_logits_kernel<1, 1><<<(warps + kWarps - 1) / kWarps, kWarps * 32, 0, stream>>>(
        normalized, gate, logit_offset, rows, experts, hidden, logits);
  }
  return cudaGetLastError();
}

bool router_topk_arguments_valid(int rows, int experts, int top_k, int n_group, int topk_group) {
  return rows > 0 && experts > 0 && experts % 32 == 0 && experts <= kMaxExperts &&
         top_k > 0 && top_k <= 32 && top_k <= experts && n_group > 0 && n_group <= 32 &&
         topk_group > 0 && experts % n_group == 0;
}

cudaError_t launch_router_topk(const float* logits, const float* bias, int rows, int experts,
                               int top_k, int n_group, int topk_group, bool norm_topk_prob,
                               float routed_scaling, int32_t* top_index, float* top_weight,
                               int32_t* expert_counts, int32_t* position, int num_sms,
                               LaunchStream stream) {
  if (!router_topk_arguments_valid(rows, experts, top_k, n_group, topk_group)) {
    return cudaErrorInvalidValue;
  }
  auto run = [&](auto kernel, int per_expert) {
    const int threads = rows <= num_sms ? per_expert : 128;
    launch_kernel(kernel, rows, threads, 0, stream, logits, bias, experts, top_k, n_group, topk_group,
                                              norm_topk_prob, routed_scaling, top_index, top_weight,
                                              expert_counts, position);
  };
  constexpr int kMostPerLane = kMaxExperts / 32;
  if (experts <= 128) {
    run(router_topk_kernel<4, false>, 4 * 32);
  } else if (experts <= 256) {
    run(select_narrows(8, top_k) ? router_topk_kernel<8, true> : router_topk_kernel<8, false>, 8 * 32);
  } else {
    run(select_narrows(kMostPerLane, top_k) ? router_topk_kernel<kMostPerLane, true>
                                            : router_topk_kernel<kMostPerLane, false>, kMaxExperts);
  }
  return cudaGetLastError();
}

}  // namespace nmoe
