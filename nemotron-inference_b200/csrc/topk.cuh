// Sigmoid scores and the selection of one token's experts by one warp (csrc/router.cu describes it; the
// small-batch front end in csrc/front.cu runs the same steps).
#pragma once

#include "common.cuh"

namespace nmoe {

// Sigmoid of expert_layer.cpp:129-136.  The host evaluates std::exp on a float;
// here exp runs in double and is rounded once, which equals the correctly
// rounded single-precision exponential.
__device__ __forceinline__ float sigmoid_ref(float v) {
  const float e = static_cast<float>(exp(-fabs(static_cast<double>(v))));
  return __fdiv_rn(v >= 0.0f ? 1.0f : e, __fadd_rn(1.0f, e));
}

// Order-preserving map of a float onto unsigned integers; 0 is left for "taken or absent".
__device__ __forceinline__ uint32_t choice_key(float v) {
  const uint32_t b = __float_as_uint(v);
  const uint32_t key = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  return key == 0u ? 1u : key;
}

// By all lanes of a warp, from a token's scores and choices (score + bias) in shared memory: lane r ends
// up with the r-th selected expert and its score; returns the sum of the selected scores in selection
// order.
template <int PER_LANE>
__device__ __forceinline__ float select_experts(const float* score_smem, const float* choice_smem,
                                                int experts, int top_k, int n_group, int topk_group,
                                                int& my_index, float& my_score) {
  const int lane = threadIdx.x & 31;
  uint32_t selected_groups = 0xffffffffu;
  const int group_size = experts / n_group;
  if (n_group > 1) {
    // group score = sum of the two largest choices of the group (:299-318);
    // keep topk_group groups, zero the others' choices (:320-339)
    uint32_t group_key = 0u;
    if (lane < n_group) {
      float top1 = -INFINITY, top2 = -INFINITY;
      for (int i = 0; i < group_size; ++i) {
        const float v = choice_smem[lane * group_size + i];
        if (v > top1) {
          top2 = top1;
          top1 = v;
        } else if (v > top2) {
          top2 = v;
        }
      }
      if (!isfinite(top2)) top2 = top1;
      group_key = choice_key(__fadd_rn(top1, top2));
    }
    selected_groups = 0u;
    const int keep = min(topk_group, n_group);
    for (int r = 0; r < keep; ++r) {
      const uint32_t best = __reduce_max_sync(0xffffffffu, group_key);
      const uint32_t index =
          __reduce_min_sync(0xffffffffu, group_key == best ? static_cast<uint32_t>(lane) : 31u);
      selected_groups |= 1u << index;
      if (static_cast<uint32_t>(lane) == index) group_key = 0u;
    }
  }

  uint32_t key[PER_LANE];
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int e = lane + 32 * j;
    key[j] = 0u;
    if (e < experts) {
      float choice = choice_smem[e];
      if (n_group > 1 && ((selected_groups >> (e / group_size)) & 1u) == 0u) choice = 0.0f;
      key[j] = choice_key(choice);
    }
  }
  uint32_t local_key = 0u, local_index = 0xffffffffu;
  auto rescan = [&]() {
    local_key = 0u;
    local_index = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      if (key[j] > local_key) {  // ascending j is ascending expert index: first maximum wins
        local_key = key[j];
        local_index = static_cast<uint32_t>(lane + 32 * j);
      }
    }
  };
  rescan();
  my_index = 0;  // lane r keeps the r-th selection
  for (int r = 0; r < top_k; ++r) {
    const uint32_t best = __reduce_max_sync(0xffffffffu, local_key);
    const uint32_t index =
        __reduce_min_sync(0xffffffffu, local_key == best ? local_index : 0xffffffffu);
    if (local_index == index) {
#pragma unroll
      for (int j = 0; j < PER_LANE; ++j) {
        if (j == static_cast<int>(index >> 5)) key[j] = 0u;  // taken
      }
      rescan();
    }
    if (lane == r) my_index = static_cast<int>(index);
  }

  // weight = score (no bias) normalised over the selection in selection order
  // (:349-365)
  my_score = score_smem[my_index];
  float weight_sum = 0.0f;
  for (int r = 0; r < top_k; ++r) {
    weight_sum = __fadd_rn(weight_sum, __shfl_sync(0xffffffffu, my_score, r));
  }
  return weight_sum;
}

// The routing weight of a selected expert (expert_layer.cpp:349-365).
__device__ __forceinline__ float selected_weight(float score, float sum, bool norm_topk_prob,
                                                 float routed_scaling) {
  float w = score;
  if (norm_topk_prob) w = __fdiv_rn(w, __fadd_rn(sum, 1.0e-20f));
  return __fmul_rn(w, routed_scaling);
}

}  // namespace nmoe
