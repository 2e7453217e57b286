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

// The groups that stay (expert_layer.cpp:299-339), as bits: a group's score is the sum of its two largest
// choices, and topk_group groups are kept.
__device__ __forceinline__ uint32_t select_groups(const float* choice_smem, int experts, int n_group,
                                                  int topk_group) {
  if (n_group <= 1) return 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int group_size = experts / n_group;
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
  uint32_t selected_groups = 0u;
  const int keep = min(topk_group, n_group);
  for (int r = 0; r < keep; ++r) {
    const uint32_t best = __reduce_max_sync(0xffffffffu, group_key);
    const uint32_t index =
        __reduce_min_sync(0xffffffffu, group_key == best ? static_cast<uint32_t>(lane) : 31u);
    selected_groups |= 1u << index;
    if (static_cast<uint32_t>(lane) == index) group_key = 0u;
  }
  return selected_groups;
}

// Many experts, by all lanes of a warp: lane r returns the r-th selected one.  `keys` holds the choices and
// becomes their keys; `list` has room for kSelectList words.  The top_k-th largest of the lanes' maxima is
// a bound that top_k experts reach and few others do (512 experts, top-22: some forty), so those are picked
// out, and a round is a choice between two of a lane.  Loops, not straight lines: fetching the code is
// what a single token waits for.
constexpr int kSelectList = 128;
__device__ __forceinline__ int select_among_many(uint32_t* keys, uint32_t* list, int experts, int top_k,
                                                 int n_group, uint32_t selected_groups) {
  const int lane = threadIdx.x & 31;
  const int group_size = experts / n_group;
  uint32_t most = 0u;
#pragma unroll 1
  for (int e = lane; e < experts; e += 32) {
    float choice = __uint_as_float(keys[e]);
    if (n_group > 1 && ((selected_groups >> (e / group_size)) & 1u) == 0u) choice = 0.0f;
    const uint32_t key = choice_key(choice);
    keys[e] = key;
    most = max(most, key);
  }
  int rank = 0;  // of this lane's maximum among the lanes'
#pragma unroll 4
  for (int r = 0; r < 32; ++r) {
    const uint32_t other = __shfl_sync(0xffffffffu, most, r);
    rank += other > most || (other == most && r < lane) ? 1 : 0;
  }
  const int from = __ffs(__ballot_sync(0xffffffffu, rank == top_k - 1)) - 1;
  const uint32_t bound = __shfl_sync(0xffffffffu, most, from);
  int total = 0;
#pragma unroll 1
  for (int e = lane; e < experts; e += 32) {
    const bool reaches = keys[e] >= bound;
    const uint32_t lanes = __ballot_sync(0xffffffffu, reaches);
    const int at = total + __popc(lanes & ((1u << lane) - 1u));
    if (reaches && at < kSelectList / 2) {
      list[at] = keys[e];
      list[kSelectList / 2 + at] = static_cast<uint32_t>(e);
    }
    total += __popc(lanes);
  }
  __syncwarp();
  int my_index = 0;
  if (total <= kSelectList / 2) {
    uint32_t first = 0u, first_at = 0xffffffffu, second = 0u, second_at = 0xffffffffu;
    if (lane < total) first = list[lane], first_at = list[kSelectList / 2 + lane];
    if (lane + 32 < total) second = list[32 + lane], second_at = list[kSelectList / 2 + 32 + lane];
#pragma unroll 1
    for (int r = 0; r < top_k; ++r) {
      const bool swap = second > first || (second == first && second_at < first_at);
      const uint32_t key = swap ? second : first, at = swap ? second_at : first_at;
      const uint32_t best = __reduce_max_sync(0xffffffffu, key);
      const uint32_t index = __reduce_min_sync(0xffffffffu, key == best ? at : 0xffffffffu);
      if (lane == r) my_index = static_cast<int>(index);
      if (at != index) continue;
      (swap ? second : first) = 0u;
      (swap ? second_at : first_at) = 0xffffffffu;
    }
    return my_index;
  }
  // too many of the same choice: every lane looks through all of its own
#pragma unroll 1
  for (int r = 0; r < top_k; ++r) {
    uint32_t key = 0u, at = 0xffffffffu;
#pragma unroll 1
    for (int e = lane; e < experts; e += 32) {
      if (keys[e] > key) {  // (ascending: the lower expert of equal ones)
        key = keys[e];
        at = static_cast<uint32_t>(e);
      }
    }
    const uint32_t best = __reduce_max_sync(0xffffffffu, key);
    const uint32_t index = __reduce_min_sync(0xffffffffu, key == best ? at : 0xffffffffu);
    if (at == index) keys[index] = 0u;
    if (lane == r) my_index = static_cast<int>(index);
  }
  return my_index;
}

// The same for up to 32 * PER_LANE experts: each lane holds its own, the best of which it keeps at hand.
template <int PER_LANE>
__device__ __forceinline__ int select_among_few(const float* choice_smem, int experts, int top_k,
                                                int n_group, uint32_t selected_groups) {
  constexpr int kPerLane = PER_LANE;
  const int lane = threadIdx.x & 31;
  const int group_size = experts / n_group;
  uint32_t key[kPerLane];
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
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
    for (int j = 0; j < kPerLane; ++j) {
      if (key[j] > local_key) {  // ascending j is ascending expert index: first maximum wins
        local_key = key[j];
        local_index = static_cast<uint32_t>(lane + 32 * j);
      }
    }
  };
  rescan();
  int my_index = 0;
  for (int r = 0; r < top_k; ++r) {
    const uint32_t best = __reduce_max_sync(0xffffffffu, local_key);
    const uint32_t index =
        __reduce_min_sync(0xffffffffu, local_key == best ? local_index : 0xffffffffu);
    if (local_index == index) {
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        if (j == static_cast<int>(index >> 5)) key[j] = 0u;  // taken
      }
      rescan();
    }
    if (lane == r) my_index = static_cast<int>(index);
  }
  return my_index;
}

// By all lanes of a warp, from a token's scores and choices (score + bias) in shared memory: lane r ends
// up with the r-th selected expert and its score; returns the sum of the selected scores in selection
// order.  PER_LANE: 4, 8 or 16, for up to 32 times as many experts; the choices may be overwritten.
//
// Narrowing down pays from some ten rounds on, while the lanes' maxima still leave few: the bound of 24 of 32
// lanes leaves more than the list holds for one token in a thousand of 512 experts, that of 27 for one in ten, and
// a launch waits for the slowest (9 tokens, top-27 49.6 us looked through and 62.2, top-32 53.7 and 67.8).
// Whole pass, looked through against narrowed down: 256 experts, 16 tokens, top-4 32.4 us and 33.1, top-8 35.7 and
// 36.8, top-12 39.3 and 39.5, top-16 42.6 and 41.8, top-32 51.4 and 57.6; 160 experts, 9 tokens, top-4 27.5 and
// 28.9, top-12 33.8 and 33.8, top-22 39.2 and 37.3, top-32 41.3 and 45.4.  Sixteen to a lane are narrowed down
// whatever top_k up to that (512 experts, top-22 13 us in a launch's last block looked through, 5.8 narrowed down).
constexpr int kSelectFewTopK = 10;
constexpr int kSelectMostNarrowed = 23;
__host__ __device__ constexpr bool select_narrows(int per_lane, int top_k) {
  return per_lane > 4 && (per_lane > 8 || top_k > kSelectFewTopK) && top_k <= kSelectMostNarrowed;
}
// (`narrowed`: select_narrows() of the two, a constant where a kernel is to hold only one of the ways)
template <int PER_LANE>
__device__ __forceinline__ float select_experts(const float* score_smem, float* choice_smem,
                                                uint32_t* list, int experts, int top_k, int n_group,
                                                int topk_group, bool narrowed, int& my_index,
                                                float& my_score) {
  const uint32_t groups = select_groups(choice_smem, experts, n_group, topk_group);
  __syncwarp();
  if (PER_LANE > 4 && narrowed) {
    my_index = select_among_many(reinterpret_cast<uint32_t*>(choice_smem), list, experts, top_k,
                                 n_group, groups);
  } else {
    my_index = select_among_few<PER_LANE>(choice_smem, experts, top_k, n_group, groups);
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
