// The words through which the blocks of a front-end launch (csrc/front.cu) hand a row on, and how they
// get back to zero for the next launch.  Also compiled for the host, without CUDA.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define NMOE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define NMOE_HOST_DEVICE inline
#endif

namespace nmoe {

constexpr int kFrontMaxRows = 8;
constexpr int kFrontLinears = 2;

// All zero between launches.
struct FrontWords {
  int32_t row_known[kFrontMaxRows];    // whether 1/rms is
  int32_t row_rounded[kFrontLinears];  // ... the one row as a linear multiplies with it
  int32_t finished;                    // blocks whose logits are there
  int32_t linear_finished[kFrontLinears];
  int32_t groups_finished;
};

// A launch is made of groups of blocks: each token's, each linear's rounding, the gate's and each linear's
// outputs.  A group is through once none of its blocks will announce a row or wait for one any more, and
// whichever is last takes the announcements back.  Those that announce count too: a block that waits gives
// up after a while, and what it gave up on, announced later, must not be there for the next launch.
NMOE_HOST_DEVICE constexpr int front_groups(int rows, int linears) { return rows + 1 + 2 * linears; }

// One group is through; `count` adds one to a word and returns what it held.
template <typename Count>
NMOE_HOST_DEVICE void front_group_through(FrontWords* words, int rows, int linears, Count count) {
  if (count(&words->groups_finished) != front_groups(rows, linears) - 1) return;
  for (int r = 0; r < rows; ++r) words->row_known[r] = 0;
  for (int i = 0; i < linears; ++i) words->row_rounded[i] = 0;
  words->groups_finished = 0;
}

}  // namespace nmoe
