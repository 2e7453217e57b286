// Two-pass router for large token counts.
//
// The reference computes gate logits with a sequential DOUBLE accumulation on
// the host (runtime/src/backend/linear_op.cpp:97-118) and selects experts from
// them (runtime/src/backend/expert_layer.cpp:277-367).  Matching its selected
// index sets bit for bit needs logits that round like an FP64 sum, but FP64 for
// every (token, expert) pair costs more than the expert GEMMs.  So:
//
//  pass 1  all logits on the tensor cores.  The FP32 normalised activation
//          y = (x * inv_rms) * w is recomputed in the kernel from the layer input
//          (the same two roundings as the RMSNorm kernel), split into three bf16
//          terms (hi + mid + lo carries the full 24-bit significand) that go
//          straight into shared memory in the tensor core's 128-byte swizzle;
//          the gate is bf16, products are exact and accumulate in FP32
//          (tcgen05.mma.kind::f16, accumulator in TMEM).  Nothing but the layer
//          input is read per token: no FP32 copy of y, no bf16 planes in HBM;
//  pass 2  per token, every expert whose pass-1 choice score lies within
//          `tie_margin` of the top_k-th score is re-evaluated with the FP64 sum
//          and the selection runs on those exact values.
//
// If every pass-1 score is within tie_margin/2 of its exact value, the exact
// top-k set is contained in the candidates, so indices AND weights equal the
// all-FP64 path.  tie_margin is ~20x the largest pass-1 error measured.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace nmoe {
namespace {

// ---------------------------------------------------------------------------
// pass 1: logits[128 tokens x E] per CTA, up to 256 experts
// ---------------------------------------------------------------------------
constexpr int kFastBlockK = 64;                 // bf16 elements per 128-byte row
constexpr int kFastABytes = 3 * 128 * 128;      // three planes of 128 rows x 128 B
constexpr int kSplitWarps = 8;                  // warps that build the planes, then store
constexpr int kFastThreads = (2 + kSplitWarps) * 32;

// Dynamic shared memory: the stages, a full and an empty barrier for each, one more, the TMEM
// address, and room to align.
constexpr int pass1_smem_bytes(int stages, int stage_bytes) {
  return stages * stage_bytes + (2 * stages + 1) * 8 + 16 + 1024;
}
// Stages of a launch: up to `most`, as many as fit.
constexpr int pass1_stages(int most, int stage_bytes) {
  int stages = most;
  while (stages > 1 && pass1_smem_bytes(stages, stage_bytes) > kMaxSharedBytes) --stages;
  return stages;
}

__device__ __forceinline__ void tcgen05_mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                                 uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// kind::f16 instruction descriptor: FP32 accumulate, bf16 x bf16, K-major, M=128
__host__ __device__ constexpr uint32_t make_idesc_bf16(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// Eight consecutive input elements of one row as FP32.
template <bool BF16>
__device__ __forceinline__ void load_x8(const void* x, size_t index, float (&v)[8]) {
  if constexpr (BF16) {
    const uint4 raw = *reinterpret_cast<const uint4*>(
        reinterpret_cast<const __nv_bfloat16*>(x) + index);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  } else {
    const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + index);
    const float4 b = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + index + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}

template <bool IN_BF16, int STAGES>
__global__ void __launch_bounds__(kFastThreads, 1)
router_fast_logits_kernel(const void* __restrict__ x, const float* inv_rms,
                          const float* __restrict__ norm_weight,
                          const __grid_constant__ CUtensorMap tmap_gate, int rows, int experts,
                          int hidden, int splits, float* __restrict__ logits, int32_t* error) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) &
                                             ~static_cast<uintptr_t>(1023u));
  const int b_bytes = experts * 128;
  uint8_t* sA = smem;
  uint8_t* sB = sA + STAGES * kFastABytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sB + STAGES * b_bytes);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* done_bar = empty_bar + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // `splits` CTAs share the contraction of a tile (see router_folded_logits_kernel)
  const int tile = static_cast<int>(blockIdx.x) / splits;
  const int split = static_cast<int>(blockIdx.x) - tile * splits;
  const int row0 = tile * 128;
  const int all_k_blocks = hidden / kFastBlockK;
  const int kb_begin = all_k_blocks * split / splits;
  const int k_blocks = all_k_blocks * (split + 1) / splits - kb_begin;
  const uint32_t tmem_cols = experts <= 32 ? 32 : experts <= 64 ? 64 : experts <= 128 ? 128 : 256;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      // the gate tile arrives by TMA (one arrive + bytes), the planes are written by
      // the split warps (one arrive each)
      mbar_init(&full_bar[s], 1 + kSplitWarps);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
    prefetch_tensormap(&tmap_gate);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, tmem_cols);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u)) {
          if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
          break;
        }
        mbar_arrive_expect_tx(&full_bar[stage], b_bytes);
        tma_load_2d(sB + stage * b_bytes, &tmap_gate, (kb_begin + kb) * kFastBlockK, 0,
                    &full_bar[stage]);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_bf16(static_cast<uint32_t>(experts));
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = 0; kb < k_blocks && ok; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase)) {
          if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const uint32_t a_addr = smem_u32(sA + stage * kFastABytes);
        const uint32_t b_addr = smem_u32(sB + stage * b_bytes);
        // smallest terms first, so that they are not absorbed by a large partial sum
        for (int plane = 2; plane >= 0; --plane) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {  // K = 16 bf16 = 32 bytes per MMA
            tcgen05_mma_bf16(tmem_base,
                             make_smem_desc(a_addr + plane * (128 * 128) + ks * 32, 0, 1024, 2),
                             make_smem_desc(b_addr + ks * 32, 0, 1024, 2), idesc,
                             (kb != 0 || plane != 2 || ks != 0) ? 1u : 0u);
          }
        }
        tcgen05_commit(&empty_bar[stage]);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) tcgen05_commit(done_bar);
    }
  } else {
    // ------------------------------------------------- split warps, then epilogue
    // Thread s of the 256 owns 16-byte chunk (s % 8) of rows (s / 8) + 32 j, j = 0..3,
    // of every K block: eight threads read one row's 128 (bf16) or 256 (FP32) bytes
    // together and write the row's three 128-byte plane rows, chunk c of row r at
    // position c ^ (r % 8) (the tensor core's 128-byte swizzle).
    const int s = threadIdx.x - 64;
    const int chunk = s & 7;
    float rinv[4];
    int row_of[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      row_of[j] = (s >> 3) + 32 * j;
      const int row = row0 + row_of[j];
      rinv[j] = row < rows ? inv_rms[row] : 0.0f;
    }
    // two K blocks of input stay in flight in registers: a row's 128-byte pieces are
    // 5 KB apart in memory, so each fetch pays a full memory latency
    float xv[2][4][8];
    auto fetch = [&](int kb, float (&dst)[4][8]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = min(row0 + row_of[j], rows - 1);
        load_x8<IN_BF16>(
            x, static_cast<size_t>(row) * hidden + (kb_begin + kb) * kFastBlockK + chunk * 8, dst[j]);
      }
    };
    fetch(0, xv[0]);
    if (k_blocks > 1) fetch(1, xv[1]);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = 0; kb < k_blocks; ++kb) {
      const float* w_at = norm_weight + (kb_begin + kb) * kFastBlockK + chunk * 8;
      const float4 w0 = *reinterpret_cast<const float4*>(w_at);
      const float4 w1 = *reinterpret_cast<const float4*>(w_at + 4);
      const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
      uint32_t words[4][3][4];
      auto split = [&](float (&src)[4][8]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            // y exactly as the RMSNorm kernel rounds it: (x * inv_rms) * w
            float rem[2] = {__fmul_rn(__fmul_rn(src[j][i], rinv[j]), w[i]),
                            __fmul_rn(__fmul_rn(src[j][i + 1], rinv[j]), w[i + 1])};
#pragma unroll
            for (int term = 0; term < 3; ++term) {
              const __nv_bfloat16 a = __float2bfloat16_rn(rem[0]);
              const __nv_bfloat16 b = __float2bfloat16_rn(rem[1]);
              rem[0] = __fsub_rn(rem[0], __bfloat162float(a));
              rem[1] = __fsub_rn(rem[1], __bfloat162float(b));
              words[j][term][i / 2] = static_cast<uint32_t>(__bfloat16_as_ushort(a)) |
                                      (static_cast<uint32_t>(__bfloat16_as_ushort(b)) << 16);
            }
          }
        }
      };
      // (the buffer index is resolved at compile time: registers cannot be indexed)
      if (kb & 1) {
        split(xv[1]);
        if (kb + 2 < k_blocks) fetch(kb + 2, xv[1]);
      } else {
        split(xv[0]);
        if (kb + 2 < k_blocks) fetch(kb + 2, xv[0]);
      }
      if (ok && !mbar_wait(&empty_bar[stage], phase ^ 1u)) {
        if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
        ok = false;
      }
      if (ok) {
        uint8_t* planes = sA + stage * kFastABytes;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = row_of[j];
          const int offset = r * 128 + ((chunk ^ (r & 7)) << 4);
#pragma unroll
          for (int term = 0; term < 3; ++term) {
            *reinterpret_cast<uint4*>(planes + term * (128 * 128) + offset) =
                make_uint4(words[j][term][0], words[j][term][1], words[j][term][2],
                           words[j][term][3]);
          }
        }
        fence_proxy_async_smem();  // the tensor core reads these stores
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[stage]);
      }
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1u;
      }
    }
    // epilogue: the first four split warps own one TMEM lane quarter each
    if (warp < 6) {
      const int quarter = warp & 3;
      const int row = row0 + quarter * 32 + lane;
      if (ok && mbar_wait(done_bar, 0)) {
        tcgen05_fence_after();
        const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        for (int c = 0; c < experts; c += 16) {
          float v[16];
          tmem_ld_x16(t_addr + c, v);
          if (row < rows) {
            float* dst = logits + (static_cast<size_t>(split) * rows + row) * experts + c;
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            }
          }
        }
      } else if (error != nullptr) {
        atomicCAS(error, kDevOk, kDevWaitTimeout);
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

// ---------------------------------------------------------------------------
// pass 1 for bf16 layer inputs: the RMSNorm weight is folded into the gate once,
//   logit[t][e] ~= inv_rms[t] * sum_i x[t][i] * (w[i] * gate[e][i]),
// so the bf16 input itself is the (exact, single-term) A operand, loaded by TMA, and
// the three bf16 terms of fl32(w[i] * gate[e][i]) are the B operands, split once when
// the layer is created.  Same three MMAs per K step as the kernel above, but no warp
// touches the operands: one producer lane, one MMA lane, four epilogue warps.  Against
// the reference's y = fl(fl(x * inv_rms) * w) this drops two roundings of 2^-24 per term,
// the size of the FP32 accumulation error already covered by the tie margin.
// ---------------------------------------------------------------------------
constexpr int kFoldThreads = 6 * 32;
constexpr int kFoldABytes = 128 * 128;  // 128 rows x 64 bf16

__global__ void fold_gate_kernel(const __nv_bfloat16* __restrict__ gate,
                                 const float* __restrict__ norm_weight, int experts, int hidden,
                                 __nv_bfloat16* __restrict__ planes) {
  const size_t total = static_cast<size_t>(experts) * hidden;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    float rem = __fmul_rn(norm_weight[i % hidden], __bfloat162float(gate[i]));
#pragma unroll
    for (int term = 0; term < 3; ++term) {
      const __nv_bfloat16 part = __float2bfloat16_rn(rem);
      rem = __fsub_rn(rem, __bfloat162float(part));
      planes[term * total + i] = part;
    }
  }
}

__global__ void __launch_bounds__(kFoldThreads, 1)
router_folded_logits_kernel(const __grid_constant__ CUtensorMap tmap_x,
                            const __grid_constant__ CUtensorMap tmap_planes,
                            const float* inv_rms, int rows, int experts, int hidden,
                            int stages, int splits, float* __restrict__ logits, int32_t* error) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) &
                                             ~static_cast<uintptr_t>(1023u));
  const int plane_bytes = experts * 128;
  const int b_bytes = 3 * plane_bytes;
  uint8_t* sA = smem;
  uint8_t* sB = sA + stages * kFoldABytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sB + stages * b_bytes);
  uint64_t* empty_bar = full_bar + stages;
  uint64_t* done_bar = empty_bar + stages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // With few row tiles the contraction is split over `splits` CTAs per tile (split s
  // writes its partial sums to logits + s * rows * experts; pass 2 adds them up), so that
  // a batch of a few thousand tokens still spreads over the SMs.
  const int tile = static_cast<int>(blockIdx.x) / splits;
  const int split = static_cast<int>(blockIdx.x) - tile * splits;
  const int row0 = tile * 128;
  const int all_k_blocks = hidden / kFastBlockK;
  const int kb_begin = all_k_blocks * split / splits;
  const int k_blocks = all_k_blocks * (split + 1) / splits - kb_begin;
  const uint32_t tmem_cols = experts <= 32 ? 32 : experts <= 64 ? 64 : experts <= 128 ? 128 : 256;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
    prefetch_tensormap(&tmap_x);
    prefetch_tensormap(&tmap_planes);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, tmem_cols);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1u)) {
          if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
          break;
        }
        mbar_arrive_expect_tx(&full_bar[stage], kFoldABytes + b_bytes);
        // rows past the end of the input read as zeros (the map's extent is `rows`)
        tma_load_2d(sA + stage * kFoldABytes, &tmap_x, (kb_begin + kb) * kFastBlockK, row0,
                    &full_bar[stage]);
        for (int plane = 0; plane < 3; ++plane) {
          tma_load_2d(sB + stage * b_bytes + plane * plane_bytes, &tmap_planes,
                      (kb_begin + kb) * kFastBlockK, plane * experts, &full_bar[stage]);
        }
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_bf16(static_cast<uint32_t>(experts));
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = 0; kb < k_blocks && ok; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase)) {
          if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const uint32_t a_addr = smem_u32(sA + stage * kFoldABytes);
        const uint32_t b_addr = smem_u32(sB + stage * b_bytes);
        // smallest terms first, so that they are not absorbed by a large partial sum
        for (int plane = 2; plane >= 0; --plane) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {  // K = 16 bf16 = 32 bytes per MMA
            tcgen05_mma_bf16(tmem_base, make_smem_desc(a_addr + ks * 32, 0, 1024, 2),
                             make_smem_desc(b_addr + plane * plane_bytes + ks * 32, 0, 1024, 2),
                             idesc, (kb != 0 || plane != 2 || ks != 0) ? 1u : 0u);
          }
        }
        tcgen05_commit(&empty_bar[stage]);
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) tcgen05_commit(done_bar);
    }
  } else {
    // epilogue: warp w owns TMEM lane quarter w % 4
    const int quarter = warp & 3;
    const int row = row0 + quarter * 32 + lane;
    const float rinv = row < rows ? inv_rms[row] : 0.0f;
    if (mbar_wait(done_bar, 0)) {
      tcgen05_fence_after();
      const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      for (int c = 0; c < experts; c += 16) {
        float v[16];
        tmem_ld_x16(t_addr + c, v);
        if (row < rows) {
          float* dst = logits + (static_cast<size_t>(split) * rows + row) * experts + c;
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            *reinterpret_cast<float4*>(dst + i) =
                make_float4(v[i] * rinv, v[i + 1] * rinv, v[i + 2] * rinv, v[i + 3] * rinv);
          }
        }
      }
    } else if (error != nullptr) {
      atomicCAS(error, kDevOk, kDevWaitTimeout);
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

// ---------------------------------------------------------------------------
// pass 2: candidates -> FP64 logits -> exact selection
// ---------------------------------------------------------------------------
constexpr int kSelectWarps = 4;
constexpr int kSelectMaxPerLane = 8;  // experts <= 256

__device__ __forceinline__ float sigmoid_exact(float v) {
  // Sigmoid of expert_layer.cpp:129-136 with exp evaluated in double
  if (v >= 0.0f) {
    const float e = static_cast<float>(exp(-static_cast<double>(v)));
    return __fdiv_rn(1.0f, __fadd_rn(1.0f, e));
  }
  const float e = static_cast<float>(exp(static_cast<double>(v)));
  return __fdiv_rn(e, __fadd_rn(1.0f, e));
}

// Order-preserving map of a float onto unsigned integers (0 is below every value), so
// that a warp-wide maximum is one redux instruction.
__device__ __forceinline__ uint32_t ordered_bits(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// The largest key of the warp and, among its holders, the smallest index
// (SelectTopExperts ranks by value; ties resolve to the lower expert index).
__device__ __forceinline__ void warp_arg_max(uint32_t key, uint32_t index, uint32_t& best_key,
                                             uint32_t& best_index) {
  best_key = __reduce_max_sync(0xffffffffu, key);
  best_index = __reduce_min_sync(0xffffffffu, key == best_key ? index : 0xffffffffu);
}

// A bf16 value (the upper half of `w`; the lower half is ignored) times 2^-896 as a double, in
// two integer instructions: the bits of a bf16 moved three places down are those of a double
// whose exponent field still has the 8-bit bias (subnormals included).  The conversion unit
// would be what this kernel waits for: it has a quarter of the FP64 unit's rate.
constexpr double kGateUnscale = 0x1p896;
__device__ __forceinline__ double gate_scaled(uint32_t w) {
  return __hiloint2double((static_cast<int>(w) >> 3) & static_cast<int>(0x8fffe000u), 0);
}

// WARPS warps per token: one for large batches (four tokens a block, nothing exchanged), four
// for small ones, where the chain of loads and FP64 sums of one token is what counts: they
// share the contraction and repeat the short steps around it.  BATCH candidates are evaluated
// per pass over the row (at least top_k, so that one pass is the rule).
// Measured, 128 experts, hidden 2688, bf16 in: 256 tokens 35 -> 17 us, 16384 tokens
// 143 -> 92 us.
// Bound by instructions (60 % of the issue slots, half of them the integer ones of gate_scaled) and by the
// warps there are to fill the rest: 72 registers, seven blocks to an SM, instead of 84 took 16384 tokens
// from 106 to 92 us, 1003 from 21 to 16.5; the short steps with a lane per candidate and without rounds
// that look through eight slots 119 to 106 before that.
// Up to some number of tokens the block form is the faster one, the more the longer a token's sums and the
// more its choices are.  us, block against warp, of the selection: 128 experts of 2688, top-6, 1280 tokens 22.6
// and 28.7, 2048 24.6 and 26.6, 3072 34.6 and 34.6; of 4096 2048 tokens 28.5 and 34.6; of 1024 2048 tokens 20.6
// and 22.9, 2560 24.6 and 23.3; 256 experts of 2688, top-8, 1536 tokens 32.5 and 36.6, 2048 34.6 and 34.6, 2560
// 46.9 and 44.9; of 2048 2048 tokens 30.5 and 31.0.  Of a pass: 32 experts of 512 700 tokens 52.5 and 52.8, 1280
// 59.8 and 58.2; 64 of 1024, top-4, 1024 tokens 53.8 and 55.8, 2048 74.6 and 71.7; 128 of 256 1024 tokens 50.3
// and 51.3, 1280 54.7 and 52.6; 128 of 512 1280 tokens 60.5 and 60.9, 2048 66.1 and 64.5; 256 of 512 1280 tokens
// 73.4 and 75.3, 1536 80.5 and 78.6.
int select_whole_block_rows(int experts, int hidden) {
  return std::min(2048, 600 + std::min(experts, 128) * hidden / 80);
}
template <bool IN_BF16, int WARPS, int BATCH, int kSelectPerLane>
__global__ void __launch_bounds__(kSelectWarps * 32, BATCH <= 6 ? 7 : 5)
router_select_exact_kernel(float* __restrict__ logits, int splits, const void* __restrict__ x,
                           const float* inv_rms,
                           const float* __restrict__ norm_weight,
                           const __nv_bfloat16* __restrict__ gate,
                           const float* __restrict__ logit_offset, const float* __restrict__ bias,
                           int rows, int experts, int hidden, int top_k, bool norm_topk_prob,
                           float routed_scaling, float tie_margin,
                           int32_t* __restrict__ top_index, float* __restrict__ top_weight,
                           int32_t* __restrict__ expert_counts, int32_t* __restrict__ position) {
  static_assert(WARPS == 1 || WARPS == kSelectWarps, "one warp, or the block, per token");
  __shared__ int16_t candidate_list[kSelectWarps][256];
  __shared__ float logit_smem[WARPS > 1 ? 256 : 1];
  __shared__ double partial_smem[WARPS > 1 ? kSelectWarps : 1][8];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int part = WARPS > 1 ? warp : 0;  // this warp's share of the contraction
  const int row = WARPS > 1 ? static_cast<int>(blockIdx.x) : blockIdx.x * kSelectWarps + warp;
  if (row >= rows) return;
  const int per_lane = experts / 32;
  float* row_logits = logits + static_cast<size_t>(row) * experts;

  // pass-1 logit of expert e: the partial sums of a split pass 1, in split order
  const bool changed = logit_offset != nullptr || splits > 1;
  auto pass1_logit = [&](int e) {
    float l = row_logits[e];
    const size_t step = static_cast<size_t>(rows) * experts;
    const float* next = row_logits + e;
#pragma unroll 8
    for (int sp = 1; sp < splits; ++sp) {
      next += step;
      l = __fadd_rn(l, *next);
    }
    if (logit_offset != nullptr) l = __fadd_rn(l, logit_offset[e]);
    if (changed) row_logits[e] = l;  // what the trace shows for experts not re-evaluated
    return l;
  };
  if constexpr (WARPS > 1) {
    for (int e = threadIdx.x; e < experts; e += kSelectWarps * 32) logit_smem[e] = pass1_logit(e);
    __syncthreads();
  }
  // pass-1 choice scores (single precision is enough here: the margin covers it);
  // lane L holds experts L, L + 32, ...
  float choice[kSelectPerLane];
  uint32_t key[kSelectPerLane];
#pragma unroll
  for (int j = 0; j < kSelectPerLane; ++j) {
    choice[j] = -INFINITY;
    key[j] = 0u;
    if (j < per_lane) {
      const int e = lane + 32 * j;
      const float l = WARPS > 1 ? logit_smem[e] : pass1_logit(e);
      choice[j] = __fdividef(1.0f, 1.0f + __expf(-l)) + bias[e];
      key[j] = ordered_bits(choice[j]);
    }
  }
  // the top_k-th largest pass-1 choice (equal ones are taken together)
  uint32_t kth_key = 0u;
  for (int taken = 0; taken < top_k;) {
    uint32_t most = key[0];
#pragma unroll
    for (int j = 1; j < kSelectPerLane; ++j) most = max(most, key[j]);
    kth_key = __reduce_max_sync(0xffffffffu, most);
    if (kth_key == 0u) break;  // (nothing is left)
    int mine = 0;
#pragma unroll
    for (int j = 0; j < kSelectPerLane; ++j) {
      if (key[j] == kth_key) {
        key[j] = 0u;
        ++mine;
      }
    }
    taken += __reduce_add_sync(0xffffffffu, mine);
  }
  // candidates: everything that could still be in the exact top-k (a score that is no number
  // could be anywhere, so a row of them is re-evaluated as a whole and keeps them)
  float kth = 0.0f;
  {
    const uint32_t b = (kth_key & 0x80000000u) ? (kth_key & 0x7fffffffu) : ~kth_key;
    kth = __uint_as_float(b);
  }
  const float threshold = kth - tie_margin;
  int total = 0;
#pragma unroll
  for (int j = 0; j < kSelectPerLane; ++j) {
    const bool mine = j < per_lane && !(choice[j] < threshold);
    const uint32_t lanes = __ballot_sync(0xffffffffu, mine);
    if (mine) {
      candidate_list[warp][total + __popc(lanes & ((1u << lane) - 1u))] =
          static_cast<int16_t>(lane + 32 * j);
    }
    total += __popc(lanes);
  }
  __syncwarp();

  // FP64 logits of the candidates, BATCH at a time; every lane takes eight consecutive hidden
  // elements per step.  y is rebuilt from the layer input with the RMSNorm kernel's own two
  // roundings: (x * inv_rms) * w.
  const float rinv = inv_rms[row];
  const int chunks = hidden / 8;
  for (int base = 0; base < total; base += BATCH) {
    const int batch = min(BATCH, total - base);
    uint32_t gate_row[BATCH];  // in chunks of eight values (fewer registers than addresses)
    double acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0;
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      // (past the end of the list the last candidate once more, ignored below)
      const int e = candidate_list[warp][min(base + i, total - 1)];
      gate_row[i] = static_cast<uint32_t>(e) * static_cast<uint32_t>(chunks);
    }
    for (int ch = lane + 32 * part; ch < chunks; ch += 32 * WARPS) {
      uint4 g[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
        g[i] = reinterpret_cast<const uint4*>(gate)[gate_row[i] + ch];
      }
      float xv[8];
      load_x8<IN_BF16>(x, static_cast<size_t>(row) * hidden + ch * 8, xv);
      const float4 w0 = *reinterpret_cast<const float4*>(norm_weight + ch * 8);
      const float4 w1 = *reinterpret_cast<const float4*>(norm_weight + ch * 8 + 4);
      const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double a0 =
            static_cast<double>(__fmul_rn(__fmul_rn(xv[2 * j], rinv), w[2 * j])) * kGateUnscale;
        const double a1 =
            static_cast<double>(__fmul_rn(__fmul_rn(xv[2 * j + 1], rinv), w[2 * j + 1])) *
            kGateUnscale;
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
          const uint32_t two = j == 0 ? g[i].x : j == 1 ? g[i].y : j == 2 ? g[i].z : g[i].w;
          acc[i] = fma(a0, gate_scaled(two << 16), acc[i]);
          acc[i] = fma(a1, gate_scaled(two), acc[i]);
        }
      }
    }
    double sum = warp_sum8(acc, lane);
    const int mine_of_batch = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    if constexpr (WARPS > 1) {
      if ((lane & 3) == 0) partial_smem[warp][mine_of_batch] = sum;
      __syncthreads();
      sum = 0.0;
#pragma unroll
      for (int p = 0; p < WARPS; ++p) sum += partial_smem[p][mine_of_batch];
      __syncthreads();
    }
    if ((lane & 3) == 0 && mine_of_batch < batch && part == 0) {
      const int e = candidate_list[warp][base + mine_of_batch];
      float logit = static_cast<float>(sum);
      if (logit_offset != nullptr) logit = __fadd_rn(logit, logit_offset[e]);
      row_logits[e] = logit;
    }
  }
  if (part != 0) return;
  __syncwarp();

  // Exact scores, compacted: lane L takes candidate L of the list (L, L + 32, ... where there are more),
  // so the double-precision exponential runs once per lane instead of once per expert slot.
  int my_index = -1;  // lane r: the r-th selection
  float my_score = 0.0f, weight_sum = 0.0f;
  if (total <= 32) {
    // a candidate's place is the number of those before it: nothing waits for a round before
    const int ex = candidate_list[warp][min(lane, total - 1)];
    const float score = sigmoid_exact(*reinterpret_cast<volatile float*>(row_logits + ex));
    const uint32_t score_key = ordered_bits(__fadd_rn(score, bias[ex]));
    int place = lane < total ? 0 : 32;
    for (int c = 0; c < total; ++c) {
      const uint32_t other = __shfl_sync(0xffffffffu, score_key, c);
      const int other_ex = __shfl_sync(0xffffffffu, ex, c);
      place += other > score_key || (other == score_key && other_ex < ex) ? 1 : 0;
    }
    for (int r = 0; r < top_k; ++r) {
      const int owner = __ffs(__ballot_sync(0xffffffffu, place == r)) - 1;
      const float s = __shfl_sync(0xffffffffu, score, owner);
      const int index = __shfl_sync(0xffffffffu, ex, owner);
      weight_sum = __fadd_rn(weight_sum, s);
      if (lane == r) {
        my_index = index;
        my_score = s;
      }
    }
  } else {
    float score[kSelectPerLane];
    uint32_t cand_key[kSelectPerLane];
    int cand_expert[kSelectPerLane];
    const int rounds = (total + 31) / 32;
  #pragma unroll
    for (int j = 0; j < kSelectPerLane; ++j) {
      score[j] = 0.0f;
      cand_key[j] = 0u;
      cand_expert[j] = -1;
      if (j < rounds) {
        const int slot = lane + 32 * j;
        if (slot < total) {
          const int ex = candidate_list[warp][slot];
          const float l = *reinterpret_cast<volatile float*>(row_logits + ex);
          score[j] = sigmoid_exact(l);
          cand_key[j] = ordered_bits(__fadd_rn(score[j], bias[ex]));
          cand_expert[j] = ex;
        }
      }
    }
    for (int r = 0; r < top_k; ++r) {
      uint32_t local_key = 0u, local_index = 0xffffffffu;
      float local_score = 0.0f;
      int local_slot = -1;
  #pragma unroll
      for (int j = 0; j < kSelectPerLane; ++j) {
        const uint32_t ex = static_cast<uint32_t>(cand_expert[j]);
        if (cand_key[j] > local_key || (cand_key[j] == local_key && cand_key[j] != 0u &&
                                        ex < local_index)) {
          local_key = cand_key[j];
          local_index = ex;
          local_score = score[j];
          local_slot = j;
        }
      }
      uint32_t best_key, best_index;
      warp_arg_max(local_key, local_index, best_key, best_index);
      const bool owner = local_key == best_key && local_index == best_index && local_slot >= 0;
      const int owner_lane = __ffs(__ballot_sync(0xffffffffu, owner)) - 1;
      const float s = __shfl_sync(0xffffffffu, local_score, owner_lane < 0 ? 0 : owner_lane);
      if (owner) {
  #pragma unroll
        for (int j = 0; j < kSelectPerLane; ++j) {
          if (j == local_slot) cand_key[j] = 0u;  // taken
        }
      }
      if (lane == r) {
        my_index = static_cast<int>(best_index);
        my_score = s;
      }
    }
    for (int r = 0; r < top_k; ++r) {
      weight_sum = __fadd_rn(weight_sum, __shfl_sync(0xffffffffu, my_score, r));
    }
  }
  if (lane < top_k) {
    float w = my_score;
    if (norm_topk_prob) w = __fdiv_rn(w, __fadd_rn(weight_sum, 1.0e-20f));
    w = __fmul_rn(w, routed_scaling);
    top_index[static_cast<size_t>(row) * top_k + lane] = my_index;
    top_weight[static_cast<size_t>(row) * top_k + lane] = w;
    if (expert_counts != nullptr && static_cast<uint32_t>(my_index) < static_cast<uint32_t>(experts)) {
      const int place = atomicAdd(&expert_counts[my_index], 1);
      if (position != nullptr) position[static_cast<size_t>(row) * top_k + lane] = place;
    }
  }
}

}  // namespace

cudaError_t launch_router_fast_logits(const void* x, bool x_bf16, const float* inv_rms,
                                      const float* norm_weight, const CUtensorMap& tmap_gate,
                                      int rows, int experts, int hidden, int splits,
                                      float* logits, int32_t* error, cudaStream_t stream) {
  if (rows <= 0 || experts % 16 != 0 || experts > 256 || hidden % kFastBlockK != 0 ||
      splits < 1 || hidden / kFastBlockK < splits) {
    return cudaErrorInvalidValue;
  }
  // three stages up to 192 experts, two beyond
  const int stage_bytes = kFastABytes + experts * 128;
  const int stages = pass1_stages(3, stage_bytes);
  const int grid = (rows + 127) / 128 * splits;
  auto run = [&](auto kernel) {
    const cudaError_t err = allow_shared_memory(kernel);
    if (err != cudaSuccess) return err;
    kernel<<<grid, kFastThreads, pass1_smem_bytes(stages, stage_bytes), stream>>>(
        x, inv_rms, norm_weight, tmap_gate, rows, experts, hidden, splits, logits, error);
    return cudaGetLastError();
  };
  if (x_bf16) {
    return stages == 3 ? run(router_fast_logits_kernel<true, 3>)
                       : run(router_fast_logits_kernel<true, 2>);
  }
  return stages == 3 ? run(router_fast_logits_kernel<false, 3>)
                     : run(router_fast_logits_kernel<false, 2>);
}

cudaError_t launch_fold_gate(const __nv_bfloat16* gate, const float* norm_weight, int experts,
                             int hidden, __nv_bfloat16* planes, cudaStream_t stream) {
  if (experts <= 0 || hidden <= 0) return cudaErrorInvalidValue;
  fold_gate_kernel<<<stride_blocks(static_cast<size_t>(experts) * hidden, 256), 256, 0, stream>>>(gate, norm_weight, experts, hidden, planes);
  return cudaGetLastError();
}

// As many CTAs per row tile as keep every CTA on an SM of its own, each with two K blocks at
// least: the chain of K blocks is what a CTA takes its time for (FP32 input, 256 rows: 78 us on
// two CTAs, 14 us on 42).
int router_pass1_splits(int rows, int hidden, int num_sms) {
  const int tiles = (rows + 127) / 128;
  const int most = std::max(1, hidden / kFastBlockK / 2);
  return std::min(std::max(1, num_sms / tiles), std::min(most, kMaxPass1Splits));
}

cudaError_t launch_router_folded_logits(const CUtensorMap& tmap_x, const CUtensorMap& tmap_planes,
                                        const float* inv_rms, int rows, int experts, int hidden,
                                        int splits, float* logits, int32_t* error,
                                        cudaStream_t stream) {
  if (rows <= 0 || experts % 16 != 0 || experts > 256 || hidden % kFastBlockK != 0 ||
      splits < 1 || hidden / kFastBlockK < splits) {
    return cudaErrorInvalidValue;
  }
  const int stage_bytes = kFoldABytes + 3 * experts * 128;
  const int stages = pass1_stages(4, stage_bytes);  // two at 256 experts
  const int smem = pass1_smem_bytes(stages, stage_bytes);
  cudaError_t err = allow_shared_memory(router_folded_logits_kernel);
  if (err != cudaSuccess) return err;
  router_folded_logits_kernel<<<(rows + 127) / 128 * splits, kFoldThreads, smem, stream>>>(
      tmap_x, tmap_planes, inv_rms, rows, experts, hidden, stages, splits, logits, error);
  return cudaGetLastError();
}

cudaError_t launch_router_select_exact(float* logits, int splits, const void* x, bool x_bf16,
                                       const float* inv_rms, const float* norm_weight,
                                       const __nv_bfloat16* gate, const float* logit_offset,
                                       const float* bias, int rows, int experts, int hidden,
                                       int top_k, bool norm_topk_prob, float routed_scaling,
                                       float tie_margin, int32_t* top_index, float* top_weight,
                                       int32_t* expert_counts, int32_t* position, cudaStream_t stream) {
  if (rows <= 0 || experts % 32 != 0 || experts > 32 * kSelectMaxPerLane || top_k <= 0 ||
      top_k > 32 || top_k > experts || hidden % 8 != 0 || splits < 1) {
    return cudaErrorInvalidValue;
  }
  const bool whole_block = rows <= select_whole_block_rows(experts, hidden);
  const int grid = whole_block ? rows : (rows + kSelectWarps - 1) / kSelectWarps;
  auto run = [&](auto kernel) {
    kernel<<<grid, kSelectWarps * 32, 0, stream>>>(
        logits, splits, x, inv_rms, norm_weight, gate, logit_offset, bias, rows, experts, hidden,
        top_k, norm_topk_prob, routed_scaling, tie_margin, top_index, top_weight, expert_counts,
        position);
  };
  auto run_lanes = [&](auto bf16, auto warps, auto batch) {
    constexpr bool kBf16 = decltype(bf16)::value;
    constexpr int kWarps = decltype(warps)::value, kBatch = decltype(batch)::value;
    if (experts <= 128) {
      run(router_select_exact_kernel<kBf16, kWarps, kBatch, 4>);
    } else {
      run(router_select_exact_kernel<kBf16, kWarps, kBatch, kSelectMaxPerLane>);
    }
  };
  auto run_batch = [&](auto bf16, auto warps) {
    if (top_k <= 4) {
      run_lanes(bf16, warps, std::integral_constant<int, 4>());
    } else if (top_k <= 6) {
      run_lanes(bf16, warps, std::integral_constant<int, 6>());
    } else {
      run_lanes(bf16, warps, std::integral_constant<int, 8>());
    }
  };
  using One = std::integral_constant<int, 1>;
  using Block = std::integral_constant<int, kSelectWarps>;
  if (x_bf16) {
    if (whole_block) run_batch(std::true_type(), Block()); else run_batch(std::true_type(), One());
  } else {
    if (whole_block) run_batch(std::false_type(), Block()); else run_batch(std::false_type(), One());
  }
  return cudaGetLastError();
}

}  // namespace nmoe
