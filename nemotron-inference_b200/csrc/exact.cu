// Correctly rounded linears on the tensor cores: y = x W^T with the sum the reference
// accumulates in double (UploadedLinearOp, runtime/src/backend/linear_op.cpp:97-118, and
// ScaledFp8LinearOp, runtime/src/backend/scaled_fp8_linear.cu:222-283) and rounds to FP32 once.
//
// FP64 arithmetic runs at 1/70 of the int8 tensor rate here, and widening FP32 operands for it
// is slower still (15 conversions per clock and SM), so a matrix of any size is done in integers:
//   * every row of x and of W is written once as fixed point below its own largest magnitude,
//     39 bits in five signed base-256 digits ("slices", after Ootomo, Ozaki and Yokota's use of
//     integer matrix units for FP64 products);
//   * tcgen05.mma.kind::i8 multiplies the slices and accumulates exactly in 32-bit integers:
//     digit i of W times digit j of x belongs to level i + j, the 22 products of levels 0..6 are
//     computed, the rest and the bits below the fixed point are bounded;
//   * the seven levels are put together in double, r, with a bound B on everything left out.  When
//     r - B and r + B round to the same FP32 number that number is the result (Ziv's test);
//     otherwise -- one value in tens of thousands -- the sum is formed in FP64 from the operands.
//     (Without level 6 one in a thousand stays open, and those take longer than level 6 does.)
// One token row or a handful is bound by reading W instead: exact_gemv_kernel reads W in the
// form it came in (FP8, bf16 or FP32) and sums in FP64.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "quant_row.cuh"
#include "weights.cuh"

namespace nmoe {
namespace {

constexpr int kSlices = 5;
constexpr int kLevels = 7;
constexpr int kFixedBits = 38;       // |x| < 2^e is stored as round(x * 2^(38 - e)); the top digit
                                     // then stays below 65 with the carries of the others
constexpr int kNoExponent = 1 << 20; // a row that holds an infinity or NaN

// Weight values as the reference multiplies with them: FP32, widened bf16, or
// DecodeFp8(byte) * weight_scale.
template <int KIND>
__device__ __forceinline__ float weight_value(const void* w, size_t i, float scale) {
  if constexpr (KIND == kWeightFp8) {
    return __fmul_rn(decode_e4m3(reinterpret_cast<const uint8_t*>(w)[i]), scale);
  } else if constexpr (KIND == kWeightBf16) {
    return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[i]);
  } else {
    return reinterpret_cast<const float*>(w)[i];
  }
}

// Exponent e with |v| < 2^e for every v of magnitude up to `amax`.
__device__ __forceinline__ int exponent_above(float amax) {
  if (!(amax < INFINITY)) return kNoExponent;  // infinity or NaN
  const int biased = static_cast<int>(__float_as_uint(amax) >> 23);
  return (biased == 0 ? 1 : biased) - 126;
}

// Five digits of v below 2^e, the most significant first; returns whether they hold v exactly.
__device__ __forceinline__ bool digits_of(float v, int e, int8_t (&d)[kSlices]) {
  const uint32_t bits = __float_as_uint(v);
  const int biased = static_cast<int>((bits >> 23) & 0xffu);
  const uint32_t mantissa = (bits & 0x7fffffu) | (biased != 0 ? 0x800000u : 0u);
  // v = mantissa * 2^(max(biased, 1) - 150)
  const int shift = (biased == 0 ? 1 : biased) - 150 + kFixedBits - e;
  long long m = 0;
  bool exact = true;
  if (shift >= 0) {
    m = static_cast<long long>(mantissa) << min(shift, 62 - 24);
  } else if (shift > -25) {
    m = (static_cast<long long>(mantissa) + (1ll << (-shift - 1))) >> -shift;
    exact = (mantissa & ((1u << -shift) - 1u)) == 0u;
  } else {
    exact = mantissa == 0u;
  }
  if (bits >> 31) m = -m;
#pragma unroll
  for (int i = kSlices - 1; i >= 0; --i) {
    d[i] = static_cast<int8_t>(m & 0xff);
    m = (m - d[i]) >> 8;
  }
  return exact;
}

constexpr int kExactRows = 128;  // weight rows per tile
constexpr int kExactChunk = 64;  // bytes of K per pipeline stage (64-byte swizzle)

// Where the 8 bytes of row `row`, slice `slice`, columns k .. k + 7 go.  A tile of `tile_rows` rows
// keeps every 64-byte chunk of K as one contiguous piece, [slice][row][64], already in the shared-
// memory image of the tensor core's 64-byte swizzle, so that a stage is one bulk copy.
template <int SLICES>
__device__ __forceinline__ size_t slice_offset(size_t row, int slice, int k, int K,
                                               int tile_rows) {
  const size_t tile = row / tile_rows;
  const int r = static_cast<int>(row - tile * tile_rows);
  const size_t chunk = tile * (K / kExactChunk) + k / kExactChunk;
  const int c = k & (kExactChunk - 1);
  return (chunk * SLICES + slice) * (static_cast<size_t>(tile_rows) * kExactChunk) +
         r * kExactChunk + ((((c >> 4) ^ (r >> 1)) & 3) << 4) + (c & 15);
}

constexpr int kSliceThreads = 256;

// One block per row, the row in registers (STEPS times eight consecutive values per thread): its
// largest magnitude, then the digits.  KIND < 0: FP32 activation rows, with `sums` each the sum of top_k
// rows of `in`, which is written there.
template <int KIND, int STEPS>
__global__ void __launch_bounds__(kSliceThreads)
slice_rows_kernel(const void* __restrict__ in, int K, float scale, int tile_rows,
                  int8_t* __restrict__ slices, SliceRow* __restrict__ info, int top_k,
                  float* __restrict__ sums) {
  __shared__ float warp_max[kSliceThreads / 32];
  const size_t row = blockIdx.x;
  float v[STEPS][8];
  float amax = 0.0f;
  bool bad = false;
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
    const int k = (s * kSliceThreads + static_cast<int>(threadIdx.x)) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[s][j] = 0.0f;
    if (k < K) {
      if constexpr (KIND < 0) {
        const float* first = reinterpret_cast<const float*>(in) + row * top_k * K + k;
        float raw[8];
        load8<false>(first, 0, raw);
        if (sums != nullptr) {
          // the row is a sum of parts in selection order (expert_layer.cpp:951-953)
#pragma unroll 4
          for (int p = 1; p < top_k; ++p) {
            float part[8];
            load8<false>(first, static_cast<size_t>(p) * K, part);
#pragma unroll
            for (int j = 0; j < 8; ++j) raw[j] = __fadd_rn(raw[j], part[j]);
          }
          float4* to = reinterpret_cast<float4*>(sums + row * K + k);
          to[0] = make_float4(raw[0], raw[1], raw[2], raw[3]);
          to[1] = make_float4(raw[4], raw[5], raw[6], raw[7]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) v[s][j] = input_value(raw[j], scale);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[s][j] = weight_value<KIND < 0 ? 0 : KIND>(in, row * K + k + j, scale);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float magnitude = fabsf(v[s][j]);
      bad = bad || !(magnitude < INFINITY);
      amax = fmaxf(amax, magnitude);
    }
  }
  if (bad) amax = INFINITY;
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, stride));
  }
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = amax;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kSliceThreads / 32; ++w) amax = fmaxf(amax, warp_max[w]);
  const int e = exponent_above(amax);
  int inexact = 0;
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
    const int k = (s * kSliceThreads + static_cast<int>(threadIdx.x)) * 8;
    if (k >= K) continue;
    uint32_t words[kSlices][2] = {};
    if (e != kNoExponent) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        int8_t d[kSlices];
        if (!digits_of(v[s][j], e, d)) ++inexact;
#pragma unroll
        for (int i = 0; i < kSlices; ++i) {
          words[i][j >> 2] |= static_cast<uint32_t>(static_cast<uint8_t>(d[i])) << (8 * (j & 3));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kSlices; ++i) {
      *reinterpret_cast<uint2*>(slices + slice_offset<kSlices>(row, i, k, K, tile_rows)) =
          make_uint2(words[i][0], words[i][1]);
    }
  }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    inexact += __shfl_xor_sync(0xffffffffu, inexact, stride);
  }
  __shared__ int warp_inexact[kSliceThreads / 32];
  if ((threadIdx.x & 31) == 0) warp_inexact[threadIdx.x >> 5] = inexact;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
    for (int w = 0; w < kSliceThreads / 32; ++w) total += warp_inexact[w];
    info[row] = SliceRow{e, total};
  }
}

template <int KIND>
void launch_slices(const void* in, int rows, int K, float scale, int tile_rows, int8_t* slices,
                   SliceRow* info, cudaStream_t stream, int top_k = 1, float* sums = nullptr) {
  auto run = [&](auto kernel) {
    kernel<<<rows, kSliceThreads, 0, stream>>>(in, K, scale, tile_rows, slices, info, top_k, sums);
  };
  if (K <= 2 * kSliceThreads * 8) {
    run(slice_rows_kernel<KIND, 2>);
  } else if (K <= 4 * kSliceThreads * 8) {
    run(slice_rows_kernel<KIND, 4>);
  } else {
    run(slice_rows_kernel<KIND, 8>);
  }
}

// ---------------------------------------------------------------------------
// the integer product: 128 weight rows x `nt` token rows per CTA
//
// A = the weight slices (M = 128), B = the token slices.  For weight digit i the token digits that
// meet it are the rows of one B tile, and level s of the sum lies at TMEM column s * nt, so one
// MMA of up to 256 columns multiplies digit i with several token digits and adds each product to
// the level it belongs to; A is read once for all of them.  A CTA takes one tile, or a share of
// its K range, and stores the levels put together as doubles.
// Bound by the MMAs (five digits of a weight of the checkpoint's shared_up's shape, 5376 x 4096, 1000 rows,
// under ncu: a stage takes 1740 cycles, 1420 of them on the tensor pipe, and its 672 tiles are 4.54 waves of
// 148 SMs; shared memory is at 32 % of its read and 13 % of its write rate).  With the two kernels around
// it 13,800 -> 370 us; 40 rows 381 -> 44 us.  (shared_up itself takes three digits where its rows are only
// quantised again, further down.)
// ---------------------------------------------------------------------------
constexpr int kExactThreads = 6 * 32;
// A product of matrices of SLICES digits: five of rows in fixed point (above), or the three of E4M3
// codes as whole numbers (below), whose nine products are all computed.
template <int SLICES>
struct ExactShape {
  static constexpr int kLevels = SLICES == kSlices ? nmoe::kLevels : 2 * SLICES - 1;
  static constexpr int kStages = SLICES == kSlices ? 3 : 5;
  static constexpr int kABytes = SLICES * kExactRows * kExactChunk;
  static constexpr int smem_bytes(int nt) {
    return kStages * (kABytes + SLICES * nt * kExactChunk) + (2 * kStages + 1) * 8 + 16 + 1024;
  }
};

__device__ __forceinline__ void tcgen05_mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// kind::i8 instruction descriptor: S32 accumulate, S8 x S8, K-major, M = 128
__device__ __forceinline__ uint32_t make_idesc_i8(uint32_t n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// The products of one 32-byte step of K: digit I of W times its token digits, from the given shared-
// memory descriptors.  A level that digit I is the first to reach is an MMA of its own, so that it
// can start the sum when `first`.
template <int SLICES, int NT, int I>
__device__ __forceinline__ void issue_digit(uint32_t tmem, uint64_t a_desc, uint64_t b_desc,
                                            bool first) {
  constexpr int kLevels = ExactShape<SLICES>::kLevels;
  constexpr int kMost = 256 / NT;                                      // token digits of one MMA
  constexpr int kMeet = SLICES < kLevels - I ? SLICES : kLevels - I;  // ... within the levels
  constexpr bool kStarts = I > 0 && I <= kLevels - SLICES;
  constexpr int kTogether = kStarts ? kMeet - 1 : kMeet;
  const uint64_t a = advance_smem_desc(a_desc, I * kExactRows * kExactChunk);
#pragma unroll
  for (int j = 0; j < kTogether; j += kMost) {
    constexpr int kFull = kMost < kTogether ? kMost : kTogether;
    const int count = kTogether - j < kFull ? kTogether - j : kFull;
    tcgen05_mma_i8(tmem + (I + j) * NT, a, advance_smem_desc(b_desc, j * NT * kExactChunk),
                   make_idesc_i8(static_cast<uint32_t>(count * NT)), I == 0 && first ? 0u : 1u);
  }
  if constexpr (kStarts) {
    tcgen05_mma_i8(tmem + (I + kMeet - 1) * NT, a,
                   advance_smem_desc(b_desc, (kMeet - 1) * NT * kExactChunk),
                   make_idesc_i8(static_cast<uint32_t>(NT)), first ? 0u : 1u);
  }
}

// `values` (only without splits): FP32 results, the sums times `scale`, in the place of `partial`.
template <int SLICES, int NT>
__global__ void __launch_bounds__(kExactThreads, 1)
exact_gemm_kernel(const int8_t* __restrict__ w_slices, const int8_t* __restrict__ x_slices,
                  int rows, int N, int K, int row_tiles, int splits, double* __restrict__ partial,
                  float* __restrict__ values, double scale, int32_t* error) {
  using Shape = ExactShape<SLICES>;
  constexpr int kLevels = Shape::kLevels, kStages = Shape::kStages, kABytes = Shape::kABytes;
  constexpr int nt = NT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) &
                                             ~static_cast<uintptr_t>(1023u));
  constexpr int b_bytes = SLICES * nt * kExactChunk;
  uint8_t* sA = smem;
  uint8_t* sB = sA + kStages * kABytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sB + kStages * b_bytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* done_bar = empty_bar + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);

  const int warp = warp_uniform(static_cast<int>(threadIdx.x >> 5));
  const int lane = threadIdx.x & 31;
  // consecutive CTAs share a weight tile
  int index = static_cast<int>(blockIdx.x);
  const int split = index % splits;
  index /= splits;
  const int row_tile = index % row_tiles;
  const int n0 = index / row_tiles * kExactRows;
  const int row0 = row_tile * nt;
  const int all_chunks = K / kExactChunk;
  const int chunk0 = all_chunks * split / splits;
  const int chunks = all_chunks * (split + 1) / splits - chunk0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);

  const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
  const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);

  if (warp == 0) {
    const int8_t* w_from =
        w_slices + (static_cast<size_t>(n0 / kExactRows) * all_chunks + chunk0) * kABytes;
    const int8_t* x_from =
        x_slices + (static_cast<size_t>(row_tile) * all_chunks + chunk0) * b_bytes;
    int stage = 0;
    uint32_t phase = 0;
    for (int c = 0; c < chunks; ++c) {
      if (!mbar_wait_warp(empty0 + stage * 8, phase ^ 1u)) {
        if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
        break;
      }
      if (elect_one()) {
        const uint32_t bar = full0 + stage * 8;
        mbar_arrive_expect_tx_at(bar, kABytes + b_bytes);
        bulk_load_at(a0 + stage * kABytes, w_from, kABytes, bar);
        bulk_load_at(b0 + stage * b_bytes, x_from, b_bytes, bar);
      }
      w_from += kABytes;
      x_from += b_bytes;
      if (++stage == kStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    const uint64_t a_desc0 = make_smem_desc(a0, 0, 512, 4);
    const uint64_t b_desc0 = make_smem_desc(b0, 0, 512, 4);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int c = 0; c < chunks; ++c) {
      if (!mbar_wait_warp(full0 + stage * 8, phase)) {
        if (error != nullptr) atomicCAS(error, kDevOk, kDevWaitTimeout);
        ok = false;
        break;
      }
      tcgen05_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < kExactChunk / 32; ++ks) {
          const uint64_t a_desc = advance_smem_desc(a_desc0, stage * kABytes + ks * 32);
          const uint64_t b_desc = advance_smem_desc(b_desc0, stage * b_bytes + ks * 32);
          const bool first = ks == 0 && c == 0;
          static_assert(SLICES == 5 || SLICES == 3, "one call per digit");
          issue_digit<SLICES, NT, 0>(tmem_base, a_desc, b_desc, first);
          issue_digit<SLICES, NT, 1>(tmem_base, a_desc, b_desc, first);
          issue_digit<SLICES, NT, 2>(tmem_base, a_desc, b_desc, first);
          if constexpr (SLICES == 5) {
            issue_digit<SLICES, NT, 3>(tmem_base, a_desc, b_desc, first);
            issue_digit<SLICES, NT, 4>(tmem_base, a_desc, b_desc, first);
          }
        }
        tcgen05_commit_at(empty0 + stage * 8);
      }
      if (++stage == kStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (ok && elect_one()) tcgen05_commit(done_bar);
  } else {
    // epilogue: warp w owns TMEM lane quarter w % 4; a thread owns a weight row
    const int quarter = warp & 3;
    const int n = n0 + quarter * 32 + lane;
    if (mbar_wait(done_bar, 0)) {
      tcgen05_fence_after();
      const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      double* out = partial + static_cast<size_t>(split) * rows * N;
      const bool as_values = values != nullptr;
      for (int c = 0; c < nt && row0 + c < rows; c += 16) {
        double sum[16];
#pragma unroll
        for (int s = 0; s < kLevels; ++s) {
          float raw[16];
          tmem_ld_x16(t_addr + s * nt + c, raw);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const double level = static_cast<double>(__float_as_int(raw[i]));
            sum[i] = s == 0 ? level : fma(sum[i], 256.0, level);
          }
        }
        if (n < N) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (row0 + c + i >= rows) break;
            const size_t at = static_cast<size_t>(row0 + c + i) * N + n;
            if (as_values) {
              values[at] = static_cast<float>(sum[i] * scale);
            } else {
              out[at] = sum[i];
            }
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
    tmem_dealloc(tmem_base, 512);
  }
}

__device__ __forceinline__ double two_to(int e) {
  return e < -1022 ? 0.0 : __hiloint2double((min(e, 1023) + 1023) << 20, 0);
}

constexpr int kFinishThreads = 256;

// FP32 results from the doubles of exact_gemm_kernel, VALUES per thread.
//
// B, in units of 2^(ea + ew): K * 2^-52 for the digit products of level 7 and beyond (two pairs of
// digits up to 128 at level 7, one at level 8: K * 2^-53 * 1.01); 2^-39 for every value of the two
// rows that its digits do not hold exactly; and |r| * 2^-50 for the roundings of the doubles (three
// of 2^-53: a sum of fewer than five levels is below 2^53).  The parts of a split sum may cancel, so
// there it is their magnitudes that count, for those three and for every addition of a part.
template <int KIND, int VALUES>
__global__ void __launch_bounds__(kFinishThreads)
exact_finish_kernel(const double* __restrict__ partial, int splits, int rows, int N, int K,
                    const float* __restrict__ in, float fp8_scale,
                    const SliceRow* __restrict__ in_info, const void* __restrict__ weight,
                    float weight_scale, const SliceRow* __restrict__ weight_info,
                    const float* __restrict__ offset, bool relu2, float* __restrict__ out,
                    const ExactMix mix) {
  constexpr int V = WeightVector<KIND>::kCount;
  __shared__ int open_count;
  __shared__ int open_list[kFinishThreads * VALUES];
  __shared__ double warp_sum[kFinishThreads / 32];
  if (threadIdx.x == 0) open_count = 0;
  __syncthreads();
  const int t = blockIdx.y;
  const int first_n = blockIdx.x * (kFinishThreads * VALUES) + threadIdx.x;
  const size_t first = static_cast<size_t>(t) * N + first_n;
  const size_t count = static_cast<size_t>(rows) * N;
  const SliceRow a = in_info[t];
  // (the loads of all values are on their way before the first of them is looked at)
  double r[VALUES];
  SliceRow w[VALUES];
  float x[VALUES], shared[VALUES];
#pragma unroll
  for (int v = 0; v < VALUES; ++v) {
    const size_t i = first + v * kFinishThreads;
    r[v] = 0.0;
    w[v] = SliceRow{0, 0};
    x[v] = shared[v] = 0.0f;
    if (first_n + v * kFinishThreads >= N) continue;
    r[v] = partial[i];
    w[v] = weight_info[first_n + v * kFinishThreads];
    if (mix.out != nullptr) {
      x[v] = mix.in_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(mix.in)[i])
                         : reinterpret_cast<const float*>(mix.in)[i];
      shared[v] = mix.shared[i];
    }
  }
  float result[VALUES];
#pragma unroll
  for (int v = 0; v < VALUES; ++v) {
    const size_t i = first + v * kFinishThreads;
    const int n = first_n + v * kFinishThreads;
    result[v] = 0.0f;
    if (n >= N) continue;
    double sum = r[v];
#pragma unroll 4
    for (int s = 1; s < splits; ++s) sum += partial[i + s * count];
    bool decided = a.exponent != kNoExponent && w[v].exponent != kNoExponent;
    if (decided) {
      const int e = a.exponent + w[v].exponent;
      sum *= two_to(e - (12 + 8 * (kLevels - 1)));
      const double left_out = K + 8192.0 * (a.inexact + w[v].inexact);
      double bound = left_out * two_to(e - 52) + fabs(sum) * 0x1p-50;
      if (splits > 1) {
        double magnitude = 0.0;
        for (int s = 0; s < splits; ++s) magnitude += fabs(partial[i + s * count]);
        bound += magnitude * two_to(e - (12 + 8 * (kLevels - 1)) - 53) * (splits + 7);
      }
      const float low = static_cast<float>(sum - bound), high = static_cast<float>(sum + bound);
      decided = low == high;
      result[v] = static_cast<float>(sum);
    }
    if (!decided) open_list[atomicAdd(&open_count, 1)] = n;
  }
  __syncthreads();
  // the block forms the FP64 sum of one undecided value at a time, each thread a part of it
  for (int o = 0; o < open_count; ++o) {
    const float* row = in + static_cast<size_t>(t) * K;
    const uint4* weights =
        reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(weight) +
                                       static_cast<size_t>(open_list[o]) * K * (16 / V));
    double sum = 0.0;
    for (int q = threadIdx.x; q * V < K; q += kFinishThreads) {
      float values[V];
      WeightVector<KIND>::unpack(weights[q], weight_scale, values);
#pragma unroll
      for (int j = 0; j < V; j += 4) {
        const float4 four = *reinterpret_cast<const float4*>(row + q * V + j);
        const float av[4] = {four.x, four.y, four.z, four.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          sum = fma(static_cast<double>(input_value(av[h], fp8_scale)),
                    static_cast<double>(values[j + h]), sum);
        }
      }
    }
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, stride);
    }
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = sum;
    __syncthreads();
#pragma unroll
    for (int v = 0; v < VALUES; ++v) {
      if (first_n + v * kFinishThreads != open_list[o]) continue;
      double total = 0.0;
#pragma unroll
      for (int w8 = 0; w8 < kFinishThreads / 32; ++w8) total += warp_sum[w8];
      result[v] = static_cast<float>(total);
    }
    __syncthreads();
  }
#pragma unroll
  for (int v = 0; v < VALUES; ++v) {
    const int n = first_n + v * kFinishThreads;
    if (n >= N) continue;
    const size_t i = first + v * kFinishThreads;
    float y = result[v];
    if (offset != nullptr) y = __fadd_rn(y, offset[n]);
    if (relu2) y = y > 0.0f ? __fmul_rn(y, y) : 0.0f;
    out[i] = y;
    if (mix.out != nullptr) {
      const float mixed = __fadd_rn(x[v], __fadd_rn(y, shared[v]));
      if (mix.out_bf16) {
        reinterpret_cast<__nv_bfloat16*>(mix.out)[i] = __float2bfloat16_rn(mixed);
      } else {
        reinterpret_cast<float*>(mix.out)[i] = mixed;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// E4M3 times E4M3 that only has to be quantised again
//
// The scaled-FP8 family rounds its activations to E4M3 as well, so both operands are codes times a
// scale.  A code is a whole number of 2^-9 below 2^18, three digits, and the nine products of two give
// the sum of the codes' products, S, as a whole number.  The reference multiplies FP32 values,
// RN(code * scale), which is S times the scales to within 2^-23 of the sum of the magnitudes: too far to
// say the FP32 result, but a relu^2 row that is quantised to FP4 next needs only the side of a rounding
// boundary.  So every block is quantised twice, from both ends of what its values can be, by the steps
// that are monotone in them; where the two disagree (one block in a thousand) the values in doubt are
// summed in FP64 like those that exact_finish_kernel leaves open.  Codes and scales are therefore those
// of the correctly rounded sums.
// The checkpoint's shared_up, 1000 rows (ncu, us): digits of the rows 17 -> 12, product 323 -> 146 (bound
// by what an SM takes in, 39 KB in the 720 cycles that a stage's MMAs take), rounding and quantising
// 43 + 10 -> 36.  Whole pass with the linears beside it, 1000 rows 962 -> 795 us, 40 rows 356 -> 343.
// ---------------------------------------------------------------------------
constexpr int kCodeSlices = 3;
constexpr int kCodeTile = 80;  // token rows: five levels of 80 columns in TMEM, N = 240 in one MMA

__device__ __forceinline__ int code_integer(uint32_t code) {
  const int e = (code >> 3) & 15, m = code & 7;
  const int magnitude = e == 0 ? m : (8 + m) << (e - 1);
  return code & 0x80u ? -magnitude : magnitude;
}

// One block per row: its codes, the codes as three digits, and an upper bound of their 2-norm (an infinity
// where a code is no number).  WEIGHT: the row is E4M3 codes already.
template <bool WEIGHT>
__global__ void __launch_bounds__(kSliceThreads)
code_rows_kernel(const void* __restrict__ in, int K, float scale, int tile_rows,
                 int8_t* __restrict__ slices, uint8_t* __restrict__ codes_out,
                 float* __restrict__ norm) {
  __shared__ float warp_sum[kSliceThreads / 32];
  const size_t row = blockIdx.x;
  float squares = 0.0f;
  for (int k = static_cast<int>(threadIdx.x) * 8; k < K; k += kSliceThreads * 8) {
    uint32_t codes[8];
    if constexpr (WEIGHT) {
      const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(in) +
                                                        row * K + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) codes[j] = ((j < 4 ? raw.x : raw.y) >> (8 * (j & 3))) & 0xffu;
    } else {
      const float4* from =
          reinterpret_cast<const float4*>(reinterpret_cast<const float*>(in) + row * K + k);
      const float4 a = from[0], b = from[1];
      const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) codes[j] = encode_e4m3(__fdiv_rn(v[j], scale)) & 0xffu;
      *reinterpret_cast<uint2*>(codes_out + row * K + k) =
          make_uint2(codes[0] | codes[1] << 8 | codes[2] << 16 | codes[3] << 24,
                     codes[4] | codes[5] << 8 | codes[6] << 16 | codes[7] << 24);
    }
    uint32_t words[kCodeSlices][2] = {};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const bool number = (codes[j] & 0x7fu) != 0x7fu;
      int m = number ? code_integer(codes[j]) : 0;
      squares = number ? fmaf(static_cast<float>(m), static_cast<float>(m), squares) : INFINITY;
#pragma unroll
      for (int i = kCodeSlices - 1; i >= 0; --i) {
        const int8_t d = static_cast<int8_t>(m & 0xff);
        m = (m - d) >> 8;
        words[i][j >> 2] |= static_cast<uint32_t>(static_cast<uint8_t>(d)) << (8 * (j & 3));
      }
    }
#pragma unroll
    for (int i = 0; i < kCodeSlices; ++i) {
      *reinterpret_cast<uint2*>(slices + slice_offset<kCodeSlices>(row, i, k, K, tile_rows)) =
          make_uint2(words[i][0], words[i][1]);
    }
  }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    squares += __shfl_xor_sync(0xffffffffu, squares, stride);
  }
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = squares;
  __syncthreads();
  if (threadIdx.x == 0) {
    float total = 0.0f;
    for (int w = 0; w < kSliceThreads / 32; ++w) total += warp_sum[w];
    // (K <= 16384 additions lose less than 2^-10 of the sum)
    norm[row] = sqrtf(total) * 1.002f;
  }
}

// FP64 sum of one value by a warp, from the codes of both rows.
__device__ __forceinline__ float exact_value(const uint8_t* x, float fp8_scale, const uint8_t* w,
                                             float weight_scale, int K) {
  using Vector = WeightVector<kWeightFp8>;
  double sum = 0.0;
#pragma unroll 2
  for (int q = threadIdx.x & 31; q * Vector::kCount < K; q += 32) {
    float a[Vector::kCount], v[Vector::kCount];
    Vector::unpack(reinterpret_cast<const uint4*>(x)[q], fp8_scale, a);
    Vector::unpack(reinterpret_cast<const uint4*>(w)[q], weight_scale, v);
#pragma unroll
    for (int j = 0; j < Vector::kCount; ++j) {
      sum = fma(static_cast<double>(a[j]), static_cast<double>(v[j]), sum);
    }
  }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, stride);
  }
  return static_cast<float>(sum);
}

__device__ __forceinline__ float relu_squared(float r) { return r > 0.0f ? __fmul_rn(r, r) : 0.0f; }

// Largest `v` of the block's threads (none is negative).
__device__ __forceinline__ float block_max_of(float v, float* warp_values) {
  const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) warp_values[threadIdx.x >> 5] = __uint_as_float(most);
  __syncthreads();
  float all = 0.0f;
  for (int w = 0; w < static_cast<int>(blockDim.x) / 32; ++w) all = fmaxf(all, warp_values[w]);
  return all;
}

// relu^2 and NVFP4 of a row (nvfp4_packing.cpp:119-153) from values known to within a bound; one block
// per row, one thread per 16-element block.  `values`, or the doubles of a split product.
__global__ void __launch_bounds__(1024)
coded_quant_kernel(const float* __restrict__ values,
                                   const double* __restrict__ partial, int splits, double scale,
                                   int rows, int N, int K, const uint8_t* __restrict__ in,
                                   float fp8_scale, const float* __restrict__ in_norm,
                                   const uint8_t* __restrict__ weight, float weight_scale,
                                   const float* __restrict__ weight_norm, int first_row,
                                   uint8_t* __restrict__ packed, uint8_t* __restrict__ sf_tiled,
                                   int k_tiles, float* __restrict__ tensor_scale) {
  constexpr int kListed = 256;  // values summed per round
  __shared__ float warp_values[32];
  __shared__ int list[kListed];
  __shared__ float sums[kListed];
  __shared__ int listed;
  const int row = blockIdx.x, n0 = static_cast<int>(threadIdx.x) * 16;
  const bool active = n0 < N;
  const size_t at = static_cast<size_t>(row) * N + n0;
  const uint8_t* x = in + static_cast<size_t>(row) * K;
  float low[16], high[16];
  {
    // 2^-23 of the magnitudes for the operands' roundings, 2^-24 each for those of the result and of
    // `values`; the factors make up for the roundings of the bounds
    const float unit = static_cast<float>(scale) * in_norm[row] * 1.2e-7f;
    float known_as[16], norms[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) known_as[i] = norms[i] = 0.0f;
    if (active) {
#pragma unroll
      for (int i = 0; i < 16; i += 8) load8<false>(weight_norm, n0 + i, eight_of(norms, i));
      if (values != nullptr) {
#pragma unroll
        for (int i = 0; i < 16; i += 8) load8<false>(values, at + i, eight_of(known_as, i));
      } else {
        double sums_of[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) sums_of[i] = 0.0;
        for (int p = 0; p < splits; ++p) {
          const double2* from =
              reinterpret_cast<const double2*>(partial + at + static_cast<size_t>(p) * rows * N);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const double2 two = from[i];
            sums_of[2 * i] += two.x;
            sums_of[2 * i + 1] += two.y;
          }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) known_as[i] = static_cast<float>(sums_of[i] * scale);
      }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float r = known_as[i];
      const float bound =
          active ? fmaf(fabsf(r), 1.2e-7f, fmaf(unit, norms[i], 1e-37f)) : 0.0f;
      // (a bound that is no number, or none: the value is summed)
      const bool known = bound < 1e30f;
      low[i] = known ? relu_squared(__fsub_rd(r, bound)) : 0.0f;
      high[i] = known ? relu_squared(__fadd_ru(r, bound)) : INFINITY;
    }
  }
  // Sums the values that the threads name in `which`, a warp each.
  auto settle = [&](uint32_t which) {
    while (__syncthreads_or(which != 0u)) {
      if (threadIdx.x == 0) listed = 0;
      __syncthreads();
      int first = kListed;
      bool fits = false;
      if (which != 0u) {
        first = atomicAdd(&listed, __popc(which));
        fits = first + __popc(which) <= kListed;
        int at = first;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (((which >> i) & 1u) != 0u && at < kListed) list[at++] = fits ? n0 + i : -1;
        }
      }
      __syncthreads();
      const int count = min(listed, kListed);
      for (int at = threadIdx.x >> 5; at < count; at += static_cast<int>(blockDim.x) / 32) {
        const int n = list[at];
        if (n < 0) continue;
        const float sum = exact_value(x, fp8_scale, weight + static_cast<size_t>(n) * K,
                                      weight_scale, K);
        if ((threadIdx.x & 31) == 0) sums[at] = relu_squared(sum);
      }
      __syncthreads();
      if (fits) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (((which >> i) & 1u) != 0u) low[i] = high[i] = sums[first++];
        }
        which = 0;
      }
    }
  };
  // those of this thread that are open and may be as large as `least`
  auto open_from = [&](float least) {
    uint32_t which = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) which |= (low[i] != high[i] && high[i] >= least ? 1u : 0u) << i;
    return which;
  };
  auto largest = [&](const float (&v)[16]) {
    float most = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) most = fmaxf(most, v[i]);
    return most;
  };
  // the row's tensor scale is 1 unless its largest value is beyond 6 * 448
  float ts = 1.0f;
  if (block_max_of(largest(high), warp_values) > kFp4Max * kFp8Max) {
    settle(open_from(block_max_of(largest(low), warp_values)));
    const float amax = block_max_of(largest(low), warp_values);
    if (amax > kFp4Max * kFp8Max) ts = clamp_scale(__fdiv_rn(amax, kFp4Max * kFp8Max));
  }
  const float scale_divisor = __fmul_rn(kFp4Max, ts), scale_reciprocal = __frcp_rn(scale_divisor);
  uint32_t in_doubt = 0;
  {
    const float low_scale = block_scale(largest(low), scale_divisor, scale_reciprocal);
    const float high_scale = block_scale(largest(high), scale_divisor, scale_reciprocal);
    const float low_divisor = __fmul_rn(ts, low_scale), high_divisor = __fmul_rn(ts, high_scale);
    const float low_reciprocal = __frcp_rn(low_divisor), high_reciprocal = __frcp_rn(high_divisor);
#pragma unroll
    for (int i = 0; i < 16; i += 8) {
      const uint32_t differ =
          quantize_half_block(eight_of(low, i), high_divisor, high_reciprocal) ^
          quantize_half_block(eight_of(high, i), low_divisor, low_reciprocal);
      if (differ != 0u) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          in_doubt |= (((differ >> (4 * j)) & 15u) != 0u ? 1u : 0u) << (i + j);
        }
      }
    }
    // what the scale follows from is settled with the values that hang on it
    if (encode_e4m3(low_scale) != encode_e4m3(high_scale)) in_doubt |= 0x10000u;
    if (in_doubt != 0u) in_doubt = (in_doubt & open_from(0.0f)) | open_from(largest(low));
  }
  settle(in_doubt);
  if (!active) return;
  const float bs = block_scale(largest(high), scale_divisor, scale_reciprocal);
  const float divisor = __fmul_rn(ts, bs), reciprocal = __frcp_rn(divisor);
  const size_t out_row = static_cast<size_t>(first_row) + row;
  *reinterpret_cast<uint2*>(packed + out_row * (N / 2) + n0 / 2) =
      make_uint2(quantize_half_block(eight_of(high, 0), divisor, reciprocal),
                 quantize_half_block(eight_of(high, 8), divisor, reciprocal));
  sf_tiled[swizzled_scale_offset(out_row, n0 / 16, k_tiles)] = static_cast<uint8_t>(encode_e4m3(bs));
  if (threadIdx.x == 0) tensor_scale[out_row] = ts;
}

// ---------------------------------------------------------------------------
// a few token rows: W in its own format, FP64 sums
// ---------------------------------------------------------------------------
constexpr int kGemvThreads = 256;
// xs[] of exact_gemv_kernel: 16 values and a gap, so that lanes reading their own 4, 8 or 16
// consecutive values meet no bank conflict.
__host__ __device__ constexpr int gemv_slot(int k) { return k + (k >> 4); }

// Weight rows n0 and n0 + 1 times ROWS token rows (`padded` doubles apart, in slots), by a warp: the sums
// in all its lanes.  A token value read from shared memory serves both weight rows.
template <int KIND, int ROWS>
__device__ __forceinline__ void dot_two_rows(const double* xs, int padded, const void* weight,
                                             float weight_scale, int n0, int N, int K,
                                             double (&acc)[ROWS][2]) {
  constexpr int V = WeightVector<KIND>::kCount;
  const size_t row_bytes = static_cast<size_t>(K) * (16 / V);
  const uint8_t* rows = reinterpret_cast<const uint8_t*>(weight);
  const uint4* w0 = reinterpret_cast<const uint4*>(rows + n0 * row_bytes);
  const uint4* w1 = reinterpret_cast<const uint4*>(rows + min(n0 + 1, N - 1) * row_bytes);
#pragma unroll
  for (int r = 0; r < ROWS; ++r) acc[r][0] = acc[r][1] = 0.0;
#pragma unroll 4
  for (int q = threadIdx.x & 31; q * V < K; q += 32) {
    float v0[V], v1[V];
    WeightVector<KIND>::unpack(w0[q], weight_scale, v0);
    WeightVector<KIND>::unpack(w1[q], weight_scale, v1);
    const double* x = xs + gemv_slot(q * V);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const double d0 = static_cast<double>(v0[j]), d1 = static_cast<double>(v1[j]);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const double a = x[r * padded + j];
        acc[r][0] = fma(a, d0, acc[r][0]);
        acc[r][1] = fma(a, d1, acc[r][1]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int stride = 16; stride > 0; stride >>= 1) {
        acc[r][h] += __shfl_xor_sync(0xffffffffu, acc[r][h], stride);
      }
    }
  }
}

// One warp per weight row at a time; the ROWS token rows wait in shared memory as doubles, so that
// they are widened once per block.  Bound by reading W at one row: shared_up of the checkpoint
// layer (22 MB of FP8) 37 -> 15 us.
template <int KIND, int ROWS>
__global__ void __launch_bounds__(kGemvThreads)
exact_gemv_kernel(const float* in, float fp8_scale, int N, int K,
                  const void* __restrict__ weight, float weight_scale,
                  const float* __restrict__ offset, bool relu2, float* __restrict__ out) {
  constexpr int V = WeightVector<KIND>::kCount;
  constexpr int kWarps = kGemvThreads / 32;
  extern __shared__ double xs[];
  const int lane = threadIdx.x & 31;
  const int padded = gemv_slot(K);
  release_successor();
  {
    // this warp's first two weight rows need not wait for the token rows
    const size_t row_bytes = static_cast<size_t>(K) * (16 / V);
    const int p = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (2 * p + 1 < N) {
      const uint8_t* first = reinterpret_cast<const uint8_t*>(weight) + 2 * p * row_bytes;
      for (size_t b = lane * 128; b < 2 * row_bytes; b += 32 * 128) prefetch_l2(first + b);
    }
  }
  wait_for_predecessor();
  // (the loads of four steps are issued before the stores of the first)
  for (int k0 = threadIdx.x; k0 < ROWS * K; k0 += 4 * kGemvThreads) {
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + i * kGemvThreads;
      if (k < ROWS * K) x[i] = in[k];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + i * kGemvThreads;
      const int r = k / K;
      if (k < ROWS * K) {
        xs[r * padded + gemv_slot(k - r * K)] = static_cast<double>(input_value(x[i], fp8_scale));
      }
    }
  }
  __syncthreads();
  const int pairs = (N + 1) / 2;
  for (int p = blockIdx.x * kWarps + (threadIdx.x >> 5); p < pairs; p += gridDim.x * kWarps) {
    const int n0 = 2 * p;
    double acc[ROWS][2];
    dot_two_rows<KIND, ROWS>(xs, padded, weight, weight_scale, n0, N, K, acc);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = n0 + h;
        if (lane == 0 && n < N) {
          float result = static_cast<float>(acc[r][h]);
          if (offset != nullptr) result = __fadd_rn(result, offset[n]);
          if (relu2) result = result > 0.0f ? __fmul_rn(result, result) : 0.0f;
          out[static_cast<size_t>(r) * N + n] = result;
        }
      }
    }
  }
}

// One block per weight row and ROWS token rows, for the short weights of a router's gate: every
// thread widens its own part of both.
template <int KIND, int ROWS>
__global__ void __launch_bounds__(kGemvThreads)
exact_gemv_block_kernel(const float* in, float fp8_scale, int rows, int N, int K,
                        const void* __restrict__ weight, float weight_scale,
                        const float* __restrict__ offset, bool relu2, float* __restrict__ out) {
  constexpr int V = WeightVector<KIND>::kCount;
  __shared__ double warp_sum[ROWS][kGemvThreads / 32];
  const int n = blockIdx.x;
  const int row0 = blockIdx.y * ROWS;
  const uint4* w = reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(weight) +
                                                  static_cast<size_t>(n) * K * (16 / V));
  double acc[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) acc[r] = 0.0;
  release_successor();
  if (row0 == 0) {
    // the weight row need not wait for the token rows
    for (int b = threadIdx.x * 128; b < K * (16 / V); b += kGemvThreads * 128) {
      prefetch_l2(reinterpret_cast<const uint8_t*>(w) + b);
    }
  }
  wait_for_predecessor();
#pragma unroll 2
  for (int q = threadIdx.x; q * V < K; q += kGemvThreads) {
    float v[V];
    WeightVector<KIND>::unpack(w[q], weight_scale, v);
    double d[V];
#pragma unroll
    for (int j = 0; j < V; ++j) d[j] = static_cast<double>(v[j]);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const float* x = in + static_cast<size_t>(min(row0 + r, rows - 1)) * K + q * V;
#pragma unroll
      for (int j = 0; j < V; j += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + j);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          acc[r] = fma(static_cast<double>(input_value(av[h], fp8_scale)), d[j + h], acc[r]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
#pragma unroll
    for (int stride = 16; stride > 0; stride >>= 1) {
      acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], stride);
    }
    if ((threadIdx.x & 31) == 0) warp_sum[r][threadIdx.x >> 5] = acc[r];
  }
  __syncthreads();
  const int r = threadIdx.x;
  if (r < ROWS && row0 + r < rows) {
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < kGemvThreads / 32; ++i) v += warp_sum[r][i];
    float result = static_cast<float>(v);
    if (offset != nullptr) result = __fadd_rn(result, offset[n]);
    if (relu2) result = result > 0.0f ? __fmul_rn(result, result) : 0.0f;
    out[static_cast<size_t>(row0 + r) * N + n] = result;
  }
}

// The end of a latent layer over one token in one launch: the routed sum in selection order
// (expert_layer.cpp:951-953), fc2_latent (:1047-1053), mixer and residual (:1064-1069).  Every block adds
// up the parts for itself, 32 outputs at a time, which keeps 4096 of them to one block an SM.
constexpr int kTailOutputs = 32;
template <int KIND>
__global__ void __launch_bounds__(kGemvThreads)
latent_tail_kernel(const LatentTail tail, int N, int K, const void* __restrict__ weight,
                   float weight_scale) {
  constexpr int V = WeightVector<KIND>::kCount;
  constexpr int kBatch = 8;  // loads of a part in flight
  extern __shared__ double xs[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int block_n = blockIdx.x * kTailOutputs;
  const size_t row_bytes = static_cast<size_t>(K) * (16 / V);
  release_successor();
  {
    // the weights need not wait for the experts
    const size_t bytes = min(kTailOutputs, N - block_n) * row_bytes;
    const uint8_t* first = reinterpret_cast<const uint8_t*>(weight) + block_n * row_bytes;
    for (size_t b = threadIdx.x * 128; b < bytes; b += kGemvThreads * 128) prefetch_l2(first + b);
  }
  wait_for_predecessor();
  for (int c = static_cast<int>(threadIdx.x) * 4; c < K; c += kGemvThreads * 4) {
    const float* base = tail.parts + c;
    float4 acc = *reinterpret_cast<const float4*>(base);
    for (int k0 = 1; k0 < tail.top_k; k0 += kBatch) {
      float4 p[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (k0 + k < tail.top_k) {
          p[k] = *reinterpret_cast<const float4*>(base + static_cast<size_t>(k0 + k) * K);
        }
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (k0 + k < tail.top_k) {
          acc.x = __fadd_rn(acc.x, p[k].x);
          acc.y = __fadd_rn(acc.y, p[k].y);
          acc.z = __fadd_rn(acc.z, p[k].z);
          acc.w = __fadd_rn(acc.w, p[k].w);
        }
      }
    }
    double* to = xs + gemv_slot(c);  // (four from a multiple of four: no gap between)
    to[0] = acc.x;
    to[1] = acc.y;
    to[2] = acc.z;
    to[3] = acc.w;
    if (blockIdx.x == 0) *reinterpret_cast<float4*>(tail.routed + c) = acc;
  }
  __syncthreads();
  constexpr int kPerWarp = kTailOutputs / (kGemvThreads / 32);
#pragma unroll 1
  for (int p = 0; p < kPerWarp; p += 2) {
    const int n0 = block_n + warp * kPerWarp + p;
    if (n0 >= N) break;
    double acc[1][2];
    dot_two_rows<KIND, 1>(xs, 0, weight, weight_scale, n0, N, K, acc);
    const int n = n0 + lane;
    if (lane >= 2 || n >= N) continue;
    const float projected = static_cast<float>(lane == 0 ? acc[0][0] : acc[0][1]);
    tail.projected[n] = projected;
    const float x = tail.in_bf16
                        ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(tail.in)[n])
                        : reinterpret_cast<const float*>(tail.in)[n];
    const float mixed = __fadd_rn(x, __fadd_rn(projected, tail.shared[n]));
    if (tail.out_bf16) {
      reinterpret_cast<__nv_bfloat16*>(tail.out)[n] = __float2bfloat16_rn(mixed);
    } else {
      reinterpret_cast<float*>(tail.out)[n] = mixed;
    }
  }
}

// Four values of W, from element i (a multiple of four).
template <int KIND>
__device__ __forceinline__ void weight_quad(const void* w, size_t i, float scale, float (&v)[4]) {
  if constexpr (KIND == kWeightFp8) {
    const uint32_t raw = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(w) + i);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const __half2_raw two = __nv_cvt_fp8x2_to_halfraw2(
          static_cast<__nv_fp8x2_storage_t>(raw >> (16 * h)), __NV_E4M3);
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
      v[2 * h] = __fmul_rn(f.x, scale);
      v[2 * h + 1] = __fmul_rn(f.y, scale);
    }
  } else if constexpr (KIND == kWeightBf16) {
    const uint2 raw =
        *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(w) + i);
    v[0] = __uint_as_float(raw.x << 16);
    v[1] = __uint_as_float(raw.x & 0xffff0000u);
    v[2] = __uint_as_float(raw.y << 16);
    v[3] = __uint_as_float(raw.y & 0xffff0000u);
  } else {
    const float4 raw = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(w) + i);
    v[0] = raw.x; v[1] = raw.y; v[2] = raw.z; v[3] = raw.w;
  }
}

// 8 x 8 outputs per block for a short W and more than a handful of rows: a value of either operand
// is widened once for eight products, where exact_gemv_block_kernel widens five for four.  The
// threads share K; each holds all 64 sums in registers.  Bound by the conversions (16 per 64 FMAs,
// at 15 a clock and SM), the FP64 FMAs (52) and one round of loads per step: 256 threads while every
// block has an SM, else 128, two blocks to an SM.  Between events, a gate of 128 x 2688: 64 rows
// 20.2 -> 12.1 us; 128 rows 31 (by slices) -> 14.2 (18.3 with 256 threads), 255 rows 31 -> 24.4.
constexpr int kTileOutputs = 8;
template <int KIND, int THREADS>
__global__ void __launch_bounds__(THREADS)
exact_tile_kernel(const float* in, float fp8_scale, int rows, int N, int K,
                  const void* __restrict__ weight, float weight_scale,
                  const float* __restrict__ offset, bool relu2, float* __restrict__ out) {
  constexpr int M = kTileOutputs;
  __shared__ double warp_sum[THREADS / 32][M * M];
  const int n0 = blockIdx.x * M, row0 = blockIdx.y * M;
  const int lane = threadIdx.x & 31;
  release_successor();
  wait_for_predecessor();
  double acc[M * M];
#pragma unroll
  for (int i = 0; i < M * M; ++i) acc[i] = 0.0;
#pragma unroll 1
  for (int k = static_cast<int>(threadIdx.x) * 4; k < K; k += THREADS * 4) {
    float w[M][4], x[M][4];
#pragma unroll
    for (int i = 0; i < M; ++i) {
      weight_quad<KIND>(weight, static_cast<size_t>(min(n0 + i, N - 1)) * K + k, weight_scale, w[i]);
      const float4 a = *reinterpret_cast<const float4*>(
          in + static_cast<size_t>(min(row0 + i, rows - 1)) * K + k);
      x[i][0] = a.x; x[i][1] = a.y; x[i][2] = a.z; x[i][3] = a.w;
    }
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      double d[M];
#pragma unroll
      for (int i = 0; i < M; ++i) d[i] = static_cast<double>(w[i][h]);
#pragma unroll
      for (int r = 0; r < M; ++r) {
        const double a = static_cast<double>(input_value(x[r][h], fp8_scale));
#pragma unroll
        for (int i = 0; i < M; ++i) acc[r * M + i] = fma(a, d[i], acc[r * M + i]);
      }
    }
  }
  // Across the lanes: each step adds up one half of the sums a lane still holds and hands the other
  // half to its partner; two sums per lane are left.
#pragma unroll
  for (int step = 0; step < 5; ++step) {
    const int half = M * M >> (step + 1), mask = 16 >> step;
    const bool upper = (lane & mask) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double keep = upper ? acc[i + half] : acc[i];
      const double give = upper ? acc[i] : acc[i + half];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, mask);
    }
  }
  warp_sum[threadIdx.x >> 5][2 * lane] = acc[0];
  warp_sum[threadIdx.x >> 5][2 * lane + 1] = acc[1];
  __syncthreads();
  const int o = threadIdx.x;
  const int row = row0 + o / M, n = n0 + o % M;
  if (o < M * M && row < rows && n < N) {
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) sum += warp_sum[w][o];
    float result = static_cast<float>(sum);
    if (offset != nullptr) result = __fadd_rn(result, offset[n]);
    if (relu2) result = result > 0.0f ? __fmul_rn(result, result) : 0.0f;
    out[static_cast<size_t>(row) * N + n] = result;
  }
}

// A block per output where the tiled kernel (sixteen outputs a block) would leave SMs idle; a block
// widens its token rows for itself, so with more than two of them less so (1 row, N 1024, K 4096 in
// FP8: 11.7 us tiled, 8.2 by blocks).
bool gemv_by_blocks(int rows, int N, int num_sms) {
  return N <= (rows <= 2 ? 8 : 4) * num_sms;
}

template <int KIND, int ROWS>
cudaError_t launch_gemv_rows(const float* in, float fp8_scale, int N, int K, const void* weight,
                             float weight_scale, const float* offset, bool relu2, float* out,
                             int num_sms, LaunchStream stream) {
  const int smem = ROWS * gemv_slot(K) * static_cast<int>(sizeof(double));
  auto kernel = exact_gemv_kernel<KIND, ROWS>;
  cudaError_t err = allow_shared_memory(kernel);
  if (err != cudaSuccess) return err;
  // no more blocks than are resident together: each widens the token rows for itself
  const int resident = std::min(8, std::max(1, 220 * 1024 / (smem + 1024)));
  const int per_block = 2 * (kGemvThreads / 32);
  const int grid = std::min((N + per_block - 1) / per_block, num_sms * resident);
  // not resident early: placed while another kernel's blocks hold part of the shared memory, the
  // blocks spread unevenly (a latent model's pass over 1 token 127 us, 106 in this way)
  launch_kernel(kernel, grid, kGemvThreads, smem, stream.stream, in, fp8_scale, N, K, weight,
                weight_scale, offset, relu2, out);
  return cudaGetLastError();
}

// Rows up to which a block per output is faster than a block per 8 x 8 outputs (128 x 2688: 7 rows
// 8.1 us against 12.1 for up to 64 rows, 32 rows 14.2).
constexpr int kGemvBlockRows = 16;

template <int KIND>
cudaError_t launch_gemv_kind(const float* in, float fp8_scale, int rows, int N, int K,
                             const void* weight, float weight_scale, const float* offset,
                             bool relu2, float* out, int num_sms, LaunchStream stream) {
  if (gemv_by_blocks(rows, N, num_sms)) {
    auto run = [&](auto kernel, int per_block) {
      launch_kernel(kernel, dim3(N, (rows + per_block - 1) / per_block), kGemvThreads, 0, stream,
          in, fp8_scale, rows, N, K, weight, weight_scale, offset, relu2, out);
    };
    if (rows > kGemvBlockRows) {
      const dim3 grid((N + kTileOutputs - 1) / kTileOutputs,
                      (rows + kTileOutputs - 1) / kTileOutputs);
      const bool alone = static_cast<int>(grid.x * grid.y) <= num_sms;
      launch_kernel(alone ? exact_tile_kernel<KIND, 256> : exact_tile_kernel<KIND, 128>, grid,
                    alone ? 256 : 128, 0, stream, in, fp8_scale, rows, N, K, weight, weight_scale,
                    offset, relu2, out);
    } else if (rows == 1) {
      run(exact_gemv_block_kernel<KIND, 1>, 1);
    } else if (rows == 2) {
      run(exact_gemv_block_kernel<KIND, 2>, 2);
    } else {
      run(exact_gemv_block_kernel<KIND, 4>, 4);
    }
    return cudaGetLastError();
  }
  const int fit = kExactGemvMaxK / K;  // rows whose doubles fit shared memory
  while (rows > 0) {
    cudaError_t err;
    int done;
    if (rows >= 4 && fit >= 4) {
      done = 4;
      err = launch_gemv_rows<KIND, 4>(in, fp8_scale, N, K, weight, weight_scale, offset, relu2, out,
                                      num_sms, stream);
    } else if (rows >= 2 && fit >= 2) {
      done = 2;
      err = launch_gemv_rows<KIND, 2>(in, fp8_scale, N, K, weight, weight_scale, offset, relu2, out,
                                      num_sms, stream);
    } else {
      done = 1;
      err = launch_gemv_rows<KIND, 1>(in, fp8_scale, N, K, weight, weight_scale, offset, relu2, out,
                                      num_sms, stream);
    }
    if (err != cudaSuccess) return err;
    rows -= done;
    in += static_cast<size_t>(done) * K;
    out += static_cast<size_t>(done) * N;
  }
  return cudaSuccess;
}

}  // namespace

bool exact_supported(int N, int K) {
  // K: whole chunks, 32-bit level sums (six pairs of digits up to 128), the rows of a gemv
  return N > 0 && K > 0 && K % kExactChunk == 0 && K <= kExactGemvMaxK && K <= 16384;
}

size_t slice_bytes(size_t rows, int K, int tile_rows) {
  return (rows + tile_rows - 1) / tile_rows * tile_rows * K * kSlices;
}

int exact_weight_tile_rows() { return kExactRows; }

cudaError_t launch_slice_weights(const void* weight, int kind, float scale, int N, int K,
                                 int8_t* slices, SliceRow* info, cudaStream_t stream) {
  if (kind == kWeightFp8) {
    launch_slices<kWeightFp8>(weight, N, K, scale, kExactRows, slices, info, stream);
  } else if (kind == kWeightBf16) {
    launch_slices<kWeightBf16>(weight, N, K, scale, kExactRows, slices, info, stream);
  } else {
    launch_slices<kWeightF32>(weight, N, K, scale, kExactRows, slices, info, stream);
  }
  return cudaGetLastError();
}

// Token rows per tile: as many as the seven levels leave room for in TMEM (7 * 64 columns of 512),
// fewer when there are fewer.
int exact_tile_rows(int rows) { return rows >= 49 ? 64 : (rows + 15) / 16 * 16; }

// The K range is shared by several CTAs while that still leaves an SM for each.
int exact_splits(int rows, int N, int K, int num_sms) {
  const int nt = exact_tile_rows(rows);
  const int tiles = (N + kExactRows - 1) / kExactRows * ((rows + nt - 1) / nt);
  return std::max(1, std::min(num_sms / tiles, K / kExactChunk));
}

cudaError_t launch_exact_linear(const ExactWeight& w, const float* in, int rows, float fp8_scale,
                                const float* offset, bool relu2, const ExactWorkspace& space,
                                float* out, int32_t* error, int num_sms, cudaStream_t stream,
                                const ExactSum& sum, const ExactMix& mix) {
  if (rows <= 0 || !exact_supported(w.N, w.K)) return cudaErrorInvalidValue;
  const int nt = exact_tile_rows(rows);
  if (sum.parts != nullptr) {
    launch_slices<-1>(sum.parts, rows, w.K, fp8_scale, nt, space.slices, space.info, stream, sum.top_k,
                      sum.sums);
    in = sum.sums;
  } else {
    launch_slices<-1>(in, rows, w.K, fp8_scale, nt, space.slices, space.info, stream);
  }
  const int row_tiles = (rows + nt - 1) / nt;
  const int splits = exact_splits(rows, w.N, w.K, num_sms);
  const int grid = (w.N + kExactRows - 1) / kExactRows * row_tiles * splits;
  auto multiply = [&](auto kernel, int smem) {
    const cudaError_t attribute = allow_shared_memory(kernel);
    if (attribute != cudaSuccess) return attribute;
    kernel<<<grid, kExactThreads, smem, stream>>>(w.slices, space.slices, rows, w.N, w.K, row_tiles,
                                                  splits, space.partial, nullptr, 0.0, error);
    return cudaGetLastError();
  };
  using Shape = ExactShape<kSlices>;
  const cudaError_t err =
      nt == 16   ? multiply(exact_gemm_kernel<kSlices, 16>, Shape::smem_bytes(16))
      : nt == 32 ? multiply(exact_gemm_kernel<kSlices, 32>, Shape::smem_bytes(32))
      : nt == 48 ? multiply(exact_gemm_kernel<kSlices, 48>, Shape::smem_bytes(48))
                 : multiply(exact_gemm_kernel<kSlices, 64>, Shape::smem_bytes(64));
  if (err != cudaSuccess) return err;
  auto run = [&](auto kernel, int values) {
    const int columns = kFinishThreads * values;
    kernel<<<dim3((w.N + columns - 1) / columns, rows), kFinishThreads, 0, stream>>>(
        space.partial, splits, rows, w.N, w.K, in, fp8_scale, space.info, w.weight, w.scale, w.info,
        offset, relu2, out, mix);
  };
  // Four values a thread where enough such blocks are left to an SM (four, fewer with a short contraction):
  // then their loads count, before that a block's undecided values do, which it sums one after the other, the
  // more of them and the longer each the longer the contraction.  Whole latent pass, one value a thread
  // against four: 4096 outputs, 40 rows 336 us and 341, 100 rows 389 and 393, 160 rows 416 and 416, 400 rows 552
  // and 547, 1000 rows 824 and 792; 2048 outputs, 8 rows 53.9 and 62.2, 256 rows 113 and 115, 400 rows 154 and
  // 153; 1024 outputs, 16 rows 47.5 and 55.8, 400 rows 94.3 and 96.0, 1000 rows 123.3 and 122.4.  Only fc2 that
  // wide, K = 512, 2048 outputs: 100 rows 83.0 and 85.4, 256 rows 90.2 and 89.3.
  auto run_kind = [&](auto kind) {
    constexpr int kKind = decltype(kind)::value;
    const long long blocks = static_cast<long long>(rows) * (w.N / (4 * kFinishThreads));
    if (blocks * 192 >= static_cast<long long>(num_sms) * std::min(w.K, 768)) {
      run(exact_finish_kernel<kKind, 4>, 4);
    } else {
      run(exact_finish_kernel<kKind, 1>, 1);
    }
  };
  if (w.kind == kWeightFp8) {
    run_kind(std::integral_constant<int, kWeightFp8>());
  } else if (w.kind == kWeightBf16) {
    run_kind(std::integral_constant<int, kWeightBf16>());
  } else {
    run_kind(std::integral_constant<int, kWeightF32>());
  }
  return cudaGetLastError();
}

// Whether a weight's codes times `scale` are FP32 values rounded to 24 bits, none of them subnormal or
// infinite, and a row fits one block's threads.
bool coded_supported(int N, int K, float weight_scale) {
  return exact_supported(N, K) && N % 16 == 0 && N <= 16 * 1024 && weight_scale >= 0x1p-80f &&
         weight_scale <= 0x1p60f;
}

int coded_weight_tile_rows() { return kExactRows; }
size_t coded_slice_bytes(size_t rows, int K, int tile_rows) {
  return (rows + tile_rows - 1) / tile_rows * tile_rows * K * kCodeSlices;
}

cudaError_t launch_code_weights(const void* weight, int N, int K, int8_t* slices, float* norm,
                                cudaStream_t stream) {
  code_rows_kernel<true><<<N, kSliceThreads, 0, stream>>>(weight, K, 1.0f, kExactRows, slices, nullptr,
                                                          norm);
  return cudaGetLastError();
}

// Token rows per tile: as many as there is TMEM for, fewer when there are fewer.
static int coded_tile_rows(int rows) {
  return rows > kCodeTile - 16 ? kCodeTile : (rows + 15) / 16 * 16;
}

cudaError_t launch_coded_linear(const CodedWeight& w, const float* in, int rows, float fp8_scale,
                                const ExactWorkspace& space, int first_row, uint8_t* packed,
                                uint8_t* sf_tiled, int k_tiles, float* tensor_scale, int32_t* error,
                                int num_sms, cudaStream_t stream) {
  if (rows <= 0 || !coded_supported(w.N, w.K, w.scale) || !(fp8_scale >= kMinScale) ||
      fp8_scale > 0x1p60f) {
    return cudaErrorInvalidValue;
  }
  const int nt = coded_tile_rows(rows);
  float* norm = reinterpret_cast<float*>(space.info);
  // (behind the three digits; the workspace has room for five)
  uint8_t* codes = reinterpret_cast<uint8_t*>(space.slices) + coded_slice_bytes(rows, w.K, nt);
  code_rows_kernel<false><<<rows, kSliceThreads, 0, stream>>>(in, w.K, fp8_scale, nt, space.slices,
                                                              codes, norm);
  const int row_tiles = (rows + nt - 1) / nt;
  const int tiles = (w.N + kExactRows - 1) / kExactRows * row_tiles;
  const int splits = std::max(1, std::min(num_sms / tiles, w.K / kExactChunk));
  float* values = splits == 1 ? reinterpret_cast<float*>(space.partial) : nullptr;
  const double scale = 0x1p-18 * static_cast<double>(fp8_scale) * static_cast<double>(w.scale);
  auto multiply = [&](auto kernel) {
    const cudaError_t attribute = allow_shared_memory(kernel);
    if (attribute != cudaSuccess) return attribute;
    kernel<<<tiles * splits, kExactThreads, ExactShape<kCodeSlices>::smem_bytes(nt), stream>>>(
        w.slices, space.slices, rows, w.N, w.K, row_tiles, splits, space.partial, values, scale,
        error);
    return cudaGetLastError();
  };
  const cudaError_t err = nt == 16   ? multiply(exact_gemm_kernel<kCodeSlices, 16>)
                          : nt == 32 ? multiply(exact_gemm_kernel<kCodeSlices, 32>)
                          : nt == 48 ? multiply(exact_gemm_kernel<kCodeSlices, 48>)
                          : nt == 64 ? multiply(exact_gemm_kernel<kCodeSlices, 64>)
                                     : multiply(exact_gemm_kernel<kCodeSlices, kCodeTile>);
  if (err != cudaSuccess) return err;
  coded_quant_kernel<<<rows, (w.N / 16 + 31) / 32 * 32, 0, stream>>>(
      values, space.partial, splits, scale, rows, w.N, w.K, codes, fp8_scale, norm,
      reinterpret_cast<const uint8_t*>(w.weight), w.scale, w.norm, first_row, packed, sf_tiled,
      k_tiles, tensor_scale);
  return cudaGetLastError();
}

// FP64 over the operands as they are, or integers over their slices?  The first reads W in its own
// format, which counts for few rows: up to four are no slower on a large W (22 MB of FP8 against
// 110 MB of slices for the checkpoint's shared_up).  A short W costs no more than widening and
// multiplying its values, which up to 90 million products is less than the three launches of the
// second take (between events, us, FP64 against integers: 128 x 2688, 261 rows, 90 million 26.7 and
// 29.7, 348 rows, 120 million 35.5 and 31.8; 512 x 2688, 65 rows 26.6 and 31.2, 87 rows 34.7 and
// 29.8; 512 x 4096, 38 rows, 80 million 28.8 and 27.9; 64 x 4096, 343 rows 33.0 and 33.8, 457 rows
// 34.6 and 33.8; 384 x 1024, 228 rows 26.7 and 26.6, 305 rows 33.0 and 27.4).
constexpr long long kMostFp64Products = 90000000;
bool exact_prefers_gemv(int rows, int N, int K, int num_sms) {
  if (rows <= 4) return true;
  return gemv_by_blocks(rows, N, num_sms) &&
         static_cast<long long>(rows) * N * K <= kMostFp64Products;
}

cudaError_t launch_latent_tail(const ExactWeight& w, const LatentTail& tail, LaunchStream stream) {
  if (!exact_supported(w.N, w.K) || w.kind == kWeightFp8) return cudaErrorInvalidValue;
  auto run = [&](auto kernel) {
    const cudaError_t err = allow_shared_memory(kernel);
    if (err != cudaSuccess) return err;
    return launch_kernel(kernel, (w.N + kTailOutputs - 1) / kTailOutputs, kGemvThreads,
                         gemv_slot(w.K) * sizeof(double), stream, tail, w.N, w.K, w.weight, w.scale);
  };
  return w.kind == kWeightBf16 ? run(latent_tail_kernel<kWeightBf16>)
                               : run(latent_tail_kernel<kWeightF32>);
}

cudaError_t launch_exact_gemv(const ExactWeight& w, const float* in, float fp8_scale, int rows,
                              const float* offset, bool relu2, float* out, int num_sms,
                              LaunchStream stream) {
  if (rows <= 0 || !exact_supported(w.N, w.K)) return cudaErrorInvalidValue;
  if (w.kind == kWeightFp8) {
    return launch_gemv_kind<kWeightFp8>(in, fp8_scale, rows, w.N, w.K, w.weight, w.scale, offset,
                                        relu2, out, num_sms, stream);
  }
  if (w.kind == kWeightBf16) {
    return launch_gemv_kind<kWeightBf16>(in, fp8_scale, rows, w.N, w.K, w.weight, w.scale, offset,
                                         relu2, out, num_sms, stream);
  }
  return launch_gemv_kind<kWeightF32>(in, fp8_scale, rows, w.N, w.K, w.weight, w.scale, offset,
                                      relu2, out, num_sms, stream);
}

}  // namespace nmoe
