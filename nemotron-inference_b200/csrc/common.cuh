// Shared device helpers: number formats, PTX wrappers for mbarrier / TMA /
// tcgen05, and small utilities.  sm_100a only.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace nmoe {

// Status words a kernel can leave in the layer's device error slot.
enum DeviceError : int {
  kDevOk = 0,
  kDevWaitTimeout = 1,      // a bounded mbarrier wait gave up
  kDevActivationRange = 2,  // a relu^2 row exceeded 6*448: per-row tensor scale != 1
  kDevPlanOverflow = 3,     // more row tiles than the workspace was sized for
};

constexpr int kQuantBlock = 16;
constexpr float kFp4Max = 6.0f;
constexpr float kFp8Max = 448.0f;
constexpr float kMinScale = 1.0f / 1024.0f;

// ---------------------------------------------------------------------------
// Number formats.  The reference decodes through the toolkit's __nv_fp4_e2m1 /
// __nv_fp8_e4m3 (runtime/src/backend/expert_layer.cpp:142-152) and encodes with
// __nv_cvt_float_to_fp4(.., cudaRoundNearest) / __nv_cvt_float_to_fp8(..,
// __NV_SATFINITE, __NV_E4M3) (runtime/src/backend/nvfp4_packing.cpp:37-46).
// The device side calls the same toolkit conversions, which lower to the
// cvt.rn.satfinite.e2m1x2.f32 / e4m3x2 hardware instructions on sm_100a.
// ---------------------------------------------------------------------------

__device__ __forceinline__ float decode_e2m1(uint32_t nibble) {
  // magnitudes 0, .5, 1, 1.5, 2, 3, 4, 6; bit 3 is the sign
  const uint32_t m = nibble & 7u;
  const float mag = m < 2u ? 0.5f * static_cast<float>(m)
                           : __uint_as_float((((m >> 1) + 126u) << 23) | ((m & 1u) << 22));
  return (nibble & 8u) ? -mag : mag;
}

__device__ __forceinline__ float decode_e4m3(uint32_t byte) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(byte), __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}

__device__ __forceinline__ uint32_t encode_e4m3(float v) {
  return static_cast<uint32_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}

// Two floats -> one byte, `even` in the low nibble, `odd` in the high nibble
// (nvfp4_packing.cpp:146-152).
__device__ __forceinline__ uint32_t encode_e2m1x2(float even, float odd) {
  return static_cast<uint32_t>(
      __nv_cvt_float2_to_fp4x2(make_float2(even, odd), __NV_E2M1, cudaRoundNearest));
}

// Eight floats -> four bytes, the even ones in the low nibbles.
__device__ __forceinline__ uint32_t encode_e2m1x8(float a, float b, float c, float d, float e,
                                                  float f, float g, float h) {
  uint32_t word;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(word)
      : "f"(a), "f"(b), "f"(c), "f"(d), "f"(e), "f"(f), "f"(g), "f"(h));
  return word;
}

// Two FP32 operations in one instruction, each rounded as the scalar one.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}

// ClampScale, nvfp4_packing.cpp:19-24
__device__ __forceinline__ float clamp_scale(float v) {
  return (!isfinite(v) || v < kMinScale) ? kMinScale : v;
}

inline float clamp_scale_host(float v) {
  return (!(v == v) || v > 3.0e38f || v < kMinScale) ? kMinScale : v;
}

// Quantise 16 FP32 values that share one block (per-row tensor scale `ts`):
// returns the E4M3 scale byte, writes 8 packed bytes into two 32-bit words.
// Follows nvfp4_packing.cpp:130-153 with IEEE divisions.
__device__ __forceinline__ uint32_t quantize_block16(const float (&v)[16], float ts,
                                                     uint32_t& lo_word, uint32_t& hi_word) {
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
  float bs = 1.0f;
  if (amax > 0.0f) bs = clamp_scale(__fdiv_rn(amax, __fmul_rn(kFp4Max, ts)));
  const uint32_t scale_byte = encode_e4m3(bs);
  const float divisor = __fmul_rn(ts, bs);
  uint32_t w[2] = {0u, 0u};
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const uint32_t byte = encode_e2m1x2(__fdiv_rn(v[i], divisor), __fdiv_rn(v[i + 1], divisor));
    w[i / 8] |= (byte & 0xffu) << (8 * ((i / 2) & 3));
  }
  lo_word = w[0];
  hi_word = w[1];
  return scale_byte;
}

// Correctly rounded x / d for d > 0 given r = RN(1/d): one multiply and two
// FMAs (q = RN(x r); q + r * RN(x - q d)).  The residual correction yields the
// IEEE quotient whenever r is the correctly rounded reciprocal and d's
// significand is not all ones (Markstein); the caller handles that one
// significand with a full division.
__device__ __forceinline__ float div_by_reciprocal(float x, float d, float r) {
  const float q = __fmul_rn(x, r);
  const float e = __fmaf_rn(-q, d, x);
  return __fmaf_rn(e, r, q);
}

// Scale of a block before its rounding to E4M3 (nvfp4_packing.cpp:130-139): amax / (6 * ts),
// given `divisor` = RN(6 * ts) and `reciprocal` = RN(1 / divisor).  Quotients too small for the
// residual to be exact are below the smallest scale and clamped.
__device__ __forceinline__ float block_scale(float block_max, float divisor, float reciprocal) {
  if (!(block_max > 0.0f)) return 1.0f;
  const bool exact = (__float_as_uint(divisor) & 0x007fffffu) != 0x007fffffu && block_max < 1.0e37f;
  return clamp_scale(exact ? div_by_reciprocal(block_max, divisor, reciprocal)
                           : __fdiv_rn(block_max, divisor));
}

// div_by_reciprocal of two values by the same divisor.
__device__ __forceinline__ uint64_t div2_by_reciprocal(uint64_t x, uint64_t minus_d, uint64_t r) {
  const uint64_t q = mul2(x, r);
  return fma2(fma2(q, minus_d, x), r, q);
}

// Programmatic dependent launch.  The successor on the stream may become resident once every CTA has
// called release_successor(), so a kernel that allocates TMEM calls it after that (a successor that
// took the columns first would wait for this kernel, and this kernel for the columns).  Every thread
// calls wait_for_predecessor() before it touches what other kernels write or read: it returns when
// the predecessor, and with it all that came before, is complete and visible.  Pointers to such data
// are not `const __restrict__`, so that no load of theirs moves ahead of it.
__device__ __forceinline__ void release_successor() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_predecessor() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Sums eight values over the warp: after the call lane L holds the total of value
// ((L >> 4) & 1) * 4 + ((L >> 3) & 1) * 2 + ((L >> 2) & 1).  Half of the values change hands in
// each of the first three steps, nine shuffles instead of forty.
__device__ __forceinline__ double warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int half = 4; half > 0; half >>= 1) {
    const int stride = half * 4;
    const bool upper = (lane & stride) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double send = upper ? v[i] : v[i + half];
      const double keep = upper ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, stride);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

// Asks for `bytes` (a multiple of 16, from a 16-byte boundary) to be brought into L2.
__device__ __forceinline__ void prefetch_l2_bulk(const void* from, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* from) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(from));
}

// The fused quantiser of the up-projection epilogue: 16 non-negative values in pairs whose maximum
// is `amax`, per-row tensor scale 1 (nvfp4_packing.cpp:119-153 with tensor_scale == 1.0).
// Bit-identical to quantize_block16(v, 1.0f, ..).
__device__ __forceinline__ uint32_t quantize_block16_unit_scale(const uint64_t (&v)[8], float amax,
                                                                uint32_t& lo_word,
                                                                uint32_t& hi_word) {
  const float bs = block_scale(amax, kFp4Max, 1.0f / kFp4Max);
  float q[16];
  if ((__float_as_uint(bs) & 0x007fffffu) != 0x007fffffu) {
    const float r = __frcp_rn(bs);
    const uint64_t minus_bs = pack2(-bs, -bs), r2 = pack2(r, r);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      unpack2(div2_by_reciprocal(v[i], minus_bs, r2), q[2 * i], q[2 * i + 1]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float a, b;
      unpack2(v[i], a, b);
      q[2 * i] = __fdiv_rn(a, bs);
      q[2 * i + 1] = __fdiv_rn(b, bs);
    }
  }
  lo_word = encode_e2m1x8(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7]);
  hi_word = encode_e2m1x8(q[8], q[9], q[10], q[11], q[12], q[13], q[14], q[15]);
  return encode_e4m3(bs);
}

// Offset of the scale of (row, 16-block) inside the 128-row x 4-block tiled
// layout of runtime/src/backend/nvfp4_scale_layout.cpp:14-28.  `k_tiles` is the
// number of 4-block groups each 128-row tile stores.
__host__ __device__ __forceinline__ size_t swizzled_scale_offset(size_t row, size_t block,
                                                                 size_t k_tiles) {
  return ((((row >> 7) * k_tiles) + (block >> 2)) << 9) | ((row & 31u) << 4) |
         (((row >> 5) & 3u) << 2) | (block & 3u);
}

// ---------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait: gives up after ~2^31 clock ticks (about a second) so that a
// protocol bug or a lost copy can never hang the GPU.  Returns false on
// timeout; the caller records kDevWaitTimeout and unwinds.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - start > (1ll << 31)) return false;
  }
  return true;
}

// The same operations by shared-memory address, for loops whose every instruction counts: a role
// of one thread runs a K block's bookkeeping as one dependent chain.
__device__ __forceinline__ bool mbar_try_wait_at(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

static __device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) {
  const long long start = clock64();
  while (!mbar_try_wait_at(bar, parity)) {
    if (clock64() - start > (1ll << 31)) return false;
  }
  return true;
}

// A role that issues tensor-core or copy instructions runs them from ONE lane, but the loop around
// them should be executed by the whole warp with warp-uniform values: their operands (descriptors,
// addresses) live in uniform registers, and in code that only one lane reaches the compiler has to
// move every operand there one by one (a K block of four MMAs and a commit took 690 cycles of
// issue that way).
template <typename T>
__device__ __forceinline__ T warp_uniform(T value) {
  return __shfl_sync(0xffffffffu, value, 0);
}

// True in one lane of the (converged) warp, the same one every time.
__device__ __forceinline__ bool elect_one() {
  uint32_t elected;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(elected));
  return elected != 0;
}

// The bounded wait, by all lanes of a warp; the result is the same in all of them.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity) {
  if (__all_sync(0xffffffffu, mbar_try_wait_at(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait_slow(bar, parity));
}

__device__ __forceinline__ void mbar_arrive_at(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx_at(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void tma_load_2d_at(uint32_t smem_dst, const CUtensorMap* map, int x,
                                               int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void bulk_load_at(uint32_t smem_dst, const void* gmem_src,
                                             uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(smem_dst), "l"(gmem_src), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tcgen05_commit_at(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}

// 2-D tiled TMA load (no multicast) into this CTA's shared memory.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// --- tcgen05 ---------------------------------------------------------------

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(columns)
               : "memory");
}

__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns)
               : "memory");
}

__device__ __forceinline__ void tcgen05_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tcgen05_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Arrive on an mbarrier once every tcgen05 operation this thread issued so far
// has completed.
__device__ __forceinline__ void tcgen05_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

// Shared-memory matrix descriptor (sm_100 format, version 1).
//   bits  0-13 start address >> 4      bits 16-29 leading byte offset >> 4
//   bits 32-45 stride byte offset >> 4 bits 46-47 version (1)
//   bits 61-63 swizzle (0 none, 2 = 128 B)
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes,
                                                   uint32_t sbo_bytes, uint32_t swizzle) {
  return static_cast<uint64_t>((smem_addr & 0x3ffffu) >> 4) |
         (static_cast<uint64_t>(lbo_bytes >> 4) << 16) |
         (static_cast<uint64_t>(sbo_bytes >> 4) << 32) | (1ull << 46) |
         (static_cast<uint64_t>(swizzle) << 61);
}

// The same descriptor for another address: `offset` bytes (a multiple of 16) further on.
__device__ __forceinline__ uint64_t advance_smem_desc(uint64_t desc, uint32_t offset) {
  const uint32_t low = static_cast<uint32_t>(desc) + (offset >> 4);
  return (desc & 0xffffffff00000000ull) | low;
}

// Copy 32 rows x 16 bytes of scale factors from shared memory into 4 TMEM
// columns, replicated to all four 32-lane quarters.
__device__ __forceinline__ void tcgen05_cp_32x128b_warpx4(uint32_t taddr, uint64_t smem_desc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(smem_desc)
               : "memory");
}

// D[tmem] (+)= A[smem] * B[smem] with per-16 UE4M3 block scales taken from
// TMEM; E2M1 operands, K = 64 per instruction.
__device__ __forceinline__ void tcgen05_mma_nvf4(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                                 uint32_t idesc, uint32_t sfa_tmem,
                                                 uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X"
      " [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem),
      "r"(sfb_tmem)
      : "memory");
}

// Instruction descriptor for kind::mxf4nvf4: E2M1 x E2M1, UE4M3 scales,
// both operands K-major, M = 128.
__host__ __device__ constexpr uint32_t make_idesc_nvf4(uint32_t n) {
  return (1u << 7) /* A = E2M1 */ | (1u << 10) /* B = E2M1 */ | ((n >> 3) << 17) |
         (0u << 23) /* scale format UE4M3 */ | ((128u >> 4) << 24);
}

// 32 lanes x 16 consecutive FP32 columns: thread i receives row (lane base + i).
__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  // The wait shares the asm statement with the load so that no use of the
  // destination registers can be scheduled between them.
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// The same load without its wait: several may be in flight before one tmem_ld_fence()
// per destination array.  The destination registers are undefined until then.
__device__ __forceinline__ void tmem_ld_x16_async(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// After tmem_ld_wait(): ties every later use of `r` to a volatile statement behind the
// wait, so that the compiler cannot schedule a use of the registers before it.
__device__ __forceinline__ void tmem_ld_fence(uint32_t (&r)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(r[i]));
}

// --- CTA pairs (cta_group::2) -------------------------------------------------
// Two CTAs of a cluster of size 2 drive one tcgen05.mma with M = 256: each CTA
// holds 128 rows of A and half of B's rows in its own shared memory (at the same
// offsets), each accumulates its own 128 rows in its own TMEM.  One thread of the
// leader (cluster rank 0) issues the MMAs and the scale copies for both.

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  return rank;
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void tma_load_2d_pair_at(uint32_t smem_dst, const CUtensorMap* map, int x,
                                                    int y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}

// Arrive on an mbarrier by its shared::cluster address (this CTA's or the partner's).  What it
// hands on is tensor memory, whose accesses are complete (tcgen05.wait) and fenced
// (tcgen05_fence_before) by then; releasing generic memory to the cluster as well
// (.release.cluster) made every arrival wait about 1100 cycles.
__device__ __forceinline__ void mbar_arrive_cluster_at(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

// The shared::cluster address of `local` (an address in this CTA's shared memory) in
// CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_address_of(const void* local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(remote)
               : "r"(smem_u32(local)), "r"(rank));
  return remote;
}

// TMEM allocation for a pair: one warp of EACH CTA executes it, the same columns
// are allocated in both.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(columns)
               : "memory");
}

__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns)
               : "memory");
}

// Arrive, once every tcgen05 operation this thread issued so far has completed, on
// the mbarrier at this offset in every CTA of `cta_mask` (bit i = cluster rank i).
__device__ __forceinline__ void tcgen05_commit_pair(uint64_t* bar, uint16_t cta_mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
      " [%0], %1;" ::"r"(smem_u32(bar)),
      "h"(cta_mask)
      : "memory");
}

// Scale copy in both CTAs of the pair: each copies from its own shared memory (same
// offset) into its own TMEM.
__device__ __forceinline__ void tcgen05_cp_pair_32x128b_warpx4(uint32_t taddr, uint64_t smem_desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(smem_desc)
               : "memory");
}

__device__ __forceinline__ void tcgen05_mma_pair_nvf4(uint32_t d_tmem, uint64_t a_desc,
                                                      uint64_t b_desc, uint32_t idesc,
                                                      uint32_t sfa_tmem, uint32_t sfb_tmem,
                                                      uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X"
      " [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem),
      "r"(sfb_tmem)
      : "memory");
}

// Instruction descriptor of make_idesc_nvf4 with M = 256 (a CTA pair).
__host__ __device__ constexpr uint32_t make_idesc_nvf4_pair(uint32_t n) {
  return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (0u << 23) | ((256u >> 4) << 24);
}

}  // namespace nmoe
