// Host-visible declarations of the kernel launchers.  Everything takes an
// explicit stream and returns cudaError_t from the launch.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace nmoe {

// Where a kernel is launched.  `chained`: what precedes it on the stream is a kernel of this library,
// and it may be made resident while that one still runs (programmatic dependent launch): it sets up
// and asks for weights meanwhile, then waits (wait_for_predecessor()) before it reads or writes
// anything else.  A pass over 1 token 45.0 -> 43.0 us, 7 tokens 69.6 -> 65.5, 64 tokens 147.5 -> 143.4.
struct LaunchStream {
  cudaStream_t stream = nullptr;
  bool chained = false;
  LaunchStream(cudaStream_t s, bool after_kernel = false) : stream(s), chained(after_kernel) {}
  operator cudaStream_t() const { return stream; }
};

template <typename... Params, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, int threads, size_t smem,
                                 LaunchStream stream, Args&&... args) {
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(static_cast<unsigned>(threads));
  config.dynamicSmemBytes = smem;
  config.stream = stream.stream;
  config.attrs = &attribute;
  config.numAttrs = stream.chained ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// SMs of the current device.
inline int device_sms() {
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    cudaGetLastError();  // (the launch will say what is wrong)
    return 1;
  }
  return sms;
}
// Blocks of a kernel that walks its elements with a grid-sized stride: enough to fill the GPU several
// times over, so that blocks need not be whole waves.
constexpr int kStrideBlocks = 2368;
inline int stride_blocks(size_t work, int threads) {
  const size_t blocks = (work + threads - 1) / threads;
  return static_cast<int>(blocks < 1 ? 1 : blocks > kStrideBlocks ? kStrideBlocks : blocks);
}

// Lets `kernel` (which has no static shared memory) be launched with all the dynamic shared memory a
// block can have.  The limit belongs to the kernel and not to the launch, so it never follows the
// launch's own size: a thread that lowered it between another thread's limit and launch made that
// launch fail (two threads, row tiles of 32 and 128 rows: 10 of 40000).
constexpr int kMaxSharedBytes = 227 * 1024;
template <typename Kernel>
inline cudaError_t allow_shared_memory(Kernel* kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kMaxSharedBytes);
}

// A row tile is a 128-row aligned slot of the expert-sorted activation buffer
// holding `rows` (<= 128) valid rows that all belong to `expert`.
struct RowTile {
  int32_t row0;    // first row of the slot (multiple of 128)
  int32_t rows;    // valid rows in the slot
  int32_t expert;  // index into the stacked expert weights
  int32_t reserved;
};

// Element type of the per-(token, slot) rows the down projection produces and the
// combine kernels add up: FP32, or a 16-bit type that halves the layer's largest
// write and read.  The numbering is nmoe_dtype's.
enum RowKind : int { kRowF32 = 0, kRowBf16 = 1, kRowF16 = 2 };
inline size_t row_kind_bytes(RowKind kind) { return kind == kRowF32 ? 4 : 2; }

enum GemmMode : int {
  kGemmUp = 0,    // D -> *scales -> relu^2 -> NVFP4 (packed + tiled scales)
  kGemmDown = 1,  // D -> *scales [* routing weight] -> FP32 rows scattered by dest_row
};

struct GemmArgs {
  int32_t K = 0;         // contraction length, multiple of 64
  int32_t N = 0;         // output features per expert
  int32_t n_tiles = 0;   // ceil(N / BN)
  int32_t k_blocks = 0;  // ceil(K / 256)
  int32_t kb_full = 0;   // K / 256: K blocks stored in the full-block weight region
  const uint8_t* b_full = nullptr;  // [expert][kb_full][N][128 B], 16-byte chunks pre-swizzled
  // A-side block scales, tiled: [row slot][k_blocks][2048 bytes]
  const uint8_t* sfa = nullptr;
  // weight block scales, [expert][n_tile][k_block][sfb_bytes] in the layout
  // produced by relayout_weight_scales()
  const uint8_t* sfb = nullptr;
  const float* a_tensor_scale = nullptr;  // per activation row, nullptr => 1.0
  const float* w_tensor_scale = nullptr;  // [expert]
  // schedule: grouped (row_tiles + device count) or dense (row_tiles == nullptr)
  const RowTile* row_tiles = nullptr;
  const int32_t* num_row_tiles = nullptr;
  int32_t dense_rows = 0;
  // kGemmUp outputs
  uint8_t* out_packed = nullptr;  // [row][N/2]
  uint8_t* out_sf = nullptr;      // tiled [row slot][out_k_blocks][2048]
  int32_t out_k_blocks = 0;       // ceil(N / 256)
  // kGemmDown outputs
  void* out_rows = nullptr;           // [dest][N] of out_kind elements
  int32_t out_kind = kRowF32;         // RowKind
  int32_t out_aligned = 0;            // every row of out_rows starts on a 32-byte boundary
  const int32_t* dest_row = nullptr;  // per activation row; nullptr => row*dest_mul+dest_add
  int32_t dest_mul = 1;
  int32_t dest_add = 0;
  const float* row_weight = nullptr;  // per activation row routing weight, nullptr => none
  int32_t relu2 = 0;                  // kGemmDown: store relu^2 of the scaled value (the
                                      // unfused up projection keeps its rows in FP32)
  // Expert-parallel return straight into the source ranks' memory: destination
  // index d means row (d + segment_slot0) % segment_rows of the buffer that
  // out_segments[(d + segment_slot0) / segment_rows] points to (a peer's GPU).
  const unsigned long long* out_segments = nullptr;
  int32_t segment_rows = 0;
  int32_t segment_slot0 = 0;
  int32_t* error = nullptr;           // device error slot (DeviceError)
};

// A kernel's weight tile.  The block scales of every MMA must start on a 4-column TMEM boundary, so
// a weight tile stores its scales in whole groups of 128 rows.
struct GemmTileInfo {
  int bn;          // output features per tile
  int sfb_groups;  // 32-row groups of weight scales stored per K-tile
  int sfb_bytes;   // bytes of weight scales per (n_tile, k_block)
  int b_rows;      // weight rows one CTA stages per K block (half a tile in a pair)
};

// Tensor maps of a CTA-pair GEMM launch.  `a`: activation rows, 128-byte swizzle, boxes of 16, 32, ..
// 128 rows; `b_full`: the full weight K blocks, the K-block-major panels as rows of eight weight rows'
// 128 bytes, no swizzle; `b_tail`: the partial last K block of the weights.
constexpr int kPairBoxRows = 16;
constexpr int kPairBoxes = 128 / kPairBoxRows;
struct GemmMaps {
  CUtensorMap a[kPairBoxes];
  CUtensorMap b_tail;
  CUtensorMap b_full;
  CUtensorMap sfa, sfb;  // both operands' tiled block scales as rows of 1024 bytes
};

// Up to four GEMMs whose tiles one persistent launch walks in order (csrc/expert_stream.cu): the
// batch sizes that are bound by reading the weights.
constexpr int kStreamPhases = 4;
constexpr int kStreamBoxes = 5;
struct StreamPhase {
  CUtensorMap a[kStreamBoxes];  // activation rows, boxes of 8, 16, 32, 64 and 128 rows
  CUtensorMap b_tail;  // the partial last K block of the weights
  GemmArgs gemm;
  int32_t mode = kGemmUp;  // GemmMode
  // Grouped phases whose row tiles hold all tokens in token order (csrc/front.cu): activation rows and
  // their scales are those of the tokens, and rows that `used` names negative are of no use.
  const int32_t* used = nullptr;
  // per 128-row slot: finished up tiles are counted here, down tiles wait for `wait_target` of
  // them (0 = their rows were complete before the launch)
  int32_t* ready = nullptr;
  int32_t wait_target = 0;
};
struct StreamArgs {
  StreamPhase phase[kStreamPhases];
  int32_t phases = 0;
  const RowTile* row_tiles = nullptr;  // those of the grouped phases (all have the same), and how many
  int32_t row_tile_room = 0;           // may be read
  int32_t tile_rows = 128;  // most rows a row tile holds: 32, 64 or 128
  int32_t* error = nullptr;
  // all `ready` words of the phases, the ticket the tiles are taken with and the count of CTAs that
  // are done, all zero between launches (the last CTA zeroes them); ticket == nullptr: tiles are
  // dealt out, for launches without waits
  int32_t* ready = nullptr;
  int32_t ready_count = 0;
  // the weights of phases over `dense_rows` are known before the launch's predecessor ends: fetch
  // them into L2 until it does
  bool fetch_dense = false;
  int32_t* ticket = nullptr;
  int32_t* finished = nullptr;
  // (with StreamPhase::used) words that the last CTA clears: those through which the blocks of the front end
  // (csrc/front.cu) hand rows on.  That launch cannot clear them itself: a block that waits gives up after a
  // while, and what it gave up on may be announced until the launch has ended.
  int32_t* front_words = nullptr;
  int32_t front_word_count = 0;
  // nullable, host memory: the last CTA stores there what it finds in `error`, unless that is nothing
  int32_t* error_host = nullptr;
};
inline int stream_tile_rows(int rows) { return rows <= 32 ? 32 : rows <= 64 ? 64 : 128; }
cudaError_t launch_expert_stream(const StreamArgs& args, int num_sms, LaunchStream stream);

GemmTileInfo stream_tile_info();
GemmTileInfo pair_tile_info();
// 256 x 208 tiles over pairs of CTAs (csrc/gemm.cu): the batches bound by arithmetic.  A grouped
// schedule gives every expert an even number of row tiles.  Needs two SMs.
cudaError_t launch_pair_gemm(GemmMode mode, const GemmMaps& maps, const GemmArgs& args, int num_sms,
                             cudaStream_t stream);

// Packed weights [experts][N][K/2] -> K-block-major (device to device): every
// (expert, 128-byte K block) becomes a contiguous [N][128 B] panel in `full`, so a
// weight tile of any height is ONE contiguous read; the partial last K block
// goes to `tail` as [experts * N][tail_pitch_bytes].
cudaError_t relayout_weight_packed(const uint8_t* row_major, int experts, int N, int K,
                                   int tail_pitch_bytes, uint8_t* full, uint8_t* tail,
                                   cudaStream_t stream);

// Re-tile row-major E4M3 weight block scales [experts][N][K/16] into the layout
// the GEMM variant consumes (device to device).
cudaError_t relayout_weight_scales(const uint8_t* row_major, int experts, int N, int K, int bn,
                                   int sfb_groups, uint8_t* out, cudaStream_t stream);
size_t weight_scale_layout_bytes(int experts, int N, int K, int bn, int sfb_groups);

// --- quantiser / norm ------------------------------------------------------
// RMSNorm (optional) + per-row dynamic NVFP4 quantisation.
//   in: [rows][cols] fp32 or bf16; norm_weight nullptr => no normalisation
//   normalized (optional) fp32 [rows][cols]
//   packed [rows][cols/2]; sf_row_major (optional) [rows][cols/16];
//   sf_tiled (optional) tiled layout with k_blocks*4 K-tiles per 128-row slot;
//   tensor_scale (optional) [rows]; inv_rms (optional) [rows]: 1/sqrt(mean(x^2)+eps);
//   `zero` (optional): `zero_count` words set to zero on the way (the histogram of what follows)
cudaError_t launch_norm_quant(const void* in, bool in_bf16, int rows, int cols,
                              const float* norm_weight, float eps, float* normalized,
                              uint8_t* packed, uint8_t* sf_row_major, uint8_t* sf_tiled,
                              int k_blocks, float* tensor_scale, int num_sms, LaunchStream stream,
                              float* inv_rms = nullptr, int32_t* zero = nullptr,
                              int zero_count = 0);
// Whole-matrix dynamic quantisation with ONE tensor scale (the reference
// packer's semantics for rows > 1).  `amax_scratch` is one float of device
// memory; it is overwritten.
cudaError_t launch_quant_matrix(const float* in, int rows, int cols, uint8_t* packed,
                                uint8_t* sf_row_major, float* tensor_scale,
                                float* amax_scratch, cudaStream_t stream);
cudaError_t launch_dequant(const uint8_t* packed, const uint8_t* sf_row_major,
                           const float* tensor_scale, bool per_row_scale, int rows, int cols,
                           float* out, cudaStream_t stream);
cudaError_t launch_swizzle_scales(const uint8_t* row_major, int rows, int cols, uint8_t* tiled,
                                  cudaStream_t stream);

// --- router ------------------------------------------------------------------
cudaError_t launch_router_logits(const float* normalized, const float* gate,
                                 const float* logit_offset /* nullable [experts] */, int rows,
                                 int experts, int hidden, float* logits, int num_sms,
                                 cudaStream_t stream);
// The argument rules of launch_router_topk, for callers that must know before they
// enqueue anything.
bool router_topk_arguments_valid(int rows, int experts, int top_k, int n_group, int topk_group);
cudaError_t launch_router_topk(const float* logits, const float* bias, int rows, int experts,
                               int top_k, int n_group, int topk_group, bool norm_topk_prob,
                               float routed_scaling, int32_t* top_index, float* top_weight,
                               int32_t* expert_counts /* nullable, += histogram */,
                               int32_t* position /* nullable [rows][top_k]: the count before */,
                               int num_sms, LaunchStream stream);

// Two-pass router for large batches.  Pass 1: logits on the tensor cores (FP32
// accumulate) from the bf16 gate and the normalised activations, which the kernel
// rebuilds from the layer input `x` as (x * inv_rms) * norm_weight and splits into
// three bf16 terms on the fly.  Pass 2, per token: every expert whose pass-1 choice
// score is within `tie_margin` of the top_k-th is re-evaluated in FP64 (and written
// back into `logits`), then top-k runs on the exact values.  Requires n_group == 1,
// experts % 32 == 0, experts <= 256, hidden % 64 == 0.
cudaError_t launch_router_fast_logits(const void* x, bool x_bf16, const float* inv_rms,
                                      const float* norm_weight, const CUtensorMap& tmap_gate,
                                      int rows, int experts, int hidden, int splits,
                                      float* logits, int32_t* error, cudaStream_t stream);
// Pass 1 for bf16 layer inputs: the RMSNorm weight folded into the gate (three bf16 terms of
// fl32(w[i] * gate[e][i]), `planes` = [3][experts][hidden], built once by launch_fold_gate),
// the input rows read by TMA through `tmap_x` ([rows][hidden] bf16, box 64 x 128, 128-byte
// swizzle; `tmap_planes` = [3 * experts][hidden], box 64 x experts), inv_rms applied to the sums.
cudaError_t launch_fold_gate(const __nv_bfloat16* gate, const float* norm_weight, int experts,
                             int hidden, __nv_bfloat16* planes, cudaStream_t stream);
// In both forms `splits` CTAs share the contraction of one 128-row tile; split s writes its
// partial sums to logits + s * rows * experts, and launch_router_select_exact adds them up.
// router_pass1_splits picks the split count for a batch; splits * rows stays below
// router_pass1_rows(rows).
constexpr int kMaxPass1Splits = 32;
int router_pass1_splits(int rows, int hidden, int num_sms);
// Rows of partial sums that any batch of up to `max_rows` rows may write.
inline size_t router_pass1_rows(size_t max_rows, int num_sms) {
  const size_t split_rows = static_cast<size_t>(num_sms) * 128;  // splits * tiles <= num_sms
  const size_t small = max_rows * kMaxPass1Splits;
  const size_t most = small < split_rows ? small : split_rows;
  return most > max_rows ? most : max_rows;
}
cudaError_t launch_router_folded_logits(const CUtensorMap& tmap_x, const CUtensorMap& tmap_planes,
                                        const float* inv_rms, int rows, int experts, int hidden,
                                        int splits, float* logits, int32_t* error,
                                        cudaStream_t stream);
cudaError_t launch_router_select_exact(float* logits, int splits, const void* x, bool x_bf16,
                                       const float* inv_rms, const float* norm_weight,
                                       const __nv_bfloat16* gate, const float* logit_offset,
                                       const float* bias, int rows, int experts, int hidden,
                                       int top_k, bool norm_topk_prob, float routed_scaling,
                                       float tie_margin, int32_t* top_index, float* top_weight,
                                       int32_t* expert_counts, int32_t* position,
                                       cudaStream_t stream);

// --- correctly rounded linears (csrc/exact.cu) ---------------------------------
// y[rows][N] = x[rows][K] x W[N][K]^T in FP32, each value the FP64 sum rounded once.
enum WeightKind : int { kWeightF32 = 0, kWeightBf16 = 1, kWeightFp8 = 2 };
// A row in fixed point: every value is below 2^exponent; `inexact` values have bits below the
// last digit.
struct SliceRow {
  int32_t exponent;
  int32_t inexact;
};
struct ExactWeight {
  int N = 0, K = 0;
  int kind = kWeightF32;           // how `weight` is stored; FP8 codes count times `scale`
  const void* weight = nullptr;    // [N][K], 16-byte aligned
  float scale = 1.0f;
  const int8_t* slices = nullptr;  // slice_bytes(N, K, exact_weight_tile_rows()) bytes, 16-byte
                                   // aligned, zero where no row is
  const SliceRow* info = nullptr;  // [N]
};
constexpr int kExactGemvMaxK = 25 * 1024;  // values of K whose doubles fit shared memory
bool exact_supported(int N, int K);
size_t slice_bytes(size_t rows, int K, int tile_rows);
int exact_weight_tile_rows();
int exact_tile_rows(int rows);  // token rows per tile for a batch
int exact_splits(int rows, int N, int K, int num_sms);
cudaError_t launch_slice_weights(const void* weight, int kind, float scale, int N, int K,
                                 int8_t* slices, SliceRow* info, cudaStream_t stream);
struct ExactWorkspace {
  int8_t* slices;   // slice_bytes(rows, K, exact_tile_rows(rows))
  SliceRow* info;   // [rows]
  double* partial;  // exact_splits() * rows * N
};
// What a linear may take in and hand on itself, in the place of kernels before and behind it: rows that
// are sums of `top_k` parts each ([rows][top_k][K]; written to `sums` [rows][K], which stands for `in`),
// and out = in + (y + shared), all [rows][N].
struct ExactSum {
  const float* parts = nullptr;
  int top_k = 1;
  float* sums = nullptr;
};
struct ExactMix {
  const void* in = nullptr;
  bool in_bf16 = false;
  const float* shared = nullptr;
  void* out = nullptr;
  bool out_bf16 = false;
};
// `fp8_scale` != 0: every value of `in` takes the round trip of the scaled-FP8 family first.
// `offset` (nullable [N]) is added to the rounded sum, `relu2` then squares what is positive.
cudaError_t launch_exact_linear(const ExactWeight& w, const float* in, int rows, float fp8_scale,
                                const float* offset, bool relu2, const ExactWorkspace& space,
                                float* out, int32_t* error, int num_sms, cudaStream_t stream,
                                const ExactSum& sum = ExactSum(), const ExactMix& mix = ExactMix());
bool exact_prefers_gemv(int rows, int N, int K, int num_sms);
// The same for a handful of rows: reads W once per four rows, no slices.
cudaError_t launch_exact_gemv(const ExactWeight& w, const float* in, float fp8_scale, int rows,
                              const float* offset, bool relu2, float* out, int num_sms,
                              LaunchStream stream);

// relu^2 and NVFP4 of a scaled-FP8 linear's rows (csrc/exact.cu): the codes, block scales and tensor
// scales that launch_norm_quant gives for the rows that launch_exact_linear computes.
struct CodedWeight {
  int N = 0, K = 0;
  const void* weight = nullptr;    // [N][K] E4M3 codes, times `scale`; 16-byte aligned
  float scale = 1.0f;
  const int8_t* slices = nullptr;  // coded_slice_bytes(N, K, coded_weight_tile_rows()) bytes, zero
                                   // where no row is; nullptr: not available
  const float* norm = nullptr;     // [N]
};
bool coded_supported(int N, int K, float weight_scale);
int coded_weight_tile_rows();
size_t coded_slice_bytes(size_t rows, int K, int tile_rows);
cudaError_t launch_code_weights(const void* weight, int N, int K, int8_t* slices, float* norm,
                                cudaStream_t stream);
// `in` [rows][K] gives rows first_row .. of the outputs (sf_tiled: k_tiles per 128-row slot).
cudaError_t launch_coded_linear(const CodedWeight& w, const float* in, int rows, float fp8_scale,
                                const ExactWorkspace& space, int first_row, uint8_t* packed,
                                uint8_t* sf_tiled, int k_tiles, float* tensor_scale, int32_t* error,
                                int num_sms, cudaStream_t stream);

// The end of a latent layer over one token: `routed` [K] = the sum of parts [top_k][K], `projected` [N] =
// routed x W^T (dense), out = in + (projected + shared).
struct LatentTail {
  const float* parts;
  int top_k;
  const float* shared;
  const void* in;
  bool in_bf16;
  float* routed;
  float* projected;
  void* out;
  bool out_bf16;
};
cudaError_t launch_latent_tail(const ExactWeight& w, const LatentTail& tail, LaunchStream stream);

// --- dense and scaled-FP8 linear families, latent-MoE data flow (csrc/dense.cu) -
// The dense matmul itself is launch_router_logits: out[rows][experts] =
// a[rows][hidden] x w[experts][hidden]^T, FP64 accumulation, FP32 result.
// Activation round trip through E4M3 with a per-tensor input scale.
cudaError_t launch_fp8_round_trip(const float* in, size_t count, float input_scale, float* out,
                                  cudaStream_t stream);
// E4M3 weight bytes -> FP32 values times the per-tensor weight scale.
cudaError_t launch_fp8_weight_dequant(const uint8_t* bytes, size_t count, float weight_scale,
                                      float* out, cudaStream_t stream);
cudaError_t launch_relu2(float* values, size_t count, cudaStream_t stream);
// out[t] = sum_k parts[t][k] in slot order; parts FP32 [rows][top_k][cols].
cudaError_t launch_sum_parts(const float* parts, int rows, int cols, int top_k, float* out,
                             LaunchStream stream);
// out = in + (projected + shared), all [rows][hidden].
cudaError_t launch_mixer(const void* in, bool in_bf16, const float* projected, const float* shared,
                         int rows, int hidden, void* out, bool out_bf16, LaunchStream stream);
// out[i] = rows[row_of[i]] (row_of == nullptr: identity), FP32 rows of `cols`.
cudaError_t launch_gather_rows(const float* rows, const int32_t* row_of, int count, int cols,
                               float* out, cudaStream_t stream);

// --- plan / permute / combine -------------------------------------------------
struct PlanBuffers {
  int32_t* expert_counts;   // [experts]  (input, filled by the router)
  int32_t* expert_cursor;   // [experts]  zeroed by the caller where pairs bring no position
  RowTile* row_tiles;       // [max_row_tiles]
  int32_t* num_row_tiles;   // [1]
};
// Where permute reads a (row, slot) pair from.  Quantised rows are indexed by
// source row = pair / pairs_per_row, routing weight and expert id by pair; all
// strides are in bytes.  Local routing: pairs_per_row = top_k over the token
// arrays.  Expert-parallel receive: pairs_per_row = 1 over dispatch records.
struct PermuteSource {
  const uint8_t* packed;
  size_t packed_stride;
  const uint8_t* sf;  // row-major E4M3 block scales
  size_t sf_stride;
  const float* tensor_scale;
  size_t tensor_scale_stride;
  const float* weight;
  size_t weight_stride;
  const int32_t* expert;  // index into the LOCAL expert stack
  size_t expert_stride;
  int pairs_per_row;
  const int32_t* position = nullptr;  // per pair, its place among its expert's; nullptr: any place
  // fixed-capacity receive buffers: pair i is valid iff (i % capacity) <
  // valid_counts[i / capacity]; nullptr = every pair is valid
  const int32_t* valid_counts = nullptr;
  int capacity = 0;
};
// Lays out every expert's row slots (128 rows each; `tile_multiple`: every expert gets a multiple of
// this many, 2 when CTA pairs consume them, and its rows are then spread over them evenly), writes the
// tile list, copies each pair's quantised activation row into its expert's slots and records where it
// went; sorted_dest[row] = source_row * dest_stride + slot.
cudaError_t launch_place_rows(const PlanBuffers& plan, const PermuteSource& src, int pairs,
                              int experts /* size of the local expert stack */, int tile_multiple,
                              int max_row_tiles, int cols, int k_blocks, uint8_t* sorted_packed,
                              uint8_t* sorted_sf_tiled, float* sorted_tensor_scale,
                              float* sorted_weight, int32_t* sorted_dest,
                              int32_t* pair_row /* nullable */, int dest_stride, int32_t* error,
                              int num_sms, LaunchStream stream);
// --- front end of a handful of tokens (csrc/front.cu) ---------------------------
constexpr int kFrontMaxRows = 8;
constexpr int kFrontMaxCols = 4096;
constexpr int kFrontMaxExperts = 512;     // of one token
constexpr int kFrontMaxExpertsOfRows = 256;  // of several
constexpr int kFrontRowsPerBlock = 4;        // of several, for which a block forms an expert's logits
constexpr int kFrontBlocksPerSm = 2;         // of a launch over several
constexpr int kFrontLinears = 2;
// A linear of the one token's normalised row whose FP32 row is then quantised with its tensor scale.
constexpr int kFrontLinearMaxN = 6144;
constexpr int kFrontLinearBlocksPerSm = 3;  // of a launch with linears
struct FrontLinear {
  int N = 0, kind = 0;
  const void* weight = nullptr;
  float scale = 1.0f, fp8_scale = 0.0f;
  bool relu2 = false;
  float* rounded = nullptr;  // [cols]
  float* out = nullptr;      // [N]
  uint8_t* packed = nullptr;
  uint8_t* sf_row_major = nullptr;
  uint8_t* sf_tiled = nullptr;
  int k_tiles = 0;
  float* tensor_scale = nullptr;
};
struct FrontArgs {
  const void* in = nullptr;  // [rows][cols]
  bool in_bf16 = false;
  int rows = 0, cols = 0;
  // launch_norm_quant's
  const float* norm_weight = nullptr;
  float eps = 0.0f;
  float* normalized = nullptr;
  uint8_t* packed = nullptr;
  uint8_t* sf_row_major = nullptr;
  uint8_t* sf_tiled = nullptr;
  int k_tiles = 0;
  float* tensor_scale = nullptr;
  float* inv_rms = nullptr;
  // the gate [experts][cols] and launch_router_topk's
  const void* gate = nullptr;
  bool gate_bf16 = false;
  const float* logit_offset = nullptr;
  const float* bias = nullptr;
  int experts = 0, top_k = 0, n_group = 1, topk_group = 1;
  bool norm_topk_prob = false;
  float routed_scaling = 0.0f;
  float* logits = nullptr;
  int32_t* top_index = nullptr;
  float* top_weight = nullptr;
  // A row tile per selected expert, in expert order, that holds all `rows` tokens in token order: row r
  // of tile i is row 128 * i + r of `dest` (token * dest_stride + slot, -1 where token r did not select
  // the expert) and `row_weight`; `pair_row` [rows][top_k] says where a pair went.
  RowTile* row_tiles = nullptr;
  int32_t* num_row_tiles = nullptr;
  int32_t* dest = nullptr;
  float* row_weight = nullptr;
  int32_t* pair_row = nullptr;
  int dest_stride = 0;
  FrontLinear linear[kFrontLinears];
  int linears = 0;
  int resident_blocks = 0;  // of a launch with linears, on all SMs together
  // front_scratch_bytes(), zero before the first launch; its first kFrontWords words have to be zero again
  // before every other, which is left to the kernel behind (StreamArgs::front_words)
  void* scratch = nullptr;
  int32_t* error = nullptr;
};
constexpr int kFrontWords = kFrontMaxRows + kFrontLinears;
constexpr size_t front_scratch_bytes() {
  return (kFrontWords + 1 + kFrontLinears) * sizeof(int32_t) + 2 * kFrontMaxRows * kFrontMaxExperts * sizeof(float);
}
cudaError_t launch_front(const FrontArgs& args, cudaStream_t stream);
// Whether one launch is the faster front end of `rows` tokens.
bool front_pays(int rows, int experts, int num_sms);

// --- expert-parallel dispatch / return (csrc/ep.cu) ---------------------------
int dispatch_record_bytes(int cols);
cudaError_t launch_dispatch_plan(const int32_t* expert_counts, int experts, int experts_per_rank,
                                 int world, int32_t* send_counts, int32_t* send_offsets,
                                 int32_t* rank_cursor, cudaStream_t stream);
cudaError_t launch_pack_records(const int32_t* top_index, const float* top_weight, int rows,
                                int top_k, int experts_per_rank, const uint8_t* packed,
                                const uint8_t* sf_row_major, const float* tensor_scale, int cols,
                                const int32_t* send_offsets, int32_t* rank_cursor,
                                int capacity /* per destination rank, 0 = compact */,
                                uint8_t* records,
                                const unsigned long long* windows /* nullable: per destination
                                rank, where this rank's segment starts in that rank's memory */,
                                int32_t* send_position, int32_t* error, cudaStream_t stream);
// Peer windows: a step counter on the device, flags raised in other ranks'
// memory (one thread per rank first..first+count-1), and a bounded wait.
cudaError_t launch_window_epoch(uint32_t* epoch, cudaStream_t stream);
cudaError_t launch_window_signal(const unsigned long long* flag_slots,
                                 const unsigned long long* word_slots, const int32_t* words,
                                 const uint32_t* epoch, int first, int count, cudaStream_t stream);
// `limit_ticks`: clock64 ticks after which a waiting thread gives up and records
// kDevWaitTimeout in `error`.
cudaError_t launch_window_wait(const uint32_t* flags, const uint32_t* epoch, int first, int count,
                               long long limit_ticks, int32_t* error, cudaStream_t stream);
cudaError_t launch_record_histogram(const uint8_t* records, int count, int cols,
                                    int local_experts, const int32_t* valid_counts, int capacity,
                                    int32_t* expert_counts, int32_t* error, cudaStream_t stream);
cudaError_t launch_combine_indexed(const void* in, bool in_bf16, const void* returned_rows,
                                   RowKind rows_kind, const int32_t* position,
                                   const void* shared_rows, RowKind shared_kind, int rows,
                                   int hidden, int top_k, void* out, bool out_bf16,
                                   int32_t* error, cudaStream_t stream);

// out[t] = in[t] + ((sum_k parts[t][k]) + parts[t][top_k]) with the routed
// parts (rows of `parts_kind`, [rows][top_k + 1][hidden]) added in slot order.
// `error` (nullable): kDevActivationRange when a binary16 part arrived as an infinity.
cudaError_t launch_combine(const void* in, bool in_bf16, const void* parts, RowKind parts_kind,
                           int rows, int hidden, int top_k, void* out, bool out_bf16,
                           int32_t* error, LaunchStream stream);

}  // namespace nmoe
