// Host side of the C ABI declared in include/nmoe.h: weight upload, scratch,
// tensor maps and the launch sequence of the expert layer.
//
// Mirrors ExpertLayerSlice::Create / ::Run
// (runtime/src/backend/expert_layer.cpp:494-709, :752-1092) with three
// differences that follow from running on the device: all weights are
// uploaded once (the reference keeps host pointers to the routed experts,
// :707), scratch is allocated once for `max_tokens` (the reference allocates
// six tensors per call, :782-787) and nothing synchronises inside Run.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "../../include/nmoe.h"
#include "common.cuh"
#include "kernels.h"

namespace nmoe {
namespace {

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------

struct Failure {
  nmoe_status status;
  std::string message;
};

#define NMOE_CUDA(expr)                                                                    \
  do {                                                                                     \
    const cudaError_t err__ = (expr);                                                      \
    if (err__ != cudaSuccess) {                                                            \
      cudaGetLastError(); /* reported here: it must not fail the next launch as well */    \
      throw Failure{NMOE_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(err__)}; \
    }                                                                                      \
  } while (0)

#define NMOE_REQUIRE(cond, text)                                        \
  do {                                                                  \
    if (!(cond)) throw Failure{NMOE_ERR_INVALID_ARGUMENT, (text)};      \
  } while (0)

class DeviceBuffer {
 public:
  DeviceBuffer() = default;
  DeviceBuffer(const DeviceBuffer&) = delete;
  DeviceBuffer& operator=(const DeviceBuffer&) = delete;
  ~DeviceBuffer() { reset(); }
  void allocate(size_t bytes, bool zero = false) {
    reset();
    if (bytes == 0) bytes = 16;
    NMOE_CUDA(cudaMalloc(&ptr_, bytes));
    bytes_ = bytes;
    if (zero) NMOE_CUDA(cudaMemset(ptr_, 0, bytes_));
  }
  void reset() {
    if (ptr_ != nullptr) cudaFree(ptr_);
    ptr_ = nullptr;
    bytes_ = 0;
  }
  template <typename T>
  T* as() const {
    return reinterpret_cast<T*>(ptr_);
  }
  size_t bytes() const { return bytes_; }

 private:
  void* ptr_ = nullptr;
  size_t bytes_ = 0;
};

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult query;
    NMOE_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &query));
    if (sym == nullptr || query != cudaDriverEntryPointSuccess) {
      throw Failure{NMOE_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver"};
    }
    fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// Packed E2M1 rows viewed as bytes: [rows][row_bytes], box = 128 bytes x
// box_rows, 128-byte swizzle (one box row = one K block of 256 elements).
CUtensorMap make_packed_map(const void* base, size_t rows, size_t row_bytes, int box_rows) {
  NMOE_REQUIRE(reinterpret_cast<uintptr_t>(base) % 16 == 0, "tensor map base must be 16-byte aligned");
  NMOE_REQUIRE(row_bytes % 16 == 0, "packed row pitch must be a multiple of 16 bytes (K % 32 == 0)");
  CUtensorMap map;
  const cuuint64_t dims[2] = {row_bytes, rows};
  const cuuint64_t strides[1] = {row_bytes};
  const cuuint32_t box[2] = {128u, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem_strides[2] = {1u, 1u};
  const CUresult rc = encode_tiled_fn()(
      &map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box,
      elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    throw Failure{NMOE_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(rc)};
  }
  return map;
}

// bf16 rows [rows][cols], box = 64 elements (128 bytes) x box_rows, 128-byte swizzle.
CUtensorMap make_bf16_map(const void* base, size_t rows, size_t cols, int box_rows) {
  NMOE_REQUIRE(reinterpret_cast<uintptr_t>(base) % 16 == 0, "tensor map base must be 16-byte aligned");
  NMOE_REQUIRE((cols * 2) % 16 == 0, "bf16 row pitch must be a multiple of 16 bytes");
  CUtensorMap map;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem_strides[2] = {1u, 1u};
  const CUresult rc = encode_tiled_fn()(
      &map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
      elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    throw Failure{NMOE_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(rc)};
  }
  return map;
}

// Bytes that are already in their shared-memory order, viewed as [rows][1024 B]: box = 1024 bytes x
// box_rows, no swizzle.  The CTA-pair GEMM loads its weight panels through such a map, eight weight
// rows of a K block at a time.
CUtensorMap make_raw_map(const void* base, size_t rows, int box_rows) {
  NMOE_REQUIRE(reinterpret_cast<uintptr_t>(base) % 16 == 0, "tensor map base must be 16-byte aligned");
  CUtensorMap map;
  const cuuint64_t dims[2] = {256u, rows};
  const cuuint64_t strides[1] = {1024u};
  const cuuint32_t box[2] = {256u, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem_strides[2] = {1u, 1u};
  const CUresult rc = encode_tiled_fn()(
      &map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box,
      elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    throw Failure{NMOE_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(rc)};
  }
  return map;
}

int k_blocks_of(int k) { return (k + 255) / 256; }
size_t tiled_sf_bytes(size_t row_slots, int k) { return row_slots * k_blocks_of(k) * 2048; }

// clock64 ticks in `ms` milliseconds at the device's maximum SM clock
long long ticks_from_ms(double ms) {
  int device = 0, khz = 0;
  NMOE_CUDA(cudaGetDevice(&device));
  NMOE_CUDA(cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, device));
  const double ticks = ms * static_cast<double>(khz);
  return ticks < 1.0 ? 1 : static_cast<long long>(ticks);
}

int device_sm_count() {
  int device = 0, sms = 0;
  NMOE_CUDA(cudaGetDevice(&device));
  NMOE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  return sms;
}

void validate_matrix(const nmoe_nvfp4_matrix& m, size_t rows, size_t cols, const char* name) {
  // shape checks of expert_layer.cpp:646-689 plus the byte counts of
  // DequantizeNvfp4Matrix (:162-169) and the 4-byte tensor scale (:189-195)
  const std::string n(name);
  NMOE_REQUIRE(m.output_rows == rows && m.input_cols == cols, n + ": shape mismatch");
  NMOE_REQUIRE(cols % 64 == 0, n + ": input_cols must be a multiple of 64");
  NMOE_REQUIRE(m.packed_data != nullptr && m.packed_nbytes == rows * cols / 2,
               n + ": packed bytes");
  NMOE_REQUIRE(m.block_scales_data != nullptr && m.block_scales_nbytes == rows * (cols / 16),
               n + ": block scale bytes");
  NMOE_REQUIRE(m.tensor_scale_data != nullptr && m.tensor_scale_nbytes == sizeof(float),
               n + ": tensor scale must be one FP32");
}

// ---------------------------------------------------------------------------
// A stack of same-shaped NVFP4 matrices resident in HBM with the scale layouts
// and tensor maps of every GEMM tile shape that may consume it.
// ---------------------------------------------------------------------------
// kClassPair: csrc/gemm.cu, 256 x 208 tiles over CTA pairs, the batches bound by arithmetic.
// kClassStream: csrc/expert_stream.cu, the batches bound by reading the weights.
enum TileClass : int { kClassPair = 0, kClassStream = 1 };

struct WeightStack {
  int experts = 0;
  int n = 0;  // output rows per expert
  int k = 0;  // input cols
  // K-block-major packed weights: every (expert, 256-element K block) is a
  // contiguous [n][128 B] panel, so a weight tile is one contiguous read; the
  // partial last K block lives in `packed_tail` as [experts * n][tail_pitch].
  DeviceBuffer packed;        // [experts][k/256][n][128]
  DeviceBuffer packed_tail;   // [experts][n][tail_pitch]
  int kb_full = 0;
  DeviceBuffer tensor_scale;  // [experts]
  DeviceBuffer sf_stream;     // scale layout for the BN=128 tiles
  DeviceBuffer sf_pair;       // scale layout for the CTA-pair tile
  // tensor maps exist only for the partial last K block; full K blocks are
  // plain bulk copies of contiguous, pre-swizzled panels
  CUtensorMap tail_stream;
  CUtensorMap tail_pair;
  CUtensorMap sf_pair_map;
  CUtensorMap full_pair;  // the K-block-major panels as [rows][1024 B], for the CTA-pair variant

  void upload(const nmoe_nvfp4_matrix* matrices, int count, int rows, int cols,
              const char* name, cudaStream_t stream) {
    experts = count;
    n = rows;
    k = cols;
    const size_t packed_each = static_cast<size_t>(rows) * cols / 2;
    const size_t sf_each = static_cast<size_t>(rows) * (cols / 16);
    tensor_scale.allocate(sizeof(float) * count);
    for (int e = 0; e < count; ++e) validate_matrix(matrices[e], rows, cols, name);
    const GemmTileInfo di = stream_tile_info();
    const size_t sf_stream_each = weight_scale_layout_bytes(1, rows, cols, di.bn, di.sfb_groups);
    const GemmTileInfo qi = pair_tile_info();
    const int pair_rows = qi.b_rows;
    const size_t sf_pair_each = weight_scale_layout_bytes(1, rows, cols, qi.bn, qi.sfb_groups);
    sf_stream.allocate(sf_stream_each * count);
    sf_pair.allocate(sf_pair_each * count);
    sf_pair_map = make_raw_map(sf_pair.as<uint8_t>(), sf_pair_each * count / 1024,
                               qi.sfb_bytes / 1024);
    kb_full = cols / 256;
    const int tail_bytes = (cols % 256) / 2;
    const size_t panel_rows = static_cast<size_t>(count) * rows;
    packed.allocate(panel_rows * kb_full * 128 + 256 * 128, true);  // + one tile of slack: the last
                                                                    // tile of the last panel over-reads
    // The tail map reads `tail_bytes` per row and lets TMA zero-fill the rest of
    // the 128-byte box; if the driver refuses a box wider than the tensor, the
    // tail rows are padded to 128 bytes instead.
    int tail_pitch = tail_bytes;
    bool narrow_tail = tail_bytes > 0;
    if (narrow_tail) {
      packed_tail.allocate(panel_rows * tail_pitch);
      try {
        tail_stream = make_packed_map(packed_tail.as<uint8_t>(), panel_rows, tail_pitch, di.bn);
        tail_pair = make_packed_map(packed_tail.as<uint8_t>(), panel_rows, tail_pitch, pair_rows);
      } catch (const Failure&) {
        narrow_tail = false;
      }
    }
    if (!narrow_tail && tail_bytes > 0) {
      tail_pitch = 128;
      packed_tail.allocate(panel_rows * tail_pitch, true);
      tail_stream = make_packed_map(packed_tail.as<uint8_t>(), panel_rows, tail_pitch, di.bn);
      tail_pair = make_packed_map(packed_tail.as<uint8_t>(), panel_rows, tail_pitch, pair_rows);
    }
    if (tail_bytes == 0) {
      tail_pitch = 16;
      packed_tail.allocate(16);
    }
    // One expert at a time through a staging buffer of one matrix: descriptor bytes
    // (host or device) -> staging -> K-block-major panels and per-tile scale layouts.
    // Copies and kernels share the stream, so the staging buffer is reused in order;
    // no second copy of the whole stack exists and the host waits once, at the end.
    DeviceBuffer staging_packed, staging_sf;
    staging_packed.allocate(packed_each);
    staging_sf.allocate(sf_each);
    const size_t panel_each = static_cast<size_t>(rows) * kb_full * 128;
    const size_t tail_each = static_cast<size_t>(rows) * tail_pitch;
    for (int e = 0; e < count; ++e) {
      NMOE_CUDA(cudaMemcpyAsync(staging_packed.as<void>(), matrices[e].packed_data, packed_each,
                                cudaMemcpyDefault, stream));
      NMOE_CUDA(cudaMemcpyAsync(staging_sf.as<void>(), matrices[e].block_scales_data, sf_each,
                                cudaMemcpyDefault, stream));
      NMOE_CUDA(cudaMemcpyAsync(tensor_scale.as<float>() + e, matrices[e].tensor_scale_data,
                                sizeof(float), cudaMemcpyDefault, stream));
      NMOE_CUDA(relayout_weight_packed(staging_packed.as<uint8_t>(), 1, rows, cols, tail_pitch,
                                       packed.as<uint8_t>() + panel_each * e,
                                       packed_tail.as<uint8_t>() + (tail_bytes > 0 ? tail_each * e : 0),
                                       stream));
      NMOE_CUDA(relayout_weight_scales(staging_sf.as<uint8_t>(), 1, rows, cols, di.bn,
                                       di.sfb_groups, sf_stream.as<uint8_t>() + sf_stream_each * e,
                                       stream));
      NMOE_CUDA(relayout_weight_scales(staging_sf.as<uint8_t>(), 1, rows, cols, qi.bn,
                                       qi.sfb_groups, sf_pair.as<uint8_t>() + sf_pair_each * e,
                                       stream));
    }
    NMOE_CUDA(cudaStreamSynchronize(stream));  // the staging buffers die here
    if (kb_full > 0) {
      full_pair = make_raw_map(packed.as<uint8_t>(), (panel_rows * kb_full + 256) / 8, pair_rows / 8);
    } else {
      full_pair = make_raw_map(packed.as<uint8_t>(), 256 / 8, pair_rows / 8);  // never read
    }
    if (tail_bytes == 0) {
      // never read (k_blocks == kb_full), but the kernel takes a valid map
      tail_stream = make_packed_map(packed.as<uint8_t>(), panel_rows * kb_full, 128, di.bn);
      tail_pair = make_packed_map(packed.as<uint8_t>(), panel_rows * kb_full, 128, pair_rows);
    }
  }

  const CUtensorMap& tail_map(TileClass c) const { return c == kClassPair ? tail_pair : tail_stream; }
  const uint8_t* sf(TileClass c) const {
    return (c == kClassPair ? sf_pair : sf_stream).as<uint8_t>();
  }
  static int tile_cols(TileClass c) {
    return (c == kClassPair ? pair_tile_info() : stream_tile_info()).bn;
  }
};

// Packed activation rows + tiled scales as a GEMM A operand.
struct ActivationOperand {
  const uint8_t* packed = nullptr;
  const uint8_t* sf_tiled = nullptr;
  CUtensorMap boxes[kStreamBoxes];     // 8, 16, 32, 64 and 128 rows
  CUtensorMap pair_boxes[kPairBoxes];  // 16, 32, .. 128 rows
  CUtensorMap sf_map;               // the tiled scales as rows of 1024 bytes
  void bind(const uint8_t* packed_rows, const uint8_t* sf, size_t rows, int k) {
    packed = packed_rows;
    sf_tiled = sf;
    sf_map = make_raw_map(sf, tiled_sf_bytes(rows / 128, k) / 1024, 2);
    for (int i = 0; i < kStreamBoxes; ++i) {
      boxes[i] = make_packed_map(packed_rows, rows, static_cast<size_t>(k) / 2, 8 << i);
    }
    for (int i = 0; i < kPairBoxes; ++i) {
      pair_boxes[i] = make_packed_map(packed_rows, rows, static_cast<size_t>(k) / 2,
                                      kPairBoxRows * (i + 1));
    }
  }
};

GemmMaps gemm_maps(const WeightStack& weights, const ActivationOperand& a) {
  GemmMaps maps;
  for (int i = 0; i < kPairBoxes; ++i) maps.a[i] = a.pair_boxes[i];
  maps.b_tail = weights.tail_map(kClassPair);
  maps.b_full = weights.full_pair;
  maps.sfa = a.sf_map;
  maps.sfb = weights.sf_pair_map;
  return maps;
}

// Which kernel multiplies `rows` rows with one matrix of `n` output features.  A K block of a
// 256 x 208 tile over two SMs takes 1.2 times as long as one of a 128 x 128 tile on one SM (shared
// expert of 16384 tokens: 89 us in 16 waves against 120 in 26): the fewer waves times that.
TileClass dense_tile_class(int rows, int n, int num_sms) {
  if (num_sms < 2) return kClassStream;
  auto waves = [](int tiles, int units) { return (tiles + units - 1) / units; };
  const int stream = waves((rows + 127) / 128 * ((n + 127) / 128), num_sms);
  const int bn = pair_tile_info().bn;
  const int pair = waves((rows + 255) / 256 * ((n + bn - 1) / bn), num_sms / 2);
  return 5 * stream <= 6 * pair ? kClassStream : kClassPair;
}

struct Schedule {
  int most_rows = 128;  // no row tile holds more
  const RowTile* row_tiles = nullptr;  // grouped when non-null
  const int32_t* num_row_tiles = nullptr;
  int dense_rows = 0;
};

// Where the down projection's rows go when they return straight to the ranks
// their records came from (GemmArgs::out_segments).
struct RowSegments {
  const unsigned long long* bases = nullptr;
  int rows = 0;
  int slot0 = 0;
};

// What every GEMM of a tile class takes from its weights, activations and schedule.
GemmArgs gemm_args(const WeightStack& weights, TileClass tile_class, const ActivationOperand& a,
                   const float* a_tensor_scale, const Schedule& schedule, int32_t* error) {
  GemmArgs g;
  const int bn = weights.tile_cols(tile_class);
  g.K = weights.k;
  g.N = weights.n;
  g.n_tiles = (weights.n + bn - 1) / bn;
  g.k_blocks = k_blocks_of(weights.k);
  g.kb_full = weights.kb_full;
  g.b_full = weights.packed.as<uint8_t>();
  g.sfa = a.sf_tiled;
  g.sfb = weights.sf(tile_class);
  g.a_tensor_scale = a_tensor_scale;
  g.w_tensor_scale = weights.tensor_scale.as<float>();
  g.row_tiles = schedule.row_tiles;
  g.num_row_tiles = schedule.num_row_tiles;
  g.dense_rows = schedule.dense_rows;
  g.error = error;
  return g;
}

// The row-storing epilogue's side of a down projection: rows = A x W^T times the tensor scales
// [x routing weight] [-> relu^2], scattered by dest_row.
struct RowOutput {
  void* rows = nullptr;
  RowKind kind = kRowF32;
  const int32_t* dest_row = nullptr;
  int dest_mul = 1;
  int dest_add = 0;
  const float* row_weight = nullptr;
  bool relu2 = false;
  RowSegments segments;
};

void set_row_output(GemmArgs* g, const RowOutput& out) {
  g->out_rows = out.rows;
  g->out_kind = out.kind;
  // (rows in peers' windows lie behind a 256-byte boundary, and N is a multiple of 64)
  g->out_aligned = out.segments.bases != nullptr || reinterpret_cast<uintptr_t>(out.rows) % 32 == 0;
  g->dest_row = out.dest_row;
  g->dest_mul = out.dest_mul;
  g->dest_add = out.dest_add;
  g->row_weight = out.row_weight;
  g->relu2 = out.relu2 ? 1 : 0;
  g->out_segments = out.segments.bases;
  g->segment_rows = out.segments.rows;
  g->segment_slot0 = out.segments.slot0;
}

// The quantising epilogue's side of an up projection.
void set_hidden_output(GemmArgs* g, uint8_t* hidden_packed, uint8_t* hidden_sf) {
  g->out_packed = hidden_packed;
  g->out_sf = hidden_sf;
  g->out_k_blocks = k_blocks_of(g->N);
}

void set_phase(StreamPhase* phase, GemmMode mode, const WeightStack& weights,
               const ActivationOperand& a, const GemmArgs& g) {
  for (int i = 0; i < kStreamBoxes; ++i) phase->a[i] = a.boxes[i];
  phase->b_tail = weights.tail_map(kClassStream);
  phase->gemm = g;
  phase->mode = mode;
}

void run_gemm(GemmMode mode, const WeightStack& weights, TileClass tile_class,
              const ActivationOperand& a, const GemmArgs& g, int most_rows, int num_sms,
              cudaStream_t stream) {
  if (tile_class != kClassStream) {
    NMOE_CUDA(launch_pair_gemm(mode, gemm_maps(weights, a), g, num_sms, stream));
    return;
  }
  StreamArgs args;
  set_phase(&args.phase[0], mode, weights, a, g);
  args.phases = 1;
  args.tile_rows = stream_tile_rows(most_rows);
  args.error = g.error;
  NMOE_CUDA(launch_expert_stream(args, num_sms, stream));
}

void run_down_gemm(const WeightStack& weights, TileClass tile_class, const ActivationOperand& a,
                   const float* a_tensor_scale, const Schedule& schedule, const RowOutput& out,
                   int32_t* error, int num_sms, cudaStream_t stream) {
  GemmArgs d = gemm_args(weights, tile_class, a, a_tensor_scale, schedule, error);
  set_row_output(&d, out);
  run_gemm(kGemmDown, weights, tile_class, a, d, schedule.most_rows, num_sms, stream);
}

// One expert FFN of a launch of csrc/expert_stream.cu: up (relu^2 + quantise, tensor scale 1) ->
// down.  Without `up` the hidden rows are complete before the launch.
struct StreamFfn {
  const WeightStack* up = nullptr;
  const WeightStack* down = nullptr;
  const ActivationOperand* a = nullptr;
  const float* a_tensor_scale = nullptr;
  Schedule schedule;
  uint8_t* hidden_packed = nullptr;
  uint8_t* hidden_sf = nullptr;
  const ActivationOperand* hidden = nullptr;
  const float* hidden_tensor_scale = nullptr;
  RowOutput out;
  const int32_t* used = nullptr;  // StreamPhase::used of the up projection
  int32_t* front_words = nullptr;  // StreamArgs::front_words
  int row_slots = 0;  // most 128-row slots the schedule may use
};

// Row slots' completion counts of such launches; zero whenever no launch is running.
struct StreamCounts {
  DeviceBuffer words;  // CTAs done, the tile ticket, then the counts
  int capacity = 0;
  void allocate(size_t slots) {
    capacity = static_cast<int>(slots);
    words.allocate((slots + 2) * sizeof(int32_t), true);
  }
};

// The shared expert comes first among the up projections and among the down projections: its down
// tiles are the longest, and short ones end together.
void run_stream(const StreamFfn* routed, const StreamFfn* shared, const StreamCounts& counts,
                int32_t* error, int num_sms, LaunchStream stream, int32_t* error_host = nullptr) {
  StreamArgs args;
  args.error_host = error_host;
  args.fetch_dense = stream.chained;
  args.error = error;
  args.finished = counts.words.as<int32_t>();
  args.ticket = counts.words.as<int32_t>() + 1;
  args.ready = counts.words.as<int32_t>() + 2;
  auto add = [&](const StreamFfn& ffn, bool up, int32_t* ready) {
    StreamPhase* phase = &args.phase[args.phases++];
    const WeightStack& weights = up ? *ffn.up : *ffn.down;
    const ActivationOperand& a = up ? *ffn.a : *ffn.hidden;
    GemmArgs g = gemm_args(weights, kClassStream, a, up ? ffn.a_tensor_scale : ffn.hidden_tensor_scale,
                           ffn.schedule, error);
    if (up) {
      set_hidden_output(&g, ffn.hidden_packed, ffn.hidden_sf);
    } else {
      set_row_output(&g, ffn.out);
    }
    set_phase(phase, up ? kGemmUp : kGemmDown, weights, a, g);
    if (up) phase->used = ffn.used;
    if (ffn.up != nullptr) {
      phase->ready = ready;
      if (!up) {
        const int bn = stream_tile_info().bn;
        phase->wait_target = (ffn.up->n + bn - 1) / bn;
      }
    }
  };
  if (routed != nullptr) {
    args.row_tiles = routed->schedule.row_tiles;
    args.row_tile_room = routed->row_slots;
    args.front_words = routed->front_words;
    args.front_word_count = routed->front_words != nullptr ? kFrontWords : 0;
  }
  int32_t* routed_ready = args.ready;
  int32_t* shared_ready = args.ready + (routed != nullptr ? routed->row_slots : 0);
  args.ready_count = (routed != nullptr ? routed->row_slots : 0) +
                     (shared != nullptr ? shared->row_slots : 0);
  NMOE_REQUIRE(args.ready_count <= counts.capacity, "row slots of the fused experts");
  if (shared != nullptr && shared->up != nullptr) add(*shared, true, shared_ready);
  if (routed != nullptr) add(*routed, true, routed_ready);
  if (shared != nullptr) add(*shared, false, shared_ready);
  if (routed != nullptr) add(*routed, false, routed_ready);
  args.tile_rows = stream_tile_rows(std::max(routed != nullptr ? routed->schedule.most_rows : 0,
                                             shared != nullptr ? shared->schedule.most_rows : 0));
  NMOE_CUDA(launch_expert_stream(args, num_sms, stream));
}

// up GEMM (relu^2 + quantise) followed by down GEMM (scale, weight, scatter).
void run_expert_gemms(const WeightStack& up, const WeightStack& down, TileClass tile_class,
                      const ActivationOperand& a, const float* a_tensor_scale,
                      const Schedule& schedule, uint8_t* hidden_packed, uint8_t* hidden_sf,
                      const ActivationOperand& hidden, const RowOutput& out, int32_t* error,
                      int num_sms, cudaStream_t stream, cudaEvent_t between = nullptr) {
  GemmArgs g = gemm_args(up, tile_class, a, a_tensor_scale, schedule, error);
  set_hidden_output(&g, hidden_packed, hidden_sf);
  run_gemm(kGemmUp, up, tile_class, a, g, schedule.most_rows, num_sms, stream);
  if (between != nullptr) cudaEventRecord(between, stream);
  // the fused quantiser always uses tensor scale 1
  run_down_gemm(down, tile_class, hidden, nullptr, schedule, out, error, num_sms, stream);
}

nmoe_status status_from_device(int code) {
  switch (code) {
    case kDevOk: return NMOE_OK;
    case kDevWaitTimeout: return NMOE_ERR_DEVICE_TIMEOUT;
    case kDevActivationRange: return NMOE_ERR_ACTIVATION_RANGE;
    case kDevPlanOverflow: return NMOE_ERR_CAPACITY;
    default: return NMOE_ERR_CUDA;
  }
}

// Hands the error word to the host and clears it: one launch in the place of a copy and a memset,
// whose start-up a synchronous call over few rows waits for (64 rows through one expert, measured on
// the host: 60.6 us with them, 50.7 so, 40.7 where the last CTA of the FFN's launch leaves an
// error with the host by itself).
__global__ void publish_error_kernel(int32_t* device, volatile int32_t* host) {
  *host = atomicExch(device, 0);
  __threadfence_system();
}

struct ErrorSlot {
  DeviceBuffer device;
  int32_t* host = nullptr;  // pinned, written by publish_error_kernel or a launch's last CTA
  void create() {
    device.allocate(sizeof(int32_t), true);
    NMOE_CUDA(cudaMallocHost(&host, sizeof(int32_t)));
    *host = 0;
  }
  ~ErrorSlot() {
    if (host != nullptr) cudaFreeHost(host);
  }
  // `published`: what ran last has left its word with the host, if there is one.
  nmoe_status sync(cudaStream_t stream, bool published = false) {
    if (published) {
      NMOE_CUDA(cudaStreamSynchronize(stream));
      if (*static_cast<volatile int32_t*>(host) == kDevOk) return NMOE_OK;
    }
    publish_error_kernel<<<1, 1, 0, stream>>>(device.as<int32_t>(), host);
    NMOE_CUDA(cudaGetLastError());
    NMOE_CUDA(cudaStreamSynchronize(stream));
    const int code = *static_cast<volatile int32_t*>(host);
    *host = kDevOk;
    return status_from_device(code);
  }
};

// Un-tile block scales of selected rows into row-major order (trace export).
__global__ void export_rows_kernel(const uint8_t* __restrict__ packed,
                                   const uint8_t* __restrict__ sf_tiled,
                                   const int32_t* __restrict__ row_of, int count, int cols,
                                   int k_tiles, uint8_t* __restrict__ out_packed,
                                   uint8_t* __restrict__ out_sf) {
  const int i = blockIdx.x;
  if (i >= count) return;
  const int row = row_of != nullptr ? row_of[i] : i;
  if (out_packed != nullptr) {
    for (int b = threadIdx.x; b < cols / 2; b += blockDim.x) {
      out_packed[static_cast<size_t>(i) * (cols / 2) + b] =
          packed[static_cast<size_t>(row) * (cols / 2) + b];
    }
  }
  if (out_sf != nullptr) {
    for (int b = threadIdx.x; b < cols / 16; b += blockDim.x) {
      out_sf[static_cast<size_t>(i) * (cols / 16) + b] =
          sf_tiled[swizzled_scale_offset(row, b, k_tiles)];
    }
  }
}

__global__ void widen_bf16_kernel(const __nv_bfloat16* __restrict__ in, size_t count,
                                  float* __restrict__ out) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    out[i] = __bfloat162float(in[i]);
  }
}

// ReadVectorWeightToHostFp32 / UploadVectorWeightToDeviceFp32 and the dense
// upload of linear_op.cpp:274-303: FP32 as is, bf16 widened.
void upload_dense_fp32(const nmoe_dense_tensor& t, size_t count, const char* name,
                       DeviceBuffer* out, cudaStream_t stream) {
  NMOE_REQUIRE(t.data != nullptr, std::string(name) + ": null data");
  NMOE_REQUIRE(t.rows * t.cols == count, std::string(name) + ": shape mismatch");
  out->allocate(count * sizeof(float));
  if (t.dtype == NMOE_F32) {
    NMOE_REQUIRE(t.nbytes == count * 4, std::string(name) + ": byte count");
    NMOE_CUDA(cudaMemcpyAsync(out->as<float>(), t.data, count * 4, cudaMemcpyDefault, stream));
  } else {
    NMOE_REQUIRE(t.nbytes == count * 2, std::string(name) + ": byte count");
    DeviceBuffer staging;
    staging.allocate(count * 2);
    NMOE_CUDA(cudaMemcpyAsync(staging.as<void>(), t.data, count * 2, cudaMemcpyDefault, stream));
    widen_bf16_kernel<<<stride_blocks(count, 256), 256, 0, stream>>>(staging.as<__nv_bfloat16>(), count, out->as<float>());
    NMOE_CUDA(cudaGetLastError());
    NMOE_CUDA(cudaStreamSynchronize(stream));
  }
}

// A weight of a correctly rounded linear, with its slices where the integer kernel may run.
struct ExactOperand {
  ExactWeight w;
  DeviceBuffer slices, info;
  void bind(const void* weight, int kind, float scale, int n, int k) {
    w.N = n;
    w.K = k;
    w.kind = kind;
    w.weight = weight;
    w.scale = scale;
  }
  void slice(cudaStream_t stream) {
    if (w.slices != nullptr) return;
    slices.allocate(slice_bytes(w.N, w.K, exact_weight_tile_rows()), true);
    info.allocate(static_cast<size_t>(w.N) * sizeof(SliceRow));
    NMOE_CUDA(launch_slice_weights(w.weight, w.kind, w.scale, w.N, w.K, slices.as<int8_t>(),
                                   info.as<SliceRow>(), stream));
    w.slices = slices.as<int8_t>();
    w.info = info.as<SliceRow>();
  }
};

// A dense or scaled-FP8 linear resident in HBM in the format it came in, with its fixed-point slices
// (those of one with codes as soon as the unfused path is on, which alone reads them); the values that count are FP32 [out][in], what the reference's UploadedLinearOp /
// ScaledFp8LinearOp multiply with (linear_op.cpp:274-303, scaled_fp8_linear.cu:121-139).
// Contractions too long for the slices keep the FP32 matrix itself.
struct DenseLinear {
  bool present = false;
  bool fp8 = false;
  bool exact = false;
  int out = 0, in = 0;
  float input_scale = 1.0f;
  DeviceBuffer weight;
  ExactOperand operand;
  CodedWeight coded;  // FP8 weights whose rows are only quantised again
  DeviceBuffer coded_slices, coded_norm;

  void slice(cudaStream_t stream) {
    if (present && exact) operand.slice(stream);
  }

  void prepare_coded(cudaStream_t stream) {
    if (!fp8 || !exact || !coded_supported(out, in, operand.w.scale) ||
        clamp_scale_host(input_scale) > 0x1p60f) {
      return;
    }
    coded_slices.allocate(coded_slice_bytes(out, in, coded_weight_tile_rows()), true);
    coded_norm.allocate(static_cast<size_t>(out) * sizeof(float));
    NMOE_CUDA(launch_code_weights(weight.as<void>(), out, in, coded_slices.as<int8_t>(),
                                  coded_norm.as<float>(), stream));
    coded.N = out;
    coded.K = in;
    coded.weight = weight.as<void>();
    coded.scale = operand.w.scale;
    coded.norm = coded_norm.as<float>();
    coded.slices = coded_slices.as<int8_t>();
  }

  void upload(const nmoe_linear& linear, size_t out_rows, size_t in_cols, const char* name,
              cudaStream_t stream) {
    const std::string n(name);
    out = static_cast<int>(out_rows);
    in = static_cast<int>(in_cols);
    exact = exact_supported(out, in);
    const size_t count = out_rows * in_cols;
    if (linear.family == NMOE_LINEAR_DENSE) {
      const nmoe_dense_tensor& t = linear.weight;
      NMOE_REQUIRE(t.rows == out_rows && t.cols == in_cols, n + ": shape mismatch");
      if (!exact || t.dtype == NMOE_F32) {
        upload_dense_fp32(t, count, name, &weight, stream);
        if (exact) operand.bind(weight.as<void>(), kWeightF32, 1.0f, out, in);
      } else {
        NMOE_REQUIRE(t.data != nullptr && t.nbytes == count * 2, n + ": byte count");
        weight.allocate(count * 2);
        NMOE_CUDA(cudaMemcpyAsync(weight.as<void>(), t.data, count * 2, cudaMemcpyDefault, stream));
        operand.bind(weight.as<void>(), kWeightBf16, 1.0f, out, in);
      }
    } else if (linear.family == NMOE_LINEAR_SCALED_FP8) {
      // DequantizeScaledFp8WeightToHostFp32 (scaled_fp8_linear.cu:121-139)
      NMOE_REQUIRE(linear.weight.data != nullptr && linear.weight.nbytes == count &&
                       linear.weight.rows == out_rows && linear.weight.cols == in_cols,
                   n + ": FP8 weight bytes");
      NMOE_REQUIRE(linear.weight_scale > 0.0f && linear.weight_scale < 3.0e38f,
                   n + ": weight_scale must be finite and positive");
      fp8 = true;
      input_scale = linear.input_scale;
      if (exact) {
        weight.allocate(count);
        NMOE_CUDA(cudaMemcpyAsync(weight.as<void>(), linear.weight.data, count, cudaMemcpyDefault,
                                  stream));
        operand.bind(weight.as<void>(), kWeightFp8, linear.weight_scale, out, in);
      } else {
        DeviceBuffer staging;
        staging.allocate(count);
        NMOE_CUDA(cudaMemcpyAsync(staging.as<void>(), linear.weight.data, count, cudaMemcpyDefault,
                                  stream));
        weight.allocate(count * sizeof(float));
        NMOE_CUDA(launch_fp8_weight_dequant(staging.as<uint8_t>(), count, linear.weight_scale,
                                            weight.as<float>(), stream));
        NMOE_CUDA(cudaStreamSynchronize(stream));
      }
    } else {
      throw Failure{NMOE_ERR_INVALID_ARGUMENT, n + ": unknown linear family"};
    }
    present = true;
  }
};

// Workspace of the linears that run one after the other on a stream.  Of the correctly rounded ones:
// sliced activation rows (up to `max_rows` at a time; longer batches go through in turn) and the partial
// sums.  Of scaled-FP8 ones with contractions too long for that: the rows after their round trip.
struct ExactScratch {
  int max_rows = 0;
  size_t most_n = 0, most_k = 0;  // of the exact linears it has room for
  DeviceBuffer slices, info, partial;
  DeviceBuffer round_trip;  // [tokens][in] FP32
  // `shapes`: (N, K) of every linear that will run
  void allocate(size_t tokens, const std::vector<std::pair<int, int>>& shapes, int num_sms) {
    max_rows = static_cast<int>(std::min<size_t>(tokens, 1024));
    most_n = most_k = 0;
    size_t n = 0, k = 0;
    for (const auto& shape : shapes) {
      n = std::max<size_t>(n, shape.first);
      k = std::max<size_t>(k, shape.second);
    }
    if (shapes.empty()) return;
    // (rows come in tiles of up to 64)
    slices.allocate(slice_bytes(max_rows, static_cast<int>(k), 64));
    info.allocate(max_rows * sizeof(SliceRow));
    // a split contraction has at most one tile of 128 x 80 sums per SM
    partial.allocate(std::max(max_rows * n, static_cast<size_t>(num_sms) * 128 * 80) *
                     sizeof(double));
    most_n = n;
    most_k = k;
  }
  bool holds(const ExactWeight& w) const {
    return static_cast<size_t>(w.N) <= most_n && static_cast<size_t>(w.K) <= most_k;
  }
  void allocate_round_trip(size_t tokens, const DenseLinear& linear) {
    if (!linear.fp8 || linear.exact) return;
    round_trip.allocate(tokens * static_cast<size_t>(linear.in) * sizeof(float));
  }
};

void run_exact(const ExactWeight& w, ExactScratch& scratch, const float* in, float fp8_scale,
               int rows, const float* offset, bool relu2, float* out, int32_t* error, int num_sms,
               LaunchStream stream) {
  if (exact_prefers_gemv(rows, w.N, w.K, num_sms)) {
    NMOE_CUDA(launch_exact_gemv(w, in, fp8_scale, rows, offset, relu2, out, num_sms, stream));
    return;
  }
  NMOE_REQUIRE(w.slices != nullptr && scratch.holds(w),
               "an exact linear without its slices or its workspace");
  for (int first = 0; first < rows; first += scratch.max_rows) {
    const int count = std::min(rows - first, scratch.max_rows);
    const float* from = in + static_cast<size_t>(first) * w.K;
    const ExactWorkspace space{scratch.slices.as<int8_t>(), scratch.info.as<SliceRow>(),
                               scratch.partial.as<double>()};
    NMOE_CUDA(launch_exact_linear(w, from, count, fp8_scale, offset, relu2, space,
                                  out + static_cast<size_t>(first) * w.N, error, num_sms, stream));
  }
}

}  // namespace
}  // namespace nmoe

using namespace nmoe;

// ===========================================================================
// nmoe_ffn
// ===========================================================================
struct nmoe_ffn {
  int hidden = 0;
  int inter = 0;
  int max_rows = 0;
  int num_sms = 0;
  WeightStack up, down;
  DeviceBuffer a_packed, a_sf, a_ts, h_packed, h_sf;
  ActivationOperand a_op, h_op;
  StreamCounts stream_counts;
  ErrorSlot error;
  int last_rows = 0;
  bool status_published = false;  // the last launch leaves its error word with the host
  bool pair_captured = false;     // a launch that does not is in a graph and may run at any time
  std::string last_error;
};

// Whether what is launched on `stream` goes into a graph.
static bool is_captured(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) == cudaSuccess) {
    return status != cudaStreamCaptureStatusNone;
  }
  cudaGetLastError();  // (the legacy stream, beside a capture on another one)
  return false;
}

extern "C" {

const char* nmoe_status_string(nmoe_status status) {
  switch (status) {
    case NMOE_OK: return "ok";
    case NMOE_ERR_INVALID_ARGUMENT: return "invalid argument";
    case NMOE_ERR_CUDA: return "CUDA error";
    case NMOE_ERR_UNSUPPORTED: return "unsupported configuration";
    case NMOE_ERR_DEVICE_TIMEOUT: return "a device-side wait timed out";
    case NMOE_ERR_ACTIVATION_RANGE: return "activated row exceeds the NVFP4 range for tensor scale 1";
    case NMOE_ERR_CAPACITY: return "token or row-tile capacity exceeded";
  }
  return "unknown status";
}

nmoe_status nmoe_ffn_create(const nmoe_nvfp4_matrix* up, const nmoe_nvfp4_matrix* down,
                            int32_t max_rows, nmoe_ffn** out_ffn) {
  if (up == nullptr || down == nullptr || out_ffn == nullptr || max_rows <= 0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  *out_ffn = nullptr;
  std::unique_ptr<nmoe_ffn> f(new (std::nothrow) nmoe_ffn);
  if (!f) return NMOE_ERR_CUDA;
  try {
    f->hidden = static_cast<int>(up->input_cols);
    f->inter = static_cast<int>(up->output_rows);
    f->max_rows = max_rows;
    f->num_sms = device_sm_count();
    cudaStream_t stream = nullptr;
    f->up.upload(up, 1, f->inter, f->hidden, "up_proj", stream);
    f->down.upload(down, 1, f->hidden, f->inter, "down_proj", stream);
    const size_t slots = (static_cast<size_t>(max_rows) + 127) / 128;
    f->a_packed.allocate(slots * 128 * f->hidden / 2, true);
    f->a_sf.allocate(tiled_sf_bytes(slots, f->hidden), true);
    f->a_ts.allocate(slots * 128 * sizeof(float), true);
    f->h_packed.allocate(slots * 128 * f->inter / 2, true);
    f->h_sf.allocate(tiled_sf_bytes(slots, f->inter), true);
    f->a_op.bind(f->a_packed.as<uint8_t>(), f->a_sf.as<uint8_t>(), slots * 128, f->hidden);
    f->h_op.bind(f->h_packed.as<uint8_t>(), f->h_sf.as<uint8_t>(), slots * 128, f->inter);
    f->stream_counts.allocate(slots);
    f->error.create();
    NMOE_CUDA(cudaDeviceSynchronize());
  } catch (const Failure& failure) {
    std::fprintf(stderr, "nmoe_ffn_create: %s\n", failure.message.c_str());
    return failure.status;
  }
  *out_ffn = f.release();
  return NMOE_OK;
}

void nmoe_ffn_destroy(nmoe_ffn* ffn) { delete ffn; }

nmoe_status nmoe_ffn_run(nmoe_ffn* ffn, void* stream_ptr, const void* input,
                         nmoe_dtype input_dtype, int64_t rows, float* output,
                         int32_t gemm_variant) {
  if (ffn == nullptr || input == nullptr || output == nullptr || rows <= 0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  if (rows > ffn->max_rows) return NMOE_ERR_CAPACITY;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  try {
    // (2 was a kernel for few rows; the streaming kernel behind it now has no such limit)
    if (gemm_variant == 2 && rows > 32) return NMOE_ERR_INVALID_ARGUMENT;
    const TileClass tile_class =
        gemm_variant == 1 || gemm_variant == 4 ? kClassPair
        : gemm_variant != 0                    ? kClassStream
                            : dense_tile_class(static_cast<int>(rows), ffn->inter, ffn->num_sms);
    NMOE_CUDA(launch_norm_quant(input, input_dtype == NMOE_BF16, static_cast<int>(rows),
                                ffn->hidden, nullptr, 0.0f, nullptr, ffn->a_packed.as<uint8_t>(),
                                nullptr, ffn->a_sf.as<uint8_t>(), k_blocks_of(ffn->hidden),
                                ffn->a_ts.as<float>(), ffn->num_sms, stream));
    Schedule schedule;
    schedule.dense_rows = static_cast<int>(rows);
    schedule.most_rows = std::min(128, static_cast<int>(rows));
    RowOutput out;
    out.rows = output;
    int32_t* error = ffn->error.device.as<int32_t>();
    if (tile_class == kClassStream) {
      StreamFfn both;
      both.up = &ffn->up;
      both.down = &ffn->down;
      both.a = &ffn->a_op;
      both.a_tensor_scale = ffn->a_ts.as<float>();
      both.schedule = schedule;
      both.hidden_packed = ffn->h_packed.as<uint8_t>();
      both.hidden_sf = ffn->h_sf.as<uint8_t>();
      both.hidden = &ffn->h_op;
      both.out = out;
      both.row_slots = (static_cast<int>(rows) + 127) / 128;
      run_stream(nullptr, &both, ffn->stream_counts, error, ffn->num_sms,
                 LaunchStream(stream, true), ffn->error.host);
    } else {
      run_expert_gemms(ffn->up, ffn->down, tile_class, ffn->a_op, ffn->a_ts.as<float>(), schedule,
                       ffn->h_packed.as<uint8_t>(), ffn->h_sf.as<uint8_t>(), ffn->h_op, out, error,
                       ffn->num_sms, stream);
      ffn->pair_captured = ffn->pair_captured || is_captured(stream);
    }
    ffn->last_rows = static_cast<int>(rows);
    ffn->status_published = tile_class == kClassStream;
  } catch (const Failure& failure) {
    ffn->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_ffn_sync_status(nmoe_ffn* ffn, void* stream_ptr) {
  if (ffn == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  try {
    // (the host knows what it launched last, not which graph it replayed since)
    return ffn->error.sync(static_cast<cudaStream_t>(stream_ptr),
                           ffn->status_published && !ffn->pair_captured);
  } catch (const Failure& failure) {
    ffn->last_error = failure.message;
    return failure.status;
  }
}

nmoe_status nmoe_ffn_export_hidden(nmoe_ffn* ffn, void* stream_ptr, uint8_t* packed,
                                   uint8_t* scales) {
  if (ffn == nullptr || ffn->last_rows <= 0) return NMOE_ERR_INVALID_ARGUMENT;
  export_rows_kernel<<<ffn->last_rows, 128, 0, static_cast<cudaStream_t>(stream_ptr)>>>(
      ffn->h_packed.as<uint8_t>(), ffn->h_sf.as<uint8_t>(), nullptr, ffn->last_rows, ffn->inter,
      k_blocks_of(ffn->inter) * 4, packed, scales);
  return cudaGetLastError() == cudaSuccess ? NMOE_OK : NMOE_ERR_CUDA;
}

}  // extern "C"

// ===========================================================================
// nmoe_layer
// ===========================================================================
enum { kStageCount = NMOE_STAGE_COUNT };

struct nmoe_layer {
  nmoe_config cfg{};
  int num_sms = 0;
  int local_experts = 0;
  int first_local_expert = 0;
  int max_row_tiles = 0;

  DeviceBuffer norm_weight, gate, bias, logit_offset;
  ExactOperand gate_exact;  // the router's FP64 logits of small batches
  bool has_gate_exact = false;
  ExactScratch exact;              // of the linears on the caller's stream
  ExactScratch fc1_exact, up_exact;  // of fc1_latent and shared_up, which may run beside them
  bool has_logit_offset = false;
  // two-pass router (tensor-core logits + FP64 re-evaluation of near-ties)
  bool fast_router = false;
  int fast_router_min_tokens = 256;
  float router_tie_margin = 2.0e-4f;
  DeviceBuffer gate_bf16, inv_rms;
  CUtensorMap gate_map;
  // bf16 inputs: the norm weight folded into the gate as three bf16 planes, and the map of
  // the last input the layer saw (its address and row count are part of the map)
  DeviceBuffer gate_planes;
  CUtensorMap planes_map;
  bool folded_router = false;
  CUtensorMap input_map;
  const void* input_map_base = nullptr;
  int input_map_rows = 0;
  // The FP32 normalised rows are needed by the FP64 logits kernel of small batches,
  // by the dense / scaled-FP8 linears and by the trace; the two-pass router of large
  // batches rebuilds them on the fly, so they are only written there while a trace may
  // be asked for (nmoe_layer_keep_trace).
  bool keep_trace = true;
  WeightStack up, down, shared_up, shared_down;

  // Latent projections and the dense / scaled-FP8 families (fc1_latent, fc2_latent,
  // shared_up, shared_down of expert_layer.cpp:534-617).  `latent` is the row length
  // the routed experts see; without projections it is the hidden size.
  int latent = 0;
  bool latent_mode = false;
  DenseLinear fc1, fc2, shared_up_dense, shared_down_dense;
  // fc1 output and its NVFP4 form
  DeviceBuffer latent_rows, lat_packed, lat_sf_row_major, lat_sf_tiled, lat_ts;
  DeviceBuffer routed_latent, projected, shared_rows;               // [T][latent], [T][H], [T][H]
  DeviceBuffer shared_raw;  // [T][S] FP32: shared_up output, activated in place
  DeviceBuffer sh_ts;       // per-row tensor scale of the quantised shared intermediate

  // The unfused activation path (nmoe_layer_set_unfused_activation): the up
  // projection's rows stay FP32 and are quantised in a pass of their own.
  bool unfused = false;
  DeviceBuffer u_raw, h_ts, unweighted_rows;
  int unweighted_tokens = 0;  // the unweighted down rows are kept for up to this many tokens

  // token-order scratch
  DeviceBuffer normalized, logits, top_index, top_weight;
  DeviceBuffer y_packed, y_sf_row_major, y_sf_tiled, y_ts;
  DeviceBuffer sh_packed, sh_sf;
  DeviceBuffer parts;
  // plan
  DeviceBuffer counts, cursor, position, row_tiles, num_row_tiles, pair_row;
  // expert-sorted scratch
  DeviceBuffer a_packed, a_sf, a_ts, a_weight, a_dest, h_packed, h_sf;

  // expert parallelism
  int ep_world = 1;
  int ep_rank = 0;
  int64_t max_pairs = 0;
  int64_t send_record_slots = 0;
  int record_bytes = 0;
  DeviceBuffer send_records, send_position, send_counts, send_offsets, rank_cursor, shared_out;

  // Peer window (nmoe_ep_window_*): one allocation per rank that the other
  // ranks map and write into: [records][returned rows][flags and counts].
  struct PeerWindow {
    bool attached = false;
    int64_t capacity = 0;  // pairs per (source rank, destination rank)
    RowKind rows_kind = kRowF16;
    DeviceBuffer local;
    size_t records_off = 0, rows_off = 0, flags_off = 0;
    std::vector<void*> peer_base;  // opened mappings, nullptr for this rank
    // u64[world] tables on the device: where this rank writes in rank r's window
    DeviceBuffer record_segments, row_segments, record_flag_slots, row_flag_slots, count_slots;
    DeviceBuffer epoch;  // uint32 step counter
    uint32_t* record_flags() const { return reinterpret_cast<uint32_t*>(local.as<uint8_t>() + flags_off); }
    uint32_t* row_flags() const { return record_flags() + 64; }
    int32_t* counts() const { return reinterpret_cast<int32_t*>(record_flags() + 128); }
    void close_peers() {
      for (void*& base : peer_base) {
        if (base != nullptr) cudaIpcCloseMemHandle(base);
        base = nullptr;
      }
      attached = false;
    }
  } window;

  ActivationOperand y_op, lat_op, sh_op, a_op, h_op;
  StreamCounts stream_counts;
  DeviceBuffer front_scratch, front_rounded;  // of csrc/front.cu
  bool front_words_set = false;  // a front end was launched, and nothing behind it that clears its words
  ErrorSlot error;
  int last_tokens = 0;
  std::string last_error;
  RowKind last_parts_kind = kRowF32;
  bool last_unfused = false;
  bool last_normalized = true;
  bool force_fp32_parts = false;  // NMOE_PARTS_FP32=1: FP32 rows whatever the output type
  // how long a kernel waits for a flag another GPU raises before it gives up with
  // kDevWaitTimeout (clock64 ticks; nmoe_layer_set_wait_limit_ms, NMOE_WAIT_LIMIT_MS)
  long long wait_limit_ticks = 1ll << 34;
  DeviceBuffer probe_epoch;  // nmoe_layer_wait_flag

  // Small batches: the shared expert runs on a stream of the layer's own beside the
  // router, plan and permute kernels (it needs only the quantised rows) and joins
  // before the combine.  Its GEMMs use a few dozen SMs at these sizes.
  cudaStream_t side_stream = nullptr;
  cudaEvent_t quant_done = nullptr, shared_done = nullptr;
  int fork_max_tokens = 1 << 30;  // (NMOE_FORK_MAX_TOKENS)
  // Latent layers: fc1_latent and its quantiser run on one more stream beside the router.
  cudaStream_t latent_stream = nullptr;
  cudaEvent_t latent_done = nullptr;
  bool window_fork_shared = false;    // nmoe_ep_window_fork_shared
  bool window_shared_pending = false;
  RowKind window_shared_kind = kRowF32;  // type of shared_out for the pending combine

  // Small batches are bound by launch overhead: the whole run is recorded once per
  // (token count, buffers, types) as a CUDA graph and replayed afterwards.
  // NMOE_GRAPH_MAX_TOKENS sets the largest batch handled this way (0 = never).
  struct RecordedRun {
    const void* input;
    void* output;
    int tokens;
    int in_dtype, out_dtype;
    RowKind parts_kind;
    bool normalized;
    cudaGraphExec_t exec;  // null while the run is not worth recording yet
    uint64_t last_use;
    int eager_runs = 0;
  };
  std::vector<RecordedRun> recorded;
  int graph_max_tokens = 256;
  uint64_t run_counter = 0;
  void drop_recorded() {
    for (RecordedRun& r : recorded) {
      if (r.exec != nullptr) cudaGraphExecDestroy(r.exec);
    }
    recorded.clear();
  }

  // optional per-stage CUDA events (nmoe_layer_enable_stage_timing)
  bool stage_timing = false;
  cudaEvent_t stage_events[kStageCount + 1] = {};
  ~nmoe_layer() {
    drop_recorded();
    window.close_peers();
    if (quant_done != nullptr) cudaEventDestroy(quant_done);
    if (shared_done != nullptr) cudaEventDestroy(shared_done);
    if (latent_done != nullptr) cudaEventDestroy(latent_done);
    if (side_stream != nullptr) cudaStreamDestroy(side_stream);
    if (latent_stream != nullptr) cudaStreamDestroy(latent_stream);
    for (cudaEvent_t e : stage_events)
      if (e != nullptr) cudaEventDestroy(e);
  }
  void mark(int index, cudaStream_t stream) {
    if (stage_timing) cudaEventRecord(stage_events[index], stream);
  }
};

namespace {

// Whether some call of up to `T` rows takes the gate through the integer kernel.  In front of the
// two-pass router only batches too small for it reach the gate: up to 255 rows of 128 x 2688 stay
// with the FP64 kernels, and such a layer needs 25 MB less.
bool gate_needs_slices(const nmoe_layer* L, size_t T) {
  const int most_rows = L->fast_router
                            ? std::min(static_cast<int>(T), L->fast_router_min_tokens - 1)
                            : static_cast<int>(T);
  return L->has_gate_exact &&
         !exact_prefers_gemv(most_rows, L->cfg.n_routed_experts, L->cfg.hidden_size, L->num_sms);
}

// Slices of the gate and the workspace of the exact linears on the caller's stream, for calls of up to `T`
// rows.
void allocate_exact(nmoe_layer* L, size_t T) {
  std::vector<std::pair<int, int>> linears;
  if (gate_needs_slices(L, T)) {
    L->gate_exact.slice(nullptr);
    linears.emplace_back(L->cfg.n_routed_experts, L->cfg.hidden_size);
  }
  for (const DenseLinear* linear : {&L->fc2, &L->shared_down_dense}) {
    if (linear->present && linear->exact) linears.emplace_back(linear->out, linear->in);
  }
  L->exact.allocate(T, linears, device_sm_count());
}

// ... and of those that may run beside it.
void allocate_exact_beside(nmoe_layer* L, size_t T) {
  const int sms = device_sm_count();
  if (L->fc1.present && L->fc1.exact) L->fc1_exact.allocate(T, {{L->fc1.out, L->fc1.in}}, sms);
  if (L->shared_up_dense.present && L->shared_up_dense.exact) {
    if (L->shared_up_dense.coded.slices == nullptr || L->unfused) L->shared_up_dense.slice(nullptr);
    L->up_exact.allocate(T, {{L->shared_up_dense.out, L->shared_up_dense.in}}, sms);
  }
}

// Everything whose size follows the token capacity.  Called at creation and by
// nmoe_layer_reserve_tokens; weights are not touched.
void allocate_scratch(nmoe_layer* L, size_t T) {
  L->drop_recorded();  // recorded runs hold the old buffers' addresses
  const nmoe_config& c = L->cfg;
  const int H = c.hidden_size, I = c.routed_expert_intermediate_size,
            S = c.shared_expert_intermediate_size, E = c.n_routed_experts, K = c.top_k;
  const int EL = L->local_experts, Lr = L->latent;
  const size_t token_slots = (T + 127) / 128;
  L->inv_rms.allocate(T * sizeof(float));
  L->normalized.allocate(T * H * sizeof(float));
  // (a split router pass 1 keeps several partial sums per logit)
  L->logits.allocate((L->fast_router ? router_pass1_rows(T, device_sm_count()) : T) * E * sizeof(float));
  L->top_index.allocate(T * K * sizeof(int32_t));
  L->top_weight.allocate(T * K * sizeof(float));
  L->y_packed.allocate(token_slots * 128 * H / 2, true);
  L->y_sf_row_major.allocate(T * (H / 16));
  L->y_sf_tiled.allocate(tiled_sf_bytes(token_slots, H), true);
  L->y_ts.allocate(token_slots * 128 * sizeof(float), true);
  L->sh_packed.allocate(token_slots * 128 * S / 2, true);
  L->sh_sf.allocate(tiled_sf_bytes(token_slots, S), true);
  L->sh_ts.allocate(token_slots * 128 * sizeof(float), true);
  if (L->latent_mode) {
    L->latent_rows.allocate(T * Lr * sizeof(float));
    L->lat_packed.allocate(token_slots * 128 * Lr / 2, true);
    L->lat_sf_tiled.allocate(tiled_sf_bytes(token_slots, Lr), true);
    L->lat_sf_row_major.allocate(T * (Lr / 16));
    L->lat_ts.allocate(token_slots * 128 * sizeof(float), true);
    L->routed_latent.allocate(T * Lr * sizeof(float));
    L->projected.allocate(T * H * sizeof(float));
    L->shared_rows.allocate(T * H * sizeof(float));
  }
  if (L->shared_up_dense.present || L->shared_down_dense.present || L->unfused) {
    L->shared_raw.allocate(T * S * sizeof(float));
  }
  allocate_exact(L, T);
  allocate_exact_beside(L, T);
  L->fc1_exact.allocate_round_trip(T, L->fc1);
  L->up_exact.allocate_round_trip(T, L->shared_up_dense);
  L->exact.allocate_round_trip(T, L->shared_down_dense);
  if (L->ep_world == 1) {
    L->parts.allocate(T * (K + 1) * static_cast<size_t>(std::max(H, Lr)) * sizeof(float));
  }

  // Row tiles: every expert may leave one partly filled slot of 128 rows.
  // With expert parallelism the rows come from every rank: the capacity is
  // max_recv_pairs (default: twice the local pairs, i.e. 2x the uniform share).
  const size_t local_pairs = T * K;
  const size_t pairs = L->ep_world == 1 ? local_pairs
                       : c.max_recv_pairs > 0 ? static_cast<size_t>(c.max_recv_pairs)
                                              : 2 * local_pairs;
  L->max_pairs = static_cast<int64_t>(pairs);
  // (an expert may leave a partly filled slot, and an empty one when pairs consume them)
  L->max_row_tiles = static_cast<int>(2 * static_cast<size_t>(EL) + (pairs + 127) / 128);
  L->stream_counts.allocate(L->max_row_tiles + token_slots);
  L->front_scratch.allocate(front_scratch_bytes(), true);
  if (L->latent_mode) {
    L->front_rounded.allocate(static_cast<size_t>(kFrontLinears) * H * sizeof(float));
  }
  const size_t slots = static_cast<size_t>(L->max_row_tiles);
  L->counts.allocate(E * sizeof(int32_t), true);
  L->cursor.allocate(E * sizeof(int32_t), true);
  L->position.allocate(T * K * sizeof(int32_t), true);
  L->row_tiles.allocate(slots * sizeof(RowTile), true);
  L->num_row_tiles.allocate(sizeof(int32_t), true);
  L->pair_row.allocate(pairs * sizeof(int32_t), true);
  if (L->ep_world > 1) {
    L->record_bytes = dispatch_record_bytes(H);
    // room for the compact layout and for fixed-capacity segments up to 2x the mean
    L->send_record_slots = static_cast<int64_t>(2 * local_pairs + 64 * 16);
    L->send_records.allocate(static_cast<size_t>(L->send_record_slots) * L->record_bytes, true);
    L->send_position.allocate(local_pairs * sizeof(int32_t), true);
    L->send_counts.allocate(64 * sizeof(int32_t), true);
    L->send_offsets.allocate(64 * sizeof(int32_t), true);
    L->rank_cursor.allocate(64 * sizeof(int32_t), true);
    L->shared_out.allocate(T * H * sizeof(float));
  }
  L->a_packed.allocate(slots * 128 * Lr / 2, true);
  L->a_sf.allocate(tiled_sf_bytes(slots, Lr), true);
  L->a_ts.allocate(slots * 128 * sizeof(float), true);
  L->a_weight.allocate(slots * 128 * sizeof(float), true);
  L->a_dest.allocate(slots * 128 * sizeof(int32_t), true);
  L->h_packed.allocate(slots * 128 * I / 2, true);
  L->h_sf.allocate(tiled_sf_bytes(slots, I), true);
  L->h_ts.allocate(slots * 128 * sizeof(float), true);
  if (L->unfused) {
    L->u_raw.allocate(slots * 128 * I * sizeof(float), true);
    L->unweighted_tokens = static_cast<int>(std::min<size_t>(T, 64));
    L->unweighted_rows.allocate(static_cast<size_t>(L->unweighted_tokens) * (K + 1) *
                                std::max(H, Lr) * sizeof(float), true);
  } else {
    L->u_raw.reset();  // of another size: the unfused path allocates when it is enabled
  }

  L->y_op.bind(L->y_packed.as<uint8_t>(), L->y_sf_tiled.as<uint8_t>(), token_slots * 128, H);
  if (L->latent_mode) {
    L->lat_op.bind(L->lat_packed.as<uint8_t>(), L->lat_sf_tiled.as<uint8_t>(), token_slots * 128, Lr);
  }
  L->sh_op.bind(L->sh_packed.as<uint8_t>(), L->sh_sf.as<uint8_t>(), token_slots * 128, S);
  L->a_op.bind(L->a_packed.as<uint8_t>(), L->a_sf.as<uint8_t>(), slots * 128, Lr);
  L->h_op.bind(L->h_packed.as<uint8_t>(), L->h_sf.as<uint8_t>(), slots * 128, I);
  L->cfg.max_tokens = static_cast<int32_t>(T);
  L->last_tokens = 0;
}

// Other scratch for a layer that has some.  Where there is no memory for it the layer gets back what
// it had, or, should that fail too, none (every run is then refused): no run finds a freed buffer.
void reallocate_scratch(nmoe_layer* L, size_t T, bool unfused) {
  const size_t had = static_cast<size_t>(L->cfg.max_tokens);
  const bool was_unfused = L->unfused;
  NMOE_CUDA(cudaDeviceSynchronize());
  L->cfg.max_tokens = 0;
  L->last_tokens = 0;
  L->unfused = unfused;
  try {
    allocate_scratch(L, T);
  } catch (const Failure&) {
    L->unfused = was_unfused;
    try {
      allocate_scratch(L, had);
    } catch (const Failure&) {
      L->cfg.max_tokens = 0;
    }
    throw;
  }
  NMOE_CUDA(cudaDeviceSynchronize());
}

void layer_create_impl(nmoe_layer* L, const nmoe_config& c, const nmoe_weights& w) {
  // config checks of expert_layer.cpp:505-528
  NMOE_REQUIRE(c.hidden_size > 0 && c.moe_latent_size > 0 &&
                   c.routed_expert_intermediate_size > 0 &&
                   c.shared_expert_intermediate_size > 0 && c.n_routed_experts > 0 &&
                   c.top_k > 0 && c.top_k <= c.n_routed_experts && c.n_group > 0 &&
                   c.topk_group > 0 && c.n_routed_experts % c.n_group == 0 &&
                   c.rms_epsilon > 0.0f && c.max_tokens > 0,
               "invalid config");
  const bool has_fc1 = w.fc1_latent.family != NMOE_LINEAR_ABSENT;
  const bool has_fc2 = w.fc2_latent.family != NMOE_LINEAR_ABSENT;
  NMOE_REQUIRE(has_fc1 == has_fc2, "fc1_latent and fc2_latent come together");
  NMOE_REQUIRE(has_fc1 || c.moe_latent_size == c.hidden_size,
               "moe_latent_size != hidden_size needs the fc1_latent / fc2_latent projections");
  NMOE_REQUIRE(w.fc2_latent.family != NMOE_LINEAR_SCALED_FP8,
               "fc2_latent is a dense projection (expert_layer.cpp:617-626)");
  NMOE_REQUIRE(c.n_routed_experts % 32 == 0 && c.n_routed_experts <= 512 && c.top_k <= 32 &&
                   c.n_group <= 32,
               "router limits: experts % 32 == 0, experts <= 512, top_k <= 32, n_group <= 32");
  NMOE_REQUIRE(c.hidden_size % 64 == 0 && c.moe_latent_size % 64 == 0 &&
                   c.routed_expert_intermediate_size % 64 == 0 &&
                   c.shared_expert_intermediate_size % 64 == 0,
               "hidden, latent and intermediate sizes must be multiples of 64");
  // Expert parallelism: this device holds experts [first_local_expert,
  // first_local_expert + n_local_experts), an equal share of all of them.
  NMOE_REQUIRE(w.n_local_experts > 0 && c.n_routed_experts % w.n_local_experts == 0 &&
                   w.first_local_expert >= 0 && w.first_local_expert % w.n_local_experts == 0 &&
                   w.first_local_expert + w.n_local_experts <= c.n_routed_experts &&
                   c.n_routed_experts / w.n_local_experts <= 64,
               "local experts must be an equal, aligned share of the routed experts");
  NMOE_REQUIRE(w.routed_up != nullptr && w.routed_down != nullptr, "missing routed expert weights");

  L->cfg = c;
  L->num_sms = device_sm_count();
  L->force_fp32_parts = std::getenv("NMOE_PARTS_FP32") != nullptr;
  if (const char* env = std::getenv("NMOE_GRAPH_MAX_TOKENS")) L->graph_max_tokens = std::atoi(env);
  if (const char* env = std::getenv("NMOE_WAIT_LIMIT_MS")) {
    const double ms = std::strtod(env, nullptr);
    if (ms > 0.0) L->wait_limit_ticks = ticks_from_ms(ms);
  }
  if (const char* env = std::getenv("NMOE_FORK_MAX_TOKENS")) L->fork_max_tokens = std::atoi(env);
  if (std::getenv("NMOE_NO_SHARED_FORK") == nullptr) {
    NMOE_CUDA(cudaStreamCreateWithFlags(&L->side_stream, cudaStreamNonBlocking));
    NMOE_CUDA(cudaEventCreateWithFlags(&L->quant_done, cudaEventDisableTiming));
    NMOE_CUDA(cudaEventCreateWithFlags(&L->shared_done, cudaEventDisableTiming));
    if (w.fc1_latent.family != NMOE_LINEAR_ABSENT) {
      NMOE_CUDA(cudaStreamCreateWithFlags(&L->latent_stream, cudaStreamNonBlocking));
      NMOE_CUDA(cudaEventCreateWithFlags(&L->latent_done, cudaEventDisableTiming));
    }
  }
  L->local_experts = w.n_local_experts;
  L->first_local_expert = w.first_local_expert;
  cudaStream_t stream = nullptr;
  const int H = c.hidden_size, I = c.routed_expert_intermediate_size,
            S = c.shared_expert_intermediate_size, E = c.n_routed_experts;
  const int EL = w.n_local_experts;
  L->ep_world = E / EL;
  L->ep_rank = w.first_local_expert / EL;
  L->latent = c.moe_latent_size;
  L->latent_mode = has_fc1;
  const int Lr = L->latent;
  const bool dense_shared = w.shared_up_linear.family != NMOE_LINEAR_ABSENT ||
                            w.shared_down_linear.family != NMOE_LINEAR_ABSENT;
  if (L->ep_world > 1 && (L->latent_mode || dense_shared)) {
    throw Failure{NMOE_ERR_UNSUPPORTED,
                  "expert parallelism is built for the all-NVFP4 layer without latent projections"};
  }

  upload_dense_fp32(w.input_norm_weight, H, "input_norm_weight", &L->norm_weight, stream);
  upload_dense_fp32(w.gate_weight, static_cast<size_t>(E) * H, "gate_weight", &L->gate, stream);
  upload_dense_fp32(w.gate_score_correction_bias, E, "gate_score_correction_bias", &L->bias, stream);
  if (w.gate_logit_offset != nullptr) {
    L->logit_offset.allocate(E * sizeof(float));
    NMOE_CUDA(cudaMemcpyAsync(L->logit_offset.as<float>(), w.gate_logit_offset,
                              E * sizeof(float), cudaMemcpyDefault, stream));
    L->has_logit_offset = true;
  }
  // routed experts act on latent rows: up_proj [I][latent], down_proj [latent][I]
  // (shape checks of expert_layer.cpp:646-689)
  L->up.upload(w.routed_up, EL, I, Lr, "routed up_proj", stream);
  L->down.upload(w.routed_down, EL, Lr, I, "routed down_proj", stream);
  if (L->latent_mode) {
    L->fc1.upload(w.fc1_latent, Lr, H, "fc1_latent", stream);
    L->fc2.upload(w.fc2_latent, H, Lr, "fc2_latent", stream);
    L->fc1.slice(stream);
    L->fc2.slice(stream);
  }
  if (w.shared_up_linear.family != NMOE_LINEAR_ABSENT) {
    L->shared_up_dense.upload(w.shared_up_linear, S, H, "shared up_proj", stream);
  } else {
    L->shared_up.upload(&w.shared_up, 1, S, H, "shared up_proj", stream);
  }
  if (w.shared_down_linear.family == NMOE_LINEAR_ABSENT && L->shared_up_dense.present) {
    L->shared_up_dense.prepare_coded(stream);
  }
  if (w.shared_down_linear.family != NMOE_LINEAR_ABSENT) {
    L->shared_down_dense.upload(w.shared_down_linear, H, S, "shared down_proj", stream);
    L->shared_down_dense.slice(stream);
  } else {
    L->shared_down.upload(&w.shared_down, 1, H, S, "shared down_proj", stream);
  }

  if (w.gate_weight.dtype == NMOE_BF16) {
    L->gate_bf16.allocate(static_cast<size_t>(E) * H * 2);
    NMOE_CUDA(cudaMemcpyAsync(L->gate_bf16.as<void>(), w.gate_weight.data,
                              static_cast<size_t>(E) * H * 2, cudaMemcpyDefault, stream));
  }
  L->has_gate_exact = exact_supported(E, H);
  if (L->has_gate_exact) {
    const bool bf16 = w.gate_weight.dtype == NMOE_BF16;
    L->gate_exact.bind(bf16 ? L->gate_bf16.as<void>() : L->gate.as<void>(),
                       bf16 ? kWeightBf16 : kWeightF32, 1.0f, E, H);
  }
  // The tensor-core pass needs the gate exactly in bf16.
  L->fast_router = w.gate_weight.dtype == NMOE_BF16 && c.n_group == 1 && E % 32 == 0 &&
                   E <= 256 && H % 64 == 0 && std::getenv("NMOE_ROUTER_FP64_ONLY") == nullptr;
  if (L->fast_router) {
    L->gate_map = make_bf16_map(L->gate_bf16.as<void>(), E, H, E);
    L->folded_router = std::getenv("NMOE_ROUTER_SPLIT_INPUT") == nullptr;
    if (L->folded_router) {
      L->gate_planes.allocate(static_cast<size_t>(3) * E * H * 2);
      NMOE_CUDA(launch_fold_gate(L->gate_bf16.as<__nv_bfloat16>(), L->norm_weight.as<float>(), E, H,
                                 L->gate_planes.as<__nv_bfloat16>(), stream));
      L->planes_map = make_bf16_map(L->gate_planes.as<void>(), static_cast<size_t>(3) * E, H, E);
    }
    if (const char* env = std::getenv("NMOE_ROUTER_TIE_MARGIN")) L->router_tie_margin = std::strtof(env, nullptr);
    if (const char* env = std::getenv("NMOE_ROUTER_FAST_MIN_TOKENS")) L->fast_router_min_tokens = std::atoi(env);
  }
  L->unfused = std::getenv("NMOE_UNFUSED_ACTIVATION") != nullptr;
  allocate_scratch(L, static_cast<size_t>(c.max_tokens));
  L->error.create();
  NMOE_CUDA(cudaDeviceSynchronize());
}

// y = x W^T of a dense / scaled-FP8 linear, rounded once from the FP64 sum [, relu^2 of it].
void run_linear(nmoe_layer* L, const DenseLinear& linear, ExactScratch& scratch,
                const float* in_rows, int rows, float* out_rows, bool relu2, LaunchStream stream) {
  if (linear.exact) {
    // (clamped first, scaled_fp8_linear.cu:27-33: a scale of zero means no round trip further down)
    const float fp8_scale = linear.fp8 ? clamp_scale_host(linear.input_scale) : 0.0f;
    run_exact(linear.operand.w, scratch, in_rows, fp8_scale, rows, nullptr, relu2, out_rows,
              L->error.device.as<int32_t>(), L->num_sms, stream);
    return;
  }
  const float* source = in_rows;
  if (linear.fp8) {
    NMOE_CUDA(launch_fp8_round_trip(in_rows, static_cast<size_t>(rows) * linear.in,
                                    linear.input_scale, scratch.round_trip.as<float>(), stream));
    source = scratch.round_trip.as<float>();
  }
  NMOE_CUDA(launch_router_logits(source, linear.weight.as<float>(), nullptr, rows, linear.out,
                                 linear.in, out_rows, L->num_sms, stream));
  if (relu2) {
    NMOE_CUDA(launch_relu2(out_rows, static_cast<size_t>(rows) * linear.out, stream));
  }
}

// RMSNorm + activation quantiser + router: fills normalized, y_*, logits,
// top_index / top_weight, the per-expert histogram `counts` (global ids) and each pair's position in it.
void route_tokens(nmoe_layer* L, LaunchStream stream, const void* input, nmoe_dtype in_dtype,
                  int tokens, cudaEvent_t after_quantise = nullptr,
                  bool fork_after_logits = false) {
  const nmoe_config& c = L->cfg;
  const int H = c.hidden_size, E = c.n_routed_experts, K = c.top_k;
  int32_t* error = L->error.device.as<int32_t>();
  L->mark(0, stream);
  const bool two_pass_router = L->fast_router && tokens >= L->fast_router_min_tokens;
  const bool in_bf16 = in_dtype == NMOE_BF16;
  const bool want_normalized = !two_pass_router || L->keep_trace || L->latent_mode ||
                               L->shared_up_dense.present;
  // RMSNorm (:795-796) fused with the activation quantiser every expert's
  // up_proj applies to the same normalised row (:913 -> nvfp4_packing.cpp:90)
  NMOE_CUDA(launch_norm_quant(input, in_bf16, tokens, H, L->norm_weight.as<float>(),
                              c.rms_epsilon, want_normalized ? L->normalized.as<float>() : nullptr,
                              L->y_packed.as<uint8_t>(), L->y_sf_row_major.as<uint8_t>(),
                              L->y_sf_tiled.as<uint8_t>(), k_blocks_of(H), L->y_ts.as<float>(),
                              L->num_sms, stream.stream, L->inv_rms.as<float>(), L->counts.as<int32_t>(), E));
  L->last_normalized = want_normalized;
  if (after_quantise != nullptr && !fork_after_logits) {
    NMOE_CUDA(cudaEventRecord(after_quantise, stream));
  }
  L->mark(1, stream);
  // gate projection (:797-799) and top-k (:881)
  const float* offset = L->has_logit_offset ? L->logit_offset.as<float>() : nullptr;
  if (two_pass_router) {
    const int logit_splits = router_pass1_splits(tokens, H, L->num_sms);
    if (L->folded_router && in_bf16 && reinterpret_cast<uintptr_t>(input) % 16 == 0) {
      if (L->input_map_base != input || L->input_map_rows != tokens) {
        L->input_map = make_bf16_map(input, tokens, H, 128);
        L->input_map_base = input;
        L->input_map_rows = tokens;
      }
      NMOE_CUDA(launch_router_folded_logits(L->input_map, L->planes_map, L->inv_rms.as<float>(),
                                            tokens, E, H, logit_splits, L->logits.as<float>(),
                                            error, stream));
    } else {
      NMOE_CUDA(launch_router_fast_logits(input, in_bf16, L->inv_rms.as<float>(),
                                          L->norm_weight.as<float>(), L->gate_map, tokens, E, H,
                                          logit_splits, L->logits.as<float>(), error, stream));
    }
    // A stream forked here runs the shared expert beside the selection, plan and permute
    // kernels; forked before pass 1 its persistent GEMM CTAs would hold the shared memory
    // the pass-1 CTAs need.
    if (after_quantise != nullptr && fork_after_logits) {
      NMOE_CUDA(cudaEventRecord(after_quantise, stream));
    }
    L->mark(2, stream);
    NMOE_CUDA(launch_router_select_exact(
        L->logits.as<float>(), logit_splits, input, in_bf16, L->inv_rms.as<float>(),
        L->norm_weight.as<float>(), L->gate_bf16.as<__nv_bfloat16>(), offset,
        L->bias.as<float>(), tokens, E, H, K, c.norm_topk_prob != 0, c.routed_scaling_factor,
        L->router_tie_margin, L->top_index.as<int32_t>(), L->top_weight.as<float>(),
        L->counts.as<int32_t>(), L->position.as<int32_t>(), stream));
  } else {
    if (L->has_gate_exact) {
      run_exact(L->gate_exact.w, L->exact, L->normalized.as<float>(), 0.0f, tokens, offset, false,
                L->logits.as<float>(), error, L->num_sms, stream);
    } else {
      NMOE_CUDA(launch_router_logits(L->normalized.as<float>(), L->gate.as<float>(), offset, tokens,
                                     E, H, L->logits.as<float>(), L->num_sms, stream));
    }
    L->mark(2, stream);
    NMOE_CUDA(launch_router_topk(L->logits.as<float>(), L->bias.as<float>(), tokens, E, K,
                                 c.n_group, c.topk_group, c.norm_topk_prob != 0,
                                 c.routed_scaling_factor, L->top_index.as<int32_t>(),
                                 L->top_weight.as<float>(), L->counts.as<int32_t>(),
                                 L->position.as<int32_t>(), L->num_sms, stream));
  }
  L->mark(3, stream);
}

// One expert FFN over rows that are already quantised, fused or unfused.
//   fused:   up GEMM (relu^2 + NVFP4 quantise in the epilogue, tensor scale 1) -> down GEMM
//   unfused: up GEMM keeps relu^2 rows in FP32 (`raw_rows`) -> per-row quantiser with
//            the row's own tensor scale (nvfp4_packing.cpp:119-153) -> down GEMM
struct FfnBuffers {
  uint8_t* hidden_packed;
  uint8_t* hidden_sf;
  float* hidden_ts;
  const ActivationOperand* hidden;
  float* raw_rows;  // unfused only: [row slots * 128][intermediate] FP32
  int raw_row_count;
};

void run_ffn(nmoe_layer* L, bool unfused, const WeightStack& up, const WeightStack& down,
             TileClass tile_class, const ActivationOperand& a, const float* a_ts,
             const Schedule& schedule, const FfnBuffers& buffers, const RowOutput& out,
             cudaStream_t stream, cudaEvent_t between) {
  int32_t* error = L->error.device.as<int32_t>();
  if (!unfused) {
    run_expert_gemms(up, down, tile_class, a, a_ts, schedule, buffers.hidden_packed,
                     buffers.hidden_sf, *buffers.hidden, out, error, L->num_sms, stream, between);
    return;
  }
  RowOutput raw;
  raw.rows = buffers.raw_rows;
  raw.relu2 = true;
  run_down_gemm(up, kClassStream, a, a_ts, schedule, raw, error, L->num_sms, stream);
  NMOE_CUDA(launch_norm_quant(buffers.raw_rows, false, buffers.raw_row_count, up.n, nullptr, 0.0f,
                              nullptr, buffers.hidden_packed, nullptr, buffers.hidden_sf,
                              k_blocks_of(up.n), buffers.hidden_ts, L->num_sms, stream));
  if (between != nullptr) cudaEventRecord(between, stream);
  run_down_gemm(down, tile_class, *buffers.hidden, buffers.hidden_ts, schedule, out, error,
                L->num_sms, stream);
}

// Whether the shared expert's tiles join the routed experts' launch; when they are many its GEMMs are long
// enough to be worth running beside the router.  What counts is the K blocks its 128 x 128 tiles take of each
// SM.  Whole pass, joined against beside (blocks per SM in brackets): benchmark layer 700 tokens 178.4 us and
// 187.8, 1003 [34] 199.8 and 206.9, 1280 [43] 215.5 and 224.7, 1500 [51] 217.2 and 216.7, 1800 234 and 231,
// popular and unpopular experts 246 and 241; shared expert of 1856 1500 tokens [27] 220 and 232, 2000 [36] 239
// and 244, of 7424 800 [59] 202.8 and 204.4, 1280 [84] 232 and 226; 64 experts of 1024, hidden 4096, shared 8192
// 450 tokens [55] 121 and 131, 1003 [110] 148 and 148, 1280 [138] 171 and 161; 256 experts of 768, hidden 2048,
// shared 768 2000 tokens [9] 195 and 204.  With 74 SMs the line lies lower still (benchmark layer, 640 tokens
// [43] 245 and 239).
constexpr int kSharedInLaunchBlocksPerSm = 56;
bool shared_joins(const nmoe_layer* L, int tokens) {
  const int bn = stream_tile_info().bn;
  const int H = L->cfg.hidden_size, S = L->cfg.shared_expert_intermediate_size;
  long long blocks = static_cast<long long>((H + bn - 1) / bn) * k_blocks_of(S);
  if (!L->shared_up_dense.present) blocks += static_cast<long long>((S + bn - 1) / bn) * k_blocks_of(H);
  return (tokens + 127) / 128 * blocks <= static_cast<long long>(kSharedInLaunchBlocksPerSm) * L->num_sms;
}

// Routed rows per expert (on average) up to which csrc/expert_stream.cu takes them: with more, most
// experts have a second row tile and their weights would be read twice.  Where the two meet depends
// on how even the routing is, which the host does not know: whole pass over bf16 rows, this kernel
// against CTA pairs, uniform 96 rows 262 us and 288, 120 rows 322 and 328, 144 rows 397 and 356;
// popular and unpopular experts 56 rows 218 and 230, 80 rows 250 and 248, 120 rows 331 and 309.  At
// 100 rows neither loses more than 8 % (273 and 297, 297 and 276).
constexpr int kStreamRowsPerExpert = 100;

// Which kernel takes `pairs` routed rows.
TileClass routed_tile_class(const nmoe_layer* L, int pairs) {
  if (pairs <= L->local_experts * kStreamRowsPerExpert) return kClassStream;
  return L->num_sms < 2 ? kClassStream : kClassPair;
}

// Plan + permute + the grouped GEMMs over `pairs` (row, slot) pairs whose per-local-expert
// histogram is already in `counts`.  `token_order`: csrc/front.cu has laid out the tiles, nothing is left
// to plan or permute.  `shared` (stream class only): the shared expert's tiles join
// the same launch.
void routed_experts(nmoe_layer* L, LaunchStream stream, const PermuteSource& source, int pairs,
                    int dest_stride, void* out_rows, RowKind out_kind,
                    RowSegments segments = RowSegments(), const StreamFfn* shared = nullptr,
                    bool token_order = false) {
  const int Lr = L->latent;
  int32_t* error = L->error.device.as<int32_t>();
  const TileClass routed_class = routed_tile_class(L, pairs);
  PlanBuffers plan;
  plan.expert_counts = L->counts.as<int32_t>();
  plan.expert_cursor = L->cursor.as<int32_t>();
  plan.row_tiles = L->row_tiles.as<RowTile>();
  plan.num_row_tiles = L->num_row_tiles.as<int32_t>();
  if (source.position == nullptr) {
    stream.chained = false;
    NMOE_CUDA(cudaMemsetAsync(plan.expert_cursor, 0, L->local_experts * sizeof(int32_t), stream));
  }
  L->mark(4, stream);
  if (!token_order) {
    NMOE_CUDA(launch_place_rows(plan, source, pairs, L->local_experts,
                                routed_class == kClassPair ? 2 : 1, L->max_row_tiles, Lr,
                                k_blocks_of(Lr), L->a_packed.as<uint8_t>(), L->a_sf.as<uint8_t>(),
                                L->a_ts.as<float>(), L->a_weight.as<float>(),
                                L->a_dest.as<int32_t>(),
                                L->ep_world == 1 ? L->pair_row.as<int32_t>() : nullptr, dest_stride,
                                error, L->num_sms, stream));
  }
  if (!L->stage_timing) stream.chained = true;
  L->mark(5, stream);
  // routed experts (:896-954)
  Schedule routed;
  routed.row_tiles = L->row_tiles.as<RowTile>();
  routed.num_row_tiles = L->num_row_tiles.as<int32_t>();
  // (a token selects an expert once)
  routed.most_rows = L->ep_world == 1 ? std::min(128, pairs / L->cfg.top_k) : 128;
  RowOutput out;
  out.rows = out_rows;
  out.kind = out_kind;
  out.dest_row = L->a_dest.as<int32_t>();
  out.row_weight = L->a_weight.as<float>();
  out.segments = segments;
  if (routed_class == kClassStream && !L->unfused) {
    StreamFfn ffn;
    ffn.up = &L->up;
    ffn.down = &L->down;
    ffn.a = !token_order ? &L->a_op : L->latent_mode ? &L->lat_op : &L->y_op;
    ffn.a_tensor_scale =
        (!token_order ? L->a_ts : L->latent_mode ? L->lat_ts : L->y_ts).as<float>();
    if (token_order) {
      ffn.used = L->a_dest.as<int32_t>();
      ffn.front_words = L->front_scratch.as<int32_t>();
    }
    ffn.schedule = routed;
    ffn.hidden_packed = L->h_packed.as<uint8_t>();
    ffn.hidden_sf = L->h_sf.as<uint8_t>();
    ffn.hidden = &L->h_op;
    ffn.out = out;
    ffn.row_slots = L->max_row_tiles;
    run_stream(&ffn, shared, L->stream_counts, error, L->num_sms, stream);
    if (token_order) L->front_words_set = false;
    L->mark(6, stream);  // (one launch: its time is that of the up projections' stage)
    return;
  }
  FfnBuffers buffers{L->h_packed.as<uint8_t>(), L->h_sf.as<uint8_t>(), L->h_ts.as<float>(),
                     &L->h_op, L->u_raw.as<float>(), L->max_row_tiles * 128};
  run_ffn(L, L->unfused, L->up, L->down, routed_class, L->a_op, L->a_ts.as<float>(), routed,
          buffers, out, stream, L->stage_timing ? L->stage_events[6] : nullptr);
  if (L->unfused && L->ep_world == 1 && pairs <= L->unweighted_tokens * L->cfg.top_k) {
    // the down_proj rows before the routing weight (routed_expert_outputs of the trace)
    RowOutput plain;
    plain.rows = L->unweighted_rows.as<float>();
    plain.dest_row = L->a_dest.as<int32_t>();
    run_down_gemm(L->down, routed_class, L->h_op, L->h_ts.as<float>(), routed, plain, error,
                  L->num_sms, stream);
  }
}

TileClass shared_tile_class(const nmoe_layer* L, int tokens) {
  return dense_tile_class(tokens, L->cfg.shared_expert_intermediate_size, L->num_sms);
}

// The shared expert's hidden rows in FP32: shared_up and relu^2 (:814-818, :956-964), by a dense /
// scaled-FP8 linear or an NVFP4 GEMM.
void shared_hidden_rows(nmoe_layer* L, LaunchStream stream, int tokens) {
  float* raw = L->shared_raw.as<float>();
  if (L->shared_up_dense.present) {
    run_linear(L, L->shared_up_dense, L->up_exact, L->normalized.as<float>(), tokens, raw,
               /*relu2=*/true, stream);
    return;
  }
  Schedule shared;
  shared.dense_rows = tokens;
  shared.most_rows = std::min(128, tokens);
  RowOutput out;
  out.rows = raw;
  out.relu2 = true;
  run_down_gemm(L->shared_up, kClassStream, L->y_op, L->y_ts.as<float>(), shared, out,
                L->error.device.as<int32_t>(), L->num_sms, stream);
}

// ... and quantised for an NVFP4 down projection, through the host linear's own packing step
// (:981-1005).
void quantised_shared_hidden(nmoe_layer* L, LaunchStream stream, int tokens) {
  const int S = L->cfg.shared_expert_intermediate_size;
  const DenseLinear& up = L->shared_up_dense;
  if (up.coded.slices != nullptr && !L->unfused &&
      !exact_prefers_gemv(tokens, up.out, up.in, L->num_sms)) {
    const float fp8_scale = clamp_scale_host(up.input_scale);
    const int most = L->up_exact.max_rows;
    for (int first = 0; first < tokens; first += most) {
      const ExactWorkspace space{L->up_exact.slices.as<int8_t>(), L->up_exact.info.as<SliceRow>(),
                                 L->up_exact.partial.as<double>()};
      NMOE_CUDA(launch_coded_linear(
          up.coded, L->normalized.as<float>() + static_cast<size_t>(first) * up.in,
          std::min(tokens - first, most), fp8_scale, space, first, L->sh_packed.as<uint8_t>(),
          L->sh_sf.as<uint8_t>(), k_blocks_of(S) * 4, L->sh_ts.as<float>(),
          L->error.device.as<int32_t>(), L->num_sms, stream));
    }
    return;
  }
  shared_hidden_rows(L, stream, tokens);
  NMOE_CUDA(launch_norm_quant(L->shared_raw.as<float>(), false, tokens, S, nullptr, 0.0f, nullptr,
                              L->sh_packed.as<uint8_t>(), nullptr, L->sh_sf.as<uint8_t>(),
                              k_blocks_of(S), L->sh_ts.as<float>(), L->num_sms, stream));
}

// shared expert (:814-818, :956-964, :981-1005) on the token-order rows
void shared_expert(nmoe_layer* L, cudaStream_t stream, int tokens, void* out_rows, int dest_mul,
                   int dest_add, cudaEvent_t between, RowKind out_kind = kRowF32) {
  const TileClass shared_class = shared_tile_class(L, tokens);
  Schedule shared;
  shared.dense_rows = tokens;
  shared.most_rows = std::min(128, tokens);
  RowOutput out;
  out.rows = out_rows;
  out.kind = out_kind;
  out.dest_mul = dest_mul;
  out.dest_add = dest_add;
  if (!L->shared_up_dense.present && !L->shared_down_dense.present) {
    FfnBuffers buffers{L->sh_packed.as<uint8_t>(), L->sh_sf.as<uint8_t>(), L->sh_ts.as<float>(),
                       &L->sh_op, L->shared_raw.as<float>(), tokens};
    run_ffn(L, L->unfused, L->shared_up, L->shared_down, shared_class, L->y_op,
            L->y_ts.as<float>(), shared, buffers, out, stream, between);
    return;
  }
  if (L->shared_down_dense.present) {
    shared_hidden_rows(L, stream, tokens);
    if (between != nullptr) cudaEventRecord(between, stream);
    // dense / scaled-FP8 down projection (:1006-1045) straight from the FP32 rows;
    // only the latent data flow (FP32 rows of `hidden` per token) reaches this
    NMOE_REQUIRE(dest_mul == 1 && dest_add == 0 && out_kind == kRowF32,
                 "a dense shared_down writes FP32 token rows");
    run_linear(L, L->shared_down_dense, L->exact, L->shared_raw.as<float>(), tokens,
               static_cast<float*>(out_rows), false, stream);
    return;
  }
  quantised_shared_hidden(L, stream, tokens);
  if (between != nullptr) cudaEventRecord(between, stream);
  run_down_gemm(L->shared_down, shared_class, L->sh_op, L->sh_ts.as<float>(), shared, out,
                L->error.device.as<int32_t>(), L->num_sms, stream);
}

// The shared expert as part of the routed experts' launch (csrc/expert_stream.cu); the hidden rows of
// a dense shared_up were made before it.
StreamFfn shared_stream_ffn(nmoe_layer* L, int tokens, void* out_rows, int dest_mul, int dest_add,
                            RowKind out_kind) {
  StreamFfn ffn;
  ffn.down = &L->shared_down;
  ffn.schedule.dense_rows = tokens;
  ffn.schedule.most_rows = std::min(128, tokens);
  ffn.hidden_packed = L->sh_packed.as<uint8_t>();
  ffn.hidden_sf = L->sh_sf.as<uint8_t>();
  ffn.hidden = &L->sh_op;
  ffn.out.rows = out_rows;
  ffn.out.kind = out_kind;
  ffn.out.dest_mul = dest_mul;
  ffn.out.dest_add = dest_add;
  ffn.row_slots = (tokens + 127) / 128;
  if (L->shared_up_dense.present) {
    ffn.hidden_tensor_scale = L->sh_ts.as<float>();
  } else {
    ffn.up = &L->shared_up;
    ffn.a = &L->y_op;
    ffn.a_tensor_scale = L->y_ts.as<float>();
  }
  return ffn;
}

PermuteSource local_source(nmoe_layer* L) {
  const int H = L->cfg.hidden_size;
  PermuteSource source;
  source.packed = L->y_packed.as<uint8_t>();
  source.packed_stride = static_cast<size_t>(H) / 2;
  source.sf = L->y_sf_row_major.as<uint8_t>();
  source.sf_stride = static_cast<size_t>(H) / 16;
  source.tensor_scale = L->y_ts.as<float>();
  source.tensor_scale_stride = sizeof(float);
  source.weight = L->top_weight.as<float>();
  source.weight_stride = sizeof(float);
  source.expert = L->top_index.as<int32_t>();
  source.expert_stride = sizeof(int32_t);
  source.pairs_per_row = L->cfg.top_k;
  source.position = L->position.as<int32_t>();
  return source;
}

// What follows the experts of a latent layer: routed sum in selection order (:951-953), fc2_latent
// (:1047-1053), mixer and residual (:1064-1069).
void latent_tail(nmoe_layer* L, LaunchStream stream, const void* input, nmoe_dtype in_dtype, int tokens,
                 void* output, nmoe_dtype out_dtype) {
  const int H = L->cfg.hidden_size, K = L->cfg.top_k, Lr = L->latent;
  if (tokens == 1 && L->fc2.exact && !L->stage_timing) {
    const LatentTail tail{L->parts.as<float>(),       K,
                          L->shared_rows.as<float>(), input,
                          in_dtype == NMOE_BF16,      L->routed_latent.as<float>(),
                          L->projected.as<float>(),   output,
                          out_dtype == NMOE_BF16};
    NMOE_CUDA(launch_latent_tail(L->fc2.operand.w, tail, stream));
    return;
  }
  if (L->fc2.exact && tokens <= L->exact.max_rows &&
      !exact_prefers_gemv(tokens, L->fc2.out, L->fc2.in, L->num_sms)) {
    const ExactWorkspace space{L->exact.slices.as<int8_t>(), L->exact.info.as<SliceRow>(),
                               L->exact.partial.as<double>()};
    const ExactSum sum{L->parts.as<float>(), K, L->routed_latent.as<float>()};
    const ExactMix mix{input, in_dtype == NMOE_BF16, L->shared_rows.as<float>(), output,
                       out_dtype == NMOE_BF16};
    NMOE_CUDA(launch_exact_linear(L->fc2.operand.w, nullptr, tokens, 0.0f, nullptr, false, space,
                                  L->projected.as<float>(), L->error.device.as<int32_t>(), L->num_sms,
                                  stream, sum, mix));
    return;
  }
  NMOE_CUDA(launch_sum_parts(L->parts.as<float>(), tokens, Lr, K, L->routed_latent.as<float>(),
                             stream));
  run_linear(L, L->fc2, L->exact, L->routed_latent.as<float>(), tokens, L->projected.as<float>(), false,
             stream);
  NMOE_CUDA(launch_mixer(input, in_dtype == NMOE_BF16, L->projected.as<float>(),
                         L->shared_rows.as<float>(), tokens, H, output, out_dtype == NMOE_BF16, stream));
}

// Everything in front of the experts in one launch (csrc/front.cu).
void route_few(nmoe_layer* L, cudaStream_t stream, const void* input, nmoe_dtype in_dtype,
               int tokens) {
  const nmoe_config& c = L->cfg;
  FrontArgs args;
  args.in = input;
  args.in_bf16 = in_dtype == NMOE_BF16;
  args.rows = tokens;
  args.cols = c.hidden_size;
  args.norm_weight = L->norm_weight.as<float>();
  args.eps = c.rms_epsilon;
  args.normalized = L->normalized.as<float>();
  args.packed = L->y_packed.as<uint8_t>();
  args.sf_row_major = L->y_sf_row_major.as<uint8_t>();
  args.sf_tiled = L->y_sf_tiled.as<uint8_t>();
  args.k_tiles = k_blocks_of(c.hidden_size) * 4;
  args.tensor_scale = L->y_ts.as<float>();
  args.inv_rms = L->inv_rms.as<float>();
  args.gate = L->gate_exact.w.weight;
  args.gate_bf16 = L->gate_exact.w.kind == kWeightBf16;
  args.logit_offset = L->has_logit_offset ? L->logit_offset.as<float>() : nullptr;
  args.bias = L->bias.as<float>();
  args.experts = c.n_routed_experts;
  args.top_k = c.top_k;
  args.n_group = c.n_group;
  args.topk_group = c.topk_group;
  args.norm_topk_prob = c.norm_topk_prob != 0;
  args.routed_scaling = c.routed_scaling_factor;
  args.logits = L->logits.as<float>();
  args.top_index = L->top_index.as<int32_t>();
  args.top_weight = L->top_weight.as<float>();
  args.row_tiles = L->row_tiles.as<RowTile>();
  args.num_row_tiles = L->num_row_tiles.as<int32_t>();
  args.dest = L->a_dest.as<int32_t>();
  args.row_weight = L->a_weight.as<float>();
  args.pair_row = L->pair_row.as<int32_t>();
  args.dest_stride = L->latent_mode ? c.top_k : c.top_k + 1;
  if (L->latent_mode) {
    auto add = [&](const DenseLinear& linear) -> FrontLinear& {
      FrontLinear& to = args.linear[args.linears++];
      to.N = linear.out;
      to.kind = linear.operand.w.kind;
      to.weight = linear.operand.w.weight;
      to.scale = linear.operand.w.scale;
      to.fp8_scale = linear.fp8 ? clamp_scale_host(linear.input_scale) : 0.0f;
      to.rounded = L->front_rounded.as<float>() +
                   static_cast<size_t>(args.linears - 1) * c.hidden_size;
      return to;
    };
    FrontLinear& fc1 = add(L->fc1);
    fc1.out = L->latent_rows.as<float>();
    fc1.packed = L->lat_packed.as<uint8_t>();
    fc1.sf_row_major = L->lat_sf_row_major.as<uint8_t>();
    fc1.sf_tiled = L->lat_sf_tiled.as<uint8_t>();
    fc1.k_tiles = k_blocks_of(L->latent) * 4;
    fc1.tensor_scale = L->lat_ts.as<float>();
    if (L->shared_up_dense.present) {
      FrontLinear& up = add(L->shared_up_dense);
      up.relu2 = true;
      up.out = L->shared_raw.as<float>();
      up.packed = L->sh_packed.as<uint8_t>();
      up.sf_tiled = L->sh_sf.as<uint8_t>();
      up.k_tiles = k_blocks_of(c.shared_expert_intermediate_size) * 4;
      up.tensor_scale = L->sh_ts.as<float>();
    }
  }
  args.resident_blocks = kFrontLinearBlocksPerSm * L->num_sms;
  args.scratch = L->front_scratch.as<void>();
  args.error = L->error.device.as<int32_t>();
  if (L->front_words_set) {  // (the launch that clears them was not made)
    NMOE_CUDA(cudaMemsetAsync(args.scratch, 0, front_scratch_bytes(), stream));
  }
  L->front_words_set = true;
  NMOE_CUDA(launch_front(args, stream));
  L->last_normalized = true;
}

// Whether csrc/front.cu takes a batch (with what it cannot quantise left out).
bool front_takes(const nmoe_layer* L, int tokens) {
  if (!front_pays(tokens, L->cfg.n_routed_experts, L->num_sms) ||
      L->cfg.hidden_size > kFrontMaxCols || !L->has_gate_exact) {
    return false;
  }
  if (!L->latent_mode) return !L->shared_up_dense.present && !L->shared_down_dense.present;
  auto fits = [](const DenseLinear& linear) {
    return linear.exact && linear.out <= kFrontLinearMaxN;
  };
  return tokens == 1 && fits(L->fc1) &&
         (!L->shared_up_dense.present || fits(L->shared_up_dense));
}

// A latent layer's three chains behind the norm -- gate and selection; fc1_latent and its quantiser;
// shared_up and its quantiser -- meet only in front of the experts.  On streams of their own one fills
// what another leaves idle: latency at a few tokens, SMs at a hundred, last waves at a thousand.  Whole
// pass of the checkpoint's layer, one stream against three: 1 token 77.8 us and 80.4 (the branches of
// the graph cost more than they hide), 2 tokens 101 and 91, 8 tokens 189 and 171, 64 tokens 399 and 373,
// 256 tokens 578 and 534, 1000 tokens 1075 and 962.
//
// Up to four tokens the linears are gemvs chained one to the other, and it depends on their size.  Long ones
// gain (fc1_latent and shared_up of 4096 x 4096 together with 1024 x 4096, 21 million products, bf16, 3 tokens
// 101 and 79, 4 tokens 95 and 84).  Short ones gain in a graph, where a branch costs least (1.3 million, FP32, 2
// tokens 33.2 and 29.0; 5.2 million in FP8 45.7 and 41.2), and lose a little as launches (38.1 and 39.8; 53.8 and
// 50.6, but 3 tokens 69.9 and 73.5).  Between, where a gemv by itself reads its weights with the whole GPU,
// the branches cost more than they hide (5.2 million, bf16, 2 tokens 40.3 and 42.2, FP32 42.2 and 46.9).  From
// five tokens on every shape gains in a graph (these 8 to 12 %), and none loses more than 2 % as launches.
constexpr int kBesideMinTokens = 2;
constexpr int kBesideAnyTokens = 5;
constexpr size_t kBesideLongProducts = 16000000;
constexpr size_t kBesideShortBytes = 6000000;
bool linears_beside(const nmoe_layer* L, int tokens, bool in_graph) {
  if (L->latent_stream == nullptr || tokens < kBesideMinTokens || tokens > L->fork_max_tokens) {
    return false;
  }
  if (tokens >= kBesideAnyTokens) return true;
  size_t products = 0, bytes = 0;
  for (const DenseLinear* linear : {&L->fc1, &L->shared_up_dense}) {
    if (!linear->present) continue;
    products += static_cast<size_t>(linear->out) * linear->in;
    bytes += linear->weight.bytes();
  }
  return products >= kBesideLongProducts || (in_graph && bytes <= kBesideShortBytes);
}

// `in_graph`: the launches are being recorded, by this library or by the caller.
void layer_run_impl(nmoe_layer* L, cudaStream_t stream, const void* input, nmoe_dtype in_dtype,
                    int tokens, void* output, nmoe_dtype out_dtype, bool in_graph) {
  const nmoe_config& c = L->cfg;
  const int H = c.hidden_size, K = c.top_k, Lr = L->latent;
  const bool dense_shared = L->shared_up_dense.present || L->shared_down_dense.present;
  // The per-(token, slot) rows of the down projection and the shared expert's row
  // wait in `parts` for the combine.  They carry the precision the output needs: FP32
  // rows for an FP32 result (the reference's arithmetic, bit for bit in the sums),
  // binary16 rows for a bf16 result: half the bytes of the layer's largest write and
  // read, and eight times finer than the bf16 the sum is rounded to in the end.
  const RowKind parts_kind = out_dtype == NMOE_BF16 && !L->force_fp32_parts && !L->latent_mode
                                 ? kRowF16 : kRowF32;
  // Small batches bound by reading the weights run both kinds of expert in one launch, the others
  // fork the shared expert onto a stream of its own.
  const bool one_launch = routed_tile_class(L, tokens * K) == kClassStream && !L->unfused &&
                          !L->shared_down_dense.present &&
                          (L->latent_mode || shared_joins(L, tokens));
  const bool fork = L->side_stream != nullptr && !L->stage_timing && !one_launch &&
                    tokens <= L->fork_max_tokens && !L->latent_mode && !dense_shared;
  const bool two_pass = L->fast_router && tokens >= L->fast_router_min_tokens;
  // One kernel after the other on one stream, and small enough for the gaps between them to count:
  // with the two-pass router there was nothing to gain (256 tokens 162 us either way) and at 700
  // tokens 2 to 4 us to lose.
  const LaunchStream chain(stream, !fork && !L->stage_timing && !L->unfused && !two_pass);
  const bool few = front_takes(L, tokens) && one_launch && !two_pass && !L->stage_timing;
  const bool beside = !few && one_launch && L->latent_mode && !L->stage_timing &&
                      linears_beside(L, tokens, in_graph);
  if (few) {
    route_few(L, stream, input, in_dtype, tokens);
  } else {
    route_tokens(L, chain, input, in_dtype, tokens, fork || beside ? L->quant_done : nullptr,
                 fork && two_pass);
  }
  L->last_tokens = tokens;
  L->last_parts_kind = parts_kind;
  L->last_unfused = L->unfused;
  if (L->latent_mode && few) {
    const StreamFfn shared =
        shared_stream_ffn(L, tokens, L->shared_rows.as<void>(), 1, 0, kRowF32);
    routed_experts(L, chain, local_source(L), tokens * K, K, L->parts.as<void>(), kRowF32,
                   RowSegments(), &shared, true);
    latent_tail(L, chain, input, in_dtype, tokens, output, out_dtype);
    return;
  }
  if (L->latent_mode) {
    // latent = fc1_latent(normalized) (:809-813); every routed expert's up_proj packs
    // the same latent row (:913 -> nvfp4_packing.cpp:90)
    LaunchStream latent = chain, up = chain, placing = chain;
    if (beside) {
      latent = LaunchStream(L->latent_stream);
      up = LaunchStream(L->side_stream);
      NMOE_CUDA(cudaStreamWaitEvent(L->latent_stream, L->quant_done, 0));
      if (L->shared_up_dense.present) {
        NMOE_CUDA(cudaStreamWaitEvent(L->side_stream, L->quant_done, 0));
      }
    }
    run_linear(L, L->fc1, L->fc1_exact, L->normalized.as<float>(), tokens,
               L->latent_rows.as<float>(), false, latent);
    NMOE_CUDA(launch_norm_quant(L->latent_rows.as<float>(), false, tokens, Lr, nullptr, 0.0f,
                                nullptr, L->lat_packed.as<uint8_t>(),
                                L->lat_sf_row_major.as<uint8_t>(), nullptr, 0,
                                L->lat_ts.as<float>(), L->num_sms, latent));
    if (one_launch && L->shared_up_dense.present) {
      quantised_shared_hidden(L, up, tokens);
    }
    if (beside) {
      NMOE_CUDA(cudaEventRecord(L->latent_done, L->latent_stream));
      NMOE_CUDA(cudaStreamWaitEvent(stream, L->latent_done, 0));
      if (L->shared_up_dense.present) {
        NMOE_CUDA(cudaEventRecord(L->shared_done, L->side_stream));
        NMOE_CUDA(cudaStreamWaitEvent(stream, L->shared_done, 0));
      }
      placing.chained = false;  // it has more than one predecessor
    }
    PermuteSource source = local_source(L);
    source.packed = L->lat_packed.as<uint8_t>();
    source.packed_stride = static_cast<size_t>(Lr) / 2;
    source.sf = L->lat_sf_row_major.as<uint8_t>();
    source.sf_stride = static_cast<size_t>(Lr) / 16;
    source.tensor_scale = L->lat_ts.as<float>();
    if (one_launch) {
      const StreamFfn shared =
          shared_stream_ffn(L, tokens, L->shared_rows.as<void>(), 1, 0, kRowF32);
      routed_experts(L, placing, source, tokens * K, K, L->parts.as<void>(), kRowF32, RowSegments(),
                     &shared);
      for (int i = 7; i <= 9; ++i) L->mark(i, stream);
    } else {
      routed_experts(L, chain, source, tokens * K, K, L->parts.as<void>(), kRowF32);
      L->mark(7, stream);
      shared_expert(L, stream, tokens, L->shared_rows.as<void>(), 1, 0,
                    L->stage_timing ? L->stage_events[8] : nullptr, kRowF32);
      L->mark(9, stream);
    }
    latent_tail(L, chain, input, in_dtype, tokens, output, out_dtype);
    L->mark(10, stream);
    return;
  }
  if (fork) {
    NMOE_CUDA(cudaStreamWaitEvent(L->side_stream, L->quant_done, 0));
    shared_expert(L, L->side_stream, tokens, L->parts.as<void>(), K + 1, K, nullptr, parts_kind);
    NMOE_CUDA(cudaEventRecord(L->shared_done, L->side_stream));
  }
  if (one_launch) {
    if (L->shared_up_dense.present) {
      quantised_shared_hidden(L, chain, tokens);
    }
    const StreamFfn shared =
        shared_stream_ffn(L, tokens, L->parts.as<void>(), K + 1, K, parts_kind);
    routed_experts(L, chain, local_source(L), tokens * K, K + 1, L->parts.as<void>(), parts_kind,
                   RowSegments(), &shared, few);
  } else {
    routed_experts(L, chain, local_source(L), tokens * K, K + 1, L->parts.as<void>(), parts_kind);
  }
  L->mark(7, stream);
  if (one_launch) {
    L->mark(8, stream);  // nothing left to wait for
  } else if (fork) {
    NMOE_CUDA(cudaStreamWaitEvent(stream, L->shared_done, 0));
  } else {
    shared_expert(L, stream, tokens, L->parts.as<void>(), K + 1, K,
                  L->stage_timing ? L->stage_events[8] : nullptr, parts_kind);
  }
  // routed sum in selection order, mixer and residual (:951-953, :1064-1069)
  L->mark(9, stream);
  NMOE_CUDA(launch_combine(input, in_dtype == NMOE_BF16, L->parts.as<void>(), parts_kind, tokens,
                           H, K, output, out_dtype == NMOE_BF16, L->error.device.as<int32_t>(),
                           chain));
  L->mark(10, stream);
}

// A latent layer's graph has three branches, and recording it costs a new pair of buffers 420 us more
// than launching the pass (40 tokens: 784 us and 366 from an idle device; 2 tokens 415 and 115), while
// a replay saves 9 to 12 us over the launches (40 tokens 342 and 354 us a pass, 2 tokens 90 and 100).
// So it is recorded when the launches have cost as much as that.  Where the linears stay on one stream, as
// for one token, and in every layer without a latent form, a run is recorded at once.
constexpr int kEagerRunsOfBranches = 32;

// nmoe_layer_run: small batches replay a recorded CUDA graph of the same run.
void run_recorded_or_eager(nmoe_layer* L, cudaStream_t stream, const void* input,
                           nmoe_dtype in_dtype, int tokens, void* output, nmoe_dtype out_dtype) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  const bool can_query = cudaStreamIsCapturing(stream, &capturing) == cudaSuccess;
  if (!can_query) cudaGetLastError();
  const bool eligible = tokens <= L->graph_max_tokens && !L->stage_timing && !L->unfused &&
                        can_query && capturing == cudaStreamCaptureStatusNone &&
                        stream != nullptr && stream != cudaStreamLegacy;
  if (!eligible) {
    layer_run_impl(L, stream, input, in_dtype, tokens, output, out_dtype,
                   can_query && capturing != cudaStreamCaptureStatusNone);
    return;
  }
  ++L->run_counter;
  const bool branches = linears_beside(L, tokens, true);
  nmoe_layer::RecordedRun* known = nullptr;
  for (nmoe_layer::RecordedRun& r : L->recorded) {
    if (r.input == input && r.output == output && r.tokens == tokens &&
        r.in_dtype == in_dtype && r.out_dtype == out_dtype) {
      r.last_use = L->run_counter;
      known = &r;
      if (r.exec == nullptr) break;
      NMOE_CUDA(cudaGraphLaunch(r.exec, stream));
      L->last_tokens = tokens;
      L->last_parts_kind = r.parts_kind;
      L->last_normalized = r.normalized;
      L->last_unfused = false;
      return;
    }
  }
  if (known == nullptr) {
    if (L->recorded.size() >= 16) {  // forget the run that was used longest ago
      size_t oldest = 0;
      for (size_t i = 1; i < L->recorded.size(); ++i) {
        if (L->recorded[i].last_use < L->recorded[oldest].last_use) oldest = i;
      }
      if (L->recorded[oldest].exec != nullptr) cudaGraphExecDestroy(L->recorded[oldest].exec);
      L->recorded.erase(L->recorded.begin() + static_cast<long>(oldest));
    }
    L->recorded.push_back(nmoe_layer::RecordedRun{input, output, tokens, in_dtype, out_dtype,
                                                  RowKind(), false, nullptr, L->run_counter});
    known = &L->recorded.back();
  }
  if (branches && known->eager_runs < kEagerRunsOfBranches) {
    ++known->eager_runs;
    layer_run_impl(L, stream, input, in_dtype, tokens, output, out_dtype, false);
    return;
  }
  // record: the launches below go into a graph instead of onto the stream
  if (cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();      // this stream cannot be captured (e.g. the legacy default stream)
    L->graph_max_tokens = 0;  // stay eager from now on
    layer_run_impl(L, stream, input, in_dtype, tokens, output, out_dtype, false);
    return;
  }
  cudaGraph_t graph = nullptr;
  try {
    layer_run_impl(L, stream, input, in_dtype, tokens, output, out_dtype, true);
  } catch (...) {
    cudaStreamEndCapture(stream, &graph);
    if (graph != nullptr) cudaGraphDestroy(graph);
    cudaGetLastError();
    throw;
  }
  NMOE_CUDA(cudaStreamEndCapture(stream, &graph));
  cudaGraphExec_t exec = nullptr;
  const cudaError_t made = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (made != cudaSuccess) {
    cudaGetLastError();
    L->graph_max_tokens = 0;
    layer_run_impl(L, stream, input, in_dtype, tokens, output, out_dtype, false);
    return;
  }
  known->parts_kind = L->last_parts_kind;
  known->normalized = L->last_normalized;
  known->exec = exec;
  NMOE_CUDA(cudaGraphLaunch(exec, stream));
}

}  // namespace

extern "C" {

nmoe_status nmoe_layer_create(const nmoe_config* config, const nmoe_weights* weights,
                              nmoe_layer** out_layer) {
  if (config == nullptr || weights == nullptr || out_layer == nullptr) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  *out_layer = nullptr;
  std::unique_ptr<nmoe_layer> layer(new (std::nothrow) nmoe_layer);
  if (!layer) return NMOE_ERR_CUDA;
  try {
    layer_create_impl(layer.get(), *config, *weights);
  } catch (const Failure& failure) {
    if (std::getenv("NEMOTRON_FORWARD_DEBUG") != nullptr) {
      std::fprintf(stderr, "expert_layer_create: layer %d failed: %s\n", config->layer_index,
                   failure.message.c_str());
    }
    return failure.status;
  }
  *out_layer = layer.release();
  return NMOE_OK;
}

void nmoe_layer_destroy(nmoe_layer* layer) { delete layer; }

nmoe_status nmoe_layer_run(nmoe_layer* layer, void* stream, const void* input,
                           nmoe_dtype input_dtype, int64_t tokens, void* output,
                           nmoe_dtype output_dtype) {
  if (layer == nullptr || input == nullptr || output == nullptr || tokens <= 0 ||
      input == output || (input_dtype != NMOE_F32 && input_dtype != NMOE_BF16) ||
      (output_dtype != NMOE_F32 && output_dtype != NMOE_BF16)) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  if (tokens > layer->cfg.max_tokens) return NMOE_ERR_CAPACITY;
  if (layer->ep_world != 1) return NMOE_ERR_INVALID_ARGUMENT;  // use the nmoe_ep_* stages
  try {
    run_recorded_or_eager(layer, static_cast<cudaStream_t>(stream), input, input_dtype,
                          static_cast<int>(tokens), output, output_dtype);
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    if (std::getenv("NEMOTRON_FORWARD_DEBUG") != nullptr) {
      std::fprintf(stderr, "expert_layer: %s\n", failure.message.c_str());
    }
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_layer_sync_status(nmoe_layer* layer, void* stream) {
  if (layer == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  try {
    const nmoe_status status = layer->error.sync(static_cast<cudaStream_t>(stream));
    if (status != NMOE_OK) layer->last_error = nmoe_status_string(status);
    return status;
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
}

nmoe_status nmoe_layer_reserve_sms(nmoe_layer* layer, int32_t reserved_sms) {
  if (layer == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  const int all = device_sm_count();
  if (reserved_sms < 0 || reserved_sms >= all) return NMOE_ERR_INVALID_ARGUMENT;
  layer->drop_recorded();
  const int before = layer->num_sms;
  layer->num_sms = all - reserved_sms;
  const size_t tokens = static_cast<size_t>(layer->cfg.max_tokens);
  const ExactWeight& gate = layer->gate_exact.w;
  if ((gate.slices != nullptr && layer->exact.holds(gate)) || !gate_needs_slices(layer, tokens)) {
    return NMOE_OK;
  }
  try {  // with this few SMs the gate goes through the integer kernel
    NMOE_CUDA(cudaDeviceSynchronize());
    allocate_exact(layer, tokens);
    NMOE_CUDA(cudaDeviceSynchronize());
  } catch (const Failure& failure) {
    layer->num_sms = before;
    layer->last_error = failure.message;
    try {  // the workspace it had, or none (every run is then refused): no run finds a freed buffer
      allocate_exact(layer, tokens);
    } catch (const Failure&) {
      layer->cfg.max_tokens = 0;
    }
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_layer_set_wait_limit_ms(nmoe_layer* layer, double milliseconds) {
  if (layer == nullptr || !(milliseconds > 0.0) || milliseconds > 60000.0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  try {
    layer->wait_limit_ticks = ticks_from_ms(milliseconds);
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_layer_wait_flag(nmoe_layer* layer, void* stream_ptr, const uint32_t* flag,
                                 uint32_t expected) {
  if (layer == nullptr || flag == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  try {
    if (layer->probe_epoch.bytes() == 0) layer->probe_epoch.allocate(sizeof(uint32_t), true);
    NMOE_CUDA(cudaMemcpyAsync(layer->probe_epoch.as<uint32_t>(), &expected, sizeof(uint32_t),
                              cudaMemcpyHostToDevice, stream));
    NMOE_CUDA(launch_window_wait(flag, layer->probe_epoch.as<uint32_t>(), 0, 1,
                                 layer->wait_limit_ticks, layer->error.device.as<int32_t>(),
                                 stream));
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_layer_enable_stage_timing(nmoe_layer* layer, int32_t enable) {
  if (layer == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  if (enable != 0) {
    for (cudaEvent_t& e : layer->stage_events) {
      if (e == nullptr && cudaEventCreate(&e) != cudaSuccess) return NMOE_ERR_CUDA;
    }
  }
  layer->stage_timing = enable != 0;
  return NMOE_OK;
}

nmoe_status nmoe_layer_stage_times(nmoe_layer* layer, float* milliseconds, int32_t count) {
  if (layer == nullptr || milliseconds == nullptr || count < kStageCount || !layer->stage_timing) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  // A stage the last run did not pass through (the expert-parallel stages record only
  // some of the marks) reports 0.
  for (int i = 0; i <= kStageCount; ++i) {
    const cudaError_t state = cudaEventQuery(layer->stage_events[i]);
    if (state == cudaErrorNotReady) {
      if (cudaEventSynchronize(layer->stage_events[i]) != cudaSuccess) return NMOE_ERR_CUDA;
    } else if (state != cudaSuccess) {
      cudaGetLastError();
    }
  }
  for (int i = 0; i < kStageCount; ++i) {
    if (cudaEventElapsedTime(&milliseconds[i], layer->stage_events[i],
                             layer->stage_events[i + 1]) != cudaSuccess) {
      cudaGetLastError();
      milliseconds[i] = 0.0f;
    }
  }
  return NMOE_OK;
}

// ---------------------------------------------------------------------------
// expert-parallel stages
// ---------------------------------------------------------------------------

size_t nmoe_ep_record_bytes(const nmoe_layer* layer) {
  return layer == nullptr ? 0 : static_cast<size_t>(dispatch_record_bytes(layer->cfg.hidden_size));
}

nmoe_status nmoe_ep_dispatch(nmoe_layer* layer, void* stream_ptr, const void* input,
                             nmoe_dtype input_dtype, int64_t tokens, int64_t capacity_per_rank,
                             const void** send_records, const int32_t** send_counts) {
  if (layer == nullptr || input == nullptr || send_records == nullptr || send_counts == nullptr ||
      tokens <= 0 || layer->ep_world <= 1) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  if (tokens > layer->cfg.max_tokens) return NMOE_ERR_CAPACITY;
  if (capacity_per_rank < 0 ||
      capacity_per_rank * layer->ep_world > layer->send_record_slots) {
    return NMOE_ERR_CAPACITY;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  try {
    const nmoe_config& c = layer->cfg;
    route_tokens(layer, stream, input, input_dtype, static_cast<int>(tokens));
    NMOE_CUDA(launch_dispatch_plan(layer->counts.as<int32_t>(), c.n_routed_experts,
                                   layer->local_experts, layer->ep_world,
                                   layer->send_counts.as<int32_t>(),
                                   layer->send_offsets.as<int32_t>(),
                                   layer->rank_cursor.as<int32_t>(), stream));
    NMOE_CUDA(launch_pack_records(layer->top_index.as<int32_t>(), layer->top_weight.as<float>(),
                                  static_cast<int>(tokens), c.top_k, layer->local_experts,
                                  layer->y_packed.as<uint8_t>(),
                                  layer->y_sf_row_major.as<uint8_t>(), layer->y_ts.as<float>(),
                                  c.hidden_size, layer->send_offsets.as<int32_t>(),
                                  layer->rank_cursor.as<int32_t>(),
                                  static_cast<int>(capacity_per_rank),
                                  layer->send_records.as<uint8_t>(), nullptr,
                                  layer->send_position.as<int32_t>(),
                                  layer->error.device.as<int32_t>(), stream));
    layer->last_tokens = static_cast<int>(tokens);
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  *send_records = layer->send_records.as<uint8_t>();
  *send_counts = layer->send_counts.as<int32_t>();
  return NMOE_OK;
}

nmoe_status nmoe_ep_experts(nmoe_layer* layer, void* stream_ptr, const void* recv_records,
                            int64_t count, const int32_t* valid_counts, int64_t capacity_per_rank,
                            void* out_rows, nmoe_dtype rows_dtype) {
  if (layer == nullptr || layer->ep_world <= 1 || count < 0 ||
      (count > 0 && (recv_records == nullptr || out_rows == nullptr))) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  if (rows_dtype != NMOE_F32 && rows_dtype != NMOE_BF16 && rows_dtype != NMOE_F16) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  if (count > layer->max_pairs) return NMOE_ERR_CAPACITY;
  if (count == 0) return NMOE_OK;
  if (valid_counts != nullptr && capacity_per_rank <= 0) return NMOE_ERR_INVALID_ARGUMENT;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  try {
    const int H = layer->cfg.hidden_size;
    NMOE_CUDA(cudaMemsetAsync(layer->counts.as<int32_t>(), 0,
                              layer->local_experts * sizeof(int32_t), stream));
    NMOE_CUDA(launch_record_histogram(static_cast<const uint8_t*>(recv_records),
                                      static_cast<int>(count), H, layer->local_experts,
                                      valid_counts, static_cast<int>(capacity_per_rank),
                                      layer->counts.as<int32_t>(),
                                      layer->error.device.as<int32_t>(), stream));
    const uint8_t* records = static_cast<const uint8_t*>(recv_records);
    const size_t stride = static_cast<size_t>(layer->record_bytes);
    const size_t tail = static_cast<size_t>(H) / 2 + static_cast<size_t>(H) / 16;
    PermuteSource source;
    source.packed = records;
    source.packed_stride = stride;
    source.sf = records + H / 2;
    source.sf_stride = stride;
    source.tensor_scale = reinterpret_cast<const float*>(records + tail);
    source.tensor_scale_stride = stride;
    source.weight = reinterpret_cast<const float*>(records + tail + 4);
    source.weight_stride = stride;
    source.expert = reinterpret_cast<const int32_t*>(records + tail + 8);
    source.expert_stride = stride;
    source.pairs_per_row = 1;
    source.valid_counts = valid_counts;
    source.capacity = static_cast<int>(capacity_per_rank);
    routed_experts(layer, stream, source, static_cast<int>(count), 1, out_rows,
                   static_cast<RowKind>(rows_dtype));
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_ep_shared(nmoe_layer* layer, void* stream_ptr) {
  if (layer == nullptr || layer->ep_world <= 1 || layer->last_tokens <= 0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  try {
    shared_expert(layer, static_cast<cudaStream_t>(stream_ptr), layer->last_tokens,
                  layer->shared_out.as<float>(), 1, 0, nullptr);
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_ep_combine(nmoe_layer* layer, void* stream_ptr, const void* input,
                            nmoe_dtype input_dtype, const void* returned_rows,
                            nmoe_dtype rows_dtype, void* output, nmoe_dtype output_dtype) {
  if (layer == nullptr || layer->ep_world <= 1 || layer->last_tokens <= 0 || input == nullptr ||
      returned_rows == nullptr || output == nullptr) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  const cudaError_t err = launch_combine_indexed(
      input, input_dtype == NMOE_BF16, returned_rows, static_cast<RowKind>(rows_dtype),
      layer->send_position.as<int32_t>(), layer->shared_out.as<void>(), kRowF32, layer->last_tokens,
      layer->cfg.hidden_size, layer->cfg.top_k, output, output_dtype == NMOE_BF16,
      layer->error.device.as<int32_t>(), static_cast<cudaStream_t>(stream_ptr));
  return err == cudaSuccess ? NMOE_OK : NMOE_ERR_CUDA;
}


// --- peer windows: the exchanges done by the stages' own kernels ------------

namespace {

// the part of nmoe_ep_experts after the records are known to be in place
void experts_over_records(nmoe_layer* layer, cudaStream_t stream, const uint8_t* records,
                          int count, const int32_t* valid_counts, int capacity, void* out_rows,
                          RowKind rows_kind, RowSegments segments) {
  const int H = layer->cfg.hidden_size;
  NMOE_CUDA(cudaMemsetAsync(layer->counts.as<int32_t>(), 0,
                            layer->local_experts * sizeof(int32_t), stream));
  NMOE_CUDA(launch_record_histogram(records, count, H, layer->local_experts, valid_counts,
                                    capacity, layer->counts.as<int32_t>(),
                                    layer->error.device.as<int32_t>(), stream));
  const size_t stride = static_cast<size_t>(layer->record_bytes);
  const size_t tail = static_cast<size_t>(H) / 2 + static_cast<size_t>(H) / 16;
  PermuteSource source;
  source.packed = records;
  source.packed_stride = stride;
  source.sf = records + H / 2;
  source.sf_stride = stride;
  source.tensor_scale = reinterpret_cast<const float*>(records + tail);
  source.tensor_scale_stride = stride;
  source.weight = reinterpret_cast<const float*>(records + tail + 4);
  source.weight_stride = stride;
  source.expert = reinterpret_cast<const int32_t*>(records + tail + 8);
  source.expert_stride = stride;
  source.pairs_per_row = 1;
  source.valid_counts = valid_counts;
  source.capacity = capacity;
  routed_experts(layer, stream, source, count, 1, out_rows, rows_kind, segments);
}

}  // namespace

nmoe_status nmoe_ep_window_create(nmoe_layer* layer, int64_t capacity_per_rank,
                                  nmoe_dtype rows_dtype, void* handle_out) {
  if (layer == nullptr || handle_out == nullptr || layer->ep_world <= 1 ||
      layer->ep_world > 64 || capacity_per_rank <= 0 ||
      (rows_dtype != NMOE_F32 && rows_dtype != NMOE_BF16 && rows_dtype != NMOE_F16)) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  static_assert(sizeof(cudaIpcMemHandle_t) == NMOE_EP_WINDOW_HANDLE_BYTES, "handle size");
  const int64_t slots = capacity_per_rank * layer->ep_world;
  if (slots > layer->max_pairs) return NMOE_ERR_CAPACITY;
  try {
    auto& w = layer->window;
    w.close_peers();
    w.capacity = capacity_per_rank;
    w.rows_kind = static_cast<RowKind>(rows_dtype);
    const size_t H = static_cast<size_t>(layer->cfg.hidden_size);
    auto round_up = [](size_t v) { return (v + 255) / 256 * 256; };
    w.records_off = 0;
    w.rows_off = round_up(static_cast<size_t>(slots) * layer->record_bytes);
    w.flags_off = w.rows_off + round_up(static_cast<size_t>(slots) * H * row_kind_bytes(w.rows_kind));
    w.local.allocate(w.flags_off + 3 * 64 * sizeof(uint32_t), true);
    w.epoch.allocate(sizeof(uint32_t), true);
    NMOE_CUDA(cudaDeviceSynchronize());  // the zeroes are in place before any peer maps it
    cudaIpcMemHandle_t handle;
    NMOE_CUDA(cudaIpcGetMemHandle(&handle, w.local.as<void>()));
    std::memcpy(handle_out, &handle, sizeof(handle));
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_ep_window_attach(nmoe_layer* layer, const void* handles) {
  if (layer == nullptr || handles == nullptr || layer->ep_world <= 1 ||
      layer->window.capacity <= 0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  try {
    auto& w = layer->window;
    const int W = layer->ep_world, me = layer->ep_rank;
    w.close_peers();
    w.peer_base.assign(W, nullptr);
    std::vector<unsigned long long> record_segments(W), row_segments(W), record_flags(W),
        row_flags(W), counts(W);
    const size_t H = static_cast<size_t>(layer->cfg.hidden_size);
    const size_t row_bytes = H * row_kind_bytes(w.rows_kind);
    for (int r = 0; r < W; ++r) {
      uint8_t* base = w.local.as<uint8_t>();
      if (r != me) {
        cudaIpcMemHandle_t handle;
        std::memcpy(&handle, static_cast<const uint8_t*>(handles) + r * sizeof(handle),
                    sizeof(handle));
        void* mapped = nullptr;
        NMOE_CUDA(cudaIpcOpenMemHandle(&mapped, handle, cudaIpcMemLazyEnablePeerAccess));
        w.peer_base[r] = mapped;
        base = static_cast<uint8_t*>(mapped);
      }
      // in rank r's window this rank owns segment `me` of every region
      const size_t segment = static_cast<size_t>(me) * w.capacity;
      record_segments[r] = reinterpret_cast<unsigned long long>(
          base + w.records_off + segment * layer->record_bytes);
      row_segments[r] =
          reinterpret_cast<unsigned long long>(base + w.rows_off + segment * row_bytes);
      uint32_t* flags = reinterpret_cast<uint32_t*>(base + w.flags_off);
      record_flags[r] = reinterpret_cast<unsigned long long>(flags + me);
      row_flags[r] = reinterpret_cast<unsigned long long>(flags + 64 + me);
      counts[r] = reinterpret_cast<unsigned long long>(flags + 128 + me);
    }
    auto upload = [&](DeviceBuffer& buffer, const std::vector<unsigned long long>& host) {
      buffer.allocate(host.size() * sizeof(unsigned long long));
      NMOE_CUDA(cudaMemcpy(buffer.as<void>(), host.data(),
                           host.size() * sizeof(unsigned long long), cudaMemcpyHostToDevice));
    };
    upload(w.record_segments, record_segments);
    upload(w.row_segments, row_segments);
    upload(w.record_flag_slots, record_flags);
    upload(w.row_flag_slots, row_flags);
    upload(w.count_slots, counts);
    w.attached = true;
  } catch (const Failure& failure) {
    layer->window.close_peers();
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_ep_window_detach(nmoe_layer* layer) {
  if (layer == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  cudaDeviceSynchronize();
  layer->window.close_peers();
  return NMOE_OK;
}

nmoe_status nmoe_ep_window_fork_shared(nmoe_layer* layer, int32_t enable) {
  if (layer == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  if (enable != 0 && layer->side_stream == nullptr) return NMOE_ERR_UNSUPPORTED;
  layer->window_fork_shared = enable != 0;
  return NMOE_OK;
}

nmoe_status nmoe_ep_window_dispatch(nmoe_layer* layer, void* stream_ptr, const void* input,
                                    nmoe_dtype input_dtype, int64_t tokens) {
  if (layer == nullptr || input == nullptr || tokens <= 0 || !layer->window.attached) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  if (tokens > layer->cfg.max_tokens) return NMOE_ERR_CAPACITY;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  try {
    const nmoe_config& c = layer->cfg;
    auto& w = layer->window;
    NMOE_CUDA(launch_window_epoch(w.epoch.as<uint32_t>(), stream));
    // The shared expert needs only the quantised rows: with `fork_shared` it starts on
    // the layer's own stream right after the quantiser and runs beside the router and
    // the packing; nmoe_ep_window_combine joins it.
    const bool fork = layer->side_stream != nullptr && layer->window_fork_shared;
    route_tokens(layer, stream, input, input_dtype, static_cast<int>(tokens),
                 fork ? layer->quant_done : nullptr);
    if (fork) {
      NMOE_CUDA(cudaStreamWaitEvent(layer->side_stream, layer->quant_done, 0));
      // the shared expert's rows take the type of the returned rows, so that the
      // combine adds what the single-device layer adds for the same output type
      shared_expert(layer, layer->side_stream, static_cast<int>(tokens),
                    layer->shared_out.as<void>(), 1, 0, nullptr, w.rows_kind);
      NMOE_CUDA(cudaEventRecord(layer->shared_done, layer->side_stream));
    }
    layer->window_shared_pending = fork;
    layer->window_shared_kind = fork ? w.rows_kind : kRowF32;
    NMOE_CUDA(launch_dispatch_plan(layer->counts.as<int32_t>(), c.n_routed_experts,
                                   layer->local_experts, layer->ep_world,
                                   layer->send_counts.as<int32_t>(),
                                   layer->send_offsets.as<int32_t>(),
                                   layer->rank_cursor.as<int32_t>(), stream));
    NMOE_CUDA(launch_pack_records(layer->top_index.as<int32_t>(), layer->top_weight.as<float>(),
                                  static_cast<int>(tokens), c.top_k, layer->local_experts,
                                  layer->y_packed.as<uint8_t>(),
                                  layer->y_sf_row_major.as<uint8_t>(), layer->y_ts.as<float>(),
                                  c.hidden_size, layer->send_offsets.as<int32_t>(),
                                  layer->rank_cursor.as<int32_t>(), static_cast<int>(w.capacity),
                                  nullptr, w.record_segments.as<unsigned long long>(),
                                  layer->send_position.as<int32_t>(),
                                  layer->error.device.as<int32_t>(), stream));
    // every destination learns its record count and that the records are there
    NMOE_CUDA(launch_window_signal(w.record_flag_slots.as<unsigned long long>(),
                                   w.count_slots.as<unsigned long long>(),
                                   layer->send_counts.as<int32_t>(), w.epoch.as<uint32_t>(), 0,
                                   layer->ep_world, stream));
    layer->last_tokens = static_cast<int>(tokens);
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_ep_window_experts(nmoe_layer* layer, void* stream_ptr, int32_t first_source_rank,
                                   int32_t source_ranks) {
  if (layer == nullptr || !layer->window.attached || first_source_rank < 0 ||
      source_ranks <= 0 || first_source_rank + source_ranks > layer->ep_world) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  try {
    auto& w = layer->window;
    const int cap = static_cast<int>(w.capacity);
    NMOE_CUDA(launch_window_wait(w.record_flags(), w.epoch.as<uint32_t>(), first_source_rank,
                                 source_ranks, layer->wait_limit_ticks,
                                 layer->error.device.as<int32_t>(), stream));
    RowSegments segments;
    segments.bases = w.row_segments.as<unsigned long long>();
    segments.rows = cap;
    segments.slot0 = first_source_rank * cap;
    const uint8_t* records = w.local.as<uint8_t>() + w.records_off +
                             static_cast<size_t>(first_source_rank) * cap * layer->record_bytes;
    experts_over_records(layer, stream, records, source_ranks * cap,
                         w.counts() + first_source_rank, cap, nullptr, w.rows_kind, segments);
    NMOE_CUDA(launch_window_signal(w.row_flag_slots.as<unsigned long long>(), nullptr, nullptr,
                                   w.epoch.as<uint32_t>(), first_source_rank, source_ranks,
                                   stream));
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_ep_window_combine(nmoe_layer* layer, void* stream_ptr, const void* input,
                                   nmoe_dtype input_dtype, void* output,
                                   nmoe_dtype output_dtype) {
  if (layer == nullptr || !layer->window.attached || layer->last_tokens <= 0 ||
      input == nullptr || output == nullptr) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  auto& w = layer->window;
  cudaError_t err = launch_window_wait(w.row_flags(), w.epoch.as<uint32_t>(), 0, layer->ep_world,
                                       layer->wait_limit_ticks,
                                       layer->error.device.as<int32_t>(), stream);
  if (err == cudaSuccess && layer->window_shared_pending) {
    err = cudaStreamWaitEvent(stream, layer->shared_done, 0);
    layer->window_shared_pending = false;
  }
  if (err == cudaSuccess) {
    err = launch_combine_indexed(input, input_dtype == NMOE_BF16,
                                 w.local.as<uint8_t>() + w.rows_off, w.rows_kind,
                                 layer->send_position.as<int32_t>(), layer->shared_out.as<void>(),
                                 layer->window_shared_kind, layer->last_tokens, layer->cfg.hidden_size, layer->cfg.top_k,
                                 output, output_dtype == NMOE_BF16,
                                 layer->error.device.as<int32_t>(), stream);
  }
  return err == cudaSuccess ? NMOE_OK : NMOE_ERR_CUDA;
}

const char* nmoe_layer_last_error(const nmoe_layer* layer) {
  return layer == nullptr ? "null layer" : layer->last_error.c_str();
}

nmoe_status nmoe_layer_trace_view(nmoe_layer* layer, nmoe_trace_view* out) {
  if (layer == nullptr || out == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  out->normalized_input = layer->last_normalized ? layer->normalized.as<float>() : nullptr;
  out->router_logits = layer->logits.as<float>();
  out->selected_index = layer->top_index.as<int32_t>();
  out->selected_weight = layer->top_weight.as<float>();
  const bool lat = layer->latent_mode;
  out->act_packed = lat ? layer->lat_packed.as<uint8_t>() : layer->y_packed.as<uint8_t>();
  out->act_scales = lat ? layer->lat_sf_row_major.as<uint8_t>() : layer->y_sf_row_major.as<uint8_t>();
  out->act_tensor_scale = lat ? layer->lat_ts.as<float>() : layer->y_ts.as<float>();
  out->parts = layer->last_parts_kind != kRowF32 ? nullptr : layer->parts.as<float>();
  out->latent_output = lat ? layer->latent_rows.as<float>() : nullptr;
  out->routed_latent_output = lat ? layer->routed_latent.as<float>() : nullptr;
  out->projected_routed_output = lat ? layer->projected.as<float>() : nullptr;
  out->shared_output = lat ? layer->shared_rows.as<float>() : nullptr;
  return NMOE_OK;
}

nmoe_status nmoe_layer_copy_trace_field(nmoe_layer* layer, void* stream, int32_t field, void* dst,
                                        size_t nbytes) {
  if (layer == nullptr || dst == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  nmoe_trace_view view;
  nmoe_layer_trace_view(layer, &view);
  const void* sources[12] = {view.normalized_input, view.router_logits, view.selected_index,
                             view.selected_weight,  view.act_packed,    view.act_scales,
                             view.act_tensor_scale, view.parts,         view.latent_output,
                             view.routed_latent_output, view.projected_routed_output,
                             view.shared_output};
  if (field < 0 || field >= 12 || sources[field] == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  return cudaMemcpyAsync(dst, sources[field], nbytes, cudaMemcpyDefault,
                         static_cast<cudaStream_t>(stream)) == cudaSuccess
             ? NMOE_OK
             : NMOE_ERR_CUDA;
}

nmoe_status nmoe_layer_keep_trace(nmoe_layer* layer, int32_t enable) {
  if (layer == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  if (layer->keep_trace != (enable != 0)) layer->drop_recorded();
  layer->keep_trace = enable != 0;
  return NMOE_OK;
}

nmoe_status nmoe_layer_reserve_tokens(nmoe_layer* layer, int32_t max_tokens) {
  if (layer == nullptr || max_tokens <= 0) return NMOE_ERR_INVALID_ARGUMENT;
  if (max_tokens <= layer->cfg.max_tokens) return NMOE_OK;
  if (layer->window.attached) return NMOE_ERR_INVALID_ARGUMENT;  // peers hold the old window
  try {
    reallocate_scratch(layer, static_cast<size_t>(max_tokens), layer->unfused);
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_layer_set_unfused_activation(nmoe_layer* layer, int32_t enable) {
  if (layer == nullptr) return NMOE_ERR_INVALID_ARGUMENT;
  const bool want = enable != 0;
  if (want == layer->unfused) return NMOE_OK;
  if (want && layer->ep_world > 1) return NMOE_ERR_UNSUPPORTED;
  try {
    if (want && layer->u_raw.bytes() == 0) {
      reallocate_scratch(layer, static_cast<size_t>(layer->cfg.max_tokens), true);
    } else {
      NMOE_CUDA(cudaDeviceSynchronize());
      layer->unfused = want;
    }
  } catch (const Failure& failure) {
    layer->last_error = failure.message;
    return failure.status;
  }
  return NMOE_OK;
}

nmoe_status nmoe_layer_export_unfused(nmoe_layer* layer, void* stream_ptr, float* routed_activated,
                                      float* routed_outputs, float* shared_activated) {
  if (layer == nullptr || layer->last_tokens <= 0 || !layer->last_unfused) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const nmoe_config& c = layer->cfg;
  const int tokens = layer->last_tokens, pairs = tokens * c.top_k;
  cudaError_t err = cudaSuccess;
  if (routed_activated != nullptr) {
    err = launch_gather_rows(layer->u_raw.as<float>(), layer->pair_row.as<int32_t>(), pairs,
                             c.routed_expert_intermediate_size, routed_activated, stream);
  }
  if (err == cudaSuccess && routed_outputs != nullptr) {
    if (tokens > layer->unweighted_tokens) return NMOE_ERR_CAPACITY;
    // kept in the layout of `parts`: [token][top_k (+1 unless latent)][row]
    const int stride = layer->latent_mode ? c.top_k : c.top_k + 1;
    const int cols = layer->latent;
    for (int t = 0; t < tokens && err == cudaSuccess; ++t) {
      err = cudaMemcpyAsync(routed_outputs + static_cast<size_t>(t) * c.top_k * cols,
                            layer->unweighted_rows.as<float>() +
                                static_cast<size_t>(t) * stride * cols,
                            static_cast<size_t>(c.top_k) * cols * sizeof(float),
                            cudaMemcpyDefault, stream);
    }
  }
  if (err == cudaSuccess && shared_activated != nullptr) {
    err = cudaMemcpyAsync(shared_activated, layer->shared_raw.as<float>(),
                          static_cast<size_t>(tokens) * c.shared_expert_intermediate_size *
                              sizeof(float),
                          cudaMemcpyDefault, stream);
  }
  return err == cudaSuccess ? NMOE_OK : NMOE_ERR_CUDA;
}

nmoe_status nmoe_layer_export_hidden(nmoe_layer* layer, void* stream_ptr, uint8_t* routed_packed,
                                     uint8_t* routed_scales, uint8_t* shared_packed,
                                     uint8_t* shared_scales) {
  if (layer == nullptr || layer->last_tokens <= 0) return NMOE_ERR_INVALID_ARGUMENT;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const nmoe_config& c = layer->cfg;
  const int pairs = layer->last_tokens * c.top_k;
  if (routed_packed != nullptr || routed_scales != nullptr) {
    export_rows_kernel<<<pairs, 128, 0, stream>>>(
        layer->h_packed.as<uint8_t>(), layer->h_sf.as<uint8_t>(), layer->pair_row.as<int32_t>(),
        pairs, c.routed_expert_intermediate_size,
        k_blocks_of(c.routed_expert_intermediate_size) * 4, routed_packed, routed_scales);
  }
  if (shared_packed != nullptr || shared_scales != nullptr) {
    export_rows_kernel<<<layer->last_tokens, 128, 0, stream>>>(
        layer->sh_packed.as<uint8_t>(), layer->sh_sf.as<uint8_t>(), nullptr, layer->last_tokens,
        c.shared_expert_intermediate_size, k_blocks_of(c.shared_expert_intermediate_size) * 4,
        shared_packed, shared_scales);
  }
  return cudaGetLastError() == cudaSuccess ? NMOE_OK : NMOE_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// unit operators
// ---------------------------------------------------------------------------

nmoe_status nmoe_quantize_nvfp4(void* stream_ptr, const void* input, nmoe_dtype dtype,
                                int64_t rows, int64_t cols, int32_t per_row, uint8_t* packed,
                                uint8_t* scales_row_major, uint8_t* scales_swizzled,
                                float* tensor_scale) {
  // argument checks of nvfp4_packing.cpp:95-97
  if (input == nullptr || packed == nullptr || scales_row_major == nullptr ||
      tensor_scale == nullptr || rows <= 0 || cols <= 0 || cols % 16 != 0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  cudaError_t err;
  if (per_row != 0) {
    if (scales_swizzled != nullptr) {
      err = cudaMemsetAsync(scales_swizzled, 0, nmoe_swizzled_scale_bytes(rows, cols), stream);
      if (err != cudaSuccess) return NMOE_ERR_CUDA;
    }
    // the tiled layout of this entry point pads blocks to 4, not to a K block
    err = launch_norm_quant(input, dtype == NMOE_BF16, static_cast<int>(rows),
                            static_cast<int>(cols), nullptr, 0.0f, nullptr, packed,
                            scales_row_major, nullptr, 0, tensor_scale, device_sms(), stream);
    if (err == cudaSuccess && scales_swizzled != nullptr) {
      err = launch_swizzle_scales(scales_row_major, static_cast<int>(rows),
                                  static_cast<int>(cols), scales_swizzled, stream);
    }
  } else {
    if (dtype != NMOE_F32) return NMOE_ERR_INVALID_ARGUMENT;
    float* scratch = nullptr;
    if (cudaMallocAsync(reinterpret_cast<void**>(&scratch), sizeof(float), stream) != cudaSuccess) {
      return NMOE_ERR_CUDA;
    }
    err = launch_quant_matrix(static_cast<const float*>(input), static_cast<int>(rows),
                              static_cast<int>(cols), packed, scales_row_major, tensor_scale,
                              scratch, stream);
    cudaFreeAsync(scratch, stream);
    if (err == cudaSuccess && scales_swizzled != nullptr) {
      err = launch_swizzle_scales(scales_row_major, static_cast<int>(rows),
                                  static_cast<int>(cols), scales_swizzled, stream);
    }
  }
  return err == cudaSuccess ? NMOE_OK : NMOE_ERR_CUDA;
}

nmoe_status nmoe_dequant_nvfp4(void* stream, const uint8_t* packed,
                               const uint8_t* scales_row_major, const float* tensor_scale,
                               int32_t per_row, int64_t rows, int64_t cols, float* output) {
  if (packed == nullptr || scales_row_major == nullptr || tensor_scale == nullptr ||
      output == nullptr || rows <= 0 || cols <= 0 || cols % 16 != 0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  return launch_dequant(packed, scales_row_major, tensor_scale, per_row != 0,
                        static_cast<int>(rows), static_cast<int>(cols), output,
                        static_cast<cudaStream_t>(stream)) == cudaSuccess
             ? NMOE_OK
             : NMOE_ERR_CUDA;
}

size_t nmoe_swizzled_scale_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0 || cols % 16 != 0) return 0;
  const size_t padded_rows = (static_cast<size_t>(rows) + 127) / 128 * 128;
  const size_t padded_blocks = (static_cast<size_t>(cols) / 16 + 3) / 4 * 4;
  return padded_rows * padded_blocks;
}

nmoe_status nmoe_swizzle_scales(void* stream, const uint8_t* scales_row_major, int64_t rows,
                                int64_t cols, uint8_t* scales_swizzled) {
  if (scales_row_major == nullptr || scales_swizzled == nullptr || rows <= 0 || cols <= 0 ||
      cols % 16 != 0) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  return launch_swizzle_scales(scales_row_major, static_cast<int>(rows), static_cast<int>(cols),
                               scales_swizzled, static_cast<cudaStream_t>(stream)) == cudaSuccess
             ? NMOE_OK
             : NMOE_ERR_CUDA;
}

nmoe_status nmoe_rmsnorm(void* stream_ptr, const void* input, nmoe_dtype dtype, int64_t rows,
                         int64_t hidden, const float* weight, float epsilon, float* output) {
  if (input == nullptr || weight == nullptr || output == nullptr || rows <= 0 || hidden <= 0 ||
      hidden % 16 != 0 || !(epsilon > 0.0f)) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const cudaError_t err = launch_norm_quant(input, dtype == NMOE_BF16, static_cast<int>(rows),
                                            static_cast<int>(hidden), weight, epsilon, output,
                                            nullptr, nullptr, nullptr, 0, nullptr, device_sms(),
                                            stream);
  return err == cudaSuccess ? NMOE_OK : NMOE_ERR_CUDA;
}

nmoe_status nmoe_router_logits(void* stream, const float* normalized, const float* gate,
                               int64_t rows, int32_t experts, int32_t hidden, float* logits) {
  if (normalized == nullptr || gate == nullptr || logits == nullptr) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  return launch_router_logits(normalized, gate, nullptr, static_cast<int>(rows), experts, hidden,
                              logits, device_sms(),
                              static_cast<cudaStream_t>(stream)) == cudaSuccess
             ? NMOE_OK
             : NMOE_ERR_INVALID_ARGUMENT;
}

nmoe_status nmoe_router_topk(void* stream, const float* logits, const float* bias, int64_t rows,
                             int32_t experts, int32_t top_k, int32_t n_group, int32_t topk_group,
                             int32_t norm_topk_prob, float routed_scaling, int32_t* top_index,
                             float* top_weight) {
  if (logits == nullptr || bias == nullptr || top_index == nullptr || top_weight == nullptr) {
    return NMOE_ERR_INVALID_ARGUMENT;
  }
  return launch_router_topk(logits, bias, static_cast<int>(rows), experts, top_k, n_group,
                            topk_group, norm_topk_prob != 0, routed_scaling, top_index,
                            top_weight, nullptr, nullptr, device_sms(),
                            static_cast<cudaStream_t>(stream)) == cudaSuccess
             ? NMOE_OK
             : NMOE_ERR_INVALID_ARGUMENT;
}

}  // extern "C"
