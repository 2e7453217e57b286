// Expert FFNs of batches that are bound by reading the weights: up and down projections of the
// routed experts and of the shared expert as the tiles of ONE persistent launch.
//
// As four launches (up and down, routed and shared) these sizes paid for every launch's start and
// for every launch's last wave with idle HBM: 64 tokens took 72 + 75 us of routed GEMMs for 670 MB.
// Here the CTAs take tiles from one list -- shared up, routed up, shared down, routed down -- and
// their loads do not stop in between: a down tile needs the quantised hidden rows of its row tile
// only for its A operand, so its weights are on their way before those rows are complete.  A row
// tile's completed up tiles are counted in global memory; the producer of a down tile waits for the
// count (bounded, like every wait here).  Tiles are taken in order with an atomic ticket, so a tile
// that others wait for is always in the hands of a running CTA, however many CTAs of the grid are
// resident beside other work.
//
// Tiles are 128 weight rows (B, BN = 128) of one row tile of up to 128 activation rows (A); the
// activation box is 8 to 128 rows high, by the rows the tile holds, and the last weight tile of
// a matrix loads the rows that exist.  At 148 SMs and the measured copy rate a K block's 18 KB of
// weights take 800 cycles to arrive; its eight scale copies and four MMAs, issued in order by one
// warp, take about 300.
//
// Roles: warp 0 takes tiles and loads weights, warp 11 loads activation rows (and waits for them:
// finding out and ordering the copies behind it takes over 1000 cycles a tile, which must not hold
// up the weights), warp 1 issues scale copies and MMAs, warps 2-9 run epilogues, warp 10 hands
// finished tiles on.
// Measured, whole pass of the benchmark layer: 64 tokens 196 -> 154 us, 256 tokens 205 -> 166,
// 1003 tokens 240 -> 209.
#include <algorithm>

#include "common.cuh"
#include "gemm_common.cuh"
#include "kernels.h"

namespace nmoe {
namespace {

constexpr int kBN = 128;
constexpr int kMaxStages = 8;
constexpr int kEpilogueWarps = 8;  // two per TMEM lane quarter
constexpr int kSignalWarp = 2 + kEpilogueWarps;
constexpr int kRowWarp = kSignalWarp + 1;
constexpr int kThreads = (kRowWarp + 1) * 32;
constexpr int kBBytes = kBN * 128;
constexpr int kSfaBytes = 2048;
constexpr int kSfbBytes = 2048;     // four groups of 32 weight rows x four MMAs x 16 bytes
constexpr int kSfBufs = 2;
constexpr int kSfBufCols = 32;      // TMEM columns of one K block's scales: 16 for A, 16 for B
constexpr int kSfCol = 2 * kBN;     // behind the two accumulators
constexpr int kTmemCols = 512;
static_assert(kSfCol + kSfBufs * kSfBufCols <= kTmemCols, "TMEM budget");

// Where a tile of the list lies.
struct Tile {
  int phase;   // -1: no more tiles
  int row0;    // first row of its 128-row slot
  int rows;    // valid rows in it
  int expert;
  int nt;      // weight tile
};

// The producer hands tiles to the other roles through a ring in shared memory.
constexpr int kRing = 4;
constexpr int kRingReaders = 1 + kEpilogueWarps + 1 + 1;
constexpr int kBarBytes =
    ((2 * kMaxStages + 6 + 2 * kRing) * 8 + kRing * static_cast<int>(sizeof(Tile)) + 16 + 15) / 16 *
    16;

// Tiles of up to kFewRows rows hand their accumulator over through shared memory: a thread per row
// would leave most lanes of the two warps that can read those rows idle and the others with four
// chunks in turn.
constexpr int kFewRows = 16;
constexpr int kFewStride = kBN / 2 + 4;  // floats per row of one warp's half of the columns
constexpr int kFewRowsBytes = 2 * kFewRows * kFewStride * 4;

// The room for activation rows in a stage is no larger than the launch's tiles (32, 64 or 128 rows).
constexpr int stage_bytes(int tile_rows) {
  return tile_rows * 128 + kBBytes + kSfaBytes + kSfbBytes;
}
constexpr int stages_for(int tile_rows) { return tile_rows <= 32 ? 8 : tile_rows <= 64 ? 7 : 6; }
constexpr int smem_bytes(int tile_rows) {
  return stages_for(tile_rows) * stage_bytes(tile_rows) + kBarBytes + kFewRowsBytes + 1024;
}
static_assert(smem_bytes(32) <= kMaxSharedBytes && smem_bytes(64) <= kMaxSharedBytes &&
                  smem_bytes(128) <= kMaxSharedBytes,
              "shared memory budget");
// The MMA always reads 128 A rows: behind a stage of fewer rows it reads what follows (those output
// rows are never stored), which must lie inside the allocation.
static_assert(stages_for(32) * kBBytes >= 128 * 128, "A over-read stays inside shared memory");

struct TileList {
  int first[kStreamPhases + 1];  // first tile of each phase, then the end
  // The first row tiles of the grouped phases, two to a lane: a launch's first tile is looked up without
  // another trip to memory, while its ticket is fetched (64 tokens 132.5 -> 131.3 us, 7 tokens 53.5 -> 53.2).
  RowTile kept[2];
  int kept_count;
  // By all lanes of a warp; `ticket` is on its way meanwhile.
  __device__ __forceinline__ void load(const StreamArgs& args) {
    const int lane = threadIdx.x & 31;
    kept_count = min(64, args.row_tile_room);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      kept[i] = RowTile{};
      if (lane + 32 * i < kept_count) kept[i] = args.row_tiles[lane + 32 * i];
    }
    int running = 0;
#pragma unroll
    for (int p = 0; p < kStreamPhases; ++p) {
      first[p] = running;
      if (p < args.phases) {
        const GemmArgs& g = args.phase[p].gemm;
        const int row_tiles =
            warp_uniform(g.row_tiles != nullptr ? *g.num_row_tiles : (g.dense_rows + 127) / 128);
        running += row_tiles * g.n_tiles;
      }
    }
    first[kStreamPhases] = running;
  }
  __device__ __forceinline__ int total() const { return first[kStreamPhases]; }
  __device__ __forceinline__ Tile locate(const StreamArgs& args, int t) const {
    Tile tile;
    tile.phase = t < total() ? 0 : -1;
    tile.row0 = tile.rows = tile.expert = tile.nt = 0;
    if (tile.phase < 0) return tile;
    int base = 0;
#pragma unroll
    for (int p = 1; p < kStreamPhases; ++p) {
      if (t >= first[p] && p < args.phases) {
        tile.phase = p;
        base = first[p];
      }
    }
    const GemmArgs& g = args.phase[tile.phase].gemm;
    const int index = t - base;
    const int rt = index / g.n_tiles;
    tile.nt = index - rt * g.n_tiles;
    if (g.row_tiles != nullptr) {
      RowTile row_tile = rt < 32 ? kept[0] : kept[1];
      const int from = rt < kept_count ? rt & 31 : 0;
      if (rt >= kept_count) row_tile = g.row_tiles[rt];
      tile.row0 = __shfl_sync(0xffffffffu, row_tile.row0, from);
      tile.rows = __shfl_sync(0xffffffffu, row_tile.rows, from);
      tile.expert = __shfl_sync(0xffffffffu, row_tile.expert, from);
    } else {
      tile.row0 = rt * 128;
      tile.rows = min(128, g.dense_rows - tile.row0);
      tile.expert = 0;
    }
    return tile;
  }
};

__device__ __forceinline__ int load_acquire(const int32_t* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// What it held.  (With a fence behind it in the place of the acquire every short launch took 0.6 us more.)
__device__ __forceinline__ int add_acquire(int32_t* p, int v) {
  int before;
  asm volatile("atom.acquire.gpu.global.add.s32 %0, [%1], %2;" : "=r"(before) : "l"(p), "r"(v) : "memory");
  return before;
}

__device__ __forceinline__ void add_release(int32_t* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Orders generic accesses (other SMs' stores, once they have been acquired) before those of the async
// proxy (bulk and tensor copies).
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

// The smallest activation box (8 << box rows) that holds `rows`.
__device__ __forceinline__ int box_of(int rows) { return rows <= 8 ? 0 : 29 - __clz(rows - 1); }

// Waits (about a second at most) until *count >= target; by all lanes of a warp.
__device__ __forceinline__ bool wait_count(const int32_t* count, int target) {
  const long long start = clock64();
  while (!__all_sync(0xffffffffu, load_acquire(count) >= target)) {
    if (__any_sync(0xffffffffu, clock64() - start > (1ll << 31))) return false;
  }
  return true;
}

// The next tile from the ring, by all lanes of a warp.
struct RingReader {
  const volatile Tile* ring;
  uint32_t full0, empty0;
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ bool next(Tile& tile) {
    if (!mbar_wait_warp(full0 + slot * 8, phase)) return false;
    tile.phase = warp_uniform(static_cast<int>(ring[slot].phase));
    tile.row0 = warp_uniform(static_cast<int>(ring[slot].row0));
    tile.rows = warp_uniform(static_cast<int>(ring[slot].rows));
    tile.expert = warp_uniform(static_cast<int>(ring[slot].expert));
    tile.nt = warp_uniform(static_cast<int>(ring[slot].nt));
    __syncwarp();
    if (elect_one()) mbar_arrive_at(empty0 + slot * 8);
    if (++slot == kRing) {
      slot = 0;
      phase ^= 1u;
    }
    return true;
  }
};

// The scale copies and MMAs of a K block that holds MMAS times 64 elements (copies and MMAs of one
// thread execute in order).
template <int MMAS>
__device__ __forceinline__ void issue_block(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                            uint64_t sfa_desc, uint64_t sfb_desc, uint32_t sf_tmem,
                                            uint32_t idesc, int kb) {
#pragma unroll
  for (int c = 0; c < MMAS; ++c) {
    tcgen05_cp_32x128b_warpx4(sf_tmem + 4 * c, advance_smem_desc(sfa_desc, c * 512));
    tcgen05_cp_32x128b_warpx4(sf_tmem + 16 + 4 * c, advance_smem_desc(sfb_desc, c * 512));
  }
#pragma unroll
  for (int kt = 0; kt < MMAS; ++kt) {
    tcgen05_mma_nvf4(d_tmem, advance_smem_desc(a_desc, kt * 32), advance_smem_desc(b_desc, kt * 32),
                     idesc, sf_tmem + 4 * kt, sf_tmem + 16 + 4 * kt, kt != 0 ? 1u : kb != 0 ? 1u : 0u);
  }
}

// The weights of the shared expert's (dense) phases into L2, tile by tile over all CTAs: HBM is idle
// while the small kernels before this one route the tokens.
__device__ __forceinline__ void fetch_dense_weights(const StreamArgs& args, int unit, int units,
                                                    int lane) {
  for (int p = 0; p < args.phases; ++p) {
    const GemmArgs& g = args.phase[p].gemm;
    if (g.row_tiles != nullptr) continue;
    for (int nt = unit; nt < g.n_tiles; nt += units) {
      const int b_row = nt * kBN;
      const uint32_t b_bytes = static_cast<uint32_t>(min(kBN, g.N - b_row)) * 128u;
      for (int kb = lane; kb < g.kb_full; kb += 32) {
        prefetch_l2_bulk(g.b_full + (static_cast<size_t>(kb) * g.N + b_row) * 128, b_bytes);
      }
      if (lane == 0) {
        prefetch_l2_bulk(g.sfb + static_cast<size_t>(nt) * g.k_blocks * kSfbBytes,
                         static_cast<uint32_t>(g.k_blocks) * kSfbBytes);
      }
    }
  }
}

// TOKEN_ORDER: some phase's row tiles hold all tokens in token order (StreamPhase::used).  A kernel of its
// own, since layers of many small experts have some fifty tiles an SM and looking it up in each of them
// showed (384 experts of 512 at 400 tokens 166.5 us without and 168.4 with it, 256 of 768 at 64 tokens 99.8
// and 101.1).
template <bool TOKEN_ORDER>
__global__ void __launch_bounds__(kThreads, 1)
expert_stream_kernel(const __grid_constant__ StreamArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) &
                                             ~static_cast<uintptr_t>(1023u));
  uint8_t* sA = smem;
  const int stages = stages_for(args.tile_rows);
  const int a_room = args.tile_rows * 128;
  uint8_t* sB = sA + stages * a_room;
  uint8_t* sSFA = sB + stages * kBBytes;
  uint8_t* sSFB = sSFA + stages * kSfaBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sSFB + stages * kSfbBytes);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* tmem_full_bar = empty_bar + kMaxStages;
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;
  uint64_t* stored_bar = tmem_empty_bar + 2;
  uint64_t* ring_full_bar = stored_bar + 2;
  uint64_t* ring_empty_bar = ring_full_bar + kRing;
  volatile Tile* ring = reinterpret_cast<volatile Tile*>(ring_empty_bar + kRing);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(
      reinterpret_cast<uint8_t*>(ring_empty_bar + kRing) + kRing * sizeof(Tile));

  const int warp = warp_uniform(static_cast<int>(threadIdx.x >> 5));
  const int lane = threadIdx.x & 31;
  const int unit = static_cast<int>(blockIdx.x);
  const int units = static_cast<int>(gridDim.x);

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full_bar[a], 1);
      mbar_init(&tmem_empty_bar[a], 1);
      mbar_init(&stored_bar[a], kEpilogueWarps);
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&ring_full_bar[i], 1);
      mbar_init(&ring_empty_bar[i], kRingReaders);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  release_successor();
  if (warp == 0 && args.fetch_dense) fetch_dense_weights(args, unit, units, lane);
  wait_for_predecessor();

  float* few_rows = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(full_bar) + kBarBytes);
  const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB), sfa0 = smem_u32(sSFA), sfb0 = smem_u32(sSFB);
  const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
  RingReader reader{ring, smem_u32(ring_full_bar), smem_u32(ring_empty_bar)};

  if (warp == 0) {
    // ------------------------------------------------------- tiles and weights
    TileList list;
    int slot = 0;
    uint32_t slot_phase = 0;
    int stage = 0;
    uint32_t phase = 0;
    // without a ticket word (nothing waits for another tile then) the tiles are dealt out
    auto take = [&](int dealt) {
      return args.ticket != nullptr && lane == 0 ? atomicAdd(args.ticket, 1) : dealt;
    };
    bool ok = true;
    const int first = take(unit);
    list.load(args);
    int t = warp_uniform(first);
    while (ok) {
      const Tile tile = list.locate(args, t);
      if (!mbar_wait_warp(reader.empty0 + slot * 8, slot_phase ^ 1u)) {
        report_timeout(args.error);
        break;
      }
      if (elect_one()) {
        ring[slot].phase = tile.phase;
        ring[slot].row0 = tile.row0;
        ring[slot].rows = tile.rows;
        ring[slot].expert = tile.expert;
        ring[slot].nt = tile.nt;
        mbar_arrive_at(reader.full0 + slot * 8);
      }
      if (++slot == kRing) {
        slot = 0;
        slot_phase ^= 1u;
      }
      if (tile.phase < 0) break;
      // The next ticket is on its way while this tile's loads are issued.  (A CTA that waits for
      // hidden rows holds no up tile then: those come first in the list.)
      const int next = take(t + units);
      const StreamPhase& ph = args.phase[tile.phase];
      const GemmArgs& g = ph.gemm;
      const int k_blocks = g.k_blocks;
      const uint32_t a_bytes = 8u * 128u << box_of(tile.rows);
      const int b_row = tile.nt * kBN;
      const uint32_t b_bytes = static_cast<uint32_t>(min(kBN, g.N - b_row)) * 128u;
      const uint8_t* sfb_src =
          g.sfb + (static_cast<size_t>(tile.expert) * g.n_tiles + tile.nt) * k_blocks * kSfbBytes;
      const uint8_t* b_src =
          g.b_full + (static_cast<size_t>(tile.expert) * g.kb_full * g.N + b_row) * 128;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_warp(empty0 + stage * 8, phase ^ 1u)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t bar = full0 + stage * 8;
          const bool full_block = kb < g.kb_full;
          // (the bytes of warp kRowWarp's copies are counted here too)
          mbar_arrive_expect_tx_at(bar, a_bytes + (full_block ? b_bytes : kBBytes) + kSfaBytes +
                                            kSfbBytes);
          if (full_block) {
            // one contiguous, pre-swizzled panel slice: a single bulk copy
            bulk_load_at(b0 + stage * kBBytes, b_src + static_cast<size_t>(kb) * g.N * 128, b_bytes,
                         bar);
          } else {
            tma_load_2d_at(b0 + stage * kBBytes, &ph.b_tail, 0, tile.expert * g.N + b_row, bar);
          }
          bulk_load_at(sfb0 + stage * kSfbBytes, sfb_src + kb * kSfbBytes, kSfbBytes, bar);
        }
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) report_timeout(args.error);
      t = warp_uniform(next);
    }
  } else if (warp == kRowWarp) {
    // --------------------------------------------------------- activation rows
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    while (ok) {
      Tile tile;
      if (!reader.next(tile)) {
        report_timeout(args.error);
        break;
      }
      if (tile.phase < 0) break;
      const StreamPhase& ph = args.phase[tile.phase];
      const GemmArgs& g = ph.gemm;
      const int k_blocks = g.k_blocks;
      const int box = box_of(tile.rows);
      const int a_row0 = TOKEN_ORDER && ph.used != nullptr ? 0 : tile.row0;
      const uint8_t* sfa_src = g.sfa + static_cast<size_t>(a_row0 >> 7) * k_blocks * kSfaBytes;
      if (ph.wait_target > 0) {
        ok = wait_count(ph.ready + (tile.row0 >> 7), ph.wait_target);
        fence_proxy_async();
      }
      for (int kb = 0; kb < k_blocks && ok; ++kb) {
        ok = mbar_wait_warp(empty0 + stage * 8, phase ^ 1u);
        if (ok && elect_one()) {
          const uint32_t bar = full0 + stage * 8;
          tma_load_2d_at(a0 + stage * a_room, &ph.a[box], kb * 128, a_row0, bar);
          bulk_load_at(sfa0 + stage * kSfaBytes, sfa_src + kb * kSfaBytes, kSfaBytes, bar);
        }
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) report_timeout(args.error);
    }
  } else if (warp == 1) {
    // -------------------------------------------------- scale copies and MMAs
    constexpr uint32_t idesc = make_idesc_nvf4(kBN);
    const uint64_t a_desc0 = make_smem_desc(a0, 0, 1024, 2);
    const uint64_t b_desc0 = make_smem_desc(b0, 0, 1024, 2);
    const uint64_t sfa_desc0 = make_smem_desc(sfa0, 0, 128, 0);
    const uint64_t sfb_desc0 = make_smem_desc(sfb0, 0, 128, 0);
    int stage = 0;
    uint32_t phase = 0;
    uint32_t sf_buf = 0;
    bool ok = true;
    for (int local = 0; ok; ++local) {
      Tile tile;
      const int acc = local & 1;
      if (!reader.next(tile)) {
        report_timeout(args.error);
        break;
      }
      if (tile.phase < 0) break;
      if (!mbar_wait_warp(smem_u32(&tmem_empty_bar[acc]), ((local >> 1) & 1u) ^ 1u)) {
        report_timeout(args.error);
        break;
      }
      const GemmArgs& g = args.phase[tile.phase].gemm;
      const int k_blocks = g.k_blocks, last_mmas = g.K / 64 - 4 * (k_blocks - 1);
      tcgen05_fence_after();
      const uint32_t d_tmem = tmem_base + acc * kBN;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_warp(full0 + stage * 8, phase)) {
          report_timeout(args.error);
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const uint64_t a_desc = advance_smem_desc(a_desc0, stage * a_room);
        const uint64_t b_desc = advance_smem_desc(b_desc0, stage * kBBytes);
        const uint64_t sfa_desc = advance_smem_desc(sfa_desc0, stage * kSfaBytes);
        const uint64_t sfb_desc = advance_smem_desc(sfb_desc0, stage * kSfbBytes);
        const uint32_t sf_tmem = tmem_base + kSfCol + sf_buf * kSfBufCols;
        if (elect_one()) {
          if (kb + 1 < k_blocks || last_mmas == 4) {
            issue_block<4>(d_tmem, a_desc, b_desc, sfa_desc, sfb_desc, sf_tmem, idesc, kb);
          } else if (last_mmas == 3) {
            issue_block<3>(d_tmem, a_desc, b_desc, sfa_desc, sfb_desc, sf_tmem, idesc, kb);
          } else if (last_mmas == 2) {
            issue_block<2>(d_tmem, a_desc, b_desc, sfa_desc, sfb_desc, sf_tmem, idesc, kb);
          } else {
            issue_block<1>(d_tmem, a_desc, b_desc, sfa_desc, sfb_desc, sf_tmem, idesc, kb);
          }
          tcgen05_commit_at(empty0 + stage * 8);
        }
        sf_buf ^= 1u;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok && elect_one()) tcgen05_commit(&tmem_full_bar[acc]);
    }
  } else if (warp == kSignalWarp) {
    // ---------------------------------------------------------------- signals
    // Once the epilogue warps have stored a tile: give its accumulator back, and count the tile
    // for the down projection.  Making the stores visible first takes some 1500 cycles, which here
    // nobody waits for.
    for (int local = 0;; ++local) {
      Tile tile;
      const int acc = local & 1;
      if (!reader.next(tile)) {
        report_timeout(args.error);
        break;
      }
      if (tile.phase < 0) break;
      if (!mbar_wait_warp(smem_u32(&stored_bar[acc]), (local >> 1) & 1u)) {
        report_timeout(args.error);
        break;
      }
      const StreamPhase& ph = args.phase[tile.phase];
      if (lane == 0) {
        mbar_arrive(&tmem_empty_bar[acc]);
        if (ph.mode == kGemmUp && ph.ready != nullptr) {
          __threadfence();
          add_release(ph.ready + (tile.row0 >> 7), 1);
        }
      }
      __syncwarp();
    }
  } else {
    // -------------------------------------------------------------- epilogue
    const int quarter = warp & 3;           // TMEM lanes a warp may read: 32 * (warp % 4)
    const int half = (warp - 2) >> 2;       // which half of the tile's columns
    const int r = quarter * 32 + lane;      // row inside the tile == TMEM lane
    constexpr int kHalfChunks = kBN / 16 / 2;
    for (int local = 0;; ++local) {
      const int acc = local & 1;
      const uint32_t acc_phase = (local >> 1) & 1u;
      Tile tile;
      if (!reader.next(tile)) {
        report_timeout(args.error);
        break;
      }
      if (tile.phase < 0) break;
      const StreamPhase& ph = args.phase[tile.phase];
      const GemmArgs& g = ph.gemm;
      const int grow = tile.row0 + r;
      const int32_t* used = TOKEN_ORDER ? ph.used : nullptr;
      const bool row_valid = r < tile.rows && (used == nullptr || used[grow] >= 0);
      float scale = g.w_tensor_scale[tile.expert];
      if (g.a_tensor_scale != nullptr && row_valid) {
        scale *= g.a_tensor_scale[used != nullptr ? r : grow];
      }
      unsigned long long dest = row_valid ? 1 : 0;  // (up: whether the row counts)
      float wt = 1.0f;
      if (ph.mode == kGemmDown && row_valid) {
        dest = output_row_address(g, grow);
        if (g.row_weight != nullptr) wt = g.row_weight[grow];
      }
      if (!mbar_wait(&tmem_full_bar[acc], acc_phase)) {
        report_timeout(args.error);
        break;
      }
      const int n0 = tile.nt * kBN;
      const uint32_t t_addr =
          tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * kBN;
      if (tile.rows <= kFewRows) {
        if (quarter == 0) {
          tcgen05_fence_after();
          const int columns = min(kBN / 2, g.N - n0 - half * (kBN / 2));  // may be none
          float* few = few_rows + half * (kFewRows * kFewStride);
#pragma unroll 1
          for (int c = 0; c < columns; c += 16) {
            float v[16];
            tmem_ld_x16(t_addr + half * (kBN / 2) + c, v);
            if (row_valid) {
#pragma unroll
              for (int i = 0; i < 16; i += 4) {
                *reinterpret_cast<float4*>(few + r * kFewStride + c + i) =
                    make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
              }
            }
          }
          tcgen05_fence_before();
          __syncwarp();
          // one 16-column chunk of one row per lane and round, four chunks to a row
#pragma unroll 1
          for (int first = 0; first < tile.rows * 4; first += 32) {
            const int from = (first + lane) >> 2, chunk = lane & 3;
            const float row_scale = __shfl_sync(0xffffffffu, scale, from & 31);
            const float row_wt = __shfl_sync(0xffffffffu, wt, from & 31);
            const unsigned long long row_dest = __shfl_sync(0xffffffffu, dest, from & 31);
            const int n = n0 + half * (kBN / 2) + chunk * 16;
            if (from >= tile.rows || chunk * 16 >= columns) continue;
            if ((TOKEN_ORDER || ph.mode == kGemmDown) && row_dest == 0) continue;
            float v[16];
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 four = *reinterpret_cast<const float4*>(
                  few + from * kFewStride + chunk * 16 + i);
              v[i] = four.x;
              v[i + 1] = four.y;
              v[i + 2] = four.z;
              v[i + 3] = four.w;
            }
            if (ph.mode == kGemmUp) {
              uint32_t lo, hi, sf;
              report_range(g, quantise_chunk(v, row_scale, lo, hi, sf));
              *reinterpret_cast<uint2*>(hidden_codes(g, tile.row0 + from, n / 16)) =
                  make_uint2(lo, hi);
              *hidden_scale(g, tile.row0 + from, n / 16) = static_cast<uint8_t>(sf);
            } else {
              store_chunk(g, v, n, row_dest, row_scale, row_wt);
            }
          }
        }
      } else if (quarter * 32 < tile.rows) {  // (else none of the warp's rows exist)
        tcgen05_fence_after();
        if (ph.mode == kGemmUp) {
          epilogue_quantise<2>(g, t_addr, n0, half * kHalfChunks, (half + 1) * kHalfChunks, grow,
                               row_valid, scale);
        } else {
          epilogue_rows_direct<2>(g, t_addr, n0, half * kHalfChunks, (half + 1) * kHalfChunks, dest,
                                  scale, wt);
        }
        tcgen05_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&stored_bar[acc]);
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  } else if (warp == 0 && args.ticket != nullptr) {
    // the last CTA leaves the counts at zero for the next launch, and the words of the front end before it
    int ticket = 0;
    if (lane == 0) {
      __threadfence();
      ticket = add_acquire(args.finished, 1);
    }
    ticket = __shfl_sync(0xffffffffu, ticket, 0);
    if (ticket == units - 1) {
      if (lane == 0 && args.error_host != nullptr) {
        const int code = *static_cast<volatile int32_t*>(args.error);
        if (code != kDevOk) {
          *static_cast<volatile int32_t*>(args.error_host) = code;
          __threadfence_system();
        }
      }
      for (int i = lane; i < args.ready_count; i += 32) args.ready[i] = 0;
      if (TOKEN_ORDER && lane < args.front_word_count) args.front_words[lane] = 0;
      if (lane == 0) {
        *args.ticket = 0;
        *args.finished = 0;
      }
    }
  }
}

}  // namespace

GemmTileInfo stream_tile_info() { return GemmTileInfo{kBN, 4, kSfbBytes, kBN}; }

cudaError_t launch_expert_stream(const StreamArgs& args, int num_sms, LaunchStream stream) {
  if (args.phases < 1 || args.phases > kStreamPhases || num_sms < 1 ||
      (args.tile_rows != 32 && args.tile_rows != 64 && args.tile_rows != 128)) {
    return cudaErrorInvalidValue;
  }
  // one persistent CTA per SM, fewer when the tiles are known to be fewer
  int grid = num_sms;
  int dense_tiles = 0;
  bool grouped = false, token_order = false;
  for (int p = 0; p < args.phases; ++p) {
    const GemmArgs& g = args.phase[p].gemm;
    grouped = grouped || g.row_tiles != nullptr;
    token_order = token_order || args.phase[p].used != nullptr;
    dense_tiles += (g.dense_rows + 127) / 128 * g.n_tiles;
  }
  if (!grouped) grid = std::max(1, std::min(grid, dense_tiles));
  auto run = [&](auto kernel) {
    const cudaError_t err = allow_shared_memory(kernel);
    if (err != cudaSuccess) return err;
    return launch_kernel(kernel, grid, kThreads, smem_bytes(args.tile_rows), stream, args);
  };
  return token_order ? run(expert_stream_kernel<true>) : run(expert_stream_kernel<false>);
}

}  // namespace nmoe
