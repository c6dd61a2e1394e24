// Ranks the rows of a batch (rank_pack.h) with LANE = FEATURE, for rows of more than 64 features whose
// rank tables are small enough: 32 neighbouring features (a slab) lie interleaved in shared memory, word
// lane of every 128-byte line belonging to feature lane, so a look-up or a search step of a warp is one
// wavefront whatever its lanes ask for -- with a feature's table to itself (rank_rows.cuh) 32 rows that ask
// for 32 buckets meet in the banks, about 3.4 wavefronts.  A row's 32 values are one 128-byte request, and
// nothing has to be turned around before it is ranked; the ranks are, 32 rows at a time, on their way out.
//
// A block keeps one slab's table (one bulk copy, laid out by make_slab_tables) and takes a range of the tiles; the blocks of
// neighbouring slabs go through the rows side by side, so that the 128-byte pieces of a row are asked for at about the same time.
// A warp ranks a tile of 32 rows at a time; the values of its next tile are asked for as soon as registers are free, 24 to
// 32 rows ahead, without a branch or a copy that would wait for them.
// Bound: issue, 71 % busy with 26 instructions per 32 values (three search steps); the table's copy and the first rows'
// way to the block for small batches.  50003 rows x 90 features of about 440 thresholds: 13.7 us, with tables apart and rows
// turned around first (tb_rank_rows) 28.3; 18944 rows x 2000 features of about 130: 51 us, 3.0 TB/s of row values.
//
// Reference counterpart: none (the reference compares fp32 values; see rank_pack.h).
#pragma once
#include "rank_rows.cuh"
#include "walk_quant.cuh"

namespace tb {

constexpr int kSlabWarps = 16, kSlabHeadBytes = 512; // per feature: scale, bias, largest threshold, lattice
constexpr int32_t kStatusRanking = 5; // status of a wait that gave up here (walks: 4)
constexpr int kSlabTurnBytes = 32 * 17 * 4;          // per warp: 32 rows x 32 ranks, rows 17 words apart (bytes: 9)
constexpr int slab_smem_bytes(uint32_t table_bytes) { return 128 + kSlabWarps * kSlabTurnBytes + (int)table_bytes; }

struct SlabParams {
  const float *rows;
  long long n_rows;
  uint32_t ld_bytes; // (32 rows within 32 bits; where a tile starts is a matter of 64)
  const unsigned char *tables; // a table per slab
  unsigned char *keys;         // tiles of tile_bytes
  uint32_t table_bytes, buckets, tile_bytes;
  int32_t num_features, steps;
  unsigned long long *searched; // statistics, as in rank_rows.cuh
  int32_t used;
  int32_t *status;
  int32_t skip_copy;   // failure drill: the tables are never copied, so the wait for them expires
  uint32_t wait_tries; // polls before the wait gives up (0 = kQWaitTries)
};

// BYTES: keys of one byte (rank_pack.h).  STEPS: search steps of a bucket (0: p.steps of them).  LATTICE: some features are
// lattice features, whose whole numbers the statistics leave out (a variant of its own: 0.5 % for all forests otherwise).
template <bool BYTES, int STEPS, bool LATTICE> __global__ void __launch_bounds__(32 * kSlabWarps, 1) tb_rank_slabs(const SlabParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw);
  const uint32_t turn = smem_u32(smem_raw) + 128u + (uint32_t)(warp * kSlabTurnBytes);
  unsigned char *table = smem_raw + 128 + kSlabWarps * kSlabTurnBytes;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const uint32_t tries = p.wait_tries ? p.wait_tries : kQWaitTries;
  const uint32_t mine = smem_u32(table) + (uint32_t)lane * 4u;
  const uint32_t bucket0 = mine + kSlabHeadBytes, thr0 = bucket0 + 128u * p.buckets; // the first bucket, the first threshold
  const int slab = blockIdx.x, f = slab * 32 + lane;
  const bool used = f < p.num_features;
  const int n_rows = (int)p.n_rows, tiles = (n_rows + 31) / 32;
  int tile = (int)((long long)tiles * blockIdx.y / gridDim.y) + warp;
  const int end = (int)((long long)tiles * (blockIdx.y + 1) / gridDim.y);
  if (threadIdx.x == 0) mbar_expect_tx(bar, p.table_bytes);
  __syncthreads();
  if (warp == 0 && lane < 8 && !p.skip_copy) { // (copies of one thread queue up)
    const uint32_t piece = (p.table_bytes / 128u + 7u) / 8u * 128u, at = min(piece * (uint32_t)lane, p.table_bytes);
    const uint32_t bytes = min(piece, p.table_bytes - at);
    if (bytes) bulk_g2s(table + at, p.tables + (size_t)slab * p.table_bytes + at, bytes, bar);
  }
  const char *column = reinterpret_cast<const char *>(p.rows + (used ? f : p.num_features - 1));
  // rows c .. c + 7 of tile t, as far as there are any (the others keep the values of rows before)
  float x[32];
  auto fetch = [&](int t, auto first) {
    constexpr int c = decltype(first)::value;
    const int rows = t < end ? n_rows - t * 32 : 0;
    const char *tile_at = column + (long long)t * (32ll * p.ld_bytes);
    uint32_t at = c * p.ld_bytes;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %2, %3;\n @p ld.global.nc.f32 %0, [%1];\n}" : "+f"(x[c + k]) : "l"(tile_at + at), "r"(rows), "r"(c + k));
      at += p.ld_bytes;
    }
  };
#pragma unroll
  for (int r = 0; r < 32; ++r) x[r] = 0.f;
  fetch(tile, std::integral_constant<int, 0>());
  fetch(tile, std::integral_constant<int, 8>());
  fetch(tile, std::integral_constant<int, 16>());
  fetch(tile, std::integral_constant<int, 24>());
  const bool ok = mbar_wait_all_lanes(smem_u32(bar), 0, tries);
  if (__syncthreads_or(!ok)) { // (no copy may land after the block is gone)
    mbar_wait_all_lanes(smem_u32(bar), 0, tries);
    if (threadIdx.x == 0) set_status(p.status, kStatusRanking);
    return;
  }
  const float scale = lds_f32(mine), bias = lds_f32(mine + 128u), most = lds_f32(mine + 256u);
  [[maybe_unused]] const bool lattice = lds_u32(mine + 384u) != 0;
  unsigned looked_up = 0;
  for (; tile < end; tile += kSlabWarps) {
    auto rank8 = [&](auto first) {
      constexpr int c = decltype(first)::value;
      if constexpr (LATTICE) {
#pragma unroll
        for (int k = 0; k < 8; ++k) looked_up += lattice && tile * 32 + c + k < n_rows && x[c + k] == floorf(x[c + k]);
      }
      uint32_t at[8]; // address of the first threshold that may be above the value
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        // (the largest threshold stands for all that is above it and for NaN; a conversion to an unsigned number takes
        // what is below zero to zero)
        x[c + k] = fminf(x[c + k], most);
        const uint32_t b = __float2uint_rz(__fmaf_rn(x[c + k], scale, bias));
        at[k] = thr0 + lds_u32(bucket0 + 128u * b);
      }
      auto step = [&](uint32_t lines) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (!(x[c + k] < lds_f32(at[k] + 128u * (lines - 1u)))) at[k] += 128u * lines;
      };
      if constexpr (STEPS == 0)
        for (uint32_t lines = 1u << (p.steps - 1); lines; lines >>= 1) step(lines);
      if constexpr (STEPS > 2) step(4u);
      if constexpr (STEPS > 1) step(2u);
      if constexpr (STEPS > 0) step(1u);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t rank = (at[k] - thr0) >> 7;
        if constexpr (BYTES) sts_u8(turn + (uint32_t)((c + k) * 36 + lane), rank);
        else sts_u16(turn + (uint32_t)((c + k) * 68 + lane * 2), rank);
      }
      fetch(tile + kSlabWarps, first);
    };
    rank8(std::integral_constant<int, 0>());
    rank8(std::integral_constant<int, 8>());
    rank8(std::integral_constant<int, 16>());
    rank8(std::integral_constant<int, 24>());
    __syncwarp();
    // word j of line m of the tile: the keys of features 2m and 2m + 1, or 4m .. 4m + 3, of row j
    constexpr int PER = BYTES ? 4 : 2, LINES = 32 / PER;
    unsigned char *out = p.keys + (size_t)tile * p.tile_bytes + (size_t)slab * (LINES * 128) + lane * 4;
    const int lines = min(LINES, (p.num_features - slab * 32 + PER - 1) / PER);
#pragma unroll
    for (int m = 0; m < LINES; ++m)
      if (m < lines) *reinterpret_cast<uint32_t *>(out + m * 128) = lds_u32(turn + (uint32_t)(lane * (BYTES ? 36 : 68) + m * 4));
    __syncwarp();
  }
  count_searched(p.searched, p.n_rows, p.used, looked_up, blockIdx.x == 0 && blockIdx.y == 0 && warp == 0);
}

} // namespace tb
