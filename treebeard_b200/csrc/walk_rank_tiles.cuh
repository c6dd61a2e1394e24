// Walk kernel for rank keys (rank_pack.h) over rows of more than 64 features: the words of a row's
// keys no longer have a bank each, so here LANE = ROW.  Keys come in tiles of 32 rows: line m (128
// bytes) of a tile holds in word j the keys of features 2m and 2m+1 of row j, so a key load touches
// 32 banks whatever the features are; at step i of a group lane l walks column (l + i) mod 32,
// which makes node and leaf loads conflict-free.
//
// A warp walks four tiles in lock-step through two columns at a time: eight independent chains of
// loads per lane keep the shared-memory pipe busy with 12 to 20 warps (one column at a time left it
// a third idle; 68 % busy over a whole launch of 50003 rows x 467 trees of 7 levels, whose last round of quads
// fills only some blocks).  The widest rows under the deepest trees leave room for 8 or 4 warps.  The nodes of a column's two topmost levels are loaded once for the four tiles; a tree of 8
// levels costs 15.75 wavefronts per 32 rows.  Sums stay in the lane that owns the row.
//
// Rows of more than 511 features have keys of one byte: line m holds in word j the keys of features 4m .. 4m+3 of row j,
// so that four tiles fit up to about 1000 features under 8 levels (1600 under 6), and pairs of tiles up to 2024 (2044 under 7 levels and fewer).  A pair with
// rows of 2000 features leaves three ring slots of 32 KB: 18944 rows x 1000 trees of 8 levels take 70 us, 17.4 wavefronts and
// 68 instructions per 32 rows and tree, pipe 53 % and issue 55 % busy -- every group's 64 KB are asked for only once the group
// before is walked.  (Walking four groups before looking up their leaf values, with node planes two ahead: 82 us; 8 warps of
// four columns each instead of 16 of two: 73.)
//
// A block has `quads` x `shares` walker warps (T x quads tiles at a time; the shares of a quad split
// the 32 columns of every group), a warp that streams the groups (node plane and leaf plane take a
// ring slot each) and a warp that fetches the keys of the next batch of tiles.  Quads of tiles are
// dealt to the blocks evenly; blockIdx.y is a chunk of the trees, combined by the last block to
// finish as in walk_rank.cuh.  All waits are bounded.
//
// Reference counterparts: as for walk_rank.cuh; the row tile of a thread block is
// src/gpu/GPURepresentations.cpp:279-399.
#pragma once
#include "walk_rank.cuh"

namespace tb {

constexpr int kRTMaxWalkers = 20, kRTBarBytes = 512, kRTMaxSlots = 16;
// shared memory: barriers, what the shares of a quad hand over, the keys of T * quads tiles, the ring
__host__ __device__ constexpr int rank_tiles_smem_bytes(int tile_bytes, int tiles, int walkers, int lockstep, int slots, uint32_t slot_bytes) {
  return kRTBarBytes + walkers * lockstep * 128 + tiles * tile_bytes + slots * (int)slot_bytes;
}

// T tiles through C columns (addresses col[c] in the node plane); kb[t]: this lane's keys in
// tile t.  off: where the walks end, as offsets into the leaf plane plus the node plane's address.
template <int D, int T, int C, bool BYTES> __device__ __forceinline__ void rank_tiles_walk(uint32_t (&off)[T * C], const uint32_t *col, const uint32_t *kb) {
  constexpr int W = T * C;
  uint32_t node[W], key[W], root[C];
  [[maybe_unused]] uint32_t left[C], right[C];
#define TBT_ALL(...)                                                                                                \
  {                                                                                                                 \
    _Pragma("unroll") for (int q = 0; q < W; ++q) {                                                                 \
      [[maybe_unused]] const int t = q % T, c = q / T;                                                              \
      __VA_ARGS__;                                                                                                  \
    }                                                                                                               \
  }
  auto key_at = [](uint32_t a) { return BYTES ? lds_u8(a) : lds_u16_imm<0>(a); };
#pragma unroll
  for (int c = 0; c < C; ++c) {
    root[c] = lds_u32_imm<0>(col[c]);
    if constexpr (D > 1) { // shared by the tiles: both nodes of level 1 are loaded
      left[c] = lds_u32_imm<128>(col[c]);
      right[c] = lds_u32_imm<256>(col[c]);
    }
  }
  TBT_ALL(key[q] = key_at((root[c] >> 16) + kb[t]))
  if constexpr (D > 1) {
    TBT_ALL(asm volatile("{\n .reg .pred p, q;\n setp.ge.f16x2 p|q, %2, %3;\n selp.b32 %0, %5, %4, p;\n selp.b32 %1, %7, %6, p;\n}"
                         : "=&r"(off[q]), "=&r"(node[q])
                         : "r"(key[q]), "r"(root[c]), "r"(col[c]), "r"(col[c] + 128u), "r"(left[c]), "r"(right[c])))
  } else {
    TBT_ALL(off[q] = col[c]; (rank_step<false, 128u>(off[q], key[q], root[c])))
  }
#define TBT_LEVEL(level)                                                                                            \
  if constexpr (D > level) {                                                                                        \
    if constexpr (level > 1) TBT_ALL(node[q] = lds_u32_imm<128 * ((1 << level) - 1)>(off[q]))              \
    TBT_ALL(key[q] = key_at((node[q] >> 16) + kb[t]))                                                       \
    TBT_ALL((rank_step<false, (128u << level)>(off[q], key[q], node[q])))                                           \
  }
  TBT_LEVEL(1) TBT_LEVEL(2) TBT_LEVEL(3) TBT_LEVEL(4) TBT_LEVEL(5) TBT_LEVEL(6) TBT_LEVEL(7)
#undef TBT_LEVEL
#undef TBT_ALL
}
template <int T, int C, bool BYTES>
__device__ __forceinline__ void rank_tiles_walk_any(uint32_t depth, uint32_t (&off)[T * C], const uint32_t *col, const uint32_t *kb) {
  switch (depth) {
  case 1: return rank_tiles_walk<1, T, C, BYTES>(off, col, kb);
  case 2: return rank_tiles_walk<2, T, C, BYTES>(off, col, kb);
  case 3: return rank_tiles_walk<3, T, C, BYTES>(off, col, kb);
  case 4: return rank_tiles_walk<4, T, C, BYTES>(off, col, kb);
  case 5: return rank_tiles_walk<5, T, C, BYTES>(off, col, kb);
  case 6: return rank_tiles_walk<6, T, C, BYTES>(off, col, kb);
  case 7: return rank_tiles_walk<7, T, C, BYTES>(off, col, kb);
  default: return rank_tiles_walk<8, T, C, BYTES>(off, col, kb);
  }
}

// T: tiles that a warp walks in lock-step (4, or 2 where four do not fit); BYTES: keys of one byte.
template <int T, bool BYTES, bool LEAF_IDS>
__global__ void __launch_bounds__(32 * (kRTMaxWalkers + 2), 1) tb_walk_rank_tiles_kernel(const __grid_constant__ RankWalkParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr int C = 2, W = T * C;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int NW = (int)(blockDim.x >> 5) - 2, Q = p.quads, shares = NW / Q;
  const uint32_t bars_s = smem_u32(smem_raw);
  // barriers: full[16] @0, empty[16] @128, keys_full @256, keys_empty @264; flag @272
  const uint32_t full_s = bars_s, empty_s = bars_s + 128u, keys_full_s = bars_s + 256u, keys_empty_s = bars_s + 264u;
  volatile uint32_t *last_flag = reinterpret_cast<volatile uint32_t *>(smem_raw + 272);
  float *shared_sums = reinterpret_cast<float *>(smem_raw + kRTBarBytes); // [share][quad][t][row]
  unsigned char *keys = smem_raw + kRTBarBytes + NW * T * 128;
  unsigned char *ring = keys + (size_t)Q * T * p.tile_bytes;
  const long long tiles = (p.n_rows + 31) / 32, quads = (tiles + T - 1) / T;
  const int quad0 = (int)(quads * blockIdx.x / gridDim.x), quad1 = (int)(quads * (blockIdx.x + 1) / gridDim.x);
  const int my_batches = (quad1 - quad0 + Q - 1) / Q;
  const int g0 = (int)blockIdx.y * p.groups_per_chunk, g1 = min(p.num_groups, g0 + p.groups_per_chunk);
  const int NG = g1 - g0;

  if (tid == 0) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw);
    for (int i = 0; i < kRTMaxSlots; ++i) mbar_init(bars + i, 1);
    for (int i = 0; i < kRTMaxSlots; ++i) mbar_init(bars + 16 + i, NW);
    mbar_init(bars + 32, 1);
    mbar_init(bars + 33, NW);
    fence_barrier_init();
  }
  __syncthreads();

  bool ok = true;
  [[maybe_unused]] uint32_t issued = 0;
  const uint32_t tries = p.wait_tries ? p.wait_tries : kQWaitTries;
  auto wait = [tries](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait_all_lanes(bar, parity, tries)) != 0; };
  auto depth_of = [&](int k) { return p.uniform_depth ? (uint32_t)p.uniform_depth : p.groups[g0 + k].depth; };

  if (warp == NW) {
    // ---- tree groups: piece 2k = node plane of group k, piece 2k + 1 = its leaf plane
    const uint64_t keep = l2_policy_keep();
    int slot = 0;
    uint32_t round = 0;
    for (int it = 0; it < my_batches && ok; ++it)
      for (int piece = 0; piece < 2 * NG && ok; ++piece) {
        if (round > 0) ok = wait(empty_s + 8u * (uint32_t)slot, (round - 1u) & 1u);
        issued += ok;
        if (ok && lane == 0 && !(p.skip_first_copy && it == 0 && piece == 0)) {
          const uint32_t d = p.uniform_depth;
          const int g = g0 + (piece >> 1);
          const unsigned long long elem = d ? (unsigned long long)g << (d + 5) : p.groups[g].elem_off;
          const uint32_t bytes = 128u << depth_of(piece >> 1);
          uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw) + slot;
          mbar_expect_tx(bar, bytes);
          bulk_g2s_hint(ring + (size_t)slot * p.stage_bytes, ((piece & 1) ? p.leaf_plane : p.node_plane) + elem, bytes, bar, keep);
        }
        if (++slot == p.stages) {
          slot = 0;
          ++round;
        }
      }
  } else if (warp == NW + 1) {
    // ---- the batches' keys (the kernel that ranks the rows may still be running)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint64_t stream = l2_policy_stream();
    for (int it = 0; it < my_batches && ok; ++it) {
      if (it > 0) ok = wait(keys_empty_s, (uint32_t)(it - 1) & 1u);
      issued += ok;
      if (ok && lane == 0) {
        const int u = quad0 + it * Q;
        const long long first = (long long)u * T, end = min(tiles, (long long)min(quad1, u + Q) * T);
        uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw) + 32;
        mbar_expect_tx(bar, (uint32_t)(end - first) * (uint32_t)p.tile_bytes);
        for (long long t = first; t < end; ++t)
          bulk_g2s_hint(keys + (size_t)(t - first) * p.tile_bytes, p.keys + t * p.tile_bytes, (uint32_t)p.tile_bytes, bar, stream);
      }
    }
  } else {
    // ---- the walkers
    const int quad = warp % Q, share = warp / Q, cols = 32 / shares;
    const bool elected = lane == 0;
    uint32_t kb[T];
#pragma unroll
    for (int t = 0; t < T; ++t) kb[t] = smem_u32(keys) + (uint32_t)((quad * T + t) * p.tile_bytes) + (uint32_t)lane * 4u;
    constexpr bool ONCE = T == 2; // (16 walkers share a pair of tiles: a warp walks two columns of a group)
    [[maybe_unused]] uint32_t first_col[C];
#pragma unroll
    for (int c = 0; c < C; ++c) first_col[c] = ((uint32_t)(lane + share * C + c) & 31u) * 4u;
    int slot = 0, it = 0;
    uint32_t parity = 0;
    for (; it < my_batches; ++it) {
      const bool busy = quad0 + it * Q + quad < quad1; // (the last batch may be short)
      const long long row0 = (long long)(quad0 + it * Q + quad) * T * 32 + lane;
      ok = wait(keys_full_s, (uint32_t)it & 1u);
      if (!ok) break;
      float acc[T];
#pragma unroll
      for (int t = 0; t < T; ++t) acc[t] = 0.f;
      uint32_t next_depth = depth_of(0);
      for (int k = 0; k < NG; ++k) {
        const uint32_t depth = next_depth;
        next_depth = depth_of(min(k + 1, NG - 1));
        const uint32_t sn = (uint32_t)slot, pn = parity;
        if (++slot == p.stages) { slot = 0; parity ^= 1u; }
        const uint32_t sl = (uint32_t)slot, pl = parity;
        if (++slot == p.stages) { slot = 0; parity ^= 1u; }
        ok = wait(full_s + 8u * sn, pn);
        if (!ok) break;
        const uint32_t nodes = smem_u32(ring) + sn * p.stage_bytes, leaves = smem_u32(ring) + sl * p.stage_bytes - nodes;
        float sum[T]; // of the group: short sums keep the rounding error down
#pragma unroll
        for (int t = 0; t < T; ++t) sum[t] = 0.f;
        bool leaves_here = false;
        if (busy)
#pragma unroll 1
          for (int i = 0; i < (ONCE ? C : cols); i += C) {
            uint32_t col[C], off[W];
#pragma unroll
            for (int c = 0; c < C; ++c) col[c] = nodes + (ONCE ? first_col[c] : ((uint32_t)(lane + share * cols + i + c) & 31u) * 4u);
            rank_tiles_walk_any<T, C, BYTES>(depth, off, col, kb);
            if (ONCE) { // done with the node plane: its slot takes the next group's while leaf values are looked up
              __syncwarp();
              if (elected) mbar_arrive(empty_s + 8u * sn);
            }
            if (!leaves_here) {
              leaves_here = ok = wait(full_s + 8u * sl, pl);
              if (!ok) break;
            }
            uint32_t v[W];
#pragma unroll
            for (int q = 0; q < W; ++q) v[q] = lds_u32(off[q] + leaves);
            if constexpr (LEAF_IDS) {
#pragma unroll
              for (int q = 0; q < W; ++q) {
                const int tree = p.tree_index[(g0 + k) * 32 + (int)((uint32_t)(lane + share * cols + i + q / T) & 31u)];
                const long long row = row0 + (q % T) * 32;
                if (tree >= 0 && row < p.n_rows) p.leaf_ids[row * p.num_trees + tree] = (int32_t)v[q];
              }
            } else {
#pragma unroll
              for (int q = 0; q < W; ++q) sum[q % T] += __uint_as_float(v[q]);
            }
          }
        else {
          ok = wait(full_s + 8u * sl, pl);
          if (ONCE && elected) mbar_arrive(empty_s + 8u * sn);
        }
        if (!ok) break;
#pragma unroll
        for (int t = 0; t < T; ++t) acc[t] += sum[t];
        __syncwarp();
        if (elected) {
          if (!ONCE) mbar_arrive(empty_s + 8u * sn);
          mbar_arrive(empty_s + 8u * sl);
        }
      }
      if (!ok) break;
      // ---- the batch's results: the shares of a quad add up
      if constexpr (!LEAF_IDS) {
        if (shares > 1) {
#pragma unroll
          for (int t = 0; t < T; ++t) shared_sums[(warp * T + t) * 32 + lane] = acc[t]; // (warp = share * Q + quad)
          asm volatile("bar.sync 1, %0;" ::"r"(32 * NW) : "memory");
        }
        for (int t = share; t < T; t += shares) { // a share finishes every shares-th tile
          float s = 0.f;
          if (shares > 1)
            for (int h = 0; h < shares; ++h) s += shared_sums[((h * Q + quad) * T + t) * 32 + lane];
          else
#pragma unroll
            for (int u = 0; u < T; ++u) s = u == t ? acc[u] : s;
          const long long row = row0 + t * 32;
          if (busy && row < p.n_rows) {
            if (gridDim.y > 1) p.scratch[(long long)blockIdx.y * p.n_rows + row] = s;
            else if (p.write_partial) p.partial[row] = s;
            else reinterpret_cast<float *>(p.out)[row] = apply_transform(p.initial_value + s, p.transform);
          }
        }
      }
      __syncwarp();
      if (elected) mbar_arrive(keys_empty_s);
    }
    // a warp whose wait gave up still meets the others at the barriers of the batches it skips
    if (!LEAF_IDS && shares > 1)
      for (; it < my_batches; ++it) asm volatile("bar.sync 1, %0;" ::"r"(32 * NW) : "memory");
  }
  // every wait above is bounded: a wait that gave up ends the launch with a status word
  const bool chunked = gridDim.y > 1 && !LEAF_IDS;
  if (chunked) __threadfence();
  if (__syncthreads_or(!ok)) {
    if (tid == 0) set_status(p.status, 4);
    if (warp >= NW) { // no copy may land after the block is gone
      const uint32_t bars = warp == NW ? full_s : keys_full_s, n = warp == NW ? (uint32_t)p.stages : 1u;
      for (uint32_t s = 0; s < min(n, issued); ++s) wait(bars + 8u * s, ((issued - 1u - s) / n) & 1u);
    }
  }
  if (!chunked) return;
  if (tid == 0) {
    const bool last = atomicAdd(p.arrivals + blockIdx.x, 1u) + 1u == gridDim.y;
    if (last) p.arrivals[blockIdx.x] = 0; // for the next launch
    *last_flag = last;
  }
  __syncthreads();
  if (!*last_flag) return;
  __threadfence();
  const long long end = min(p.n_rows, (long long)quad1 * T * 32);
  for (long long row = (long long)quad0 * T * 32 + tid; row < end; row += blockDim.x) {
    const float s = rank_sum_chunks(p, row);
    if (p.write_partial) p.partial[row] = s;
    else reinterpret_cast<float *>(p.out)[row] = apply_transform(p.initial_value + s, p.transform);
  }
}

} // namespace tb
