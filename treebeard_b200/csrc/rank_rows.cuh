// Ranks the rows of a batch (rank_pack.h): fp32 row values -> 16-bit keys in the order in which the
// walk (walk_rank.cuh) copies them into shared memory: rows of at most 32 features in pairs
// (word f of a line = keys of feature f of rows 2i and 2i + 1), rows of at most 64 one by one, wider
// rows in tiles of 32 (word j of line m = keys of features 2m and 2m + 1 of row j).
//
// A thread ranks FW neighbouring features of a row or of a pair of rows, all in lock-step: the
// look-ups and search steps of different values are independent, so their latencies overlap.
//  * SMEM = false: the tables are read through L1/L2.  A gather there costs one wavefront per
//    lane, too much for large batches, but nothing has to be loaded first.
//  * SMEM = true: a block keeps the tables of its features in shared memory (blockIdx.y = slab of
//    `pieces` pieces of FW features) and takes a range of the rows.
#pragma once
#include "walk_kernels.cuh"

namespace tb {

struct DevRankFeature { // = RankFeature
  float lo, scale, top; // top: the last bucket
  uint32_t lut_off, thr_off, n, buckets, lattice;
};

struct RankRowsParams {
  const float *rows;
  long long n_rows, ld;
  const DevRankFeature *features;
  const uint16_t *lut;
  const float *thr;
  uint16_t *keys;
  int32_t num_features, stride; // stride: bytes per row of keys
  int32_t pieces;               // pieces per slab
  int32_t vec4_ok;
  int32_t lattice;              // some feature is a lattice feature
  int32_t bytes;                // tiles of one-byte keys (tables in global memory only)
  uint32_t turn_off;            // tiles: the warps' buffers, behind the tables
  int32_t used;                 // features with thresholds (here the struct grows no larger: 8 bytes more of parameters cost small host batches 0.4 us)
  unsigned long long *searched; // statistics: values whose rank the feature's look-up table alone doesn't give (rank_of)
};

// The statistics of a launch or block that ranks `rows` rows: the values of features with thresholds, less those (of this
// thread) that the look-up table gave.  The warp is complete.
__device__ __forceinline__ void count_searched(unsigned long long *searched, long long rows, int used, unsigned looked_up, bool whole_rows) {
  looked_up = __reduce_add_sync(0xffffffffu, looked_up);
  const long long n = (whole_rows ? rows * used : 0ll) - (long long)looked_up;
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(searched, (unsigned long long)n);
}

// Ranks up to N values of a block's rows, tables in global memory: number i0, i0 + stride, ... of `count`, counted
// row by row.  value(row, feature) gives one, use(row, feature, rank) takes its rank.  They go through their
// look-ups and search steps in lock-step, as in tb_rank_rows: each of these is an L2 round trip that depends
// on the last one.
template <int N, typename Value, typename Use>
__device__ __forceinline__ void rank_values(const RankRowsParams &r, uint32_t i0, uint32_t stride, uint32_t count, unsigned &looked_up,
                                            Value value, Use use) {
  const uint32_t F = (uint32_t)r.num_features, rows = stride / F, rest = stride - rows * F; // (from one value to the next)
  float x[N];
  uint32_t row[N], f[N], s[N], e[N], longest = 0;
  const float *thr[N]; // of the feature, less one
#pragma unroll
  for (int k = 0; k < N; ++k) {
    if (k == 0) {
      row[k] = i0 / F;
      f[k] = i0 - row[k] * F;
    } else {
      const bool over = f[k - 1] + rest >= F;
      row[k] = row[k - 1] + rows + (over ? 1u : 0u);
      f[k] = f[k - 1] + rest - (over ? F : 0u);
    }
    x[k] = 0.f;
    s[k] = e[k] = 0;
    thr[k] = r.thr;
    if (i0 + k * stride < count) {
      const uint4 *feature = reinterpret_cast<const uint4 *>(r.features + f[k]);
      const uint4 a = __ldg(feature), b = __ldg(feature + 1);
      x[k] = value(row[k], f[k]);
      const float lo = __uint_as_float(a.x), scale = __uint_as_float(a.y), top = __uint_as_float(a.z);
      const float y = fmaxf(fminf(__fmul_rn(__fsub_rn(x[k], lo), scale), top), 0.f);
      const uint16_t *l = r.lut + a.w + (uint32_t)y;
      s[k] = __ldg(l);
      e[k] = __ldg(l + 1);
      thr[k] = r.thr + b.x - 1;
      if (b.w && x[k] == floorf(x[k])) {
        s[k] = e[k] = x[k] < lo ? 0u : e[k];
        ++looked_up;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < N; ++k) longest = max(longest, e[k] - s[k]);
  for (uint32_t step = longest ? 1u << (31 - __clz(longest)) : 0u; step; step >>= 1) {
    float t[N];
#pragma unroll
    for (int k = 0; k < N; ++k) t[k] = s[k] + step <= e[k] ? __ldg(thr[k] + s[k] + step) : INFINITY;
#pragma unroll
    for (int k = 0; k < N; ++k)
      if (s[k] + step <= e[k] && !(x[k] < t[k])) s[k] += step;
  }
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (i0 + k * stride < count) use(row[k], f[k], s[k]);
}

// A warp that ranks a piece of a tile reads its 32 x 8 values as 32-byte stretches of rows and turns
// them around in a buffer of its own: one row per lane would take 32 wavefronts a load.
constexpr int kRankTurnBytes = 32 * 32 * 9 * 4;

enum RankLayout { kRankPairs, kRankRows, kRankTiles };

template <int FW, int LAYOUT, bool SMEM>
__global__ void __launch_bounds__(SMEM ? 1024 : 256, 1) tb_rank_rows(const RankRowsParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int F = p.num_features;
  const int f_first = SMEM ? (int)blockIdx.y * p.pieces * FW : 0;
  const int f_end = SMEM ? min(F, f_first + p.pieces * FW) : F;
  const DevRankFeature *feat = p.features;
  const unsigned char *lut = reinterpret_cast<const unsigned char *>(p.lut), *thr = reinterpret_cast<const unsigned char *>(p.thr);
  [[maybe_unused]] uint32_t thr_lane = 0; // shared-memory address of the threshold before offset 0
  if constexpr (SMEM) {
    // the block's own copies: descriptors (offsets now from smem_raw), thresholds, bucket tables
    const DevRankFeature a = p.features[f_first], z = p.features[f_end - 1];
    const uint32_t lut0 = a.lut_off, lut_n = z.lut_off + (z.buckets + 1 + 7) / 8 * 8 - lut0;
    const uint32_t thr0 = a.thr_off, thr_n = z.thr_off + (z.n + 3) / 4 * 4 - thr0;
    auto *feat_s = reinterpret_cast<DevRankFeature *>(smem_raw);
    const uint32_t thr_s = (uint32_t)(f_end - f_first) * (uint32_t)sizeof(DevRankFeature), lut_s = thr_s + 4u * thr_n;
    for (int i = threadIdx.x; i < f_end - f_first; i += blockDim.x) {
      DevRankFeature d = p.features[f_first + i];
      d.lut_off = lut_s / 2 + d.lut_off - lut0;
      d.thr_off = thr_s / 4 + d.thr_off - thr0;
      feat_s[i] = d;
    }
    for (uint32_t i = threadIdx.x; i < thr_n / 4; i += blockDim.x)
      *reinterpret_cast<float4 *>(smem_raw + thr_s + 16 * i) = __ldg(reinterpret_cast<const float4 *>(p.thr + thr0) + i);
    for (uint32_t i = threadIdx.x; i < lut_n / 8; i += blockDim.x)
      *reinterpret_cast<uint4 *>(smem_raw + lut_s + 16 * i) = __ldg(reinterpret_cast<const uint4 *>(p.lut + lut0) + i);
    feat = feat_s - f_first;
    lut = thr = smem_raw;
    thr_lane = smem_u32(smem_raw) - 4u;
    __syncthreads();
  }
  const int pieces = p.pieces; // without tables in shared memory: of the whole row
  constexpr bool PAIR = LAYOUT == kRankPairs, TILES = LAYOUT == kRankTiles;
  constexpr int RPT = PAIR ? 2 : 1, N = RPT * FW; // rows and values per thread
  const uint32_t n_rows = (uint32_t)p.n_rows;     // (the host bounds a batch by the bytes of its keys)
  // lines: rows, or pairs of rows, or all rows of the tiles; a warp takes one piece of a tile's rows
  const uint32_t items = (TILES ? (n_rows + 31) & ~31u : (n_rows + RPT - 1) / RPT) * (uint32_t)pieces;
  constexpr float kNowhere = 0.5f; // in the places of features and rows that there are not: no whole number
  unsigned looked_up = 0;
  for (uint32_t it = blockIdx.x * blockDim.x + threadIdx.x; it < items; it += gridDim.x * blockDim.x) {
    const uint32_t unit = TILES ? it >> 5 : it, whole = pieces == 1 ? unit : unit / (uint32_t)pieces;
    const uint32_t line = TILES ? whole * 32u + (it & 31u) : whole;
    const int f0 = f_first + (int)(unit - whole * (uint32_t)pieces) * FW;
    if (f0 >= F) continue;
    float x[N];
    if constexpr (TILES && SMEM) {
      static_assert(FW == 8, "a piece is 8 features");
      float *turn = reinterpret_cast<float *>(smem_raw + p.turn_off) + (threadIdx.x >> 5) * (32 * 9);
      const uint32_t lane = it & 31u, i = lane & 7u;
      const bool in = f0 + (int)i < F;
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t r = 4u * k + (lane >> 3), row = min(whole * 32u + r, n_rows - 1);
        turn[r * 9 + i] = in ? __ldg(p.rows + (long long)row * p.ld + f0 + i) : kNowhere;
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = turn[lane * 9 + k];
    } else
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const float *src = p.rows + (long long)min(line * RPT + r, n_rows - 1) * p.ld + f0;
      if (FW >= 4 && p.vec4_ok) {
#pragma unroll
        for (int i = 0; i + 3 < FW; i += 4) {
          const float4 v = f0 + i < F ? __ldg(reinterpret_cast<const float4 *>(src + i)) : make_float4(kNowhere, kNowhere, kNowhere, kNowhere);
          x[r * FW + i] = v.x;
          x[r * FW + i + 1] = v.y;
          x[r * FW + i + 2] = v.z;
          x[r * FW + i + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < FW; ++i) x[r * FW + i] = f0 + i < F ? __ldg(src + i) : kNowhere;
      }
    }
    if (line * RPT + RPT > n_rows) { // the second row of the last pair, or rows that fill up a tile
#pragma unroll
      for (int k = (int)(PAIR) * FW; k < N; ++k) x[k] = kNowhere;
    }
    uint32_t s[N], e[N], first[FW]; // byte offsets of thresholds
    uint32_t longest = 0;
#pragma unroll
    for (int i = 0; i < FW; ++i) {
      const uint4 *d4 = reinterpret_cast<const uint4 *>(feat + min(f0 + i, F - 1));
      uint4 a, b;
      if (SMEM) {
        a = d4[0];
        b = d4[1];
      } else {
        a = __ldg(d4);
        b = __ldg(d4 + 1);
      }
      const float lo = __uint_as_float(a.x), scale = __uint_as_float(a.y), top = __uint_as_float(a.z);
      first[i] = 4u * b.x;
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int k = r * FW + i;
        // Both roundings as on the host.  Values below every threshold land in the first bucket,
        // values above in the last one, and so does NaN (the inner minimum drops it): the search
        // then finds 0 or n.
        const float y = fmaxf(fminf(__fmul_rn(__fsub_rn(x[k], lo), scale), top), 0.f);
        const uint16_t *l = reinterpret_cast<const uint16_t *>(lut + 2u * (a.w + (uint32_t)y));
        s[k] = SMEM ? l[0] : __ldg(l);
        e[k] = SMEM ? l[1] : __ldg(l + 1);
        if (p.lattice && b.w && x[k] == floorf(x[k])) { // a bucket's threshold is at or below its whole number
          s[k] = x[k] < lo ? 0u : e[k];
          e[k] = s[k];
          ++looked_up;
        }
        longest = max(longest, e[k] - s[k]);
        s[k] = first[i] + 4u * s[k];
        e[k] = first[i] + 4u * e[k];
      }
    }
    // rank = s + thresholds among the bucket's e - s that are at or below x: s grows by powers of
    // two, largest first, in lock-step for all the values of the warp
    longest = __reduce_max_sync(__activemask(), longest);
    for (uint32_t step = longest ? 4u << (31 - __clz(longest)) : 0u; step >= 4u; step >>= 1) {
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const uint32_t m = s[k] + step;
        if constexpr (SMEM) { // (without a branch: a value's next threshold, the comparison, the step)
          asm volatile("{\n .reg .pred p, q;\n .reg .f32 t;\n setp.le.u32 p, %1, %2;\n mov.f32 t, 0f00000000;\n"
                       " @p ld.shared.f32 t, [%3];\n setp.geu.and.f32 q, %4, t, p;\n @q mov.b32 %0, %1;\n}"
                       : "+r"(s[k]) : "r"(m), "r"(e[k]), "r"(thr_lane + m), "f"(x[k]));
        } else if (m <= e[k]) {
          const float *t = reinterpret_cast<const float *>(thr + m - 4u);
          if (!(x[k] < __ldg(t))) s[k] = m;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) s[k] = (s[k] - first[k % FW]) >> 2;
    unsigned char *dst = reinterpret_cast<unsigned char *>(p.keys) + (size_t)line * (RPT * p.stride) + f0 * (2 * RPT);
    uint32_t w[(N + 1) / 2]; // keys in the order of memory: feature by feature, the pair's rows side by side
#pragma unroll
    for (int k = 0; k < (N + 1) / 2; ++k) {
      if constexpr (PAIR) w[k] = s[k] | s[FW + k] << 16;
      else w[k] = 2 * k + 1 < N ? s[2 * k] | s[2 * k + 1] << 16 : s[2 * k];
    }
    if constexpr (TILES) {
      unsigned char *tile = reinterpret_cast<unsigned char *>(p.keys) + (size_t)whole * (32 * p.stride) + (it & 31u) * 4u;
      if constexpr (FW == 1) {
        if (p.bytes) tile[(f0 >> 2) * 128 + (f0 & 3)] = (unsigned char)s[0];
        else *reinterpret_cast<uint16_t *>(tile + (f0 >> 1) * 128 + (f0 & 1) * 2) = (uint16_t)s[0];
      } else {
#pragma unroll
        for (int k = 0; k < N / 2; ++k)
          if (f0 + 2 * k < F) *reinterpret_cast<uint32_t *>(tile + (f0 / 2 + k) * 128) = w[k];
      }
    } else if constexpr (N == 8) *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    else if constexpr (N == 4) *reinterpret_cast<uint2 *>(dst) = make_uint2(w[0], w[1]);
    else if constexpr (N == 2) *reinterpret_cast<uint32_t *>(dst) = w[0];
    else *reinterpret_cast<uint16_t *>(dst) = (uint16_t)w[0];
  }
  count_searched(p.searched, p.n_rows, p.used, looked_up, blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 32);
}

} // namespace tb
