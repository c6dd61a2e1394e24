// Ranks the rows of a batch (rank_pack.h): fp32 row values -> 16-bit keys, row after row in
// `stride` bytes each, which is how the walk (walk_rank.cuh) copies them into shared memory.
//
// A thread ranks a piece of W neighbouring features of one row, all of them in lock-step (the
// table look-ups and search steps of the features are independent, so their latencies overlap).
//  * tb_rank_rows<8, false>: the tables are read through L1/L2.  A gather there costs one
//    wavefront per lane, which is too much for large batches, but nothing has to be loaded first.
//  * tb_rank_rows<W, true>: a block keeps the tables of its features in shared memory (blockIdx.y
//    = slab of pieces) and takes a range of the rows.
#pragma once
#include "walk_kernels.cuh"

namespace tb {

struct DevRankFeature { // = RankFeature
  float lo, hi, scale;
  uint32_t buckets, lut_off, thr_off, n, lattice;
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
  unsigned long long *searched; // statistics: values that were compared with thresholds
};

// Pieces of a block's tables in shared memory: its features' descriptors, bucket tables, thresholds.
template <int W, bool SMEM>
__global__ void __launch_bounds__(SMEM ? 1024 : 256) tb_rank_rows(const RankRowsParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int F = p.num_features;
  const int f_first = SMEM ? (int)blockIdx.y * p.pieces * W : 0;
  const int f_end = SMEM ? min(F, f_first + p.pieces * W) : F;
  const DevRankFeature *feat = p.features;
  const uint16_t *lut = p.lut;
  const float *thr = p.thr;
  if constexpr (SMEM) {
    // descriptors with offsets into the block's own copies of the tables
    const DevRankFeature a = p.features[f_first], z = p.features[f_end - 1];
    const uint32_t lut0 = a.lut_off, lut1 = z.lut_off + (z.buckets + 1 + 7) / 8 * 8;
    const uint32_t thr0 = a.thr_off, thr1 = z.thr_off + (z.n + 3) / 4 * 4;
    auto *feat_s = reinterpret_cast<DevRankFeature *>(smem_raw);
    auto *thr_s = reinterpret_cast<float4 *>(smem_raw + (size_t)(f_end - f_first) * sizeof(DevRankFeature));
    auto *lut_s = reinterpret_cast<uint4 *>(thr_s + (thr1 - thr0) / 4);
    for (int i = threadIdx.x; i < f_end - f_first; i += blockDim.x) {
      DevRankFeature d = p.features[f_first + i];
      d.lut_off -= lut0;
      d.thr_off -= thr0;
      feat_s[i] = d;
    }
    for (uint32_t i = threadIdx.x; i < (thr1 - thr0) / 4; i += blockDim.x) thr_s[i] = __ldg(reinterpret_cast<const float4 *>(p.thr + thr0) + i);
    for (uint32_t i = threadIdx.x; i < (lut1 - lut0) / 8; i += blockDim.x) lut_s[i] = __ldg(reinterpret_cast<const uint4 *>(p.lut + lut0) + i);
    feat = feat_s - f_first;
    lut = reinterpret_cast<const uint16_t *>(lut_s);
    thr = reinterpret_cast<const float *>(thr_s);
    __syncthreads();
  }
  const int pieces = p.pieces; // without tables in shared memory: of the whole row
  const uint32_t items = (uint32_t)p.n_rows * (uint32_t)pieces; // (the host bounds a batch by the bytes of its keys)
  unsigned searched = 0;
  for (uint32_t it = blockIdx.x * blockDim.x + threadIdx.x; it < items; it += gridDim.x * blockDim.x) {
    const uint32_t row = pieces == 1 ? it : it / (uint32_t)pieces;
    const int f0 = f_first + (int)(it - row * (uint32_t)pieces) * W;
    if (f0 >= F) continue;
    const float *src = p.rows + (long long)row * p.ld + f0;
    float x[W];
    if (p.vec4_ok && W >= 4) {
#pragma unroll
      for (int i = 0; i < W; i += 4) {
        const float4 v = f0 + i < F ? __ldg(reinterpret_cast<const float4 *>(src + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[i] = v.x;
        if (i + 1 < W) x[i + 1] = v.y;
        if (i + 2 < W) x[i + 2] = v.z;
        if (i + 3 < W) x[i + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < W; ++i) x[i] = f0 + i < F ? __ldg(src + i) : 0.f;
    }
    uint32_t s[W], e[W], off[W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
      s[i] = e[i] = off[i] = 0;
      if (f0 + i < F) {
        const uint4 *d4 = reinterpret_cast<const uint4 *>(feat + f0 + i);
        uint4 a, b;
        if (SMEM) {
          a = d4[0];
          b = d4[1];
        } else {
          a = __ldg(d4);
          b = __ldg(d4 + 1);
        }
        const float lo = __uint_as_float(a.x), hi = __uint_as_float(a.y), scale = __uint_as_float(a.z);
        off[i] = b.y;
        if (!(x[i] < hi)) { // at or above every threshold, or NaN
          s[i] = e[i] = b.z;
        } else if (x[i] >= lo) {
          // (both roundings as on the host: nothing to contract into one operation)
          const uint32_t bucket = min((uint32_t)__fmul_rn(__fsub_rn(x[i], lo), scale), a.w - 1u);
          const uint16_t *l = lut + b.x + bucket;
          s[i] = SMEM ? l[0] : __ldg(l);
          e[i] = SMEM ? l[1] : __ldg(l + 1);
          if (b.w && x[i] == floorf(x[i])) s[i] = e[i]; // lattice: one threshold at most, at or below a whole number
          searched += s[i] < e[i];
        }
      }
    }
    bool more = true;
    while (more) {
      more = false;
#pragma unroll
      for (int i = 0; i < W; ++i)
        if (s[i] < e[i]) {
          const uint32_t m = (s[i] + e[i]) >> 1;
          const float t = SMEM ? thr[off[i] + m] : __ldg(thr + off[i] + m);
          if (x[i] < t) e[i] = m;
          else s[i] = m + 1;
          more |= s[i] < e[i];
        }
    }
    unsigned char *dst = reinterpret_cast<unsigned char *>(p.keys) + (size_t)row * p.stride + f0 * 2;
    if constexpr (W == 8)
      *reinterpret_cast<uint4 *>(dst) = make_uint4(s[0] | s[1] << 16, s[2] | s[3] << 16, s[4] | s[5] << 16, s[6] | s[7] << 16);
    else if constexpr (W == 4)
      *reinterpret_cast<uint2 *>(dst) = make_uint2(s[0] | s[1] << 16, s[2] | s[3] << 16);
    else if constexpr (W == 2)
      *reinterpret_cast<uint32_t *>(dst) = s[0] | s[1] << 16;
    else
      *reinterpret_cast<uint16_t *>(dst) = (uint16_t)s[0];
  }
  searched = __reduce_add_sync(0xffffffffu, searched);
  if ((threadIdx.x & 31) == 0 && searched) atomicAdd(p.searched, (unsigned long long)searched);
}

} // namespace tb
