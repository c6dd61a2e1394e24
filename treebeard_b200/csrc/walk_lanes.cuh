// Walk kernel for the lane layout (lane_pack.h): every lane takes its row through the trees of a
// range at its own pace.  A step follows the node's distance -- to a child, or from a leaf to the
// next tree's root -- so a lane spends no step below a leaf and needs no tree counter; a fixed-depth
// walk takes every row to the depth of the deepest tree of the group (16 steps where trees grown
// until their leaves are pure need 5).  65536 rows through 200 such trees of up to 16 levels: 207 us at
// fixed depth from interleaved groups, 83.5 us here.
//
// A warp = 32 rows and one of `shares` ranges of the trees; the row tile (transposed, bank = row) is
// shared by the warps that split the trees, and their sums meet in shared memory in share order.
// What bounds the kernel is the nodes' gathers: 19 sectors of L1 a load, 93 % of them hits, 18 warps waiting for
// one per instruction issued, the load pipe 68 % and issue 49 % busy (65536 rows x 200 trees).  So blocks are
// small and many fit an SM: the trees being walked stay in L1.  blockIdx.y splits the trees further for small batches, those of
// every class alike (3000 rows, 3 classes of 30 trees: 50.2 us with whole classes to a warp, 22.6 so); a
// second kernel adds those partial sums (walk_kernels.cuh).
//
// Reference counterparts: the scalar walk that stops at a leaf, src/mlir/CodeGenStateMachine.cpp:
// 149-243; the tie rule of class ids, src/reduction/LowerReduceOps.cpp:148-189.
#pragma once
#include "walk_kernels.cuh"

#include <type_traits>

namespace tb {

// A lane adds its leaves one after another.  Against 64 bits (2-norm over 4096 of 65536 rows; one fp32 sum of 50 and
// of 250 trees: 1.1e-7 and 3.8e-7, a double one 3.0e-8 and 3.5e-8) the fp32 sum of a short chain is as
// good as that of a fixed-depth walk (1.0e-7 and 1.4e-7), a long one is not.  The double one costs 6 % of
// the kernel at 50 trees (83.5 -> 89.9 us, 65536 rows x 200 trees), 5 % at 250 (425 -> 445 us, 1000 trees).
constexpr int kLaneShortChain = 64;

struct LaneParams {
  const uint2 *nodes;
  const uint32_t *root;       // [num_trees + 1]
  const int32_t *tree_index;
  const int32_t *orig_node;
  const uint32_t *class_end;  // multiclass: end of every class's nodes, of its trees
  const uint32_t *class_tree;
  const float *rows;
  long long n_rows, ld;
  float *partial;             // write_partial: [chunks][n_rows], or [chunks][n_rows][classes]
  void *out;
  int32_t *leaf_ids;
  long long num_trees;
  int32_t num_features, num_classes, transform, out_kind, write_partial;
  float initial_value;
  int32_t tiles, shares;      // of a block: row tiles, warps that split the trees of a tile
  int32_t vec4_ok;
};

// all * i / n in 32 bits (n: at most 1024)
__device__ __forceinline__ uint32_t lane_share(uint32_t all, uint32_t i, uint32_t n) { return all / n * i + all % n * i / n; }

// Where part `i` of `n` of the trees begins; parts of a multiclass forest are whole classes.
template <bool WHOLE_CLASSES> __device__ __forceinline__ uint32_t lane_part(const LaneParams &p, uint32_t i, uint32_t n) {
  if constexpr (!WHOLE_CLASSES) return p.root[lane_share((uint32_t)p.num_trees, i, n)];
  const uint32_t c = lane_share((uint32_t)p.num_classes, i, n);
  return c == 0 ? 0u : p.class_end[c - 1];
}

// LONG: chains of more than kLaneShortChain trees, summed in a double accumulator.
template <bool CLASSES, bool LEAF_IDS, bool LONG>
__global__ void __launch_bounds__(512) tb_walk_lanes_kernel(const LaneParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tile = warp % p.tiles, share = warp / p.tiles;
  const int F = p.num_features;
  float *xs = reinterpret_cast<float *>(smem_raw) + (size_t)tile * (F + 1) * 32;
  float *sums = reinterpret_cast<float *>(smem_raw) + (size_t)p.tiles * (F + 1) * 32; // [warp][row], classes: [warp][2][row]
  const long long row = ((long long)blockIdx.x * p.tiles + tile) * 32 + lane;
  const bool live = row < p.n_rows;
  {
    const float *src = p.rows + (live ? row : 0) * p.ld;
    if (p.vec4_ok) {
      for (int k = share; k < F / 4; k += p.shares) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(src) + k);
        xs[(4 * k + 0) * 32 + lane] = v.x;
        xs[(4 * k + 1) * 32 + lane] = v.y;
        xs[(4 * k + 2) * 32 + lane] = v.z;
        xs[(4 * k + 3) * 32 + lane] = v.w;
      }
    } else {
      for (int k = share; k < F; k += p.shares) xs[k * 32 + lane] = __ldg(src + k);
    }
    if (share == 0) xs[F * 32 + lane] = -INFINITY; // a leaf's feature: on to the next tree
  }
  __syncthreads();

  constexpr bool WHOLE_CLASSES = CLASSES && !LEAF_IDS;
  const int part = WHOLE_CLASSES ? share : (int)blockIdx.y * p.shares + share;
  const int parts = WHOLE_CLASSES ? p.shares : (int)gridDim.y * p.shares;
  uint32_t n = lane_part<WHOLE_CLASSES>(p, part, parts);
  const uint32_t end = lane_part<WHOLE_CLASSES>(p, part + 1, parts);
  const float *mine = xs + lane;
  using Sum = std::conditional_t<LONG, double, float>;
  Sum acc = 0;
  [[maybe_unused]] float best = -INFINITY;
  [[maybe_unused]] int cls = 0, best_class = 0, last_class = 0;
  [[maybe_unused]] uint32_t class_end = 0, tree = 0;
  if constexpr (WHOLE_CLASSES) {
    cls = (int)lane_share(p.num_classes, part, parts);
    last_class = (int)lane_share(p.num_classes, part + 1, parts);
    if (gridDim.y > 1) { // this block's part of every class
      for (; cls < last_class; ++cls) {
        const uint32_t a = cls > 0 ? p.class_tree[cls - 1] : 0u, trees = p.class_tree[cls] - a;
        const uint32_t stop = p.root[a + lane_share(trees, blockIdx.y + 1, gridDim.y)];
        acc = 0;
        for (n = p.root[a + lane_share(trees, blockIdx.y, gridDim.y)]; n < stop;) {
          const uint2 node = __ldg(p.nodes + n);
          const uint32_t f = node.y & 0xffffu;
          const float t = __uint_as_float(node.x), x = mine[f * 32];
          const bool leaf = f == (uint32_t)F;
          acc += leaf ? (Sum)t : (Sum)0;
          n += (node.y >> 16) + (x < t || leaf ? 0u : 1u);
        }
        if (live) p.partial[((long long)blockIdx.y * p.n_rows + row) * p.num_classes + cls] = (float)acc;
      }
      return;
    }
    class_end = cls < last_class ? p.class_end[cls] : end;
  }
  // the sum of class `cls` is complete (ties go to the higher class)
  [[maybe_unused]] auto close = [&]() {
    const float sum = (float)acc;
    if (p.write_partial && live) p.partial[row * p.num_classes + cls] = sum;
    if (sum >= best) {
      best = sum;
      best_class = cls;
    }
    acc = 0;
    ++cls;
    class_end = cls < last_class ? p.class_end[cls] : 0xffffffffu;
  };
  if constexpr (LEAF_IDS) { // the tree that this part begins with
    uint32_t lo = 0, hi = (uint32_t)p.num_trees;
    while (lo < hi) {
      const uint32_t m = (lo + hi) / 2;
      if (p.root[m] < n) lo = m + 1;
      else hi = m;
    }
    tree = lo;
  }
  while (n < end) {
    if constexpr (WHOLE_CLASSES)
      while (n >= class_end) close();
    const uint2 node = __ldg(p.nodes + n);
    const uint32_t f = node.y & 0xffffu;
    const float t = __uint_as_float(node.x), x = mine[f * 32];
    const bool leaf = f == (uint32_t)F;
    if constexpr (LEAF_IDS) {
      if (leaf) {
        if (live) p.leaf_ids[row * p.num_trees + p.tree_index[tree]] = p.orig_node[n];
        ++tree;
      }
    } else {
      acc += leaf ? (Sum)t : (Sum)0;
    }
    n += (node.y >> 16) + (x < t || leaf ? 0u : 1u);
  }
  if constexpr (LEAF_IDS) return;
  if constexpr (CLASSES) {
    const bool empty = (int)lane_share(p.num_classes, part, parts) == last_class; // (a part without classes wins nothing)
    while (cls < last_class) close();
    if (p.write_partial) return;
    sums[(2 * warp) * 32 + lane] = empty ? __int_as_float(0x7fffffff) : best;
    sums[(2 * warp + 1) * 32 + lane] = __int_as_float(best_class);
    __syncthreads();
    if (share != 0 || !live) return;
    for (int s = 1; s < p.shares; ++s) { // (classes rise with the shares)
      const float b = sums[2 * (s * p.tiles + tile) * 32 + lane];
      if (b >= best) {
        best = b;
        best_class = __float_as_int(sums[(2 * (s * p.tiles + tile) + 1) * 32 + lane]);
      }
    }
    if (p.out_kind == 1) reinterpret_cast<int8_t *>(p.out)[row] = (int8_t)best_class;
    else reinterpret_cast<float *>(p.out)[row] = (float)best_class;
  } else {
    sums[warp * 32 + lane] = (float)acc;
    __syncthreads();
    if (share != 0 || !live) return;
    double all = acc;
    for (int s = 1; s < p.shares; ++s) all += (double)sums[(s * p.tiles + tile) * 32 + lane];
    if (p.write_partial) p.partial[(long long)blockIdx.y * p.n_rows + row] = (float)all;
    else reinterpret_cast<float *>(p.out)[row] = apply_transform((float)((double)p.initial_value + all), p.transform);
  }
}

} // namespace tb
