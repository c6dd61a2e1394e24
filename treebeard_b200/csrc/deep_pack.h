// "One tree per stage": the packed layout for forests of DEEP trees (9 .. 12 decision
// levels), whose 16-tree groups are far too large for the shared-memory stages of the
// general kernel -- the reference then walks such trees from global memory
// (src/gpu/GPURepresentations.cpp:630-715 caches a tree only when it fits).
//
// Every tree becomes a complete tree of its pair's depth D (trees are sorted by depth and
// taken two at a time; a pair is what one thread walks in lock-step), stored as planes of
// deep_tree_words(D) elements per tree, 16.5 KB at D = 12.  Nodes are numbered IN ORDER: the node
// that prefix p of decisions leads to on level d has number (2p + 1) 2^(D-1-d), leaf l number l; so
// a walk that keeps the number of the leftmost leaf below it finds the node 2^(D-1-d) further on,
// and a right turn adds just that.  Positions are numbers with one element of padding after every
// 32 and one after every 1024: still additive bit by bit, but the nodes of the upper levels and the
// siblings of the lower ones spread over all shared-memory banks (19.2 wavefronts for the 12 node
// loads of a warp on random trees; 21.4 in level order):
//
//   node plane   u32  (feature code << 16) | threshold key.  Feature code: the byte offset of the
//                     feature's line in a key tile (128 f), or f itself where that does not fit 16 bits
//   leaf plane   f32  leaf values
//   exact plane  f32  fp32 thresholds, laid out like the node plane (global memory only)
//
// Rows are staged as the 15-bit order-preserving keys of quant_pack.h, so a block holds
// 32 x row_warps rows (512 for 128 features) next to a ring of whole-tree pieces; key ties
// are resolved on the exact fp32 values, which keeps leaf selection that of the fp32 walk.
// A leaf above the bottom level is a chain of pass-through nodes (key 0, below every row key:
// always left) ending in the leaf slot that holds its value.
#pragma once
#include "forest.h"
#include "quant_pack.h"

#include <cstdint>
#include <string>
#include <vector>

#ifdef __CUDACC__
#define TB_BOTH_SIDES __host__ __device__
#else
#define TB_BOTH_SIDES
#endif

namespace tb {

constexpr int kDeepMaxDepth = 12;
constexpr int kDeepMinDepth = 2; // pieces of at least 16 bytes
TB_BOTH_SIDES constexpr uint32_t deep_position(uint32_t number) { return number + (number >> 5) + (number >> 10); }
TB_BOTH_SIDES constexpr uint32_t deep_tree_words(uint32_t depth) { return (deep_position((1u << depth) - 1) + 1 + 3) / 4 * 4; }
constexpr int kDeepNarrowFeatures = 511; // feature codes up to here are byte offsets
inline uint32_t deep_feature_code(int32_t num_features, uint32_t f) { return num_features <= kDeepNarrowFeatures ? 128 * f : f; }

struct DeepForest {
  int32_t num_features = 0, transform = 0;
  double initial_value = 0.0;
  int64_t num_trees = 0, num_nodes = 0;
  int32_t max_depth = 0;
  std::vector<QuantGroup> pairs;    // elem_off of tree 0 of the pair; tree 1 follows at + slots = deep_tree_words(depth)
  std::vector<uint32_t> node_plane; // key field is filled on the device at upload
  std::vector<float> leaf_plane;
  std::vector<float> exact_plane;
  std::vector<int32_t> orig_leaf;   // original node id per leaf-plane element
  std::vector<int32_t> tree_index;  // [pairs*2] original tree index, -1 = filler
  std::vector<float> lo, scale;     // per feature (+ sentinel entry)
};

// Empty string on success; fails for multiclass forests, trees deeper than kDeepMaxDepth
// or non-finite thresholds.
std::string pack_deep(const Forest &f, DeepForest *out);

// Host interpreter of the packed planes (layout verification only).
void walk_deep_on_host(const DeepForest &q, const float *rows, int64_t n_rows, int64_t ld,
                       int32_t *leaf_ids, float *sums, int64_t *ties);

} // namespace tb
