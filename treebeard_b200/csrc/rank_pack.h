// "Rank keys": the packed layout for forests of at most 8 levels over rows that are narrow
// enough for the rank kernels (walk_rank.cuh, walk_rank_tiles.cuh).
//
// A threshold is compared with one feature only, so all that a walk needs to know of a row value
// x is its RANK among the feature's distinct thresholds t_0 < t_1 < ...:
//     rank(x) = number of thresholds with !(x < t)          (NaN: all of them)
//     x < t_j  <=>  rank(x) < j + 1
// A row is ranked once per batch (tb_rank_rows); from then on a decision is ONE comparison of
// 16-bit whole numbers that is never in doubt -- there are no ties to flag and to walk again, as
// there are with the rounded keys of quant_pack.h.
//
// Ranking uses a table per feature: the range of its thresholds is cut into equal buckets,
// lut[b] = thresholds in the buckets before b, and the thresholds of the value's own bucket are
// searched.  Bucket numbers are computed with one subtraction and one multiplication, both
// monotone, on the host and on the device alike, so a bucket separates values exactly.  A
// LATTICE feature (whole-number thresholds close together) has one bucket per whole number; a
// whole-number row value is ranked by the table alone.
//
// Planes, per group of 32 trees of (padded) depth D, 2^D slots x 32 columns each:
//   node plane  u32  (key offset << 16) | (j + 1); the offset is the byte offset of the feature's
//                    key in a row of keys (2 f), in a pair of rows (up to 32 features: 4 f) or in
//                    a tile of 32 rows (more than 64 features: (f / 2) 128 + (f mod 2) 2; more than 511,
//                    whose keys are bytes: (f / 4) 128 + f mod 4)
//   leaf plane  f32  leaf values
// Slots: node on level d reached by the decisions r_0 .. r_(d-1) (1 = right) is slot
// 2^d - 1 + sum r_i 2^i, leaf sum r_i 2^i.  With the decision of level i worth 2^i slots on EVERY
// level below, a walk keeps one offset that a right turn adds 2^i * 128 bytes to, and the start of
// a level is an immediate of the load: a comparison and a predicated addition advance the walk.
// A leaf above the bottom level fills the all-left path below it with nodes that always go left
// (key offset 0, threshold rank kRankAlwaysLeft).
//
// Columns are trees ordered by depth; for a multiclass forest by (class, depth) WITHOUT padding
// the classes to whole groups: class c owns the columns class_begin[c] .. class_begin[c+1] - 1.
#pragma once
#include "forest.h"
#include "quant_pack.h"

#include <memory>

namespace tb {

constexpr int kRankCols = 32, kRankMaxDepth = 8;
// A forest all of whose ranks fit the positive half-precision numbers is compared by the half2
// comparison, which needs no masking (one instruction per decision less than whole numbers).
constexpr uint32_t kRankHalfMax = 31742, kRankMax = 65534;
constexpr int kRankPairFeatures = 32; // up to here the keys of two rows lie side by side
constexpr int kRankRowFeatures = 64;  // up to here the keys of a row have a bank each
constexpr int kRankMaxFeatures = 511; // up to here four tiles of keys fit beside the ring and four walker warps (walk_rank_tiles.cuh)
// Wider rows: keys of one byte, for features of at most kRankByteMax distinct thresholds.
constexpr int kRankMaxByteFeatures = 2044; // (offsets in a tile have 16 bits)
constexpr uint32_t kRankByteMax = 255;
constexpr bool rank_bytes(int32_t num_features) { return num_features > kRankMaxFeatures; }
inline uint32_t rank_key_offset(int32_t num_features, uint32_t feature) {
  if (rank_bytes(num_features)) return (feature >> 2) * 128 + (feature & 3);
  if (num_features > kRankRowFeatures) return (feature >> 1) * 128 + (feature & 1) * 2;
  return num_features <= kRankPairFeatures ? 4 * feature : 2 * feature;
}
inline uint32_t rank_feature_at(int32_t num_features, uint32_t offset) {
  if (rank_bytes(num_features)) return (offset >> 7) * 4 + (offset & 3);
  if (num_features > kRankRowFeatures) return (offset >> 7) * 2 + (offset >> 1 & 1);
  return num_features <= kRankPairFeatures ? offset / 4 : offset / 2;
}

struct RankFeature { // 32 bytes, the same on the device
  float lo;          // smallest threshold
  float scale;       // buckets per unit
  float top;         // buckets - 1
  uint32_t lut_off;  // first of buckets + 1 entries
  uint32_t thr_off;  // first of n thresholds
  uint32_t n;        // distinct thresholds (0: the feature is not used)
  uint32_t buckets;
  uint32_t lattice;
};

struct RankForest {
  int32_t num_features = 0, transform = 0, num_classes = 0;
  double initial_value = 0.0;
  int64_t num_trees = 0, num_nodes = 0;
  int32_t max_depth = 0;   // at least 1
  int32_t lattice = 0;       // some feature is a lattice feature
  int32_t whole_compare = 0; // some rank exceeds kRankHalfMax: compare as whole numbers
  std::vector<QuantGroup> groups; // elem_off in elements of either plane
  std::vector<uint32_t> node_plane;
  std::vector<float> leaf_plane;
  std::vector<int32_t> orig_leaf;   // original node id per leaf-plane element
  std::vector<int32_t> tree_index;  // [groups*32] original tree index, -1 = filler
  std::vector<int32_t> class_begin; // multiclass: [num_classes + 1] first column of every class
  std::vector<RankFeature> features;
  std::vector<uint16_t> lut;
  std::vector<float> thresholds;
};

// Empty string on success; fails (so that the caller can take another layout) for trees deeper
// than 8 levels, more than kRankMaxByteFeatures features (kRankRowFeatures for multiclass forests),
// non-finite thresholds or leaves, or a feature with more than kRankMax distinct thresholds
// (kRankHalfMax beyond kRankRowFeatures features, kRankByteMax beyond kRankMaxFeatures).
std::string pack_rank(const Forest &f, RankForest *out);

// The rank tables of 32 neighbouring features each, interleaved for rank_slabs.cuh: 128-byte lines whose word i belongs to
// feature 32 s + i.  Four lines (buckets per unit, bucket of zero, largest threshold, lattice), then a line per bucket (128 times the
// thresholds before it), then a line per threshold and 2^steps - 1 of infinity.  Bucket of x: fma(min(x, largest threshold),
// scale, bias), below zero bucket zero; no bucket holds more than 2^steps - 1 thresholds.
struct SlabTables {
  uint32_t buckets = 0; // lines of each slab
  int32_t steps = 0;
  uint32_t bytes = 0; // per slab
  std::unique_ptr<uint32_t[]> words;
  size_t num_words = 0;
};
// False where a slab takes more than `room` bytes.  One to eight buckets per threshold of the feature that has most.
bool make_slab_tables(const RankForest &q, uint32_t room, SlabTables *out);

// Rank of a row value; *searched: the look-up table alone doesn't give it (a feature with thresholds, and not a whole number
// on a lattice feature).
uint32_t rank_of(const RankForest &q, int32_t feature, float x, bool *searched);

// Host interpreter of the packed planes (layout verification only).
void walk_rank_on_host(const RankForest &q, const float *rows, int64_t n_rows, int64_t ld, int32_t *leaf_ids, float *sums,
                       int64_t *searched);

} // namespace tb
