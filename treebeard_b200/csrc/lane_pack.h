// "Lane" layout: forests that no other layout takes -- trees too deep for whole-tree stages, or
// several classes on deep trees -- whose groups fit no shared-memory stage either.  The nodes are
// read from global memory, so what counts is that the walk reads few of them and that they lie
// together (walk_lanes.cuh):
//
//   node  8 bytes  { f32 threshold or leaf value, (distance << 16) | feature }
//
// Trees lie one after another, each in level order with siblings adjacent; `distance` leads from a
// split to its left child and from a leaf -- feature num_features, whose row value is -inf, so that
// the leaf "goes left" -- to the root of the NEXT tree.  A lane that follows distances walks all
// trees of a range without ever looking anything else up, and never takes a step below a leaf.
// Trees are ordered by class for a multiclass forest (class c owns the nodes class_end[c-1] ..
// class_end[c] - 1), else as they come.
#pragma once
#include "forest.h"

#include <cstdint>
#include <string>
#include <vector>

namespace tb {

struct LaneNode {
  float value;
  uint32_t link;
};

struct LaneForest {
  int32_t num_features = 0, transform = 0, num_classes = 0;
  double initial_value = 0.0;
  int64_t num_trees = 0, num_nodes = 0;
  int32_t max_depth = 0;
  std::vector<LaneNode> nodes;
  std::vector<uint32_t> root;      // [num_trees + 1] position of every tree, in walking order, and the end
  std::vector<int32_t> tree_index; // original index of the tree at that position
  std::vector<int32_t> orig_node;  // original node id per node
  std::vector<uint32_t> class_end; // multiclass: end of every class's nodes
};

// Empty string on success; fails where a distance does not fit 16 bits (trees of more than 65535
// nodes) or the forest has 2^31 nodes or 65535 features.
std::string pack_lanes(const Forest &f, LaneForest *out);

} // namespace tb
