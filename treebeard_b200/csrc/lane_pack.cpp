#include "lane_pack.h"

#include <algorithm>
#include <atomic>
#include <numeric>

namespace tb {

std::string pack_lanes(const Forest &f, LaneForest *out) {
  const int64_t T = f.num_trees(), N = f.num_nodes();
  if (N >= INT32_MAX) return "more than 2^31 nodes";
  if (f.num_features >= 65535) return "more than 65534 features";
  LaneForest &q = *out;
  q = LaneForest();
  q.num_features = f.num_features;
  q.transform = f.transform;
  q.num_classes = f.num_classes;
  q.initial_value = f.initial_value;
  q.num_trees = T;
  q.num_nodes = N;
  std::vector<int32_t> order(T);
  std::iota(order.begin(), order.end(), 0);
  if (f.num_classes > 0)
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return f.class_id[a] < f.class_id[b]; });
  q.tree_index = order;
  q.root.assign(T + 1, 0);
  for (int64_t k = 0; k < T; ++k) q.root[k + 1] = q.root[k] + (uint32_t)(f.tree_off[order[k] + 1] - f.tree_off[order[k]]);
  if (f.num_classes > 0) {
    q.class_end.assign(f.num_classes, 0);
    for (int64_t k = 0; k < T; ++k) q.class_end[f.class_id[order[k]]] = q.root[k + 1];
    for (int32_t c = 1; c < f.num_classes; ++c) q.class_end[c] = std::max(q.class_end[c], q.class_end[c - 1]);
  }
  q.nodes.resize(N);
  q.orig_node.resize(N);
  std::atomic<bool> far{false};
  std::atomic<int32_t> deepest{0};
#pragma omp parallel for schedule(dynamic, 16) num_threads(pack_threads()) if (N > 1 << 15)
  for (int64_t k = 0; k < T; ++k) {
    const int64_t a = f.tree_off[order[k]];
    const uint32_t base = q.root[k], end = q.root[k + 1];
    struct Item { int32_t node, level; };
    std::vector<Item> queue{{0, 0}}; // queue[i]: the node at position base + i
    queue.reserve(end - base);
    int32_t levels = 0;
    for (size_t i = 0; i < queue.size(); ++i) {
      const Item it = queue[i];
      const int64_t n = a + it.node;
      const bool leaf = f.left[n] < 0;
      const uint64_t distance = leaf ? end - (base + i) : queue.size() - i;
      if (distance > 65535) far = true;
      q.nodes[base + i] = LaneNode{f.thr[n], (uint32_t)(distance & 0xffff) << 16 | (uint32_t)(leaf ? f.num_features : f.feat[n])};
      q.orig_node[base + i] = it.node;
      levels = std::max(levels, it.level);
      if (!leaf) {
        queue.push_back({f.left[n], it.level + 1});
        queue.push_back({f.right[n], it.level + 1});
      }
    }
    int32_t seen = deepest.load();
    while (levels > seen && !deepest.compare_exchange_weak(seen, levels)) {}
  }
  q.max_depth = deepest;
  return far ? "a tree has more than 65535 nodes" : "";
}

} // namespace tb
