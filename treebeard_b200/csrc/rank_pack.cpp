#include "rank_pack.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <numeric>
#include <utility>

namespace tb {

namespace {

// Bucket of a value; the device computes the same two roundings.
uint32_t bucket_of(const RankFeature &f, float x) {
  const float d = x - f.lo;
  const float y = d * f.scale;
  return (uint32_t)std::fmax(std::fmin(y, f.top), 0.f); // (NaN: the last bucket)
}

uint32_t bits_of(float x) {
  uint32_t u;
  std::memcpy(&u, &x, 4);
  return u;
}

// The bucket table of one feature whose sorted distinct thresholds are t[0..n).
void fill_table(RankFeature *f, const float *t, uint16_t *lut) {
  for (uint32_t b = 0; b <= f->buckets; ++b) lut[b] = 0;
  for (uint32_t i = 0; i < f->n; ++i) ++lut[bucket_of(*f, t[i]) + 1];
  for (uint32_t b = 1; b <= f->buckets; ++b) lut[b] = (uint16_t)(lut[b] + lut[b - 1]);
}

// Has this feature more than `limit` distinct thresholds?  Asked of the most used one it settles most forests that have
// too many for one-byte keys before all splits are sorted: 2000 trees of 8 levels over 520 features
// 1.9 ms instead of 12.0 (8 cores).
bool crowded(const Forest &f, int32_t feature, uint32_t limit) {
  std::vector<float> thr;
  for (int64_t g = 0; g < f.num_nodes() && thr.size() < 2 * limit; ++g)
    if (f.feat[g] == feature && !f.is_leaf(g)) thr.push_back(f.thr[g]);
  std::sort(thr.begin(), thr.end());
  return std::unique(thr.begin(), thr.end()) - thr.begin() > (int64_t)limit;
}

} // namespace

std::string pack_rank(const Forest &f, RankForest *out) {
  const int64_t T = f.num_trees(), N = f.num_nodes();
  const int F = f.num_features;
  if (F > kRankMaxByteFeatures) return "more than " + std::to_string(kRankMaxByteFeatures) + " features";
  const bool tiles = F > kRankRowFeatures;
  if (tiles && f.num_classes > 0) return "multiclass forests over more than " + std::to_string(kRankRowFeatures) + " features";
  RankForest &q = *out;
  q = RankForest();
  q.num_features = F;
  q.transform = f.transform;
  q.num_classes = f.num_classes;
  q.initial_value = f.initial_value;
  q.num_trees = T;
  q.num_nodes = N;

  // ---- distinct thresholds per feature, and every split's rank among them
  if (N > INT32_MAX) return "more than 2^31 nodes";
  // (counted and put in their places by several threads, each with a range of the nodes: in the nodes' order)
  const int parts = N > 1 << 15 ? pack_threads() : 1;
  std::vector<int64_t> first(F + 1, 0), at((size_t)parts * F, 0); // at[part * F + feature]
  bool finite = true;
#pragma omp parallel for schedule(static, 1) reduction(&& : finite) num_threads(parts)
  for (int p = 0; p < parts; ++p) {
    int64_t *const mine = at.data() + (size_t)p * F;
    for (int64_t g = N * p / parts; g < N * (p + 1) / parts; ++g) {
      finite = finite && std::isfinite(f.thr[g]);
      if (!f.is_leaf(g)) ++mine[f.feat[g]];
    }
  }
  if (!finite) return "non-finite threshold or leaf value";
  int32_t most_used = 0;
  for (int i = 0; i < F; ++i) {
    int64_t end = first[i];
    for (int p = 0; p < parts; ++p) end += std::exchange(at[(size_t)p * F + i], end);
    first[i + 1] = end;
    if (end - first[i] > first[most_used + 1] - first[most_used]) most_used = i;
  }
  const uint32_t limit = rank_bytes(F) ? kRankByteMax : tiles ? kRankHalfMax : kRankMax;
  const std::string too_many = "a feature has more than " + std::to_string(limit) + " distinct thresholds";
  if (rank_bytes(F) && first[most_used + 1] - first[most_used] > (int64_t)limit && crowded(f, most_used, limit)) return too_many;
  struct Split { // (by threshold, then node)
    float threshold;
    int32_t node;
    bool operator<(const Split &o) const { return threshold < o.threshold || (!(o.threshold < threshold) && node < o.node); }
  };
  const std::unique_ptr<Split[]> split(new Split[first[F]]); // by feature
#pragma omp parallel for schedule(static, 1) num_threads(parts)
  for (int p = 0; p < parts; ++p) {
    int64_t *const mine = at.data() + (size_t)p * F;
    for (int64_t g = N * p / parts; g < N * (p + 1) / parts; ++g)
      if (!f.is_leaf(g)) split[mine[f.feat[g]]++] = Split{f.thr[g], (int32_t)g};
  }
  std::vector<uint16_t> rank(N, 0);
  std::vector<std::vector<float>> distinct(F);
  std::atomic<uint32_t> most{0};
#pragma omp parallel for schedule(dynamic, 1) num_threads(pack_threads()) if (N > 1 << 15)
  for (int i = 0; i < F; ++i) {
    std::sort(split.get() + first[i], split.get() + first[i + 1]);
    auto &d = distinct[i];
    for (int64_t k = first[i]; k < first[i + 1]; ++k) {
      if (d.empty() || d.back() != split[k].threshold) d.push_back(split[k].threshold);
      rank[split[k].node] = (uint16_t)std::min<size_t>(d.size(), kRankMax + 1);
    }
    uint32_t seen = most.load();
    while (d.size() > seen && !most.compare_exchange_weak(seen, (uint32_t)d.size())) {}
  }
  if (most > limit) return too_many;
  q.whole_compare = most > kRankHalfMax;

  // ---- rank tables
  q.features.resize(F);
  uint32_t lut_size = 0, thr_size = 0;
  for (int i = 0; i < F; ++i) {
    const auto &d = distinct[i];
    RankFeature &rf = q.features[i];
    rf = RankFeature{0.f, 0.f, 0.f, lut_size, thr_size, (uint32_t)d.size(), 1, 0};
    if (!d.empty()) {
      rf.lo = d.front();
      const float hi = d.back();
      bool whole = std::fabs(rf.lo) <= 0x1p22f && std::fabs(hi) <= 0x1p22f && hi - rf.lo <= std::max(4096.f, 4.f * (float)d.size());
      for (size_t k = 0; k < d.size() && whole; ++k) whole = d[k] == std::floor(d[k]);
      if (whole) {
        rf.lattice = 1;
        q.lattice = 1;
        rf.buckets = (uint32_t)(hi - rf.lo) + 1;
        rf.scale = 1.f;
      } else {
        // two buckets per threshold: the table takes as much room as the thresholds, and three steps
        // finish the search of the fullest bucket that a warp usually meets
        rf.buckets = 2 * (uint32_t)d.size();
        const float range = hi - rf.lo;
        rf.scale = range > 0.f && std::isfinite(range) ? (float)rf.buckets / range : 0.f;
        if (!std::isfinite(rf.scale) || rf.scale == 0.f) { // a range that fp32 cannot cut up: one bucket
          rf.scale = 0.f;
          rf.buckets = 1;
        }
      }
    }
    rf.top = (float)(rf.buckets - 1);
    lut_size += (rf.buckets + 1 + 7) / 8 * 8; // (tables start on 16-byte boundaries)
    thr_size += ((uint32_t)d.size() + 3) / 4 * 4;
  }
  q.lut.assign(lut_size, 0);
  q.thresholds.assign(thr_size, 0.f);
#pragma omp parallel for schedule(dynamic, 1) num_threads(pack_threads()) if (N > 1 << 15)
  for (int i = 0; i < F; ++i) {
    RankFeature &rf = q.features[i];
    std::copy(distinct[i].begin(), distinct[i].end(), q.thresholds.begin() + rf.thr_off);
    fill_table(&rf, distinct[i].data(), q.lut.data() + rf.lut_off);
  }

  // ---- columns: trees by (class,) depth
  std::vector<int32_t> depth(T);
  int32_t deepest = 0;
#pragma omp parallel for schedule(dynamic, 64) reduction(max : deepest) num_threads(pack_threads()) if (N > 1 << 15)
  for (int64_t t = 0; t < T; ++t) {
    depth[t] = tree_depth(f, t);
    deepest = std::max(deepest, depth[t]);
  }
  q.max_depth = std::max(1, deepest);
  if (deepest > kRankMaxDepth) return "trees deeper than " + std::to_string(kRankMaxDepth) + " levels";
  std::vector<int64_t> order(T);
  std::iota(order.begin(), order.end(), 0);
  const bool multi = f.num_classes > 0;
  std::stable_sort(order.begin(), order.end(), [&](int64_t a, int64_t b) {
    if (multi && f.class_id[a] != f.class_id[b]) return f.class_id[a] < f.class_id[b];
    return depth[a] < depth[b];
  });
  if (multi) {
    q.class_begin.assign(f.num_classes + 1, 0);
    for (int64_t t = 0; t < T; ++t) ++q.class_begin[f.class_id[t] + 1];
    for (int32_t c = 0; c < f.num_classes; ++c) q.class_begin[c + 1] += q.class_begin[c];
  }
  const int64_t G = (T + kRankCols - 1) / kRankCols;
  q.groups.resize(G);
  q.tree_index.assign(G * kRankCols, -1);
  uint64_t elems = 0;
  for (int64_t g = 0; g < G; ++g) {
    uint32_t d = 1;
    for (int64_t k = g * kRankCols; k < std::min(T, (g + 1) * kRankCols); ++k) d = std::max<uint32_t>(d, depth[order[k]]);
    q.groups[g] = QuantGroup{elems, d, 1u << d};
    elems += (uint64_t)(1u << d) * kRankCols;
  }
  const uint32_t always_left = q.whole_compare ? 0xffffu : kRankHalfMax + 1;
  q.node_plane.assign(elems, always_left);
  q.leaf_plane.assign(elems, 0.f);
  q.orig_leaf.assign(elems, -1);
#pragma omp parallel for schedule(dynamic, 1) num_threads(pack_threads()) if (N > 1 << 15)
  for (int64_t g = 0; g < G; ++g) {
    const QuantGroup &gm = q.groups[g];
    struct Item { int32_t node; uint32_t path, level; };
    std::vector<Item> stack;
    for (int c = 0; c < kRankCols && g * kRankCols + c < T; ++c) {
      const int64_t t = order[g * kRankCols + c], a = f.tree_off[t];
      q.tree_index[g * kRankCols + c] = (int32_t)t;
      stack.assign(1, Item{0, 0, 0});
      while (!stack.empty()) {
        const Item it = stack.back();
        stack.pop_back();
        const int64_t n = a + it.node;
        if (f.left[n] < 0) { // all-left from here on
          const uint64_t e = gm.elem_off + (uint64_t)it.path * kRankCols + c;
          q.leaf_plane[e] = f.thr[n];
          q.orig_leaf[e] = it.node;
          continue;
        }
        const uint64_t e = gm.elem_off + (uint64_t)((1u << it.level) - 1 + it.path) * kRankCols + c;
        q.node_plane[e] = (rank_key_offset(F, (uint32_t)f.feat[n]) << 16) | rank[n];
        stack.push_back({f.left[n], it.path, it.level + 1});
        stack.push_back({f.right[n], it.path | (1u << it.level), it.level + 1});
      }
    }
  }
  return "";
}

namespace {

struct SlabFeature { // buckets of a feature (rank_slabs.cuh)
  float scale = 0.f, bias = 0.f, most = 0.f;
  SlabFeature(const float *t, uint32_t n, uint32_t buckets) {
    if (n == 0) return;
    most = t[n - 1];
    const float range = most - t[0];
    scale = range > 0.f && std::isfinite(range) ? ((float)buckets - 0.5f) / range : 0.f;
    bias = -(t[0] * scale);
    // (a range that fp32 cannot cut up: one bucket)
    if (!std::isfinite(scale) || !std::isfinite(bias) || !(std::fma(most, scale, bias) < (float)buckets)) scale = bias = 0.f;
  }
  uint32_t bucket(float x) const { // (as the device: never decreasing in x)
    const float y = std::fma(std::fmin(x, most), scale, bias);
    return y > 0.f ? (uint32_t)y : 0u;
  }
};

} // namespace

bool make_slab_tables(const RankForest &q, uint32_t room, SlabTables *out) {
  const int F = q.num_features, slabs = (F + 31) / 32;
  uint32_t most = 1; // thresholds of a feature
  for (const RankFeature &f : q.features) most = std::max(most, f.n);
  SlabTables &t = *out;
  t = SlabTables();
  for (const uint32_t per : {1u, 2u, 3u, 4u, 6u, 8u}) {
    if (512 + 128ull * (per + 1) * most > room) break;
    const uint32_t buckets = per * most;
    uint32_t fullest = 1;
#pragma omp parallel for schedule(dynamic, 8) reduction(max : fullest) num_threads(pack_threads()) if ((int64_t)F * most > 1 << 15)
    for (int i = 0; i < F; ++i) {
      const RankFeature &f = q.features[i];
      const float *thr = q.thresholds.data() + f.thr_off;
      const SlabFeature b(thr, f.n, buckets);
      for (uint32_t k = 0, here = 0, last = buckets; k < f.n; ++k) {
        const uint32_t bucket = b.bucket(thr[k]);
        here = bucket == last ? here + 1 : 1;
        last = bucket;
        fullest = std::max(fullest, here);
      }
    }
    int32_t steps = 1;
    while ((1u << steps) - 1 < fullest) ++steps;
    const uint64_t bytes = 512 + 128ull * buckets + 128ull * (most + (1u << steps) - 1);
    // a step is paid for by every value, the table's copy by every block: about the same for 64 KB
    if (bytes > room || (t.bytes && steps + (double)bytes / 65536 >= t.steps + (double)t.bytes / 65536)) continue;
    t.buckets = buckets;
    t.steps = steps;
    t.bytes = (uint32_t)bytes;
  }
  if (!t.bytes) return false;
  t.words.reset(new uint32_t[t.num_words = (size_t)slabs * (t.bytes / 4)]); // (each of them is written below)
#pragma omp parallel for schedule(dynamic, 8) num_threads(pack_threads()) if ((int64_t)F * most > 1 << 15)
  for (int i = 0; i < slabs * 32; ++i) {
    uint32_t *w = t.words.get() + (size_t)(i / 32) * (t.bytes / 4) + i % 32;
    uint32_t *const thr_words = w + 128 + 32 * (size_t)t.buckets;
    const uint32_t n = i < F ? q.features[i].n : 0, lines = t.bytes / 128 - 4 - t.buckets;
    for (uint32_t k = n; k < lines; ++k) thr_words[32 * (size_t)k] = bits_of(INFINITY);
    if (n == 0) { // one bucket, no thresholds
      for (uint32_t k = 0; k < 4 + t.buckets; ++k) w[32 * (size_t)k] = 0;
      continue;
    }
    const RankFeature &f = q.features[i];
    const float *thr = q.thresholds.data() + f.thr_off;
    const SlabFeature b(thr, n, t.buckets);
    w[0] = bits_of(b.scale);
    w[32] = bits_of(b.bias);
    w[64] = bits_of(b.most);
    w[96] = f.lattice;
    uint32_t before = 0;
    uint32_t first = b.bucket(thr[0]); // of the threshold number `before`
    for (uint32_t bucket = 0; bucket < t.buckets; ++bucket) {
      while (before < n && first < bucket)
        if (++before < n) first = b.bucket(thr[before]);
      w[128 + 32 * (size_t)bucket] = 128 * before;
    }
    for (uint32_t k = 0; k < n; ++k) thr_words[32 * (size_t)k] = bits_of(thr[k]);
  }
  return true;
}

uint32_t rank_of(const RankForest &q, int32_t feature, float x, bool *searched) {
  const RankFeature &f = q.features[feature];
  const uint32_t b = bucket_of(f, x);
  uint32_t s = q.lut[f.lut_off + b], e = q.lut[f.lut_off + b + 1];
  const bool looked_up = f.lattice && x == std::floor(x);
  if (looked_up) s = e = x < f.lo ? 0 : e;
  *searched = f.n > 0 && !looked_up;
  while (s < e) {
    const uint32_t m = (s + e) >> 1;
    if (x < q.thresholds[f.thr_off + m]) e = m;
    else s = m + 1;
  }
  return s;
}

void walk_rank_on_host(const RankForest &q, const float *rows, int64_t n_rows, int64_t ld, int32_t *leaf_ids, float *sums,
                       int64_t *searched) {
  const int C = std::max(1, q.num_classes);
  std::vector<uint32_t> key(q.num_features + 1, 0);
  int64_t count = 0;
  for (int64_t r = 0; r < n_rows; ++r) {
    for (int i = 0; i < q.num_features; ++i) {
      bool s;
      key[i] = rank_of(q, i, rows[r * ld + i], &s);
      count += s;
    }
    if (sums) std::fill(sums + r * C, sums + (r + 1) * C, 0.f);
    int32_t cls = 0;
    for (size_t k = 0; k < q.tree_index.size(); ++k) {
      if (q.tree_index[k] < 0) continue;
      const QuantGroup &gm = q.groups[k / kRankCols];
      const uint64_t base = gm.elem_off + k % kRankCols;
      uint32_t path = 0;
      for (uint32_t d = 0; d < gm.depth; ++d) {
        const uint32_t node = q.node_plane[base + (uint64_t)((1u << d) - 1 + path) * kRankCols];
        if (key[rank_feature_at(q.num_features, node >> 16)] >= (node & 0xffffu)) path |= 1u << d;
      }
      const uint64_t e = base + (uint64_t)path * kRankCols;
      while (q.num_classes > 0 && (int32_t)k >= q.class_begin[cls + 1]) ++cls;
      if (sums) sums[r * C + cls] += q.leaf_plane[e];
      if (leaf_ids) leaf_ids[r * q.num_trees + q.tree_index[k]] = q.orig_leaf[e];
    }
  }
  if (searched) *searched = count;
}

} // namespace tb
