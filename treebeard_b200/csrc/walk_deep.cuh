// Walk kernel for the one-tree-per-stage layout (deep_pack.h): forests of deep trees.
//
// One block = RW warps = one tile of 32*RW rows, staged ONCE as 15-bit keys and kept for
// the whole forest.  Lane = row: every thread walks its own row through BOTH trees of a
// pair in lock-step (two independent dependence chains per thread), so all threads of the
// block read the same two node planes.  The node planes stream through a ring of whole-tree
// pieces (16 KB each at 12 levels) filled by cp.async.bulk copies that one extra PRODUCER warp
// issues, the next pair's always in flight while a pair is walked; a row warp frees a slot
// with one arrival on the slot's "empty" mbarrier and the producer refills it when all row
// warps have arrived, so the row warps never meet at a block barrier and may drift apart by a
// pair.  Leaf values come straight from L2 (32 scattered
// sectors per warp whatever the layout), by asynchronous copies, and are consumed one pair later.  Sums stay in the
// owning thread's register: there is no cross-thread reduction.
//
// The kernel is bound by latency and, since nothing else waits any more, the shared-memory pipe: 71 % busy, issue
// 50 %, 53.3 wavefronts per walk of 32 rows through 12 levels (24 loads, 4 of bank conflicts of nodes, 23 of leaf
// values; 85248 rows, one wave of 18 row warps, x 400 trees).  (Where all pairs have one depth, tb_walk_deep_staged_kernel
// has the leaf values cheaper.)  A warp that stops for anything but its two chains stops
// the others two pairs later, so nothing in the loop waits for global memory: leaf values are copied to
// shared memory asynchronously (as loads, every pair waited some 600 of 2970 clocks for them, however
// far ahead they were issued), and a tree behind a key tie is put off until the row's other
// trees are done.  1048576 rows x 2000 trees of 12 levels over 128 features: 17.65 -> 16.0 ms; either
// change without the other gains nothing.
//
// Every two row warps have a key tile of their own (128 bytes per feature: word j = row j of the even
// warp | row j of the odd warp << 16), so a warp's key load touches 32 distinct banks and the
// upper half of a node word -- the byte offset of the feature's line -- is one shift-add away from
// the key's address.  The in-order numbering of deep_pack.h makes a right turn one addition that
// depends on the level alone.  A key tie is only flagged on the fast path; the flagged (row, tree) is
// walked again at the end, with exact fp32 comparisons at the tied steps.
//
// Reference counterparts: src/mlir/CodeGenStateMachine.cpp:149-243 (scalar walk),
// src/mlir/WalkDecisionTreeLoweringPass.cpp:24-53 (fixed-depth walk of padded trees),
// src/gpu/GPURepresentations.cpp:279-399 (row cache) and :630-715 (tree cache).
#pragma once
#include "walk_quant.cuh"

namespace tb {

struct DeepParams {
  const uint32_t *node_plane;
  const float *leaf_plane;
  const float *exact_plane;
  const DevQuantGroup *pairs;
  const int32_t *tree_index;
  const int32_t *orig_leaf;
  const float *lo;
  const float *scale;
  const float *rows;
  long long n_rows, ld;
  float *partial;
  void *out;
  int32_t write_partial;
  int32_t *leaf_ids;
  long long num_trees;
  int32_t num_pairs, pairs_per_chunk, num_features, transform;
  float initial_value;
  int32_t ring_slots;  // 4 .. 8
  uint32_t slot_bytes; // of a tree of the forest's depth
  uint32_t tree_words; // the same in words
  uint32_t key_tile;   // bytes of the key tile of two row warps
  uint32_t leaf_off;   // where the leaf values on their way are in shared memory
  int32_t *status;
  unsigned long long *tie_count;
  int32_t skip_first_copy; // failure drill: the first piece's copy is never issued, so its wait expires
  uint32_t wait_tries;     // polls before a wait gives up (0 = kQWaitTries)
};

constexpr int kDeepMaxSlots = 8;
constexpr uint32_t kDeepNoLeaf = 0xffffffffu;
constexpr int kDeepLeafBytes = 512; // per row warp: the leaf values of two pairs
// Trees behind a key tie that a thread puts off.  On continuous features one comparison in some 24000 ties:
// 1.0 per row in 2000 trees of 12 levels, 8.2 in 16000.  A tie walked in place holds up its warp, and with it
// the block two pairs later.  4194304 rows with room for four: 60.0 ms through 2000 trees, 551.5 through
// 16000; with room for 32: 60.2 and 475.1.
constexpr int kDeepTied = 32;

// Fast walk of DEPTH levels of two trees in lock-step, in PTX (the step of walk_quant.cuh: keys
// are 15-bit integers that compare as fp16 numbers, so one half2 comparison of (key, node word)
// picks the child and a second one accumulates the tie flag).  On a level whose distance to the
// leaves is s (deep_position of a power of two, in bytes) the node lies s behind the current
// address, and a right turn moves the address on by s.
// base0 / base1: shared-memory addresses of the node planes; returns the leaf positions reached and
// whether any key comparison on either path tied.
//   %0, %1  addresses (updated)   %2, %3  node words (scratch)   %4  tie flags (out)
//   %5  the thread's base in its key tile
#define TBD_DECL ".reg .b32 ka0, ka1, kx0, kx1;\n .reg .pred p0, p1, t0, t1, q;\n"
#define TBD_KEY(i, n)                                                                                               \
  "shr.u32 ka" #i ", " n ", 16;\n add.u32 ka" #i ", ka" #i ", %5;\n ld.shared.u16 kx" #i ", [ka" #i "];\n"
// WIDE: the upper half of a node word is the feature's number, its line 128 bytes for each
#define TBD_KEYW(i, n)                                                                                              \
  "shr.u32 ka" #i ", " n ", 16;\n mad.lo.u32 ka" #i ", ka" #i ", 128, %5;\n ld.shared.u16 kx" #i ", [ka" #i "];\n"
#define TBD_CMP0(i, n) "setp.lt.f16x2 p" #i "|q, kx" #i ", " n ";\n setp.eq.f16x2 t" #i "|q, kx" #i ", " n ";\n"
#define TBD_CMP(i, n) "setp.lt.f16x2 p" #i "|q, kx" #i ", " n ";\n setp.eq.or.f16x2 t" #i "|q, kx" #i ", " n ", t" #i ";\n"
#define TBD_LEVEL(K, C, step)                                                                                       \
  "ld.shared.u32 %2, [%0+" step "];\n ld.shared.u32 %3, [%1+" step "];\n" K(0, "%2") K(1, "%3") C(0, "%2") C(1, "%3") \
  "@p0 add.u32 %0, %0, " step ";\n @p1 add.u32 %1, %1, " step ";\n"
#define TBD_R1(K) TBD_LEVEL(K, TBD_CMP, "4")
#define TBD_R2(K) TBD_LEVEL(K, TBD_CMP, "8") TBD_R1(K)
#define TBD_R3(K) TBD_LEVEL(K, TBD_CMP, "16") TBD_R2(K)
#define TBD_R4(K) TBD_LEVEL(K, TBD_CMP, "32") TBD_R3(K)
#define TBD_R5(K) TBD_LEVEL(K, TBD_CMP, "64") TBD_R4(K)
#define TBD_R6(K) TBD_LEVEL(K, TBD_CMP, "132") TBD_R5(K)
#define TBD_R7(K) TBD_LEVEL(K, TBD_CMP, "264") TBD_R6(K)
#define TBD_R8(K) TBD_LEVEL(K, TBD_CMP, "528") TBD_R7(K)
#define TBD_R9(K) TBD_LEVEL(K, TBD_CMP, "1056") TBD_R8(K)
#define TBD_R10(K) TBD_LEVEL(K, TBD_CMP, "2112") TBD_R9(K)
#define TBD_R11(K) TBD_LEVEL(K, TBD_CMP, "4228") TBD_R10(K)
#define TBD_L2(K) TBD_LEVEL(K, TBD_CMP0, "8") TBD_R1(K)
#define TBD_L3(K) TBD_LEVEL(K, TBD_CMP0, "16") TBD_R2(K)
#define TBD_L4(K) TBD_LEVEL(K, TBD_CMP0, "32") TBD_R3(K)
#define TBD_L5(K) TBD_LEVEL(K, TBD_CMP0, "64") TBD_R4(K)
#define TBD_L6(K) TBD_LEVEL(K, TBD_CMP0, "132") TBD_R5(K)
#define TBD_L7(K) TBD_LEVEL(K, TBD_CMP0, "264") TBD_R6(K)
#define TBD_L8(K) TBD_LEVEL(K, TBD_CMP0, "528") TBD_R7(K)
#define TBD_L9(K) TBD_LEVEL(K, TBD_CMP0, "1056") TBD_R8(K)
#define TBD_L10(K) TBD_LEVEL(K, TBD_CMP0, "2112") TBD_R9(K)
#define TBD_L11(K) TBD_LEVEL(K, TBD_CMP0, "4228") TBD_R10(K)
#define TBD_L12(K) TBD_LEVEL(K, TBD_CMP0, "8456") TBD_R11(K)
#define TBD_TIES "selp.u32 %4, 1, 0, t0;\n @t1 or.b32 %4, %4, 2;\n"
template <int DEPTH, bool WIDE>
__device__ __forceinline__ void deep_walk(uint32_t base0, uint32_t base1, uint32_t key_lane, uint32_t *j0, uint32_t *j1,
                                          bool *tie0, bool *tie1) {
  static_assert(DEPTH >= 2 && DEPTH <= 12, "two to twelve levels");
  uint32_t a0 = base0, a1 = base1, tb;
  [[maybe_unused]] uint32_t n0, n1;
#define TBD_ASM(levels) asm volatile("{\n" TBD_DECL levels TBD_TIES "}" : "+r"(a0), "+r"(a1), "=&r"(n0), "=&r"(n1), "=&r"(tb) : "r"(key_lane))
#define TBD_CASE(n)                                                                                                 \
  if constexpr (DEPTH == n) {                                                                                       \
    if constexpr (WIDE) TBD_ASM(TBD_L##n(TBD_KEYW));                                                                \
    else TBD_ASM(TBD_L##n(TBD_KEY));                                                                                \
  }
  TBD_CASE(2) TBD_CASE(3) TBD_CASE(4) TBD_CASE(5) TBD_CASE(6) TBD_CASE(7) TBD_CASE(8) TBD_CASE(9) TBD_CASE(10) TBD_CASE(11) TBD_CASE(12)
#undef TBD_CASE
#undef TBD_ASM
  *j0 = (a0 - base0) >> 2;
  *j1 = (a1 - base1) >> 2;
  *tie0 = tb & 1u;
  *tie1 = tb & 2u;
}

template <bool WIDE>
__device__ __forceinline__ void deep_walk_any(uint32_t depth, uint32_t base0, uint32_t base1, uint32_t key_lane, uint32_t *j0,
                                              uint32_t *j1, bool *t0, bool *t1) {
  switch (depth) {
  case 2: return deep_walk<2, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 3: return deep_walk<3, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 4: return deep_walk<4, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 5: return deep_walk<5, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 6: return deep_walk<6, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 7: return deep_walk<7, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 8: return deep_walk<8, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 9: return deep_walk<9, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 10: return deep_walk<10, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  case 11: return deep_walk<11, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  default: return deep_walk<12, WIDE>(base0, base1, key_lane, j0, j1, t0, t1);
  }
}

// Re-walk of one (row, tree) behind a key tie: the staged keys decide wherever they can,
// the tied comparisons read the exact fp32 values from global memory.  Returns the leaf position.
// `nodes`: the tree in global memory, or null to read it from the ring at `base`.
static __device__ __noinline__ uint32_t deep_walk_exact(uint32_t base, const uint32_t *nodes, uint32_t key_lane, bool wide, uint32_t depth,
                                                 const float *exact_tree, const float *rowp) {
  uint32_t at = 0;
  for (uint32_t d = 0; d < depth; ++d) {
    const uint32_t x = 1u << (depth - 1 - d), step = x + (x >> 5) + (x >> 10); // (deep_position)
    const uint32_t node = nodes ? __ldg(nodes + at + step) : lds_u32(base + (at + step) * 4u);
    const uint32_t f = wide ? node >> 16 : node >> 23, kt = node & 0x7fffu;
    const uint32_t kx = lds_u16(key_lane + f * 128u);
    bool right = kx < kt;
    if (kx == kt) right = !(__ldg(rowp + f) < __ldg(exact_tree + at + step));
    at += right ? step : 0u;
  }
  return at;
}

// A word from global to shared memory behind the thread's back, and the wait for all such copies.
__device__ __forceinline__ void copy_word(uint32_t dst, const float *src, bool read) { // (zero without reading otherwise)
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(read ? 4u : 0u) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void sts_f32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

// Stages the thread's row as keys; each thread reads back only the keys it wrote, so no barrier is needed.
__device__ __forceinline__ void deep_stage_row(const DeepParams &p, int F, const float *rowp, bool live, uint32_t key_lane) {
  constexpr uint32_t ks = 128;
  const bool vec = (F % 4 == 0) && (p.ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.rows) & 15) == 0);
  if (vec) {
    for (int f = 0; f < F; f += 4) {
      const float4 x = live ? __ldg(reinterpret_cast<const float4 *>(rowp + f)) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 lo = __ldg(reinterpret_cast<const float4 *>(p.lo + f));
      const float4 sc = __ldg(reinterpret_cast<const float4 *>(p.scale + f));
      sts_u16(key_lane + (uint32_t)f * ks, quant_key15_lattice_dev(x.x, lo.x, sc.x));
      sts_u16(key_lane + (uint32_t)(f + 1) * ks, quant_key15_lattice_dev(x.y, lo.y, sc.y));
      sts_u16(key_lane + (uint32_t)(f + 2) * ks, quant_key15_lattice_dev(x.z, lo.z, sc.z));
      sts_u16(key_lane + (uint32_t)(f + 3) * ks, quant_key15_lattice_dev(x.w, lo.w, sc.w));
    }
  } else {
    for (int f = 0; f < F; ++f)
      sts_u16(key_lane + (uint32_t)f * ks, quant_key15_lattice_dev(live ? __ldg(rowp + f) : 0.f, __ldg(p.lo + f), __ldg(p.scale + f)));
  }
}

// The value of one tree of a pair, walked again.
__device__ __forceinline__ float deep_exact_value(const DeepParams &p, uint32_t depth, int pair, uint32_t c, uint32_t key_lane, const float *rowp) {
  const unsigned long long off = (2ull * (unsigned long long)pair + c) * p.tree_words;
  return __ldg(p.leaf_plane + off + deep_walk_exact(0, p.node_plane + off, key_lane, false, depth, p.exact_plane + off, rowp));
}

// UD: depth shared by every pair of the forest (0 = mixed, decided per pair at run time).
// LEAF_IDS: the launch records leaf ids instead of predictions.
// WIDE: more features than the byte offset of a 128-byte line in 16 bits reaches.
template <int MAX_THREADS, int UD, bool WIDE, bool LEAF_IDS>
__global__ void __launch_bounds__(MAX_THREADS, 1) tb_walk_deep_kernel(const DeepParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int RW = (blockDim.x >> 5) - 1; // row warps; the last warp is the ring producer
  const int F = p.num_features;
  const int S = p.ring_slots;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw); // [S], then empty[S]
  unsigned char *ring = smem_raw + 128;
  const uint32_t ring_s = smem_u32(ring);
  const uint32_t keys_s = ring_s + (uint32_t)S * p.slot_bytes;
  const uint32_t key_lane = keys_s + (uint32_t)(warp >> 1) * p.key_tile + (uint32_t)lane * 4u + (uint32_t)(warp & 1) * 2u;

  const long long row = ((long long)blockIdx.x * RW + warp) * 32 + lane;
  const bool live = row < p.n_rows;
  const float *rowp = p.rows + (live ? row : 0) * p.ld;
  const int g0 = blockIdx.y * p.pairs_per_chunk;
  const int g1 = min(p.num_pairs, g0 + p.pairs_per_chunk);
  const int P = 2 * (g1 - g0); // pieces of this block: the node planes of every tree
  // (a last block's warps without a row have no part in the walk: one warp of 22 with rows, 300 trees x 60 features, took
  // its block 250 us instead of 212)
  const int live_warps = (int)min((long long)RW, (p.n_rows - (long long)blockIdx.x * RW * 32 + 31) / 32);

  if (tid == 0) {
    for (int i = 0; i < S; ++i) mbar_init(&full[i], 1);
    for (int i = 0; i < S; ++i) mbar_init(&full[S + i], live_warps); // empty: one arrival per row warp
    fence_barrier_init();
  }
  __syncthreads();
  const uint32_t full_s = smem_u32(full), empty_s = full_s + 8u * (uint32_t)S;
  const uint32_t tries = p.wait_tries ? p.wait_tries : kQWaitTries;

  // piece 2k + j of the block: node plane of tree j of pair k.  Pieces are consumed in order,
  // so slots and barrier phases advance by counters (S and RW are run-time values: no
  // division on the hot path).
  auto issue = [&](int piece, int slot) {
    const DevQuantGroup gm = p.pairs[g0 + (piece >> 1)];
    const size_t off = (size_t)gm.elem_off + ((piece & 1) ? gm.slots : 0u);
    uint64_t *bar = &full[slot];
    mbar_expect_tx(bar, gm.slots * 4u);
    bulk_g2s(ring + (size_t)slot * p.slot_bytes, p.node_plane + off, gm.slots * 4u, bar);
  };
  if (warp == RW) {
    // ---- the producer: piece q goes to slot q mod S, once every row warp has released
    // the piece that was there
    bool ok = true;
    int slot = 0, issued = 0;
    uint32_t round = 0;
    for (int piece = 0; piece < P && ok; ++piece) {
      if (round > 0) ok = mbar_wait_all_lanes(empty_s + 8u * (uint32_t)slot, (round - 1u) & 1u, tries);
      if (ok && lane == 0 && !(p.skip_first_copy && piece == 0)) issue(piece, slot);
      issued += ok;
      if (++slot == S) {
        slot = 0;
        ++round;
      }
    }
    if (__syncthreads_or(!ok)) {
      if (lane == 0) set_status(p.status, 4);
      for (int q = max(0, issued - S); q < issued; ++q) // no copy may land after the block is gone
        mbar_wait_all_lanes(full_s + 8u * (uint32_t)(q % S), (uint32_t)(q / S) & 1u, tries);
    }
    return;
  }

  if (warp >= live_warps) {
    __syncthreads_or(0); // (the one at the end)
    return;
  }
  deep_stage_row(p, F, rowp, live, key_lane);
  // (each thread reads back only the keys it wrote: no barrier is needed for the tile)

  // thousands of leaf values per row: a double accumulator keeps the sum within the
  // fp32 rounding of the exact result (one conversion and one add per tree)
  double acc = 0.0;
  // leaf values of the last pair on their way from L2, two words of this thread for each parity of a pair
  [[maybe_unused]] const uint32_t leaf_s = smem_u32(smem_raw) + p.leaf_off + (uint32_t)warp * kDeepLeafBytes + (uint32_t)lane * 4u;
  if constexpr (!LEAF_IDS) {
    sts_f32(leaf_s + 256u, 0.f);
    sts_f32(leaf_s + 384u, 0.f);
  }
  // trees behind a key tie, walked after all others: up to four numbers (plus one) of 16 bits, and, in
  // local memory, the fours before them
  [[maybe_unused]] unsigned long long tied = 0, more_tied[kDeepTied / 4 - 1];
  [[maybe_unused]] int num_more = 0;
  bool ok = true;
  unsigned ties = 0;
  int slot = 0;          // ring slot of the next piece to consume
  uint32_t parity = 0;   // phase of that slot's barrier

  // Takes the next piece: waits for it and returns its shared-memory address.
  auto take = [&](int *slot_out) -> uint32_t {
    const int s = slot;
    if (ok) ok = mbar_wait_all_lanes(full_s + 8u * (uint32_t)s, parity, tries);
    *slot_out = s;
    if (++slot == S) {
      slot = 0;
      parity ^= 1u;
    }
    return ring_s + (uint32_t)s * p.slot_bytes;
  };

  // where pair k's planes start and its depth: computed where all pairs have the same depth, else
  // loaded a pair ahead
  auto pair_of = [&](int k) -> DevQuantGroup {
    if constexpr (UD > 0) return DevQuantGroup{(unsigned long long)(g0 + k) * (2u * p.tree_words), (uint32_t)UD, p.tree_words};
    return p.pairs[min(g0 + k, g1 - 1)];
  };
  DevQuantGroup next = pair_of(0);
  for (int k = 0; k < g1 - g0 && ok; ++k) {
    const DevQuantGroup gm = next;
    next = pair_of(k + 1);
    const uint32_t depth = gm.depth;
    uint32_t j0 = 0, j1 = 0;
    int sl[2];

    const uint32_t n0 = take(&sl[0]), n1 = take(&sl[1]);
    if (ok) {
      bool t0, t1;
      if constexpr (UD > 0)
        deep_walk<UD, WIDE>(n0, n1, key_lane, &j0, &j1, &t0, &t1);
      else
        deep_walk_any<WIDE>(depth, n0, n1, key_lane, &j0, &j1, &t0, &t1);
      // a tied tree waits for the end, where it holds up nobody; beyond kDeepTied it is walked here
      auto resolve = [&](bool tie, int c, uint32_t base, uint32_t &at) {
        if (!tie) return;
        ++ties;
        const uint32_t number = 2u * (uint32_t)k + (uint32_t)c + 1u;
        if (LEAF_IDS || number > 0xffffu || (tied >> 48 && num_more == kDeepTied / 4 - 1)) {
          at = deep_walk_exact(base, nullptr, key_lane, WIDE, depth, p.exact_plane + gm.elem_off + (c ? gm.slots : 0u), rowp);
          return;
        }
        at = kDeepNoLeaf;
        if (tied >> 48) {
          more_tied[num_more++] = tied;
          tied = 0;
        }
        tied = tied << 16 | number;
      };
      resolve(t0, 0, n0, j0);
      resolve(t1, 1, n1, j1);
    }
    // a warp's 32 leaves are scattered over the leaf plane (one sector each), which moves the same
    // bytes as staging the plane would, without taking ring slots
    if (ok) {
      if (!LEAF_IDS) {
        const uint32_t here = leaf_s + ((uint32_t)k & 1u) * 256u, last = leaf_s + ((uint32_t)(k + 1) & 1u) * 256u;
        copies_wait();
        acc += (double)lds_f32(last) + (double)lds_f32(last + 128u);
        copy_word(here, p.leaf_plane + gm.elem_off + (j0 == kDeepNoLeaf ? 0u : j0), j0 != kDeepNoLeaf);
        copy_word(here + 128u, p.leaf_plane + gm.elem_off + gm.slots + (j1 == kDeepNoLeaf ? 0u : j1), j1 != kDeepNoLeaf);
      }
      if (LEAF_IDS && live) {
        const int t0 = p.tree_index[(g0 + k) * 2], t1 = p.tree_index[(g0 + k) * 2 + 1];
        if (t0 >= 0) p.leaf_ids[row * p.num_trees + t0] = p.orig_leaf[gm.elem_off + j0];
        if (t1 >= 0) p.leaf_ids[row * p.num_trees + t1] = p.orig_leaf[gm.elem_off + gm.slots + j1];
      }
    }
    // this warp is done with the pair's two node planes
    __syncwarp();
    if (ok && lane == 0) {
      mbar_arrive(empty_s + 8u * (uint32_t)sl[0]);
      mbar_arrive(empty_s + 8u * (uint32_t)sl[1]);
    }
  }
  // every wait above is bounded: a wait that gave up ends the launch with a status word
  const bool failed = __syncthreads_or(!ok) != 0;
  if (failed) {
    copies_wait();
    if (tid == 0) set_status(p.status, 4);
    return;
  }
  if constexpr (!LEAF_IDS) {
    const uint32_t last = leaf_s + ((uint32_t)(g1 - g0 + 1) & 1u) * 256u;
    copies_wait();
    acc += (double)lds_f32(last) + (double)lds_f32(last + 128u);
    for (; tied || num_more; tied >>= 16) {
      if (!tied) tied = more_tied[--num_more];
      const uint32_t number = (uint32_t)(tied & 0xffff) - 1u;
      const DevQuantGroup gm = p.pairs[g0 + (int)(number >> 1)];
      const unsigned long long off = gm.elem_off + (number & 1u ? gm.slots : 0u);
      acc += (double)__ldg(p.leaf_plane + off + deep_walk_exact(0, p.node_plane + off, key_lane, WIDE, gm.depth, p.exact_plane + off, rowp));
    }
  }
  if (p.tie_count != nullptr && ties) atomicAdd(p.tie_count, (unsigned long long)ties);
  if (LEAF_IDS || !live) return;
  if (p.write_partial)
    p.partial[(long long)blockIdx.y * p.n_rows + row] = (float)acc;
  else
    reinterpret_cast<float *>(p.out)[row] = apply_transform((float)((double)p.initial_value + acc), p.transform);
}

// ---------------------------------------------------------------------------
// Forests whose pairs all have UD levels, predictions: the leaf planes go through the ring too.  Gathered from L2 a leaf
// value costs 23 wavefronts of the shared-memory pipe per 32 rows (32 sectors that arrive one by one), nearly as many as
// the walk itself; from shared memory it is one load of 3.4.  So that a pair's planes fit the ring, the bottom level is a
// plane of its own, needed only at the end, and so are the left and the right leaves (tb_deep_split):
//   A  the UD - 1 upper levels, an in-order tree whose leaf positions are those of
//   B  the nodes of the bottom level and
//   L  two half planes, the leaves to the left and to the right of these nodes.
// A pair takes four ring slots of two planes each: A of both trees, B of both, L of the first, L of the second; five slots
// keep the copy of every piece about a pair ahead of its use.
// 85248 rows x 400 trees of 12 levels over 128 features: 53.3 -> 35.2 wavefronts per 32 rows and tree, pipe 71 -> 50 % busy,
// 252 -> 251 us; 1048576 rows x 2000 trees 15.05 -> 14.52 ms; 100000 rows x 500 trees of 10 levels over 30 features
// 306 -> 285 us.  Where it is not the faster one, and why: deep_staged_pays (tbk_api.cu).  (Both L of a pair are looked for at once: 14.55
// instead of 14.30 ms one after the other; with B 14.62.)  Bound: the chain of a walk, about 100 clocks a level, times too few of them: two trees of 18 row warps
// are what fits.  (Leaf values as plain loads, consumed a pair later: 15.9 ms.)
struct DeepStagedParams : DeepParams {
  const uint32_t *split; // per pair: A0 A1 B0 B1 L0 (left, right) L1 (left, right)
};
constexpr int kDeepStagedMinSlots = 5;

// Re-orders a forest's planes; a thread handles a position of the planes of a tree.
__global__ void tb_deep_split(const uint32_t *node_plane, const float *leaf_plane, uint32_t *split, long long trees, uint32_t depth,
                              uint32_t tree_words, uint32_t half_words) {
  const uint32_t half = 1u << (depth - 1);
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long tree = i >> (depth - 1);
  const uint32_t k = (uint32_t)i & (half - 1);
  if (tree >= trees) return;
  const uint32_t *node = node_plane + tree * tree_words;
  const float *leaf = leaf_plane + tree * tree_words;
  uint32_t *pair = split + (tree >> 1) * 8ll * half_words;
  const uint32_t c = (uint32_t)tree & 1u, at = deep_position(k);
  pair[c * half_words + at] = node[deep_position(2 * k)];
  pair[(2 + c) * half_words + at] = node[deep_position(2 * k + 1)];
  pair[(4 + 2 * c) * half_words + at] = __float_as_uint(leaf[deep_position(2 * k)]);
  pair[(5 + 2 * c) * half_words + at] = __float_as_uint(leaf[deep_position(2 * k + 1)]);
}

template <int MAX_THREADS, int UD> __global__ void __launch_bounds__(MAX_THREADS, 1) tb_walk_deep_staged_kernel(const DeepStagedParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int RW = (blockDim.x >> 5) - 1; // row warps; the last warp is the ring producer
  const int F = p.num_features, S = p.ring_slots;
  constexpr uint32_t H = deep_tree_words(UD - 1) * 4u, SLOT = 2u * H; // bytes of a plane and of a ring slot
  uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw); // [S], then empty[S]
  unsigned char *ring = smem_raw + 128;
  const uint32_t ring_s = smem_u32(ring), full_s = smem_u32(full), empty_s = full_s + 8u * (uint32_t)S;
  const uint32_t key_lane = ring_s + (uint32_t)S * SLOT + (uint32_t)(warp >> 1) * p.key_tile + (uint32_t)lane * 4u + (uint32_t)(warp & 1) * 2u;
  const long long row = ((long long)blockIdx.x * RW + warp) * 32 + lane;
  const bool live = row < p.n_rows;
  const float *rowp = p.rows + (live ? row : 0) * p.ld;
  const int g0 = blockIdx.y * p.pairs_per_chunk, pairs = min(p.num_pairs - g0, p.pairs_per_chunk);
  if (tid == 0) {
    for (int i = 0; i < S; ++i) mbar_init(&full[i], 1);
    for (int i = 0; i < S; ++i) mbar_init(&full[S + i], RW);
    fence_barrier_init();
  }
  __syncthreads();
  const uint32_t tries = p.wait_tries ? p.wait_tries : kQWaitTries;
  bool ok = true;
  int slot = 0;
  if (warp == RW) {
    // ---- the producer: piece q goes to slot q mod S once every row warp has released the one that was there
    uint32_t round = 0;
    int issued = 0;
    for (int piece = 0; piece < 4 * pairs && ok; ++piece) {
      if (round > 0) ok = mbar_wait_all_lanes(empty_s + 8u * (uint32_t)slot, (round - 1u) & 1u, tries);
      if (ok && !(p.skip_first_copy && piece == 0)) {
        if (lane == 0) {
          mbar_expect_tx(&full[slot], SLOT);
          bulk_g2s(ring + (size_t)slot * SLOT, p.split + ((size_t)g0 * 4 + (size_t)piece) * (SLOT / 4), SLOT, &full[slot]);
        }
      }
      issued += ok;
      if (++slot == S) {
        slot = 0;
        ++round;
      }
    }
    if (__syncthreads_or(!ok)) {
      if (lane == 0) set_status(p.status, 4);
      for (int q = max(0, issued - S); q < issued; ++q) // no copy may land after the block is gone
        mbar_wait_all_lanes(full_s + 8u * (uint32_t)(q % S), (uint32_t)(q / S) & 1u, tries);
    }
    return;
  }
  deep_stage_row(p, F, rowp, live, key_lane);

  double acc = 0.0; // (as in tb_walk_deep_kernel)
  unsigned long long tied = 0, more_tied[kDeepTied / 4 - 1];
  int num_more = 0;
  unsigned ties = 0;
  uint32_t parity = 0;
  // the next piece's slot
  auto next_slot = [&](uint32_t *phase) {
    const uint32_t s = (uint32_t)slot;
    *phase = parity;
    if (++slot == S) {
      slot = 0;
      parity ^= 1u;
    }
    return s;
  };
  auto arrived = [&](uint32_t s, uint32_t phase) { // (the warp agrees)
    return __all_sync(0xffffffffu, mbar_wait_all_lanes(full_s + 8u * s, phase, tries)) != 0;
  };
  for (int k = 0; k < pairs; ++k) {
    uint32_t j0, j1, pa, pb, p0, p1;
    bool t0, t1;
    const uint32_t sa = next_slot(&pa), sb = next_slot(&pb), s0 = next_slot(&p0), s1 = next_slot(&p1);
    ok = arrived(sa, pa);
    if (!ok) break;
    deep_walk<UD - 1, false>(ring_s + sa * SLOT, ring_s + sa * SLOT + H, key_lane, &j0, &j1, &t0, &t1);
    __syncwarp();
    if (lane == 0) mbar_arrive(empty_s + 8u * sa);
    ok = arrived(sb, pb);
    if (!ok) break;
    const uint32_t n0 = lds_u32(ring_s + sb * SLOT + 4u * j0), n1 = lds_u32(ring_s + sb * SLOT + H + 4u * j1);
    const uint32_t k0 = lds_u16((n0 >> 16) + key_lane), k1 = lds_u16((n1 >> 16) + key_lane);
    const bool r0 = k0 < (n0 & 0x7fffu), r1 = k1 < (n1 & 0x7fffu);
    t0 |= k0 == (n0 & 0x7fffu);
    t1 |= k1 == (n1 & 0x7fffu);
    __syncwarp();
    if (lane == 0) mbar_arrive(empty_s + 8u * sb);
    // both L: one look at two barriers, which as a rule are complete
    uint32_t here;
    asm volatile("{\n .reg .pred p, q;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n and.pred p, p, q;\n"
                 " vote.sync.all.pred p, p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(here)
                 : "r"(full_s + 8u * s0), "r"(p0), "r"(full_s + 8u * s1), "r"(p1)
                 : "memory");
    if (!here) {
      ok = arrived(s0, p0) && arrived(s1, p1);
      if (!ok) break;
    }
    float v0 = lds_f32(ring_s + s0 * SLOT + 4u * j0 + (r0 ? H : 0u));
    float v1 = lds_f32(ring_s + s1 * SLOT + 4u * j1 + (r1 ? H : 0u));
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(empty_s + 8u * s0);
      mbar_arrive(empty_s + 8u * s1);
    }
    // a tree behind a key tie waits for the end, where it holds up nobody; beyond kDeepTied it is walked here
    auto resolve = [&](bool tie, uint32_t c, float &v) {
      if (!tie) return;
      ++ties;
      const uint32_t number = 2u * (uint32_t)k + c + 1u;
      if (number > 0xffffu || (tied >> 48 && num_more == kDeepTied / 4 - 1)) {
        v = deep_exact_value(p, UD, g0 + k, c, key_lane, rowp);
        return;
      }
      v = 0.f;
      if (tied >> 48) {
        more_tied[num_more++] = tied;
        tied = 0;
      }
      tied = tied << 16 | number;
    };
    resolve(t0, 0, v0);
    resolve(t1, 1, v1);
    acc += (double)v0 + (double)v1;
  }
  // every wait above is bounded: a wait that gave up ends the launch with a status word
  if (__syncthreads_or(!ok)) {
    if (tid == 0) set_status(p.status, 4);
    return;
  }
  for (; tied || num_more; tied >>= 16) {
    if (!tied) tied = more_tied[--num_more];
    const uint32_t number = (uint32_t)(tied & 0xffff) - 1u;
    acc += (double)deep_exact_value(p, UD, g0 + (int)(number >> 1), number & 1u, key_lane, rowp);
  }
  if (p.tie_count != nullptr && ties) atomicAdd(p.tie_count, (unsigned long long)ties);
  if (!live) return;
  if (p.write_partial)
    p.partial[(long long)blockIdx.y * p.n_rows + row] = (float)acc;
  else
    reinterpret_cast<float *>(p.out)[row] = apply_transform((float)((double)p.initial_value + acc), p.transform);
}

} // namespace tb
