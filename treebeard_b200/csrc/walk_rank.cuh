// Walk kernel for rank keys (rank_pack.h): forests of at most 8 levels over rows of at most 64
// features.
//
// LANE = TREE.  A warp owns up to 16 rows of the batch and walks them through the 32 trees of a
// group, one tree per lane, four rows in lock-step.  What that buys over lane = row:
//  * a lane's tree is the same for all its rows, so the nodes of its three topmost levels live in
//    registers and cost no shared-memory load (RankTop);
//  * the keys of one row are read by all lanes at once: 16-bit keys of up to 64 features lie in
//    32 words, so whatever features the 32 trees ask for, the load is one wavefront;
//  * leaf values are added to 16 running sums per lane and meet across lanes once per batch, not
//    once per tree: no table of leaf numbers, no second set of warps, and every sum has only
//    trees / 32 terms;
//  * a warp's work is 4 to 16 rows, not 32: small batches still spread over the GPU.
// Node loads are conflict-free (32 columns = 32 banks).  A level costs a node load, a shift-add to
// the key's address, a key load, a comparison and a predicated add (rank_pack.h on the slot
// numbering); a tree of 8 levels 14.0 shared-memory wavefronts and 44.7 instructions.  Bound:
// the shared-memory pipe, 94 % busy (1048576 rows through 1000 trees of 8 levels).
//
// A block = 20 walker warps, a warp that streams the tree groups (node plane and leaf plane of a
// group = one stage, as many stages as fit) and a warp that fetches the keys of the next batch of
// rows while the current one is walked.  All hand-offs are mbarriers with bounded waits; a
// wait that gives up ends the launch with a status word.  The rows are dealt to the blocks of a
// row (blockIdx.x) evenly in units of 80 (4 per warp), so that all end at the same time; a block
// takes its share in batches of up to 4 units, 16 rows per warp.  blockIdx.y is a chunk of the
// trees: with several chunks a block has one batch, leaves its partial sums in scratch memory, and
// the last block to finish with a batch adds them up in chunk order -- one launch, and the same
// result every time.
//
// The smallest batches are ranked by the walkers themselves (every tree chunk's blocks rank their
// rows again): a launch of its own takes longer than two values per thread.  They also take a
// variant of the kernel (NR = 4) with at most 20 walker warps of four rows each and every loop
// rolled up: the code of such a launch is executed once.
//
// Multiclass: the running sums belong to one class at a time (a class owns consecutive columns);
// when the class changes they are combined across the lanes -- afterwards a lane holds the class
// sum of ONE row -- and the best class so far is updated with the reference's tie rule (ties go
// to the higher class index, src/reduction/LowerReduceOps.cpp:148-189).  Tree chunks are then
// ranges of whole classes.
//
// Reference counterparts: the scalar walk src/mlir/CodeGenStateMachine.cpp:149-243, the row and
// tree caches src/gpu/GPURepresentations.cpp:279-399, :630-715, the cross-thread reduction
// src/reduction/LowerReduceOps.cpp:921-1003.
#pragma once
#include "rank_rows.cuh"
#include "walk_quant.cuh"

#include <type_traits>

namespace tb {

constexpr int kRankInline = 256; // row values that travel with the launch
// Row values that a thread of the walk ranks itself: two, in lock-step.  With more of them the ranking kernel is
// faster, launched ahead of a walk that sets up meanwhile: 64 trees of 8 levels over 28 features, 300 rows, calls
// back to back, 12.3 us with four values inside one after another, 10.3 in two pairs, 8.3 apart; over 10 features
// 8.5 inside and 8.2 apart, but 11.7 against 13.1 for a call by itself.  252 shapes of 30 to 400 trees, 10 to
// 60 features, 100 to 30000 rows, back to back and as single calls: 3228 and 4080 us with all ranked apart, 3214 and
// 4055 with up to two values inside, 3247 and 4077 with up to four.
constexpr int kRankInside = 2;

struct RankWalkParams {
  const uint32_t *node_plane;
  const uint32_t *leaf_plane; // leaf values, or original node ids where leaf ids are recorded
  const DevQuantGroup *groups;
  const int32_t *tree_index;
  const int32_t *class_begin; // multiclass
  const unsigned char *keys;  // [n_rows][S]
  RankRowsParams ranking;     // rows != null: a block ranks the rows of its only batch itself
  long long n_rows;
  float *partial;             // where write_partial asks for raw sums
  float *scratch;             // [chunks][n_rows] partial sums, or (best sum, class) pairs
  void *out;
  int32_t *leaf_ids;
  unsigned int *arrivals;     // per row batch: chunks that are done (zero between launches)
  long long num_trees;
  int32_t num_groups, groups_per_chunk, num_classes, classes_per_chunk;
  int32_t uniform_depth;      // of all groups; 0: they differ
  int32_t quads, tile_bytes;  // tiles of rows (walk_rank_tiles.cuh)
  int32_t write_partial, out_kind, transform;
  float initial_value;
  int32_t stages;
  uint32_t stage_bytes;
  int32_t *status;
  int32_t skip_first_copy; // failure drill
  uint32_t wait_tries;
};
// With the rows themselves, one after another.  (A kilobyte of parameters costs a launch 0.7 us: 64 trees over
// 10 features, 300 device rows, 13.4 us with them and 12.8 without.)
struct RankWalkInlineParams : RankWalkParams {
  float inline_rows[kRankInline];
};

constexpr int kRWWalkers = 20, kRWThreads = 32 * (kRWWalkers + 2);
constexpr int kRWUnitRows = 4 * kRWWalkers, kRWBatchUnits = 4, kRWBatchRows = kRWUnitRows * kRWBatchUnits;
constexpr int kRWBarBytes = 256; // full[8], empty[8], keys_full[2], keys_empty[2]; flag at 192
constexpr int kRWMaxStages = 8;
constexpr int kRankArrivals = 4096;                    // row batches of a launch with several tree chunks
constexpr size_t kRankArrivalBytes = 4 * kRankArrivals;

__host__ __device__ constexpr int rank_walk_smem_bytes(int stride, int stages, uint32_t stage_bytes) {
  return kRWBarBytes + 2 * kRWBatchRows * stride + stages * (int)stage_bytes;
}

template <int IMM> __device__ __forceinline__ uint32_t lds_u32_imm(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(IMM));
  return v;
}
template <int IMM> __device__ __forceinline__ uint32_t lds_u16_imm(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u16 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(IMM));
  return v;
}
// One decision: where key >= threshold rank (the low half of the node word), `off` moves on by IMM.
// WHOLE = false compares the low halves as half-precision numbers (ranks up to kRankHalfMax).
template <bool WHOLE, uint32_t IMM> __device__ __forceinline__ void rank_step(uint32_t &off, uint32_t key, uint32_t node) {
  if constexpr (WHOLE)
    asm volatile("{\n .reg .pred p;\n .reg .b32 t;\n and.b32 t, %2, 0xffff;\n setp.ge.u32 p, %1, t;\n @p add.u32 %0, %0, %3;\n}"
                 : "+r"(off) : "r"(key), "r"(node), "n"(IMM));
  else
    asm volatile("{\n .reg .pred p, q;\n setp.ge.f16x2 p|q, %1, %2;\n @p add.u32 %0, %0, %3;\n}"
                 : "+r"(off) : "r"(key), "r"(node), "n"(IMM));
}
// The nodes of a lane's tree that live in registers: levels 0 to 2.
struct RankTop {
  uint32_t root;   // the root's threshold rank, in both halves where two rows are decided together
  uint32_t ka0;    // address of the root's key of row 0
  uint32_t n1[2];  // level 1
  uint32_t n2[4];  // level 2
};
// What the decision at the root leaves of them: the node of level 1, the two of level 2 that are
// still possible, the offset.
struct RankPath {
  uint32_t off, node, lo2, hi2;
};
#define TBR_ROOT_SELECTS(p, off, node, lo2, hi2)                                                                    \
  " selp.b32 " off ", %11, %10, " p ";\n selp.b32 " node ", %13, %12, " p ";\n"                                    \
  " selp.b32 " lo2 ", %15, %14, " p ";\n selp.b32 " hi2 ", %17, %16, " p ";\n"
#define TBR_ROOT_OPERANDS                                                                                           \
  "r"(t.root), "r"(col), "r"(col + 128u), "r"(t.n1[0]), "r"(t.n1[1]), "r"(t.n2[0]), "r"(t.n2[1]), "r"(t.n2[2]), "r"(t.n2[3])
// Two rows whose keys share a word: one comparison decides both.
__device__ __forceinline__ void rank_root_pair(RankPath &a, RankPath &b, uint32_t keys, const RankTop &t, uint32_t col) {
  asm volatile("{\n .reg .pred p, q;\n setp.ge.f16x2 p|q, %8, %9;\n"
               TBR_ROOT_SELECTS("p", "%0", "%1", "%2", "%3") TBR_ROOT_SELECTS("q", "%4", "%5", "%6", "%7") "}"
               : "=&r"(a.off), "=&r"(a.node), "=&r"(a.lo2), "=&r"(a.hi2), "=&r"(b.off), "=&r"(b.node), "=&r"(b.lo2), "=&r"(b.hi2)
               : "r"(keys), TBR_ROOT_OPERANDS);
}
template <bool WHOLE> __device__ __forceinline__ void rank_root_one(RankPath &a, uint32_t key, const RankTop &t, uint32_t col) {
  const bool right = WHOLE ? key >= (t.root & 0xffffu) : false;
  if constexpr (WHOLE) {
    a.off = right ? col + 128u : col;
    a.node = right ? t.n1[1] : t.n1[0];
    a.lo2 = right ? t.n2[1] : t.n2[0];
    a.hi2 = right ? t.n2[3] : t.n2[2];
  } else {
    [[maybe_unused]] uint32_t x0, x1, x2, x3;
    asm volatile("{\n .reg .pred p, q;\n setp.ge.f16x2 p|q, %8, %9;\n" TBR_ROOT_SELECTS("p", "%0", "%1", "%2", "%3")
                 " mov.b32 %4, 0;\n mov.b32 %5, 0;\n mov.b32 %6, 0;\n mov.b32 %7, 0;\n}"
                 : "=&r"(a.off), "=&r"(a.node), "=&r"(a.lo2), "=&r"(a.hi2), "=r"(x0), "=r"(x1), "=r"(x2), "=r"(x3)
                 : "r"(key), TBR_ROOT_OPERANDS);
  }
}
// The decision on level 1 also picks the node of level 2.
template <bool WHOLE> __device__ __forceinline__ void rank_step1(RankPath &a, uint32_t key) {
  if constexpr (WHOLE)
    asm volatile("{\n .reg .pred p;\n .reg .b32 t;\n and.b32 t, %1, 0xffff;\n setp.ge.u32 p, %2, t;\n @p add.u32 %0, %0, 256;\n"
                 " selp.b32 %1, %4, %3, p;\n}"
                 : "+r"(a.off), "+r"(a.node) : "r"(key), "r"(a.lo2), "r"(a.hi2));
  else
    asm volatile("{\n .reg .pred p, q;\n setp.ge.f16x2 p|q, %2, %1;\n @p add.u32 %0, %0, 256;\n selp.b32 %1, %4, %3, p;\n}"
                 : "+r"(a.off), "+r"(a.node) : "r"(key), "r"(a.lo2), "r"(a.hi2));
}

// Offset of row r's keys from row 0's: rows in pairs share the words of a 128-byte line.
template <int S> __host__ __device__ constexpr int rank_row_offset(int r) { return S == 64 ? (r >> 1) * 128 + (r & 1) * 2 : r * S; }

// Walks rows ROW0 .. ROW0 + 3 (row 0's keys at kb) through this lane's tree of depth D, whose
// column starts at `col` (node plane; leaf plane 2^D * 128 bytes on); v = leaf words.
template <int D, int S, int ROW0, bool WHOLE>
__device__ __forceinline__ void rank_walk4(uint32_t (&v)[4], uint32_t col, uint32_t kb, const RankTop &t) {
  RankPath a[4];
  uint32_t key[4];
#define TBR_ROWS(stmt)                                                                                              \
  { { constexpr int q = 0; stmt; } { constexpr int q = 1; stmt; } { constexpr int q = 2; stmt; } { constexpr int q = 3; stmt; } }
  if constexpr (S == 64 && !WHOLE) {
    key[0] = lds_u32_imm<rank_row_offset<S>(ROW0)>(t.ka0);
    key[2] = lds_u32_imm<rank_row_offset<S>(ROW0 + 2)>(t.ka0);
    rank_root_pair(a[0], a[1], key[0], t, col);
    rank_root_pair(a[2], a[3], key[2], t, col);
  } else {
    TBR_ROWS(key[q] = lds_u16_imm<rank_row_offset<S>(ROW0 + q)>(t.ka0))
    TBR_ROWS(rank_root_one<WHOLE>(a[q], key[q], t, col))
  }
#define TBR_DECIDE(level)                                                                                           \
  if constexpr (D > level) {                                                                                        \
    if constexpr (level > 2) TBR_ROWS(a[q].node = lds_u32_imm<128 * ((1 << level) - 1)>(a[q].off))                  \
    TBR_ROWS(key[q] = lds_u16_imm<rank_row_offset<S>(ROW0 + q)>((a[q].node >> 16) + kb))                            \
    if constexpr (level == 1) TBR_ROWS(rank_step1<WHOLE>(a[q], key[q]))                                             \
    else TBR_ROWS((rank_step<WHOLE, (128u << level)>(a[q].off, key[q], a[q].node)))                                 \
  }
  TBR_DECIDE(1) TBR_DECIDE(2) TBR_DECIDE(3) TBR_DECIDE(4) TBR_DECIDE(5) TBR_DECIDE(6) TBR_DECIDE(7)
  TBR_ROWS(v[q] = lds_u32_imm<(128 << D)>(a[q].off))
#undef TBR_DECIDE
#undef TBR_ROWS
}

// The same walk with the levels rolled up; the offset moves from level to level with the loop.
template <int S> __device__ __forceinline__ void rank_walk4_rolled(uint32_t (&v)[4], uint32_t depth, uint32_t col, uint32_t kb) {
  uint32_t off[4] = {col, col, col, col}, step = 128;
#pragma unroll 1
  for (uint32_t d = 0; d < depth; ++d, step *= 2) {
    uint32_t node[4], key[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) node[q] = lds_u32(off[q]);
    key[0] = lds_u16_imm<rank_row_offset<S>(0)>((node[0] >> 16) + kb);
    key[1] = lds_u16_imm<rank_row_offset<S>(1)>((node[1] >> 16) + kb);
    key[2] = lds_u16_imm<rank_row_offset<S>(2)>((node[2] >> 16) + kb);
    key[3] = lds_u16_imm<rank_row_offset<S>(3)>((node[3] >> 16) + kb);
#pragma unroll
    for (int q = 0; q < 4; ++q) off[q] += step + (key[q] >= (node[q] & 0xffffu) ? step : 0u);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = lds_u32_imm<128>(off[q]); // past the node plane's last, unused slot
}

// Adds up v over the 32 lanes for every of NR rows: afterwards lane l holds the sum of row
// l * NR / 32 (32 / NR neighbouring lanes hold the same row).
template <int NR> __device__ __forceinline__ float rank_reduce_rows(float (&v)[NR], int lane) {
  int bit = 16;
#pragma unroll
  for (int half = NR / 2; half >= 1; half /= 2, bit /= 2) {
    const bool up = lane & bit;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = up ? v[i + half] : v[i], give = up ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
  }
  float s = v[0];
  for (; bit >= 1; bit /= 2) s += __shfl_xor_sync(0xffffffffu, s, bit);
  return s;
}
// One group of depth D for the warp's rows, four times `fours` of them; use(c, v) takes the leaf
// words of rows 4c .. 4c+3.
template <int D, int S, bool WHOLE, typename Use>
__device__ __forceinline__ void rank_walk_rows(int fours, uint32_t col, uint32_t kb, Use use) {
  RankTop t{};
  uint32_t v[4];
  t.root = lds_u32_imm<0>(col);
  t.ka0 = (t.root >> 16) + kb;
  if constexpr (S == 64 && !WHOLE) t.root = __byte_perm(t.root, t.root, 0x1010);
  if constexpr (D > 1) {
    t.n1[0] = lds_u32_imm<128>(col);
    t.n1[1] = lds_u32_imm<256>(col);
  }
  if constexpr (D > 2) {
    t.n2[0] = lds_u32_imm<384>(col);
    t.n2[1] = lds_u32_imm<512>(col);
    t.n2[2] = lds_u32_imm<640>(col);
    t.n2[3] = lds_u32_imm<768>(col);
  }
  rank_walk4<D, S, 0, WHOLE>(v, col, kb, t);
  use(0, v);
  if (fours == 1) return;
  rank_walk4<D, S, 4, WHOLE>(v, col, kb, t);
  use(1, v);
  if (fours == 2) return;
  rank_walk4<D, S, 8, WHOLE>(v, col, kb, t);
  use(2, v);
  if (fours == 3) return;
  rank_walk4<D, S, 12, WHOLE>(v, col, kb, t);
  use(3, v);
}
template <int S, int NR, bool WHOLE, typename Use>
__device__ __forceinline__ void rank_walk_group(uint32_t depth, int fours, uint32_t col, uint32_t kb, Use use) {
  if constexpr (NR == 4) {
    uint32_t v[4];
    rank_walk4_rolled<S>(v, depth, col, kb);
    return use(0, v);
  }
  switch (depth) {
  case 1: return rank_walk_rows<1, S, WHOLE>(fours, col, kb, use);
  case 2: return rank_walk_rows<2, S, WHOLE>(fours, col, kb, use);
  case 3: return rank_walk_rows<3, S, WHOLE>(fours, col, kb, use);
  case 4: return rank_walk_rows<4, S, WHOLE>(fours, col, kb, use);
  case 5: return rank_walk_rows<5, S, WHOLE>(fours, col, kb, use);
  case 6: return rank_walk_rows<6, S, WHOLE>(fours, col, kb, use);
  case 7: return rank_walk_rows<7, S, WHOLE>(fours, col, kb, use);
  default: return rank_walk_rows<8, S, WHOLE>(fours, col, kb, use);
  }
}

// The chunks' partial sums of a row, in chunk order.  (Many loads at a time: their round trip is
// what this costs.)
__device__ __forceinline__ float rank_sum_chunks(const RankWalkParams &p, long long row) {
  float s = 0.f;
  for (int y = 0; y < (int)gridDim.y; y += 16) {
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = y + i < (int)gridDim.y ? __ldcg(p.scratch + (long long)(y + i) * p.n_rows + row) : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) s += v[i];
  }
  return s;
}

enum RankMode { kRankSums, kRankClasses, kRankLeafIds };

// S: bytes per row of keys; NR: most rows per warp (16, or 4 where a block has one unit of rows;
// that variant compares whole numbers whatever the ranks).
// INLINE: the rows travel with the launch.
template <int S, int NR, bool WHOLE, int MODE, bool INLINE>
__global__ void __launch_bounds__(kRWThreads, 1)
    tb_walk_rank_kernel(const __grid_constant__ std::conditional_t<INLINE, RankWalkInlineParams, RankWalkParams> p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0); // uniform by construction
  const int NW = NR == 4 ? (int)(blockDim.x >> 5) - 2 : kRWWalkers; // walker warps
  const int UR = 4 * NW;                                           // rows per unit
  const uint32_t bars_s = smem_u32(smem_raw);
  const uint32_t full_s = bars_s, empty_s = bars_s + 64u, keys_full_s = bars_s + 128u, keys_empty_s = bars_s + 144u;
  volatile uint32_t *last_flag = reinterpret_cast<volatile uint32_t *>(smem_raw + 192);
  unsigned char *keys = smem_raw + kRWBarBytes;           // two batches of keys
  unsigned char *ring = keys + 2 * kRWBatchRows * S;
  // this block's units of rows, in batches of up to four
  const long long units = (p.n_rows + UR - 1) / UR;
  const int unit0 = (int)(units * blockIdx.x / gridDim.x), unit1 = (int)(units * (blockIdx.x + 1) / gridDim.x);
  const int my_batches = (unit1 - unit0 + kRWBatchUnits - 1) / kRWBatchUnits;
  // this chunk's groups; with classes: those that hold the columns of classes c0 .. c1 - 1
  int g0 = (int)blockIdx.y * p.groups_per_chunk, g1 = min(p.num_groups, g0 + p.groups_per_chunk);
  [[maybe_unused]] int c0 = 0, c1 = 0, col0 = 0;
  if constexpr (MODE == kRankClasses) {
    c0 = (int)blockIdx.y * p.classes_per_chunk;
    c1 = min(p.num_classes, c0 + p.classes_per_chunk);
    col0 = p.class_begin[c0];
    const int col1 = p.class_begin[c1];
    g0 = col0 / 32;
    g1 = col1 > col0 ? (col1 + 31) / 32 : g0;
  }
  const int NG = g1 - g0;

  if (tid == 0) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw);
    for (int i = 0; i < kRWMaxStages; ++i) mbar_init(bars + i, 1);              // full: the copies' bytes
    for (int i = 0; i < kRWMaxStages; ++i) mbar_init(bars + 8 + i, NW); // empty: one arrival per walker warp
    for (int i = 0; i < 2; ++i) mbar_init(bars + 16 + i, 1);                    // keys_full
    for (int i = 0; i < 2; ++i) mbar_init(bars + 18 + i, NW);           // keys_empty
    fence_barrier_init();
  }
  __syncthreads();

  bool ok = true;
  [[maybe_unused]] uint32_t issued = 0; // copies (of a stage, of a batch's keys) this producer warp has started
  const uint32_t tries = p.wait_tries ? p.wait_tries : kQWaitTries;
  // (the warp agrees on the outcome: shuffles follow)
  auto wait = [tries](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait_all_lanes(bar, parity, tries)) != 0; };

  if (warp == NW) {
    // ---- tree groups, batch after batch
    const uint64_t keep = l2_policy_keep();
    int slot = 0;
    uint32_t round = 0;
    for (int it = 0; it < my_batches && ok; ++it)
      for (int k = 0; k < NG && ok; ++k) {
        if (round > 0) ok = wait(empty_s + 8u * (uint32_t)slot, (round - 1u) & 1u);
        issued += ok;
        if (ok && lane == 0 && !(p.skip_first_copy && it == 0 && k == 0)) {
          const uint32_t d = p.uniform_depth;
          const unsigned long long elem = d ? (unsigned long long)(g0 + k) << (d + 5) : p.groups[g0 + k].elem_off;
          const uint32_t bytes = 128u << (d ? d : p.groups[g0 + k].depth);
          unsigned char *dst = ring + (size_t)slot * p.stage_bytes;
          uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw) + slot;
          mbar_expect_tx(bar, 2u * bytes);
          bulk_g2s_hint(dst, p.node_plane + elem, bytes, bar, keep);
          bulk_g2s_hint(dst + bytes, p.leaf_plane + elem, bytes, bar, keep);
        }
        if (++slot == p.stages) {
          slot = 0;
          ++round;
        }
      }
  } else if (warp == NW + 1) {
    // ---- the batches' keys, one batch ahead of the walk; the kernel that ranks the rows may
    // still be running when this one starts
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint64_t stream = l2_policy_stream();
    for (int it = 0; it < my_batches && ok && !p.ranking.rows; ++it) {
      const uint32_t buf = (uint32_t)it & 1u;
      if (it >= 2) ok = wait(keys_empty_s + 8u * buf, (uint32_t)((it >> 1) - 1) & 1u);
      issued += ok;
      if (ok && lane == 0) {
        const int u = unit0 + it * kRWBatchUnits;
        const long long row0 = (long long)u * UR, end = (long long)min(unit1, u + kRWBatchUnits) * UR;
        const uint32_t bytes = ((uint32_t)(min(end, p.n_rows) - row0) + 1u & ~1u) * (uint32_t)S; // (rows may lie in pairs)
        uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw) + 16 + buf;
        mbar_expect_tx(bar, bytes);
        bulk_g2s_hint(keys + (size_t)buf * kRWBatchRows * S, p.keys + row0 * S, bytes, bar, stream);
      }
    }
  } else {
    // ---- the walkers
    const bool elected = lane == 0;
    const uint32_t ring_col = smem_u32(ring) + (uint32_t)lane * 4u;
    int slot = 0;
    uint32_t parity = 0;
    for (int it = 0; it < my_batches && ok; ++it) {
      const int fours = min(unit1 - unit0 - it * kRWBatchUnits, kRWBatchUnits); // rows per warp / 4
      const long long row0 = (long long)(unit0 + it * kRWBatchUnits) * UR + warp * fours * 4;
      const long long row = row0 + lane * NR / 32; // the row whose sum this lane ends up with
      const bool live = (lane & (32 / NR - 1)) == 0 && lane * NR / 32 < 4 * fours && row < p.n_rows;
      if (p.ranking.rows) {
        const RankRowsParams &r = p.ranking;
        const int F = r.num_features;
        const uint32_t values = (uint32_t)(min((long long)unit1 * UR, p.n_rows) - (long long)unit0 * UR) * (uint32_t)F;
        unsigned looked_up = 0;
        rank_values<kRankInside>(r, (uint32_t)tid, 32u * NW, values, looked_up,
                       [&](uint32_t q, uint32_t f) {
                         if constexpr (INLINE) return p.inline_rows[((uint32_t)(unit0 * UR) + q) * (uint32_t)F + f];
                         else return __ldg(r.rows + ((long long)unit0 * UR + q) * r.ld + f);
                       },
                       [&](uint32_t q, uint32_t f, uint32_t rank) {
                         const uint32_t at = S == 64 ? (q >> 1) * 128u + 4u * f + (q & 1u) * 2u : q * S + 2u * f;
                         sts_u16(smem_u32(keys) + at, rank);
                       });
        if (blockIdx.y == 0) count_searched(r.searched, values / (uint32_t)F, r.used, looked_up, warp == 0);
        asm volatile("bar.sync 1, %0;" ::"r"(32 * NW) : "memory");
      } else {
        ok = wait(keys_full_s + 8u * ((uint32_t)it & 1u), (uint32_t)(it >> 1) & 1u);
        if (!ok) break;
      }
      const uint32_t kb = smem_u32(keys) + ((uint32_t)it & 1u) * (uint32_t)(kRWBatchRows * S) + (uint32_t)(warp * fours * 4 * S);
      float acc[NR];
#pragma unroll
      for (int i = 0; i < NR; ++i) acc[i] = 0.f;
      [[maybe_unused]] int cls = c0, lo = col0 & 31, best_class = c0;
      [[maybe_unused]] float sum = 0.f, best = -INFINITY;
      // class `cls` is complete, its sum for this lane's row in `sum`
      [[maybe_unused]] auto finish = [&]() {
        if (p.write_partial) {
          if (live) p.partial[row * p.num_classes + cls] = sum;
        }
        if (sum >= best) {
          best = sum;
          best_class = cls;
        }
        sum = 0.f;
        ++cls;
      };
      uint32_t next_depth = p.uniform_depth ? (uint32_t)p.uniform_depth : NG > 0 ? p.groups[g0].depth : 0u;
      for (int k = 0; k < NG; ++k) {
        const uint32_t depth = next_depth;
        if (!p.uniform_depth) next_depth = p.groups[min(g0 + k + 1, g1 - 1)].depth;
        ok = wait(full_s + 8u * (uint32_t)slot, parity);
        if (!ok) break;
        const uint32_t col = ring_col + (uint32_t)slot * p.stage_bytes;
        if constexpr (MODE == kRankLeafIds) {
          const int t = p.tree_index[(g0 + k) * 32 + lane];
          int32_t *dst = p.leaf_ids + row0 * p.num_trees + t;
          const int rows = (int)min((long long)NR, p.n_rows - row0);
          rank_walk_group<S, NR, WHOLE>(depth, fours, col, kb, [&](int c, const uint32_t(&v)[4]) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (t >= 0 && 4 * c + q < rows) dst[(4 * c + q) * p.num_trees] = (int32_t)v[q];
          });
        } else {
          auto add = [&](int c, const uint32_t(&v)[4]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[4 * c + q] += __uint_as_float(v[q]);
          };
          if constexpr (MODE == kRankClasses) {
            int next = p.class_begin[cls + 1] - (g0 + k) * 32; // first column of the next class
            auto combine = [&](float(&v)[NR]) { sum += rank_reduce_rows<NR>(v, lane); };
            if (NR > 4 && lo == 0 && next >= 32) { // one class
              rank_walk_group<S, NR, WHOLE>(depth, fours, col, kb, add);
              if (next == 32) {
                combine(acc);
                finish();
#pragma unroll
                for (int i = 0; i < NR; ++i) acc[i] = 0.f;
              }
            } else if (NR > 4 && lo == 0 && cls + 1 < c1 && p.class_begin[cls + 2] - (g0 + k) * 32 > 32) {
              // two classes: this one's columns complete its sums, the others start the next one's
              float other[NR];
#pragma unroll
              for (int i = 0; i < NR; ++i) other[i] = 0.f;
              rank_walk_group<S, NR, WHOLE>(depth, fours, col, kb, [&](int c, const uint32_t(&v)[4]) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  acc[4 * c + q] += lane < next ? __uint_as_float(v[q]) : 0.f;
                  other[4 * c + q] = lane < next ? 0.f : __uint_as_float(v[q]);
                }
              });
              combine(acc);
              finish();
#pragma unroll
              for (int i = 0; i < NR; ++i) acc[i] = other[i];
            } else { // several, or a chunk that starts or ends inside the group
              if (lo == 0) combine(acc);
#pragma unroll
              for (int i = 0; i < NR; ++i) acc[i] = 0.f;
              rank_walk_group<S, NR, WHOLE>(depth, fours, col, kb, add);
              while (cls < c1 && next <= 32) { // classes that end in this group
                float part[NR];
#pragma unroll
                for (int i = 0; i < NR; ++i) part[i] = lane >= lo && lane < next ? acc[i] : 0.f;
                combine(part);
                finish();
                lo = next;
                if (cls < c1) next = p.class_begin[cls + 1] - (g0 + k) * 32;
              }
#pragma unroll
              for (int i = 0; i < NR; ++i) acc[i] = lane >= lo ? acc[i] : 0.f;
              lo = 0;
            }
          } else {
            rank_walk_group<S, NR, WHOLE>(depth, fours, col, kb, add);
          }
        }
        __syncwarp();
        if (elected) mbar_arrive(empty_s + 8u * (uint32_t)slot);
        if (++slot == p.stages) {
          slot = 0;
          parity ^= 1u;
        }
      }
      if (!ok) break;
      if (elected) mbar_arrive(keys_empty_s + 8u * ((uint32_t)it & 1u));
      // ---- the batch's results
      if constexpr (MODE == kRankSums) {
        const float s = rank_reduce_rows<NR>(acc, lane);
        if (live) {
          if (gridDim.y > 1) p.scratch[(long long)blockIdx.y * p.n_rows + row] = s;
          else if (p.write_partial) p.partial[row] = s;
          else reinterpret_cast<float *>(p.out)[row] = apply_transform(p.initial_value + s, p.transform);
        }
      } else if constexpr (MODE == kRankClasses) {
        while (cls < c1) finish(); // classes without trees
        if (live && !p.write_partial) {
          if (gridDim.y > 1)
            reinterpret_cast<float2 *>(p.scratch)[(long long)blockIdx.y * p.n_rows + row] = make_float2(best, __int_as_float(best_class));
          else if (p.out_kind == 1) reinterpret_cast<int8_t *>(p.out)[row] = (int8_t)best_class;
          else reinterpret_cast<float *>(p.out)[row] = (float)best_class;
        }
      }
    }
  }
  // every wait above is bounded: a wait that gave up ends the launch with a status word
  const bool chunked = gridDim.y > 1 && MODE != kRankLeafIds && !(MODE == kRankClasses && p.write_partial);
  if (chunked) __threadfence();
  if (__syncthreads_or(!ok)) {
    if (tid == 0) set_status(p.status, 4);
    if (warp >= NW) { // no copy may land after the block is gone
      const uint32_t bars = warp == NW ? full_s : keys_full_s, n = warp == NW ? (uint32_t)p.stages : 2u;
      for (uint32_t s = 0; s < min(n, issued); ++s) wait(bars + 8u * s, ((issued - 1u - s) / n) & 1u);
    }
  }
  if (!chunked) return;
  // ---- tree chunks: the last block to finish with this row batch combines them
  if (tid == 0) {
    const bool last = atomicAdd(p.arrivals + blockIdx.x, 1u) + 1u == gridDim.y;
    if (last) p.arrivals[blockIdx.x] = 0; // for the next launch
    *last_flag = last;
  }
  __syncthreads();
  if (!*last_flag) return;
  __threadfence();
  const long long row = (long long)unit0 * UR + tid;
  if (row >= min((long long)unit1 * UR, p.n_rows)) return;
  if constexpr (MODE == kRankClasses) {
    float best = -INFINITY;
    int best_class = 0;
    for (int y = 0; y < (int)gridDim.y; y += 8) {
      float2 b[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        b[i] = y + i < (int)gridDim.y ? __ldcg(reinterpret_cast<const float2 *>(p.scratch) + (long long)(y + i) * p.n_rows + row)
                                      : make_float2(__int_as_float(0x7fffffff), 0.f); // (NaN wins nothing)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (b[i].x >= best) { // (classes rise with the chunks: a later one wins ties)
          best = b[i].x;
          best_class = __float_as_int(b[i].y);
        }
    }
    if (p.out_kind == 1) reinterpret_cast<int8_t *>(p.out)[row] = (int8_t)best_class;
    else reinterpret_cast<float *>(p.out)[row] = (float)best_class;
  } else {
    const float s = rank_sum_chunks(p, row);
    if (p.write_partial) p.partial[row] = s;
    else reinterpret_cast<float *>(p.out)[row] = apply_transform(p.initial_value + s, p.transform);
  }
}

} // namespace tb
