// Tree-walk kernels for sm_100a.
//
// Work decomposition (what the reference expresses as a schedule over the (row, tree)
// iteration space, src/mlir/GPUAutoSchedule.cpp:355-403):
//   grid.x  -> row tiles of (row_warps * 32 * RPL) rows
//   grid.y  -> tree chunks (ranges of 16-tree groups); partial sums of the chunks are
//              combined by a second, atomic-free pass
//   block   -> row_warps * tree_threads warps.  A warp owns 32*RPL rows (lane = row,
//              RPL rows per lane walked in lock-step for instruction-level
//              parallelism); the tree_threads warps that share a row tile split the 16
//              columns of every group between them.
//
// The walk (reference: src/mlir/CodeGenStateMachine.cpp:149-243 scalar step,
// :284-507 tile step with look-up table, src/mlir/WalkDecisionTreeLoweringPass.cpp:24-53
// fixed-depth walk of padded trees) is branch-free: every tree of a group is walked
// for exactly the group's depth; leaves route back to themselves through the sentinel
// feature (see pack.h).  At shift s lane j walks column (j + s) mod 16, so the 32
// lanes of a warp always address 16 distinct tile columns (bank-conflict free in the
// slot-major interleaved layout) and, in the transposed row tile xs[feature][row],
// 32 distinct banks.
//
// Tree groups are staged into shared memory with cp.async.bulk (the TMA unit's
// untiled bulk copy) into a ring of two stages, or one, guarded by mbarriers; feature rows are
// transposed on their way into shared memory (large batches: stage_pieces).  The reference's
// counterparts are the cooperative row cache (src/gpu/GPURepresentations.cpp:279-399)
// and tree cache (:630-715).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace tb {

struct DevGroupMeta {
  unsigned long long byte_off;
  uint32_t slots;
  uint32_t depth;
};

struct WalkParams {
  const uint8_t *blob;
  const DevGroupMeta *groups;
  const int16_t *tree_class;
  const int32_t *tree_index;
  const int32_t *orig_node;
  const unsigned long long *orig_off;
  const int8_t *lut;
  int32_t lut_bytes;
  const float *rows;
  long long n_rows;
  long long ld;
  float *partial;      // [chunks][n_rows][W]; used when write_partial != 0
  void *out;
  int32_t out_kind;
  int32_t write_partial;
  int32_t *leaf_ids;   // [n_rows][num_trees] or null
  long long num_trees;
  int32_t num_groups;
  int32_t groups_per_chunk;
  int32_t num_features;
  int32_t num_classes;
  int32_t transform;
  float initial_value;
  int32_t row_warps;
  int32_t tree_threads;
  uint32_t stage_bytes; // capacity of one stage (0 when not staged)
  int32_t stages;       // 1 or 2: groups that fit only once are copied and walked by turns
  int32_t vec4_ok;      // rows can be read with 16-byte loads
  int32_t class_regs;   // multiclass: class sums in registers, arg-max decided on the fly
  int32_t *status;      // device status word, 0 = ok
  uint32_t wait_limit;  // polls before a wait on a stage gives up (0 = kWaitLimit)
  int32_t skip_first_copy; // failure drill: the first stage's copy is never issued, so its wait expires
};

constexpr int kCols = 16;
constexpr uint32_t kWaitLimit = 1u << 22;

// --------------------------------------------------------------------------
// mbarrier / bulk-copy primitives

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
               " selp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok)
               : "r"(smem_u32(bar)), "r"(parity)
               : "memory");
  return ok != 0;
}
// Bounded wait: gives up after kWaitLimit polls instead of spinning for ever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, uint32_t limit = kWaitLimit) {
  for (uint32_t it = 0; it < limit; ++it) {
    if (mbar_test(bar, parity)) return true;
    if (it > 64) __nanosleep(64);
  }
  return false;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// The status word lies in mapped host memory: the host reads it after a synchronisation it needs
// anyway, without a copy.
__device__ __forceinline__ void set_status(int32_t *status, int32_t value) {
  *reinterpret_cast<volatile int32_t *>(status) = value;
  __threadfence_system();
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// A wait of the block gave up; called by all threads: sets the status, and no bulk copy may land after the block is gone.
// Thread i waits for the copy that barrier i, of the `bars` ones at the start of shared memory, may expect.  Which of them
// do is not known here, so that nothing has to be kept for it on the way: a barrier that does not change its phase in a
// millisecond had none.
static __device__ __noinline__ void give_up(int32_t *status, uint32_t bars) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  if (threadIdx.x == 0) set_status(status, 4);
  if (threadIdx.x >= bars) return;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw) + threadIdx.x;
  mbar_wait_bounded(bar, mbar_test(bar, 0) ? 1 : 0, 16384);
}

// --------------------------------------------------------------------------
// tile decode: loads the tile at (slot n, column col) and returns the next slot.

template <bool SMEM> __device__ __forceinline__ uint2 ld2(const void *p) {
  if (SMEM) return *reinterpret_cast<const uint2 *>(p);
  return __ldg(reinterpret_cast<const uint2 *>(p));
}
template <bool SMEM> __device__ __forceinline__ uint4 ld4(const void *p) {
  if (SMEM) return *reinterpret_cast<const uint4 *>(p);
  return __ldg(reinterpret_cast<const uint4 *>(p));
}

struct RowAccess {
  const float *xs;      // cached: transposed tile base (+ lane offset applied)
  const float *grow;    // uncached: row base in global memory
  int32_t num_features;
};

// RT = floats between consecutive features of the transposed row tile.
template <bool CACHED, int RT> __device__ __forceinline__ float feature(const RowAccess &ra, uint32_t f) {
  if (CACHED) return ra.xs[f * RT];
  return f == (uint32_t)ra.num_features ? __int_as_float(0xff800000) : __ldg(ra.grow + f);
}

// REP: 0 sparse, 1 array, 2 reorg.  Walks NC columns in lock-step (their loads are independent, so
// that many are in flight per lane); returns the leaf values after `depth` steps and the final slots.
template <int REP, int TS, bool SMEM, bool CACHED, int RT, int NC>
__device__ __forceinline__ void walk_columns(const uint8_t *gbase, uint32_t slots, uint32_t depth, const uint32_t (&col)[NC],
                                             const RowAccess &ra, const int8_t *lut, uint32_t (&n)[NC], float (&v)[NC]) {
#define TBW_ALL _Pragma("unroll") for (int c = 0; c < NC; ++c)
  TBW_ALL n[c] = 0;
  if (REP == 2) {
    const float *thr = reinterpret_cast<const float *>(gbase);
    const uint16_t *feat = reinterpret_cast<const uint16_t *>(gbase + (size_t)slots * kCols * 4);
    for (uint32_t d = 0; d < depth; ++d) {
      float t[NC], x[NC];
      uint32_t f[NC];
      TBW_ALL {
        const uint32_t i = n[c] * kCols + col[c];
        t[c] = SMEM ? thr[i] : __ldg(thr + i);
        f[c] = SMEM ? feat[i] : __ldg(feat + i);
      }
      TBW_ALL x[c] = feature<CACHED, RT>(ra, f[c]);
      TBW_ALL n[c] = 2 * n[c] + 1 + !(x[c] < t[c]);
    }
    TBW_ALL {
      const uint32_t i = n[c] * kCols + col[c];
      v[c] = SMEM ? thr[i] : __ldg(thr + i);
    }
    return;
  }
  constexpr int TB = TS == 1 ? 8 : TS == 2 ? 16 : TS == 3 ? 24 : 32;
  for (uint32_t d = 0; d < depth; ++d) {
    uint32_t k[NC], child[NC];
    if (TS == 1) {
      uint2 t[NC];
      float x[NC];
      TBW_ALL t[c] = ld2<SMEM>(gbase + (size_t)(n[c] * kCols + col[c]) * TB);
      TBW_ALL x[c] = feature<CACHED, RT>(ra, t[c].y & 0xffffu);
      TBW_ALL {
        child[c] = t[c].y >> 16;
        k[c] = !(x[c] < __uint_as_float(t[c].x));
      }
    } else {
      float thr[NC][TS];
      uint32_t f[NC][TS], shape[NC], bits[NC];
      TBW_ALL {
        const uint8_t *tp = gbase + (size_t)(n[c] * kCols + col[c]) * TB;
        if (TS == 2) {
          const uint4 t = ld4<SMEM>(tp);
          thr[c][0] = __uint_as_float(t.x); thr[c][1] = __uint_as_float(t.y);
          f[c][0] = t.z & 0xffffu; f[c][1] = t.z >> 16;
          shape[c] = t.w & 0xffffu; child[c] = t.w >> 16;
        } else if (TS == 3) {
          const uint2 a = ld2<SMEM>(tp), b = ld2<SMEM>(tp + 8), e = ld2<SMEM>(tp + 16);
          thr[c][0] = __uint_as_float(a.x); thr[c][1] = __uint_as_float(a.y); thr[c][2] = __uint_as_float(b.x);
          f[c][0] = b.y & 0xffffu; f[c][1] = b.y >> 16; f[c][2] = e.x & 0xffffu;
          shape[c] = e.x >> 16; child[c] = e.y & 0xffffu;
        } else {
          const uint4 a = ld4<SMEM>(tp), b = ld4<SMEM>(tp + 16);
          thr[c][0] = __uint_as_float(a.x); thr[c][1] = __uint_as_float(a.y);
          thr[c][2] = __uint_as_float(a.z); thr[c][3] = __uint_as_float(a.w);
          f[c][0] = b.x & 0xffffu; f[c][1] = b.x >> 16; f[c][2] = b.y & 0xffffu; f[c][3] = b.y >> 16;
          shape[c] = b.z & 0xffffu; child[c] = b.z >> 16;
        }
      }
      TBW_ALL {
        bits[c] = 0;
#pragma unroll
        for (int i = 0; i < TS; ++i) bits[c] |= (uint32_t)(feature<CACHED, RT>(ra, f[c][i]) < thr[c][i]) << i;
      }
      TBW_ALL k[c] = (uint32_t)lut[(shape[c] << TS) + bits[c]];
    }
    TBW_ALL n[c] = REP == 0 ? child[c] + k[c] : n[c] * (TS + 1) + 1 + k[c];
  }
  TBW_ALL {
    const uint8_t *tp = gbase + (size_t)(n[c] * kCols + col[c]) * TB;
    v[c] = SMEM ? *reinterpret_cast<const float *>(tp) : __ldg(reinterpret_cast<const float *>(tp));
  }
#undef TBW_ALL
}

__device__ __forceinline__ float apply_transform(float v, int transform) {
  return transform == 1 ? 1.0f / (1.0f + expf(-v)) : v;
}

// argmax with the reference generated code's tie rule
// (src/reduction/LowerReduceOps.cpp:148-189): "if (max > v) keep else take".
template <typename Load> __device__ __forceinline__ int argmax_last(int C, Load load) {
  float best = __int_as_float(0xff800000);
  int arg = 0;
  for (int c = 0; c < C; ++c) {
    const float v = load(c);
    if (!(best > v)) { best = v; arg = c; }
  }
  return arg;
}

// Stages the features of 32 rows: pieces of 8, numbers tt, tt + TT, .. of them; a rest is the window of the last 8, staged
// before the piece that it overlaps.  A request reads 32-byte stretches of four rows: with a row per lane every 4 bytes cost
// a 32-byte sector (30 sectors a request, and a chunk of 5 groups of trees spent a quarter of its time on them at 54 features).
// A piece is turned around in the lines that it will take: the values of rows 4k .. 4k+3 lie in line k, in an order that
// meets 32 banks both ways.
// lines: the rows' place in the first line, as a shared-memory address; the next line is NEXT floats on.
template <int NEXT>
__device__ __forceinline__ void stage_pieces(const float *src, long long ld, int rows, int F, uint32_t lines, int tt, int TT) {
  const int lane = threadIdx.x & 31, i = lane & 7, r = lane >> 3, whole = F / 8;
  src += r * ld + i;
  const uint32_t to = lines + (uint32_t)r * 32u, from = lines + (uint32_t)(lane >> 2) * (NEXT * 4u) + (uint32_t)(lane & 3) * 32u;
  int f0 = F % 8 != 0 && tt == (whole - 1) % TT ? F - 8 : 8 * tt;
  for (int k = tt; k < whole;) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = 4 * q + r < rows ? __ldg(src + f0 + 4 * q * ld) : 0.f;
    const uint32_t at = (uint32_t)f0 * (NEXT * 4u);
#pragma unroll
    for (int q = 0; q < 8; ++q) asm volatile("st.shared.f32 [%0], %1;" ::"r"(to + at + (uint32_t)(q * NEXT * 4) + (uint32_t)((i ^ q) * 4)), "f"(v[q]) : "memory");
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[q]) : "r"(from + at + (uint32_t)((q ^ (lane >> 2)) * 4)) : "memory");
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q) asm volatile("st.shared.f32 [%0], %1;" ::"r"(lines + at + (uint32_t)(q * NEXT * 4) + (uint32_t)lane * 4u), "f"(v[q]) : "memory");
    __syncwarp(); // (the next piece may take some of these lines)
    if (f0 == 8 * k) k += TT; // (the window leads to the first piece)
    f0 = 8 * k;
  }
}

// --------------------------------------------------------------------------

// TURN: the rows are turned around in shared memory (stage_pieces) instead of read one per lane.
template <int REP, int TS, int RPL, bool STAGED, bool CACHED, bool TURN = false>
__global__ void __launch_bounds__(1024, 1) tb_walk_kernel(const WalkParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int RW = p.row_warps, TT = p.tree_threads;
  const int rw = warp % RW, tt = warp / RW;
  const int F = p.num_features;
  const int W = p.num_classes > 0 ? p.num_classes : 1;
  constexpr int RT = 32 * RPL; // rows per warp tile

  // shared memory carve-up
  uint64_t *mbar = reinterpret_cast<uint64_t *>(smem_raw);                 // 2 barriers
  int8_t *lut_s = reinterpret_cast<int8_t *>(smem_raw + 16);               // look-up table
  size_t off = (16 + (size_t)p.lut_bytes + 127) & ~(size_t)127;
  unsigned char *stage0 = smem_raw + off;
  off += STAGED ? (size_t)p.stages * p.stage_bytes : 0;
  float *xs_all = reinterpret_cast<float *>(smem_raw + off);
  const size_t xs_floats = CACHED ? (size_t)(F + 1) * RT : 0;
  off += (size_t)RW * xs_floats * 4;
  // per-warp class sums (multiclass) or cross-tree-thread partials
  float *acc_s = reinterpret_cast<float *>(smem_raw + off);

  const long long row_base = (long long)blockIdx.x * RW * RT + (long long)rw * RT;
  const int g0 = blockIdx.y * p.groups_per_chunk;
  const int g1 = min(p.num_groups, g0 + p.groups_per_chunk);

  if (STAGED && tid == 0) {
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
    fence_barrier_init();
  }
  for (int i = tid; i < p.lut_bytes; i += blockDim.x) lut_s[i] = p.lut[i];
  // ---- stage the row tile, transposed: xs[f][row]
  static_assert(!TURN || (CACHED && RPL == 1), "one row per lane of a cached tile");
  if (CACHED) {
    float *xs = xs_all + (size_t)rw * xs_floats;
    if constexpr (TURN) {
      const long long row0 = row_base < p.n_rows ? row_base : 0;
      stage_pieces<RT>(p.rows + row0 * p.ld, p.ld, (int)min(p.n_rows - row0, 32ll), F, smem_u32(xs), tt, TT);
    } else {
      // a row per lane
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        const long long row = row_base + q * 32 + lane;
        const bool live = row < p.n_rows;
        const float *src = p.rows + (live ? row : 0) * p.ld;
        float *dst = xs + q * 32 + lane;
        if (p.vec4_ok) {
          for (int k = tt; k < F / 4; k += TT) {
            const float4 v = live ? __ldg(reinterpret_cast<const float4 *>(src) + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            dst[(4 * k + 0) * RT] = v.x; dst[(4 * k + 1) * RT] = v.y;
            dst[(4 * k + 2) * RT] = v.z; dst[(4 * k + 3) * RT] = v.w;
          }
        } else {
          for (int k = tt; k < F; k += TT) dst[k * RT] = live ? __ldg(src + k) : 0.f;
        }
      }
    }
    if (tt == 0)
#pragma unroll
      for (int q = 0; q < RPL; ++q) xs[F * RT + q * 32 + lane] = __int_as_float(0xff800000); // sentinel feature: -inf
  }
  __syncthreads();

  if (STAGED && tid == 0) {
    for (int s = p.skip_first_copy ? 1 : 0; s < p.stages && g0 + s < g1; ++s) {
      const DevGroupMeta gm = p.groups[g0 + s];
      const uint32_t bytes = (gm.slots * kCols * (REP == 2 ? 6u : (uint32_t)(TS == 1 ? 8 : TS == 2 ? 16 : TS == 3 ? 24 : 32)) + 15u) & ~15u;
      mbar_expect_tx(&mbar[s], bytes);
      bulk_g2s(stage0 + (size_t)s * p.stage_bytes, p.blob + gm.byte_off, bytes, &mbar[s]);
    }
  }

  RowAccess ra[RPL];
#pragma unroll
  for (int q = 0; q < RPL; ++q) {
    ra[q].xs = xs_all + (size_t)rw * xs_floats + q * 32 + lane;
    const long long row = row_base + q * 32 + lane;
    ra[q].grow = p.rows + (row < p.n_rows ? row : 0) * p.ld;
    ra[q].num_features = F;
  }

  float acc[RPL];
#pragma unroll
  for (int q = 0; q < RPL; ++q) acc[q] = 0.f;
  float *cacc = acc_s + (size_t)warp * W * RT; // multiclass: [class][row in tile]
  if (p.num_classes > 0 && !p.class_regs)
    for (int i = lane; i < W * RT; i += 32) cacc[i] = 0.f;
  __syncwarp();
  // Multiclass with class sums in registers: the packer lays a multiclass forest out class
  // by class (every group belongs to one class, classes in increasing order, every class
  // present), so one register per row holds the running sum of the current class and the
  // arg-max is updated whenever the class changes -- no shared-memory class table, which
  // leaves room for a full block of row warps.
  int cur_cls = -1;
  float best[RPL];
  int arg[RPL];
#pragma unroll
  for (int q = 0; q < RPL; ++q) {
    best[q] = __int_as_float(0xff800000);
    arg[q] = 0;
  }
  auto close_class = [&]() {
    if (cur_cls < 0) return;
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      const float v = p.initial_value + acc[q];
      if (!(best[q] > v)) { // the reference's tie rule: the later class wins
        best[q] = v;
        arg[q] = cur_cls;
      }
      acc[q] = 0.f;
    }
  };

  bool failed = false; // (the way out lies behind the loop: inside it cost sparse tiles of one node 2.8 %, 167 -> 172 us)
  for (int g = g0; g < g1; ++g) {
    const DevGroupMeta gm = p.groups[g];
    if (p.class_regs) {
      const int cls = p.tree_class[g * kCols];
      if (cls != cur_cls) {
        close_class();
        cur_cls = cls;
      }
    }
    const uint8_t *gbase;
    if (STAGED) {
      const int s = p.stages == 2 ? (g - g0) & 1 : 0;
      const uint32_t parity = (p.stages == 2 ? (g - g0) >> 1 : g - g0) & 1;
      const bool ok = mbar_wait_bounded(&mbar[s], parity, p.wait_limit ? p.wait_limit : kWaitLimit);
      failed = __syncthreads_or(!ok) != 0;
      if (failed) break;
      gbase = stage0 + (size_t)s * p.stage_bytes;
    } else {
      gbase = p.blob + gm.byte_off;
    }
    // what becomes of row q's value from column `col`
    auto use = [&](uint32_t col, int q, float v, uint32_t slot) {
      const int k = g * kCols + (int)col;
      if (p.leaf_ids != nullptr) {
        const int t = p.tree_index[k];
        const long long row = row_base + q * 32 + lane;
        if (t >= 0 && row < p.n_rows)
          p.leaf_ids[row * p.num_trees + t] = p.orig_node[p.orig_off[g] + (size_t)slot * kCols + col];
      } else if (p.num_classes > 0 && !p.class_regs) {
        cacc[(int)p.tree_class[k] * RT + q * 32 + lane] += v;
      } else {
        acc[q] += v;
      }
    };
    if (TURN && TS <= 2) {
      // Large batches, fewer than four tree threads: four columns in lock-step, twice the
      // loads in flight that two have.  100000 rows of 54 features, 300 trees of 8 levels: sparse tiles of one node 198 -> 167 us, of two 305 ->
      // 265, array 232 -> 208, reorg 218 -> 201 (eight columns: 177 and 207 for one node and reorg; tiles of three lose, 463 -> 487).
      // Bound: issue, 69 % busy with two columns at 231 instructions per 32 rows and tree (tiles of two), shared-memory pipe 64 %.
      for (int s = tt; s < kCols; s += 4 * TT) {
        uint32_t col[4], slot[4];
        float v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) col[c] = (uint32_t)(lane + s + c * TT) & (kCols - 1);
        walk_columns<REP, TS, STAGED, CACHED, RT, 4>(gbase, gm.slots, gm.depth, col, ra[0], lut_s, slot, v);
#pragma unroll
        for (int c = 0; c < 4; ++c) use(col[c], 0, v[c], slot[c]);
      }
    } else if (RPL == 1 && TT < kCols) {
      // one row per lane: two columns in lock-step
      for (int s = tt; s < kCols; s += 2 * TT) {
        const uint32_t col[2] = {(uint32_t)(lane + s) & (kCols - 1), (uint32_t)(lane + s + TT) & (kCols - 1)};
        uint32_t slot[2];
        float v[2];
        walk_columns<REP, TS, STAGED, CACHED, RT, 2>(gbase, gm.slots, gm.depth, col, ra[0], lut_s, slot, v);
        use(col[0], 0, v[0], slot[0]);
        use(col[1], 0, v[1], slot[1]);
      }
    } else {
      for (int s = tt; s < kCols; s += TT) {
        const uint32_t col[1] = {(uint32_t)(lane + s) & (kCols - 1)};
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
          uint32_t slot[1];
          float v[1];
          walk_columns<REP, TS, STAGED, CACHED, RT, 1>(gbase, gm.slots, gm.depth, col, ra[q], lut_s, slot, v);
          use(col[0], q, v[0], slot[0]);
        }
      }
    }
    if (STAGED) {
      __syncthreads(); // every warp is done with this stage
      if (tid == 0 && g + p.stages < g1) {
        const int s = p.stages == 2 ? (g - g0) & 1 : 0;
        const DevGroupMeta nx = p.groups[g + p.stages];
        const uint32_t bytes = (nx.slots * kCols * (REP == 2 ? 6u : (uint32_t)(TS == 1 ? 8 : TS == 2 ? 16 : TS == 3 ? 24 : 32)) + 15u) & ~15u;
        mbar_expect_tx(&mbar[s], bytes);
        bulk_g2s(stage0 + (size_t)s * p.stage_bytes, p.blob + nx.byte_off, bytes, &mbar[s]);
      }
    }
  }
  if (failed) {
    give_up(p.status, 2);
    return;
  }
  if (p.leaf_ids != nullptr) return;

  // ---- combine the tree-thread warps that share a row tile (block-level pass)
  if (p.num_classes == 0) {
    if (TT > 1) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < RPL; ++q) acc_s[(size_t)warp * RT + q * 32 + lane] = acc[q];
      __syncthreads();
      if (tt == 0) {
        for (int o = 1; o < TT; ++o)
#pragma unroll
          for (int q = 0; q < RPL; ++q) acc[q] += acc_s[(size_t)(o * RW + rw) * RT + q * 32 + lane];
      }
    }
    if (tt != 0) return;
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      const long long row = row_base + q * 32 + lane;
      if (row >= p.n_rows) continue;
      if (p.write_partial)
        p.partial[(long long)blockIdx.y * p.n_rows + row] = acc[q];
      else
        reinterpret_cast<float *>(p.out)[row] = apply_transform(p.initial_value + acc[q], p.transform);
    }
  } else if (p.class_regs) {
    close_class();
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      const long long row = row_base + q * 32 + lane;
      if (row >= p.n_rows) continue;
      if (p.out_kind == 1) reinterpret_cast<int8_t *>(p.out)[row] = (int8_t)arg[q];
      else reinterpret_cast<float *>(p.out)[row] = (float)arg[q];
    }
  } else {
    __syncthreads();
    if (tt != 0) return;
    for (int o = 1; o < TT; ++o) {
      const float *other = acc_s + (size_t)(o * RW + rw) * W * RT;
      for (int i = lane; i < W * RT; i += 32) cacc[i] += other[i];
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      const long long row = row_base + q * 32 + lane;
      if (row >= p.n_rows) continue;
      const float *mine = cacc + q * 32 + lane;
      if (p.write_partial) {
        float *dst = p.partial + ((long long)blockIdx.y * p.n_rows + row) * W;
        for (int c = 0; c < W; ++c) dst[c] = mine[c * RT];
      } else {
        const float init = p.initial_value;
        const int arg = argmax_last(W, [&](int c) { return init + mine[c * RT]; });
        if (p.out_kind == 1) reinterpret_cast<int8_t *>(p.out)[row] = (int8_t)arg;
        else reinterpret_cast<float *>(p.out)[row] = (float)arg;
      }
    }
  }
}

using WalkKernel = void (*)(const WalkParams);
// turn: rows turned around in shared memory.  (walk_kernels.cu)
WalkKernel walk_kernel(int representation, int tile_size, int rows_per_lane, bool staged, bool cached, bool turn);

} // namespace tb
