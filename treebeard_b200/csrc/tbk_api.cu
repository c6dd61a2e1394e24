// C ABI of the kernel library (see include/tbk.h): packed-forest upload, launch-shape
// selection, kernel dispatch, the second pass, and the host-buffer pipeline.
#include "../../include/tbk.h"
#include "pack.h"
#include "quant_pack.h"
#include "rank_pack.h"
#include "deep_pack.h"
#include "lane_pack.h"
#include "schedule.h"
#include "walk_kernels.cuh"
#include "second_pass.cuh"
#include "walk_quant.cuh"
#include "quant_keys.cuh"
#include "walk_quant_batch.cuh"
#include "walk_deep.cuh"
#include "rank_rows.cuh"
#include "walk_rank.cuh"
#include "rank_slabs.cuh"
#include "walk_rank_tiles.cuh"
#include "walk_lanes.cuh"
#include "packed_image.h"

#ifdef __SSE2__
#include <emmintrin.h>
#endif
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <list>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

namespace {

thread_local std::string g_last_error;

int fail(int code, const char *fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}

#define CUDA_TRY(expr)                                                                     \
  do {                                                                                     \
    cudaError_t e__ = (expr);                                                              \
    if (e__ != cudaSuccess)                                                                \
      return fail(TBK_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__),   \
                  __FILE__, __LINE__);                                                     \
  } while (0)

} // namespace

// Pinned, mapped host memory is slow to come by (milliseconds for a few MiB), so what a forest gives
// back is kept for the next one: blocks of up to 32 MiB, 64 MiB of them in all, until the process has
// no forest any more.
class PinnedPool {
public:
  unsigned char *take(size_t bytes, size_t *capacity) { // null: none to be had
    bytes = (bytes + 65535) / 65536 * 65536;
    {
      std::lock_guard<std::mutex> lock(mu_);
      size_t best = free_.size();
      for (size_t i = 0; i < free_.size(); ++i)
        if (free_[i].second >= bytes && free_[i].second <= 4 * bytes && (best == free_.size() || free_[i].second < free_[best].second)) best = i;
      if (best < free_.size()) {
        const auto b = free_[best];
        free_.erase(free_.begin() + (ptrdiff_t)best);
        kept_ -= b.second;
        *capacity = b.second;
        return b.first;
      }
    }
    unsigned char *mem = nullptr;
    if (cudaHostAlloc(&mem, bytes, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) return nullptr;
    *capacity = bytes;
    return mem;
  }
  void give_back(unsigned char *mem, size_t capacity) {
    if (!mem) return;
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (capacity <= ((size_t)32 << 20) && kept_ + capacity <= ((size_t)64 << 20)) {
        free_.emplace_back(mem, capacity);
        kept_ += capacity;
        return;
      }
    }
    cudaFreeHost(mem);
  }
  // A status word: 64 bytes of a shared page.
  int32_t *take_status() {
    std::lock_guard<std::mutex> lock(mu_);
    if (status_.empty()) {
      unsigned char *page = nullptr;
      if (cudaHostAlloc(&page, 4096, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) return nullptr;
      pages_.push_back(page);
      for (int i = 0; i < 4096; i += 64) status_.push_back(reinterpret_cast<int32_t *>(page + i));
    }
    int32_t *word = status_.back();
    status_.pop_back();
    *word = 0;
    return word;
  }
  void give_back_status(int32_t *word) {
    if (!word) return;
    std::lock_guard<std::mutex> lock(mu_);
    status_.push_back(word);
  }

  void attach() {
    std::lock_guard<std::mutex> lock(mu_);
    ++forests_;
  }
  void detach() { // (the last forest has given back what it had)
    std::lock_guard<std::mutex> lock(mu_);
    if (--forests_ > 0) return;
    for (const auto &b : free_) cudaFreeHost(b.first);
    for (unsigned char *page : pages_) cudaFreeHost(page);
    free_.clear();
    pages_.clear();
    status_.clear();
    kept_ = 0;
  }

private:
  std::mutex mu_;
  int64_t forests_ = 0;
  std::vector<std::pair<unsigned char *, size_t>> free_;
  std::vector<unsigned char *> pages_;
  std::vector<int32_t *> status_;
  size_t kept_ = 0;
};
PinnedPool &pinned_pool() { // (never destroyed: forests may outlive static objects)
  static PinnedPool *pool = new PinnedPool();
  return *pool;
}

// Copies pageable batches into staging slots, chunk after chunk, on a few threads that a forest
// keeps from its first such batch on: one core moves about 20 GB/s, PCIe takes 55, and starting
// threads for every call costs more than the copy.  The calling thread enqueues GPU work meanwhile
// and copies pieces when it has nothing else to do.
//
// The copies bypass the caches: the DMA engine reads lines that are still dirty in some core's cache
// at a quarter of its rate (a bulk call of 524288 x 28 rows took 2.5 ms with plain copies).
void copy_past_caches(unsigned char *dst, const unsigned char *src, size_t n) {
#ifdef __SSE2__
  if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
    size_t i = 0;
    for (; i + 64 <= n; i += 64) {
      const __m128i *from = reinterpret_cast<const __m128i *>(src + i);
      __m128i *to = reinterpret_cast<__m128i *>(dst + i);
      const __m128i a = _mm_loadu_si128(from), b = _mm_loadu_si128(from + 1), c = _mm_loadu_si128(from + 2), d = _mm_loadu_si128(from + 3);
      _mm_stream_si128(to, a);
      _mm_stream_si128(to + 1, b);
      _mm_stream_si128(to + 2, c);
      _mm_stream_si128(to + 3, d);
    }
    std::memcpy(dst + i, src + i, n - i);
    _mm_sfence();
    return;
  }
#endif
  std::memcpy(dst, src, n);
}
class Stager {
public:
  explicit Stager(int threads) {
    for (int t = 0; t < threads; ++t) workers_.emplace_back([this] { work(); });
  }
  ~Stager() {
    {
      std::lock_guard<std::mutex> lock(mu_);
      quit_ = true;
    }
    wake_.notify_all();
    for (std::thread &w : workers_) w.join();
  }
  void start(const void *rows, size_t bytes, unsigned char *const *slots, int num_slots, size_t chunk_bytes) {
    std::lock_guard<std::mutex> lock(mu_);
    src_ = static_cast<const unsigned char *>(rows);
    total_ = bytes;
    slots_ = slots;
    num_slots_ = num_slots;
    chunk_bytes_ = chunk_bytes;
    per_chunk_ = (int64_t)((chunk_bytes + kPiece - 1) / kPiece);
    const size_t chunks = (bytes + chunk_bytes - 1) / chunk_bytes;
    done_ = std::vector<std::atomic<int64_t>>(chunks);
    num_pieces_ = per_chunk_ * (int64_t)chunks;
    next_ = 0;
    allowed_ = num_slots - 1;
    active_ = true;
    wake_.notify_all();
  }
  void allow(int64_t chunk) { allowed_.store(chunk, std::memory_order_release); } // chunks up to this one have a free slot
  bool ready(int64_t chunk) const { return done_[chunk].load(std::memory_order_acquire) == per_chunk_; }
  // Copies one piece, if one is left whose slot is free.
  bool copy_one() {
    int64_t p = next_.load(std::memory_order_relaxed);
    do {
      if (p >= num_pieces_ || p / per_chunk_ > allowed_.load(std::memory_order_acquire)) return false;
    } while (!next_.compare_exchange_weak(p, p + 1));
    const int64_t chunk = p / per_chunk_;
    const size_t lo = (size_t)(p % per_chunk_) * kPiece, begin = (size_t)chunk * chunk_bytes_ + lo;
    const size_t end = std::min(total_, std::min(begin + kPiece, (size_t)(chunk + 1) * chunk_bytes_));
    if (begin < end) copy_past_caches(slots_[chunk % num_slots_] + lo, src_ + begin, end - begin);
    done_[chunk].fetch_add(1, std::memory_order_release);
    return true;
  }
  // The batch is over (or given up): returns once no worker looks at it any more.
  void finish() {
    active_ = false;
    while (busy_.load() != 0) std::this_thread::yield();
  }

private:
  static constexpr size_t kPiece = (size_t)256 << 10;
  void work() {
    std::unique_lock<std::mutex> lock(mu_);
    while (!quit_) {
      if (!active_ || next_.load() >= num_pieces_) {
        wake_.wait(lock);
        continue;
      }
      ++busy_;
      lock.unlock();
      while (active_ && next_.load(std::memory_order_relaxed) < num_pieces_)
        if (!copy_one()) std::this_thread::yield();
      lock.lock();
      --busy_;
    }
  }
  std::mutex mu_;
  std::condition_variable wake_;
  std::vector<std::thread> workers_;
  const unsigned char *src_ = nullptr;
  unsigned char *const *slots_ = nullptr;
  size_t total_ = 0, chunk_bytes_ = 0;
  int num_slots_ = 0;
  int64_t per_chunk_ = 1, num_pieces_ = 0;
  std::vector<std::atomic<int64_t>> done_; // pieces of every chunk that are in place
  std::atomic<int64_t> next_{0}, allowed_{0};
  std::atomic<int> busy_{0};
  std::atomic<bool> active_{false};
  bool quit_ = false;
};

struct tbk_image {
  tb::PackedImage im;
};

struct RankPlan {
  int units = tb::kRWBatchUnits; // units of rows in a block's (first) batch
  int quads = 0, walkers = 0;    // tiled keys: quads of tiles per batch, walker warps
  int tiles = 4;                 // ... tiles of such a "quad": 4, or 2 where four do not fit
  int chunks = 1, per_chunk = 1; // per_chunk: groups, or classes of a multiclass forest
  int stages = 2, smem = 0;
  uint32_t stage_bytes = 0;
  int64_t grid_x = 1;
};

// How a batch is cut for the deep-tree kernel: blocks of 32 x row_warps rows, the first `whole` of them
// over all trees and the rest over `chunks` ranges of them.
struct DeepSplit {
  bool staged = false;
  int64_t n_rows = -1, whole = 0;
  int row_warps = 0, chunks = 1;
};

struct tbk_forest {
  tb::PackedForest packed; // host copy (orig_node kept for lazy upload)
  int device = 0;
  tbk_schedule user{};     // what the caller asked for (zeros = auto)
  tb::LaunchPlan last_plan{};
  int32_t last_ran = 0;    // TBK_RAN_*
  int64_t batch_hint = 0;
  int max_smem_optin = 0;
  int num_sms = 0;
  // device buffers
  uint8_t *d_blob = nullptr;
  tb::DevGroupMeta *d_groups = nullptr;
  int16_t *d_tree_class = nullptr;
  int32_t *d_tree_index = nullptr;
  int32_t *d_orig_node = nullptr;
  unsigned long long *d_orig_off = nullptr;
  bool orig_ready = false;
  int8_t *d_lut = nullptr;
  int32_t *h_status = nullptr, *d_status = nullptr; // status word in mapped host memory, both addresses
  // 16-bit-key layout (wide rows)
  bool quant = false;
  tb::QuantForest qf;
  uint32_t *d_qnode = nullptr;
  float *d_qleaf = nullptr, *d_qexact = nullptr, *d_qlo = nullptr, *d_qscale = nullptr;
  tb::DevQuantGroup *d_qgroups = nullptr;
  int32_t *d_qtree_index = nullptr, *d_qorig = nullptr;
  int32_t *d_qset_groups = nullptr, *d_qgroup_class = nullptr; // multiclass key layout
  int32_t qset_count[2] = {0, 0};
  unsigned long long *d_ties = nullptr;
  // rank keys (narrow rows): pointers into one block
  bool rank = false;
  unsigned char *d_rank_block = nullptr;
  tb::RankForest rf;
  uint32_t *d_rnode = nullptr;
  float *d_rleaf = nullptr, *d_rthr = nullptr;
  int32_t *d_rorig = nullptr, *d_rtree_index = nullptr, *d_rclass_begin = nullptr;
  tb::DevQuantGroup *d_rgroups = nullptr;
  tb::DevRankFeature *d_rfeatures = nullptr;
  uint16_t *d_rlut = nullptr;
  int rank_used = 0;                                     // features with thresholds
  int rank_width = 0, rank_pieces = 1, rank_smem = 0; // the ranking kernel's tables (plan_rank_tables)
  uint32_t *d_rslabs = nullptr;                       // the same interleaved (rank_slabs.cuh), where they fit
  uint32_t slab_bytes = 0, slab_buckets = 0;
  int slab_steps = 0;
  struct Workspace {
    unsigned char *mem = nullptr;
    size_t bytes = 0;
    unsigned long long stream = 0; // id of the stream that uses it
    bool used = false;
    bool marked = false;        // `done` stands behind the last use
    cudaEvent_t done = nullptr;
  };
  static constexpr int kWorkspaces = 8;
  bool mark_uses = false;
  Workspace workspace[kWorkspaces];
  unsigned next_victim = 0;
  // memory of calls that were captured, and whether a graph of such a call still exists
  struct Captured {
    Workspace memory;
    std::shared_ptr<std::atomic<bool>> alive;
  };
  std::list<Captured> captured;
  std::vector<const void *> smem_allowed;
  RankPlan rank_plan;          // of the last batch size
  int64_t rank_plan_rows = -1;
  bool rank_plan_ids = false;
  // lane layout (what is left)
  bool lanes = false;
  uint2 *d_lnodes = nullptr;
  uint32_t *d_lroot = nullptr, *d_lclass_end = nullptr, *d_lclass_tree = nullptr;
  int32_t *d_ltree_index = nullptr, *d_lorig = nullptr;
  int64_t lane_class_trees = 0; // of the largest class
  // one-tree-per-stage layout (deep trees); shares the device buffers of the key layout
  bool deep = false;
  tb::DeepForest df;
  int deep_row_warps = 0, deep_slots = 0;
  uint32_t *d_qsplit = nullptr; // deep trees of one depth: the planes in the order of the kernel that stages leaves too
  int deep_staged_warps = 0, deep_staged_slots = 0;
  DeepSplit deep_split;
  int uniform_depth = 0; // key layouts: depth shared by all groups / pairs, 0 = mixed
  // host pipeline: slots of device buffers and pinned staging that a large batch streams through,
  // and one pinned buffer that the kernels read and write directly for small batches
  static constexpr int kPipeSlots = 4;
  unsigned char *d_in[kPipeSlots] = {}, *d_res[kPipeSlots] = {}, *h_pin[kPipeSlots] = {}, *h_res[kPipeSlots] = {};
  size_t pipe_bytes = 0, pipe_rows = 0; // capacity of a slot
  std::unique_ptr<Stager> stager;
  unsigned char *h_small = nullptr, *d_small = nullptr, *d_small_in = nullptr;
  size_t small_capacity = 0, pin_capacity[kPipeSlots] = {}, res_capacity[kPipeSlots] = {};
  const float *inline_rows = nullptr; // rows of the small host batch being predicted, which may travel with the launch
  cudaStream_t streams[2] = {nullptr, nullptr};
  cudaEvent_t slot_read[kPipeSlots] = {}, slot_done[kPipeSlots] = {}; // a chunk's rows are copied / its results are there
  int64_t host_batch_rows = 0; // rows of the host batch whose chunks are being predicted
  // timing
  bool timing = false;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  bool ev_pending = false;
  int64_t launches = 0;
  bool expire_next_wait = false; // failure drill (tbk_debug_expire_next_wait)
  std::mutex mu;
};

namespace {

// Rows are turned around in shared memory where there are many of them (few tree threads per row) and a block has
// its SM to itself.  100000 rows of 54 features through 300 trees of 8 levels, two columns in
// lock-step, row per lane and turned around: sparse tiles of
// one node 266 and 198 us, of two 448 and 305, of four 698 and 614; array 395 and 232, reorg 365 and 218.  The loads in flight
// take 64 registers a thread instead of 32 to 48, which costs small blocks their company on the SM: 30000 rows of 7
// features, 200 trees, tiles of two 60.7 and 63.9 us, and 12000 rows of 40 features under 16 tree threads 26.3 and 33.5.
bool turn_rows(const tb::LaunchPlan &plan, int num_features) {
  return plan.cache_rows && plan.rows_per_lane == 1 && plan.tree_threads < 4 && num_features >= 8 &&
         2 * (plan.smem_bytes + 1024) > 228 * 1024;
}

tb::WalkKernel pick_kernel(int rep, int ts, const tb::LaunchPlan &plan, int num_features, int32_t *ran) {
  const bool turn = turn_rows(plan, num_features);
  if (turn) *ran |= TBK_RAN_ROWS_TURNED;
  return tb::walk_kernel(rep, ts, plan.rows_per_lane, plan.staged, plan.cache_rows, turn);
}

// Dynamic shared memory beyond 48 KB has to be asked for once per kernel and device.  All forests ask for
// the most there is: what one asked for just before a launch, a smaller one of another thread would take back.
int allow_smem(tbk_forest *f, const void *kernel) {
  for (const void *k : f->smem_allowed)
    if (k == kernel) return TBK_OK;
  CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, f->max_smem_optin));
  f->smem_allowed.push_back(kernel);
  return TBK_OK;
}

// Memory for a call that is being captured.  The graph may be replayed at any time, so the memory is
// the graph's: a user object of the graph, which everything instantiated from it holds as well,
// tells when the last of them is gone (and its replays done).  The memory then serves the next capture, or
// goes back when a call allocates anyway.  Sizes are powers of two, so that captures of many batch shapes
// find each other's.
int captured_acquire(tbk_forest *f, cudaStream_t stream, size_t bytes, tbk_forest::Workspace **out) {
  size_t size = (size_t)64 << 10;
  while (size < bytes) size *= 2;
  tbk_forest::Captured *c = nullptr;
  for (auto &old : f->captured)
    if (old.memory.bytes == size && !old.alive->load(std::memory_order_acquire)) c = &old;
  if (!c) {
    unsigned char *mem = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t e = cudaMalloc(&mem, size);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return fail(TBK_ERR_CUDA, "workspace of a captured call: %s", cudaGetErrorString(e));
    f->captured.emplace_back();
    c = &f->captured.back();
    c->memory.mem = mem;
    c->memory.bytes = size;
  }
  c->alive = std::make_shared<std::atomic<bool>>(false);
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  CUDA_TRY(cudaStreamGetCaptureInfo_v2(stream, &status, &id, &graph, nullptr, nullptr));
  if (!graph) return fail(TBK_ERR_CUDA, "workspace of a captured call: the capture has ended");
  using Alive = std::shared_ptr<std::atomic<bool>>;
  auto *token = new Alive(c->alive);
  cudaUserObject_t object = nullptr;
  cudaError_t e = cudaUserObjectCreate(&object, token, [](void *p) {
    auto *mine = static_cast<Alive *>(p);
    (*mine)->store(false, std::memory_order_release);
    delete mine;
  }, 1, cudaUserObjectNoDestructorSync);
  if (e != cudaSuccess) {
    delete token;
    return fail(TBK_ERR_CUDA, "workspace of a captured call: %s", cudaGetErrorString(e));
  }
  c->alive->store(true, std::memory_order_release);
  e = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) {
    cudaUserObjectRelease(object, 1);
    return fail(TBK_ERR_CUDA, "workspace of a captured call: %s", cudaGetErrorString(e));
  }
  CUDA_TRY(cudaMemsetAsync(c->memory.mem, 0, tb::kRankArrivalBytes, stream));
  *out = &c->memory;
  return TBK_OK;
}

// Device memory that a call needs from its first kernel to its last: the keys of the rows and
// the partial sums of tree chunks.  Calls on one stream are ordered and share one workspace; a call
// on a further stream gets one of its own, up to kWorkspaces, and after that waits on the device for
// the last user of the one that it takes over.  A stream is known by its id: a handle may stand for
// another stream in every thread (cudaStreamPerThread), or for a new stream once its first one is
// destroyed, with work still pending.  From the fourth stream on every use ends with an event, so that
// there are marked ones to take over by the time that all are taken; fewer streams need none.
int workspace_acquire(tbk_forest *f, cudaStream_t stream, size_t bytes, tbk_forest::Workspace **out) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  CUDA_TRY(cudaStreamIsCapturing(stream, &capturing));
  if (capturing != cudaStreamCaptureStatusNone) return captured_acquire(f, stream, bytes, out);
  unsigned long long id = 0;
  CUDA_TRY(cudaStreamGetId(stream, &id));
  tbk_forest::Workspace *w = nullptr;
  int used = 0;
  for (auto &c : f->workspace) {
    used += c.used;
    if (c.used && c.stream == id) w = &c;
  }
  if (!w) {
    for (auto &c : f->workspace)
      if (!c.used && (!w || c.bytes > w->bytes)) w = &c;
    if (w && used + 1 >= tbk_forest::kWorkspaces / 2) f->mark_uses = true;
  }
  for (int i = 0; !w && i < tbk_forest::kWorkspaces; ++i) {
    tbk_forest::Workspace &c = f->workspace[f->next_victim++ % tbk_forest::kWorkspaces];
    if (!c.marked) continue;
    CUDA_TRY(cudaStreamWaitEvent(stream, c.done, 0));
    w = &c;
  }
  if (!w) { // (no use got as far as its mark)
    CUDA_TRY(cudaDeviceSynchronize());
    w = &f->workspace[f->next_victim++ % tbk_forest::kWorkspaces];
  }
  w->stream = id;
  w->used = true;
  w->marked = false;
  if (w->bytes < bytes) {
    f->captured.remove_if([](const tbk_forest::Captured &c) {
      return !c.alive->load(std::memory_order_acquire) && cudaFree(c.memory.mem) == cudaSuccess;
    });
    if (w->mem) CUDA_TRY(cudaFree(w->mem)); // (waits for the work that uses it)
    w->mem = nullptr;
    w->bytes = 0;
    CUDA_TRY(cudaMalloc(&w->mem, bytes));
    CUDA_TRY(cudaMemsetAsync(w->mem, 0, tb::kRankArrivalBytes, stream));
    w->bytes = bytes;
  }
  *out = w;
  return TBK_OK;
}
int workspace_release(tbk_forest *f, tbk_forest::Workspace *w, cudaStream_t stream) {
  if (!f->mark_uses || !w->used) return TBK_OK; // (a captured call's is never taken over)
  if (!w->done) CUDA_TRY(cudaEventCreateWithFlags(&w->done, cudaEventDisableTiming));
  CUDA_TRY(cudaEventRecord(w->done, stream));
  w->marked = true;
  return TBK_OK;
}

// Memory for a call's tree-chunk partial sums, behind the counters that rank keys use.
int partials_acquire(tbk_forest *f, cudaStream_t stream, size_t floats, float **partials, tbk_forest::Workspace **out) {
  const int rc = workspace_acquire(f, stream, tb::kRankArrivalBytes + floats * sizeof(float), out);
  if (rc == TBK_OK) *partials = reinterpret_cast<float *>((*out)->mem + tb::kRankArrivalBytes);
  return rc;
}

// A copy from pageable memory may return before its data has reached the device, and a memset does:
// both are work of the legacy stream, which non-blocking streams don't wait for.
int uploads_done() {
  CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));
  return TBK_OK;
}

int ensure_orig(tbk_forest *f) {
  if (f->orig_ready) return TBK_OK;
  const auto &p = f->packed;
  if (!f->d_orig_node) CUDA_TRY(cudaMalloc(&f->d_orig_node, std::max<size_t>(4, p.orig_node.size() * 4)));
  CUDA_TRY(cudaMemcpy(f->d_orig_node, p.orig_node.data(), p.orig_node.size() * 4, cudaMemcpyHostToDevice));
  if (!f->d_orig_off) CUDA_TRY(cudaMalloc(&f->d_orig_off, std::max<size_t>(8, p.orig_off.size() * 8)));
  CUDA_TRY(cudaMemcpy(f->d_orig_off, p.orig_off.data(), p.orig_off.size() * 8, cudaMemcpyHostToDevice));
  const int rc = uploads_done();
  f->orig_ready = rc == TBK_OK;
  return rc;
}

enum Mode { kPredict, kPartial, kLeafIds };

int quant_smem_bytes(int num_features) {
  return tb::kQBarBytes + tb::kQRingBytes + tb::kQLeafTableBytes + tb::quant_key_tile_bytes(num_features);
}

// Tiles of 32 rows that the narrow-row kernel can stage together (0: the rows are too wide for it).
int quant_batch_tiles(const tbk_forest *f, int num_features) {
  const int room = f->max_smem_optin - tb::kQBBarBytes - tb::kQBRingBytes;
  const int fit = room / tb::quant_batch_tile_bytes(num_features);
  return fit >= 4 ? std::min(fit, tb::kQBMaxTiles) : 0;
}

// One prediction with a 15-bit-key kernel: rows whose key tiles fit shared memory several at a
// time go to the batch kernel (persistent blocks of 22 warps over batches of up to 16 tiles),
// wide rows to the kernel that holds one tile (persistent blocks of 24 warps over tiles of 32 rows).
int run_quant(tbk_forest *f, Mode mode, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out, int32_t out_kind,
              float *d_partial, int32_t *d_leaf_ids, cudaStream_t stream, float *fixed = nullptr, size_t fixed_floats = 0) {
  const auto &q = f->qf;
  const int64_t G = (int64_t)q.groups.size();
  const int64_t tiles = (n_rows + 31) / 32;
  const int max_batch = quant_batch_tiles(f, q.num_features);
  const bool batched = max_batch > 0;
  const bool multi = q.num_classes > 0;
  if (multi && !batched) return fail(TBK_ERR_UNSUPPORTED, "multiclass forests in the key layout need rows narrow enough for the batch kernel");
  // batch kernel: as many tiles per batch as still give every SM a batch
  int R = 1;
  if (batched) {
    R = max_batch;
    while (R > 1 && (tiles + R - 1) / R < (int64_t)f->num_sms) R = (R + 1) / 2;
  }
  const int64_t units = batched ? (tiles + R - 1) / R : tiles; // blocks' units of work along x
  int64_t chunks = 1;
  if (multi) chunks = 1; // a class must stay within one leaf warp's sequence of groups
  else if (f->user.tree_chunks > 0) chunks = f->user.tree_chunks;
  else if (batched) {
    if (units < (int64_t)f->num_sms) chunks = ((int64_t)f->num_sms + units - 1) / units;
  } else if (tiles < 2 * (int64_t)f->num_sms) chunks = (2 * (int64_t)f->num_sms + tiles - 1) / tiles;
  // (batch kernel: a second pass over partial sums costs about ten microseconds, more than the
  // walk of a small forest: trees are split only into chunks of at least 32 groups -- measured
  // on 4 096 rows x 32 groups: 38 us in one chunk, 47 us in two -- unless the caller asks)
  const int64_t max_chunks = !batched ? G : f->user.tree_chunks > 0 ? std::max<int64_t>(1, G / 2) : std::max<int64_t>(1, G / 32);
  chunks = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(chunks, max_chunks), 65535));
  if (fixed) chunks = std::max<int64_t>(1, std::min<int64_t>(chunks, (int64_t)fixed_floats / n_rows));
  const int gpc = (int)((G + chunks - 1) / chunks);
  chunks = (G + gpc - 1) / gpc;
  const bool vec4 = q.num_features % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(d_rows) & 15) == 0;
  // One block per SM (shared memory allows no more).  With more units than blocks a block is
  // persistent; the one-tile kernel then stages its next tile in tensor memory while it walks
  // the current one, a path that reads rows with 16-byte loads.
  const int64_t blocks_x = std::max<int64_t>(1, (int64_t)f->num_sms / chunks);
  const int64_t grid_x = batched ? std::min(units, blocks_x) : (vec4 && tiles > blocks_x) ? blocks_x : tiles;
  tb::LaunchPlan plan;
  plan.row_warps = batched ? R : 1;
  plan.tree_threads = tb::kQWalkers;
  plan.rows_per_lane = 1;
  plan.chunks = (int32_t)chunks;
  plan.groups_per_chunk = gpc;
  plan.staged = 1;
  plan.cache_rows = 1;
  plan.stage_bytes = tb::kQPiece;
  plan.smem_bytes = batched ? tb::quant_batch_smem_bytes(q.num_features, R) : quant_smem_bytes(q.num_features);
  plan.threads = batched ? tb::kQBThreads : tb::kQThreads;
  plan.grid_x = grid_x;
  f->last_plan = plan;

  const bool need_partials = mode == kPartial || (mode == kPredict && chunks > 1);
  float *partial_dst = nullptr;
  tbk_forest::Workspace *ws = nullptr;
  if (need_partials) {
    if (mode == kPartial && chunks == 1) {
      partial_dst = d_partial;
    } else if (fixed) {
      partial_dst = fixed;
    } else {
      const int rc = partials_acquire(f, stream, (size_t)chunks * n_rows, &partial_dst, &ws);
      if (rc) return rc;
    }
  }
  tb::QuantParams p{};
  p.node_plane = f->d_qnode;
  p.leaf_plane = f->d_qleaf;
  p.exact_plane = f->d_qexact;
  p.groups = f->d_qgroups;
  p.tree_index = f->d_qtree_index;
  p.orig_leaf = f->d_qorig;
  p.lo = f->d_qlo;
  p.scale = f->d_qscale;
  p.rows = d_rows;
  p.n_rows = n_rows;
  p.ld = ld;
  p.partial = partial_dst;
  p.out = d_out;
  p.write_partial = need_partials ? 1 : 0;
  p.leaf_ids = mode == kLeafIds ? d_leaf_ids : nullptr;
  p.num_trees = q.num_trees;
  p.num_groups = (int32_t)G;
  p.groups_per_chunk = gpc;
  p.num_features = q.num_features;
  p.transform = q.transform;
  p.initial_value = (float)q.initial_value;
  p.vec4_ok = vec4 ? 1 : 0;
  p.tiles_per_batch = R;
  p.set_groups = f->d_qset_groups;
  p.set_count[0] = f->qset_count[0];
  p.set_count[1] = f->qset_count[1];
  p.group_class = f->d_qgroup_class;
  p.num_classes = q.num_classes;
  p.out_kind = out_kind == TBK_OUT_I8 ? 1 : 0;
  p.status = f->d_status;
  p.tie_count = f->d_ties;
  p.skip_first_copy = f->expire_next_wait ? 1 : 0;
  p.wait_tries = f->expire_next_wait ? 2000u : 0u;
  f->expire_next_wait = false;
  // kernels specialised for forests whose groups all have 8 (or 6) levels; generic otherwise
  const bool ids = mode == kLeafIds;
  const int ud = (f->uniform_depth == 8 || f->uniform_depth == 6) ? f->uniform_depth : 0;
  const tb::QuantKernel qkernel = batched ? tb::batch_quant_kernel(ud, ids, multi) : tb::wide_quant_kernel(ud, ids);
  if (const int rc = allow_smem(f, (const void *)qkernel)) return rc;
  if (f->timing) CUDA_TRY(cudaEventRecord(f->ev0, stream));
  dim3 grid((unsigned)grid_x, (unsigned)chunks);
  qkernel<<<grid, plan.threads, plan.smem_bytes, stream>>>(p);
  CUDA_TRY(cudaGetLastError());
  ++f->launches;
  const int tpb = 256;
  if (mode == kPredict && chunks > 1) {
    tb::tb_finalize_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, stream>>>(
        partial_dst, (int)chunks, n_rows, 1, 0, (float)q.initial_value, q.transform, d_out, TBK_OUT_F32);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
  } else if (mode == kPartial && chunks > 1) {
    tb::tb_sum_partials_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, stream>>>(partial_dst, (int)chunks, n_rows, d_partial);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
  }
  if (f->timing) {
    CUDA_TRY(cudaEventRecord(f->ev1, stream));
    f->ev_pending = true;
  }
  return ws ? workspace_release(f, ws, stream) : TBK_OK;
}

// Shared-memory plan of the deep-tree kernel: the most row warps (even -- one block per SM
// either way, and more rows per tile mean fewer passes over the forest and more walks in
// flight) whose key tile leaves room for a ring of at least 4 whole-tree pieces.
bool deep_plan(int num_features, int max_depth, int smem_limit, int *row_warps, int *slots) {
  const int64_t slot = 4ll * tb::deep_tree_words((uint32_t)std::max(max_depth, tb::kDeepMinDepth));
  // four slots hold the node planes of the pair being walked and of the next one
  for (int rw = 30; rw >= 2; rw -= 2) { // (the block has one more warp, the ring producer)
    const int64_t keys = ((int64_t)num_features * 64 + tb::kDeepLeafBytes) * rw;
    const int64_t room = (int64_t)smem_limit - 128 - keys;
    const int64_t s = std::min<int64_t>(tb::kDeepMaxSlots, room / slot);
    if (s >= 4) {
      *row_warps = rw;
      *slots = (int)s;
      return true;
    }
  }
  return false;
}
int deep_smem_bytes(const tbk_forest *f) {
  return 128 + f->deep_slots * 4 * (int)tb::deep_tree_words((uint32_t)std::max(f->df.max_depth, tb::kDeepMinDepth)) +
         (f->df.num_features * 64 + tb::kDeepLeafBytes) * f->deep_row_warps;
}

template <bool WIDE> void (*pick_deep(bool small, bool d12, bool ids))(const tb::DeepParams) {
  if (small)
    return d12 ? (ids ? tb::tb_walk_deep_kernel<768, 12, WIDE, true> : tb::tb_walk_deep_kernel<768, 12, WIDE, false>)
               : (ids ? tb::tb_walk_deep_kernel<768, 0, WIDE, true> : tb::tb_walk_deep_kernel<768, 0, WIDE, false>);
  return d12 ? (ids ? tb::tb_walk_deep_kernel<1024, 12, WIDE, true> : tb::tb_walk_deep_kernel<1024, 12, WIDE, false>)
             : (ids ? tb::tb_walk_deep_kernel<1024, 0, WIDE, true> : tb::tb_walk_deep_kernel<1024, 0, WIDE, false>);
}

// Predictions of a forest of one depth (9 to 12 levels) over at most kDeepNarrowFeatures features take leaf values from
// shared memory (tb_walk_deep_staged_kernel).
template <int MAX> void (*pick_deep_staged(int depth))(const tb::DeepStagedParams) {
  return depth == 9    ? tb::tb_walk_deep_staged_kernel<MAX, 9>
         : depth == 10 ? tb::tb_walk_deep_staged_kernel<MAX, 10>
         : depth == 11 ? tb::tb_walk_deep_staged_kernel<MAX, 11>
                       : tb::tb_walk_deep_staged_kernel<MAX, 12>;
}
uint32_t deep_half_words(int depth) { return tb::deep_tree_words((uint32_t)depth - 1); }
int deep_staged_smem(int num_features, int depth, int row_warps, int slots) {
  return 128 + slots * 8 * (int)deep_half_words(depth) + num_features * 64 * row_warps;
}
bool deep_staged_plan(int num_features, int depth, int smem_limit, int *row_warps, int *slots) {
  for (int rw = 30; rw >= 2; rw -= 2)
    for (int s = tb::kDeepMaxSlots; s >= tb::kDeepStagedMinSlots; --s)
      if (deep_staged_smem(num_features, depth, rw, s) <= smem_limit) {
        *row_warps = rw;
        *slots = s;
        return true;
      }
  return false;
}

// What counts is the waves of blocks and what a pair of trees takes a block: 300 pairs of 12 levels
// 0.25 ms with 4 row warps, 0.34 with 18, 0.42 with 24, 0.50 with 30 (9 levels: 0.25, 0.31, 0.36, 0.42) -- all
// latency up to about 18, then the shared-memory pipe as well.  The blocks that fill no whole wave
// split the trees, into as many ranges as leave the least of their last wave empty.  Staging
// the rows takes a block the time of 8 pairs and more, the second pass over partial sums that of 8.
// (1048576 rows, 2000 trees, 18 row warps: 12.3 waves of blocks; 8000 rows, 387 trees of 9 levels: 63
// blocks in three ranges were two waves.)
DeepSplit split_deep(const tbk_forest *f, int64_t n_rows, bool staged) {
  const int64_t G = (int64_t)f->df.pairs.size(), row_tiles = (n_rows + 31) / 32, SMs = f->num_sms;
  DeepSplit best;
  best.n_rows = n_rows;
  best.staged = staged;
  double best_cost = -1.0;
  const int most = staged ? f->deep_staged_warps : f->deep_row_warps;
  for (int rw = std::min(4, most); rw <= most; ++rw) {
    const int64_t blocks = (row_tiles + rw - 1) / rw, rest = blocks % SMs;
    const double pair = rw <= 18 ? 0.7 + 0.0167 * rw : 1.0 + 0.02 * (rw - 18), start = 8.0 + 0.006 * f->df.num_features * rw;
    for (int64_t c = 1; c <= std::min<int64_t>(G, std::max<int64_t>(8, (SMs + blocks - 1) / blocks)); ++c) {
      const int64_t per = (G + c - 1) / c;
      if ((G + per - 1) / per != c) continue;
      const double waves = (double)((rest * c + SMs - 1) / SMs);
      const double cost = pair * ((double)(blocks / SMs) * ((double)G + start) + waves * ((double)per + start)) + (c > 1 ? 8.0 : 0.0);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best.row_warps = rw;
        best.chunks = (int)c;
        best.whole = c > 1 ? blocks - rest : 0;
      }
      if (rest == 0) break;
    }
  }
  return best;
}

// Are staged leaves the faster ones?  A pair of trees costs them one more wait, and 12 levels have a gathering kernel of their own,
// which wins where rows are so wide that few row warps fit (96 features and more; what a pair costs the shared-memory
// pipe matters less) and blocks walk enough pairs to make up for a later end -- unless a forest of 1500 trees and more
// is walked in whole waves and its gathers miss L2.  Staged / gathered, 12 levels: 1200 trees x 128 features, batches of 2500 (21 pairs
// to a block) 1.00, 7000 (55) 1.02, 24000 1.07, 76000 1.09, 170000 rows 1.03; 500 x 160: 4000 (21) 1.00, 17000 (84) 1.04, 64000 1.07;
// 2000 x 100: 12000 1.10, 33000 1.04, 125000 0.99, 170000 0.98; 2000 x 128: 17000 1.10, 100000 0.99.  500 x 60 and 30: 0.86 to 0.96
// from 4000 rows on.  9 to 11 levels: 0.90 to 1.00.
bool deep_staged_pays(const tbk_forest *f, const DeepSplit &s, int64_t n_rows) {
  const int64_t pairs = (int64_t)f->df.pairs.size(), per_block = s.whole > 0 ? pairs : (pairs + s.chunks - 1) / s.chunks;
  const bool waves = n_rows > 32ll * s.row_warps * f->num_sms;
  return f->uniform_depth < 12 || f->df.num_features < 96 || s.row_warps > f->deep_row_warps || per_block < 32 ||
         (waves && f->df.num_trees >= 1500);
}

// One launch of the deep-tree kernel over `n_rows` rows, and the second pass over chunks.
int run_deep_rows(tbk_forest *f, Mode mode, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out,
                  float *d_partial, int32_t *d_leaf_ids, cudaStream_t stream, bool staged, int rw, int64_t chunks) {
  const auto &q = f->df;
  const int64_t G = (int64_t)q.pairs.size();
  const int64_t rows_per_block = 32 * rw;
  const int64_t grid_x = (n_rows + rows_per_block - 1) / rows_per_block;
  chunks = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(chunks, G), 65535));
  const int gpc = (int)((G + chunks - 1) / chunks);
  chunks = (G + gpc - 1) / gpc;
  tb::LaunchPlan plan;
  plan.row_warps = rw;
  plan.tree_threads = 1;
  plan.rows_per_lane = 1;
  plan.chunks = (int32_t)chunks;
  plan.groups_per_chunk = gpc;
  plan.staged = 1;
  plan.cache_rows = 1;
  plan.stage_bytes = 4u * tb::deep_tree_words((uint32_t)std::max(q.max_depth, tb::kDeepMinDepth));
  plan.smem_bytes = staged ? deep_staged_smem(q.num_features, f->uniform_depth, (rw + 1) / 2 * 2, f->deep_staged_slots) : deep_smem_bytes(f);
  plan.threads = 32 * (rw + 1); // row warps + the ring producer
  plan.grid_x = grid_x;
  f->last_plan = plan;

  const bool need_partials = mode == kPartial || (mode == kPredict && chunks > 1);
  float *partial_dst = nullptr;
  tbk_forest::Workspace *ws = nullptr;
  if (need_partials) {
    if (mode == kPartial && chunks == 1) {
      partial_dst = d_partial;
    } else {
      const int rc = partials_acquire(f, stream, (size_t)chunks * n_rows, &partial_dst, &ws);
      if (rc) return rc;
    }
  }
  tb::DeepStagedParams p{};
  p.node_plane = f->d_qnode;
  p.leaf_plane = f->d_qleaf;
  p.exact_plane = f->d_qexact;
  p.pairs = f->d_qgroups;
  p.tree_index = f->d_qtree_index;
  p.orig_leaf = f->d_qorig;
  p.lo = f->d_qlo;
  p.scale = f->d_qscale;
  p.rows = d_rows;
  p.n_rows = n_rows;
  p.ld = ld;
  p.partial = partial_dst;
  p.out = d_out;
  p.write_partial = need_partials ? 1 : 0;
  p.leaf_ids = mode == kLeafIds ? d_leaf_ids : nullptr;
  p.num_trees = q.num_trees;
  p.num_pairs = (int32_t)G;
  p.pairs_per_chunk = gpc;
  p.num_features = q.num_features;
  p.transform = q.transform;
  p.initial_value = (float)q.initial_value;
  p.ring_slots = staged ? f->deep_staged_slots : f->deep_slots;
  p.slot_bytes = plan.stage_bytes;
  p.tree_words = plan.stage_bytes / 4;
  p.key_tile = 128u * (uint32_t)q.num_features;
  p.leaf_off = (uint32_t)(plan.smem_bytes - tb::kDeepLeafBytes * f->deep_row_warps);
  p.status = f->d_status;
  p.tie_count = f->d_ties;
  p.skip_first_copy = f->expire_next_wait ? 1 : 0;
  p.wait_tries = f->expire_next_wait ? 2000u : 0u;
  f->expire_next_wait = false;
  // up to 24 warps (row warps + producer) the compiler may use 80 registers per thread, beyond that 64
  // (specialised for forests whose pairs all have 12 levels; generic otherwise)
  const bool d12 = f->uniform_depth == 12, ids = mode == kLeafIds, small = plan.threads <= 768;
  dim3 grid((unsigned)grid_x, (unsigned)chunks);
  if (staged) {
    f->last_ran |= TBK_RAN_STAGED_LEAVES;
    p.split = f->d_qsplit;
    const auto kernel = small ? pick_deep_staged<768>(f->uniform_depth) : pick_deep_staged<1024>(f->uniform_depth);
    if (const int rc = allow_smem(f, (const void *)kernel)) return rc;
    kernel<<<grid, plan.threads, plan.smem_bytes, stream>>>(p);
  } else {
    const auto kernel = q.num_features > tb::kDeepNarrowFeatures ? pick_deep<true>(small, d12, ids) : pick_deep<false>(small, d12, ids);
    if (const int rc = allow_smem(f, (const void *)kernel)) return rc;
    kernel<<<grid, plan.threads, plan.smem_bytes, stream>>>(p);
  }
  CUDA_TRY(cudaGetLastError());
  ++f->launches;
  const int tpb = 256;
  if (mode == kPredict && chunks > 1) {
    tb::tb_finalize_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, stream>>>(
        partial_dst, (int)chunks, n_rows, 1, 0, (float)q.initial_value, q.transform, d_out, TBK_OUT_F32);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
  } else if (mode == kPartial && chunks > 1) {
    tb::tb_sum_partials_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, stream>>>(partial_dst, (int)chunks, n_rows, d_partial);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
  }
  return ws ? workspace_release(f, ws, stream) : TBK_OK;
}

// One prediction with the deep-tree kernel.
int run_deep(tbk_forest *f, Mode mode, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out,
             float *d_partial, int32_t *d_leaf_ids, cudaStream_t stream) {
  DeepSplit &s = f->deep_split;
  bool staged = f->d_qsplit && mode != kLeafIds;
  if (s.n_rows != n_rows || s.staged != staged) {
    s = split_deep(f, n_rows, staged);
    if (f->user.tree_chunks > 0) { // (asked for: all rows)
      s.whole = 0;
      s.chunks = f->user.tree_chunks;
    }
  }
  staged = staged && deep_staged_pays(f, s, n_rows);
  if (f->timing) CUDA_TRY(cudaEventRecord(f->ev0, stream));
  const int64_t first = std::min<int64_t>(n_rows, s.whole * s.row_warps * 32);
  if (first > 0) {
    const int rc = run_deep_rows(f, mode, d_rows, first, ld, d_out, d_partial, d_leaf_ids, stream, staged, s.row_warps, 1);
    if (rc) return rc;
  }
  if (first < n_rows) {
    const int rc = run_deep_rows(f, mode, d_rows + first * ld, n_rows - first, ld, d_out ? static_cast<float *>(d_out) + first : nullptr,
                                 d_partial ? d_partial + first : nullptr, d_leaf_ids ? d_leaf_ids + first * f->df.num_trees : nullptr,
                                 stream, staged, s.row_warps, s.chunks);
    if (rc) return rc;
  }
  if (f->timing) {
    CUDA_TRY(cudaEventRecord(f->ev1, stream));
    f->ev_pending = true;
  }
  return TBK_OK;
}

// ---------------------------------------------------------------------------
// Rank keys (rank_pack.h)

// bytes of keys per row
bool rank_tiled(int num_features) { return num_features > tb::kRankRowFeatures; }
int rank_stride(int num_features) {
  if (tb::rank_bytes(num_features)) return (num_features + 3) / 4 * 4;
  return rank_tiled(num_features) ? (num_features + 1) / 2 * 4 : num_features <= tb::kRankPairFeatures ? 64 : 128;
}

template <int S, int NR, bool WHOLE, bool INLINE> const void *pick_rank(int mode) {
  return mode == tb::kRankLeafIds   ? (const void *)tb::tb_walk_rank_kernel<S, NR, WHOLE, tb::kRankLeafIds, INLINE>
         : mode == tb::kRankClasses ? (const void *)tb::tb_walk_rank_kernel<S, NR, WHOLE, tb::kRankClasses, INLINE>
                                    : (const void *)tb::tb_walk_rank_kernel<S, NR, WHOLE, tb::kRankSums, INLINE>;
}
const void *pick_rank_kernel(int stride, bool small, bool whole, bool inlined, int mode) {
  if (inlined) return stride == 64 ? pick_rank<64, 4, true, true>(mode) : pick_rank<128, 4, true, true>(mode);
  if (small) return stride == 64 ? pick_rank<64, 4, true, false>(mode) : pick_rank<128, 4, true, false>(mode);
  if (stride == 64) return whole ? pick_rank<64, 16, true, false>(mode) : pick_rank<64, 16, false, false>(mode);
  return whole ? pick_rank<128, 16, true, false>(mode) : pick_rank<128, 16, false, false>(mode);
}

const void *pick_rank_tiles_kernel(int tiles, bool bytes, bool ids) {
  if (!bytes) return ids ? (const void *)tb::tb_walk_rank_tiles_kernel<4, false, true> : (const void *)tb::tb_walk_rank_tiles_kernel<4, false, false>;
  if (tiles == 4) return ids ? (const void *)tb::tb_walk_rank_tiles_kernel<4, true, true> : (const void *)tb::tb_walk_rank_tiles_kernel<4, true, false>;
  return ids ? (const void *)tb::tb_walk_rank_tiles_kernel<2, true, true> : (const void *)tb::tb_walk_rank_tiles_kernel<2, true, false>;
}

// How many quads of tiles a block of the tiled kernel takes at a time, with how many walker warps.
// Rows of 491 to 511 features under trees of 8 levels leave three ring slots beside one quad only with
// 8 walkers, or 4 (507 to 511).
// Rows of one-byte keys that are too wide for four tiles go in pairs of tiles.
struct RankTilesShape { int quads, walkers, tiles; };
constexpr RankTilesShape kRankTilesShapes[] = {{1, 16, 4}, {2, 16, 4}, {3, 12, 4}, {4, 16, 4}, {5, 20, 4}, {6, 12, 4}, {1, 8, 4}, {1, 4, 4}, {1, 16, 2}};
int rank_tiles_slots(const RankTilesShape &sh, int num_features, int max_depth, int smem_limit) {
  const int room = smem_limit - tb::rank_tiles_smem_bytes(32 * rank_stride(num_features), sh.tiles * sh.quads, sh.walkers, sh.tiles, 0, 0);
  return room < 0 || (sh.tiles == 2 && !tb::rank_bytes(num_features)) ? 0 : std::min(tb::kRTMaxSlots, room / (128 << max_depth));
}
constexpr int kRankTilesMinSlots = 3; // one plane more than the group being walked

// Does some launch shape hold rank keys of such rows and trees?
bool rank_fits(int num_features, int max_depth, int smem_limit) {
  if (!rank_tiled(num_features)) return tb::rank_walk_smem_bytes(rank_stride(num_features), 2, 256u << max_depth) <= smem_limit;
  for (const RankTilesShape &sh : kRankTilesShapes)
    if (rank_tiles_slots(sh, num_features, max_depth, smem_limit) >= kRankTilesMinSlots) return true;
  return false;
}

// The same for keys in tiles.
RankPlan make_rank_tiles_plan(const tbk_forest *f, int64_t n_rows) {
  const auto &q = f->rf;
  const int G = (int)q.groups.size(), D = q.max_depth;
  const int tile_bytes = 32 * rank_stride(q.num_features);
  RankPlan best;
  double best_cost = -1.0;
  for (const RankTilesShape &sh : kRankTilesShapes) {
    RankPlan p;
    p.quads = sh.quads;
    p.walkers = sh.walkers;
    p.stage_bytes = 128u << D;
    p.stages = rank_tiles_slots(sh, q.num_features, D, f->max_smem_optin);
    if (p.stages < kRankTilesMinSlots) continue;
    p.tiles = sh.tiles;
    p.smem = tb::rank_tiles_smem_bytes(tile_bytes, sh.tiles * sh.quads, sh.walkers, sh.tiles, p.stages, p.stage_bytes);
    const int64_t quads = (n_rows + 32 * sh.tiles - 1) / (32 * sh.tiles);
    // clocks of a group of trees for a batch of b quads (2 D - 0.25 wavefronts per 32 rows and tree; in pairs of tiles 2 D + 0.5)
    auto group = [&](int64_t b) {
      return std::max(1.15 * sh.tiles * 32 * (double)b * (2 * D - (sh.tiles == 4 ? 0.25 : -0.5)) + 300.0, std::max(2.0 * p.stage_bytes / (p.stages >= 5 ? 70.0 : p.stages == 4 ? 50.0 : 35.0), 32.0 / (sh.walkers / sh.quads) * (sh.walkers < 8 ? 85.0 : 50.0) * D));
    };
    auto block = [&](int64_t mine) { return (double)(mine / sh.quads) * group(sh.quads) + (mine % sh.quads ? group(mine % sh.quads) : 0.0); };
    const int most = f->user.tree_chunks > 0 ? std::min(G, f->user.tree_chunks) : std::min(G, 64);
    for (int c = f->user.tree_chunks > 0 ? most : 1; c <= most; ++c) {
      const int per = (G + c - 1) / c, chunks = (G + per - 1) / per;
      const int64_t x = chunks > 1 ? (quads + sh.quads - 1) / sh.quads : std::min<int64_t>(quads, f->num_sms);
      if (chunks > 1 && x >= f->num_sms && f->user.tree_chunks <= 0) break;
      const double waves = chunks > 1 ? (double)((x * chunks + f->num_sms - 1) / f->num_sms) : 1.0;
      const double cost = waves * (per * block((quads + x - 1) / x) + 4000.0) + (chunks > 1 ? 1500.0 : 0.0);
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best = p;
        best.chunks = chunks;
        best.per_chunk = per;
        best.grid_x = x;
      }
    }
  }
  return best;
}

// Launch shape of the walk over `n_rows` rows: blocks along the rows and tree chunks, by what the
// slowest block costs in clocks.  A group takes a warp about 2 D - 1 shared-memory wavefronts per
// row and 20 warps share the pipe; a few hundred clocks go into the hand-off and the chain of
// dependent loads, and the stage's copy needs its time too (70 bytes a clock).  A block starts up
// for about 4000 clocks, and combining chunks adds about as much (a fence, an arrival, partial sums out and
// back: 64 trees of 6 levels over 10 features, 3000 rows, 10.3 us in two chunks, 8.2 in one; with 1500 clocks
// 34 of 252 small shapes were slower than one launch over rounded keys had been, with 4000 27; 3000 to 5500
// measure within 1 % of each other over all of them, 7500 2 % slower).
constexpr double kCombineClocks = 4000.0;
RankPlan make_rank_plan(const tbk_forest *f, int64_t n_rows, bool leaf_ids) {
  const auto &q = f->rf;
  const int G = (int)q.groups.size(), S = rank_stride(q.num_features);
  const bool multi = q.num_classes > 0 && !leaf_ids;
  const int parts = multi ? q.num_classes : G; // what chunks are made of
  const int64_t units = (n_rows + tb::kRWUnitRows - 1) / tb::kRWUnitRows;
  RankPlan p;
  p.stage_bytes = 256u << q.max_depth;
  p.stages = std::min(tb::kRWMaxStages, (f->max_smem_optin - tb::rank_walk_smem_bytes(S, 0, 0)) / (int)p.stage_bytes);
  p.smem = tb::rank_walk_smem_bytes(S, p.stages, p.stage_bytes);
  auto group_clocks = [&](int batch_units) {
    return std::max(1.15 * tb::kRWUnitRows * batch_units * (2 * q.max_depth - 1) + 60.0 * q.max_depth + 200.0, p.stage_bytes / 70.0);
  };
  auto set = [&](int64_t grid_x, int chunks) {
    p.grid_x = grid_x;
    p.per_chunk = (parts + chunks - 1) / chunks;
    p.chunks = (parts + p.per_chunk - 1) / p.per_chunk;
    p.units = (int)std::min<int64_t>(tb::kRWBatchUnits, (units + grid_x - 1) / grid_x);
  };
  // one chunk, as many blocks as there are units or SMs
  const int64_t whole_x = std::min<int64_t>(units, f->num_sms);
  const int64_t whole_units = (units + whole_x - 1) / whole_x;
  double best = 4000.0 + (double)G * ((double)(whole_units / 4) * group_clocks(4) + (whole_units % 4 ? group_clocks((int)(whole_units % 4)) : 0.0));
  set(whole_x, 1);
  if (f->user.tree_chunks > 0) {
    if (f->user.tree_chunks > 1) set((units + tb::kRWBatchUnits - 1) / tb::kRWBatchUnits, std::min(parts, f->user.tree_chunks));
    return p;
  }
  for (int u = 1; u <= tb::kRWBatchUnits; ++u) {
    const int64_t x = (units + u - 1) / u;
    for (int c = 2; c <= std::min(parts, 64) && x < f->num_sms; ++c) {
      const int per = (parts + c - 1) / c, chunks = (parts + per - 1) / per;
      const double groups = multi ? (double)G * per / parts + 1.0 : per;
      const double waves = (double)((x * chunks + f->num_sms - 1) / f->num_sms);
      const double cost = waves * (4000.0 + groups * group_clocks(u)) + kCombineClocks;
      if (cost < best) {
        best = cost;
        set(x, c);
      }
    }
  }
  return p;
}

RankPlan plan_rank(tbk_forest *f, int64_t n_rows, bool leaf_ids) { // (a server's batches are mostly alike)
  if (f->rank_plan_rows != n_rows || f->rank_plan_ids != leaf_ids) {
    f->rank_plan = rank_tiled(f->rf.num_features) ? make_rank_tiles_plan(f, n_rows) : make_rank_plan(f, n_rows, leaf_ids);
    f->rank_plan_rows = n_rows;
    f->rank_plan_ids = leaf_ids;
  }
  return f->rank_plan;
}

// Walker warps of a launch over `n_rows` rows.  A batch of less than a unit gets only as many as the rows
// -- or ranking them with two values per thread -- can use.
int rank_walkers(const tbk_forest *f, const RankPlan &r, int64_t n_rows) {
  if (r.quads) return r.walkers;
  if (n_rows >= tb::kRWUnitRows) return tb::kRWWalkers;
  return (int)std::min<int64_t>(tb::kRWWalkers, std::max((n_rows + 3) / 4, (n_rows * f->rf.num_features + 63) / 64));
}

tb::LaunchPlan rank_launch_plan(const RankPlan &r, int walkers) {
  tb::LaunchPlan plan;
  plan.row_warps = r.quads ? r.quads : walkers;
  plan.rows_per_block = r.quads ? 32 * r.tiles * r.quads : 4 * walkers * r.units;
  plan.tree_threads = walkers / plan.row_warps;
  plan.rows_per_lane = 1;
  plan.chunks = r.chunks;
  plan.groups_per_chunk = r.per_chunk;
  plan.staged = 1;
  plan.cache_rows = 1;
  plan.stage_bytes = r.stage_bytes;
  plan.smem_bytes = r.smem;
  plan.threads = 32 * (walkers + 2);
  plan.grid_x = r.grid_x;
  return plan;
}

// Rows per pass: the keys of a pass stay in L2 between the two kernels, and a pass of several
// chunks has an arrival counter for every row batch.
int64_t rank_rows_per_pass(const tbk_forest *f) {
  const int64_t by_keys = ((int64_t)96 << 20) / rank_stride(f->rf.num_features);
  const int64_t round = tb::rank_bytes(f->rf.num_features)   ? (int64_t)64 * f->num_sms
                        : rank_tiled(f->rf.num_features) ? (int64_t)128 * f->num_sms : (int64_t)tb::kRWBatchRows * f->num_sms;
  return std::max(round, by_keys / round * round);
}

size_t rank_key_bytes(const tbk_forest *f, int64_t rows) { // (whole tiles)
  return ((size_t)((rows + 31) / 32 * 32) * rank_stride(f->rf.num_features) + 255) / 256 * 256;
}
size_t rank_workspace_bytes(const tbk_forest *f, const RankPlan &plan, int64_t rows) {
  size_t bytes = tb::kRankArrivalBytes + rank_key_bytes(f, rows);
  if (plan.chunks > 1) bytes += (size_t)plan.chunks * rows * (f->rf.num_classes > 0 ? 8 : 4);
  return bytes;
}

tb::RankRowsParams rank_rows_params(const tbk_forest *f, const float *rows, int64_t n, int64_t ld, uint16_t *keys) {
  const auto &q = f->rf;
  const int F = q.num_features;
  tb::RankRowsParams p{};
  p.rows = rows;
  p.n_rows = n;
  p.ld = ld;
  p.features = f->d_rfeatures;
  p.lut = f->d_rlut;
  p.thr = f->d_rthr;
  p.keys = keys;
  p.num_features = F;
  p.stride = rank_stride(F);
  p.vec4_ok = F % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(rows) & 15) == 0;
  p.lattice = q.lattice;
  p.bytes = tb::rank_bytes(F);
  p.searched = f->d_ties;
  p.used = f->rank_used;
  return p;
}

template <bool BYTES, bool LATTICE> void (*pick_rank_slabs(int steps))(const tb::SlabParams) {
  return steps == 1   ? tb::tb_rank_slabs<BYTES, 1, LATTICE>
         : steps == 2 ? tb::tb_rank_slabs<BYTES, 2, LATTICE>
         : steps == 3 ? tb::tb_rank_slabs<BYTES, 3, LATTICE>
                      : tb::tb_rank_slabs<BYTES, 0, LATTICE>;
}

// Tables in shared memory pay from here on (see launch_rank_rows).
bool slab_batch(const tbk_forest *f, int64_t n, int num_features) { return n * num_features > (int64_t)f->num_sms * 2048; }

// The kernel that ranks `n` rows into `keys`.
int launch_rank_rows(tbk_forest *f, const float *rows, int64_t n, int64_t ld, uint16_t *keys, cudaStream_t stream) {
  const int F = f->rf.num_features;
  tb::RankRowsParams p = rank_rows_params(f, rows, n, ld, keys);
  const bool pair = F <= tb::kRankPairFeatures, tiled = rank_tiled(F);
  const int64_t lines = pair ? (n + 1) / 2 : tiled ? (n + 31) / 32 * 32 : n;
  if (f->slab_bytes > 0 && slab_batch(f, n, F) && ld < (int64_t)1 << 25) {
    f->last_ran |= TBK_RAN_SLABS;
    tb::SlabParams sp{};
    sp.rows = rows;
    sp.n_rows = n;
    sp.ld_bytes = 4u * (uint32_t)ld;
    sp.tables = reinterpret_cast<const unsigned char *>(f->d_rslabs);
    sp.keys = reinterpret_cast<unsigned char *>(keys);
    sp.table_bytes = f->slab_bytes;
    sp.buckets = f->slab_buckets;
    sp.tile_bytes = 32u * (uint32_t)rank_stride(F);
    sp.num_features = F;
    sp.steps = f->slab_steps;
    sp.searched = f->d_ties;
    sp.used = f->rank_used;
    sp.status = f->d_status;
    sp.skip_copy = f->expire_next_wait ? 1 : 0;
    sp.wait_tries = f->expire_next_wait ? 2000u : 0u;
    f->expire_next_wait = false;
    const int slabs = (F + 31) / 32;
    // segments of the tiles: the last wave of blocks nearly full, at about 230 clocks a tile and 3000 for a block's start
    const int64_t tiles = (n + 31) / 32;
    int64_t segments = 1;
    double best = -1.0;
    for (int64_t c = 1; c <= std::max<int64_t>(8, f->num_sms / slabs) && c <= tiles; ++c) {
      const double cost = (double)((slabs * c + f->num_sms - 1) / f->num_sms) * ((double)(((tiles + c - 1) / c + 15) / 16 * 16) * 230.0 + 3000.0);
      if (best < 0 || cost < best) {
        best = cost;
        segments = c;
      }
    }
    const int smem = tb::slab_smem_bytes(f->slab_bytes);
    const auto kernel = tb::rank_bytes(F) ? (f->rf.lattice ? pick_rank_slabs<true, true>(f->slab_steps) : pick_rank_slabs<true, false>(f->slab_steps))
                                          : (f->rf.lattice ? pick_rank_slabs<false, true>(f->slab_steps) : pick_rank_slabs<false, false>(f->slab_steps));
    if (const int rc = allow_smem(f, (const void *)kernel)) return rc;
    const dim3 grid((unsigned)slabs, (unsigned)segments);
    kernel<<<grid, 32 * tb::kSlabWarps, smem, stream>>>(sp);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
    return TBK_OK;
  }
  // Tables in shared memory pay once every SM has a few thousand values to rank: loading them
  // takes about as long as ranking 2000 values through L2 (a gather there costs a wavefront per lane).
  if (f->rank_width > 0 && !p.bytes && n * F > (int64_t)f->num_sms * 2048) {
    const int w = f->rank_width, slabs = (F + w * f->rank_pieces - 1) / (w * f->rank_pieces);
    p.pieces = f->rank_pieces;
    p.turn_off = (uint32_t)f->rank_smem;
    const int64_t want = (lines * p.pieces + 1023) / 1024;
    const dim3 grid((unsigned)std::min<int64_t>(want, std::max(1, f->num_sms / slabs)), (unsigned)slabs);
    using K = void (*)(const tb::RankRowsParams);
    using tb::kRankPairs, tb::kRankRows, tb::kRankTiles;
    const K k = tiled  ? tb::tb_rank_rows<8, kRankTiles, true>
                : pair ? (w == 4   ? tb::tb_rank_rows<4, kRankPairs, true>
                          : w == 2 ? tb::tb_rank_rows<2, kRankPairs, true>
                                   : tb::tb_rank_rows<1, kRankPairs, true>)
                       : (w == 8   ? tb::tb_rank_rows<8, kRankRows, true>
                          : w == 4 ? tb::tb_rank_rows<4, kRankRows, true>
                          : w == 2 ? tb::tb_rank_rows<2, kRankRows, true>
                                   : tb::tb_rank_rows<1, kRankRows, true>);
    const int rc = allow_smem(f, (const void *)k);
    if (rc) return rc;
    k<<<grid, 1024, f->rank_smem + (tiled ? tb::kRankTurnBytes : 0), stream>>>(p);
  } else {
    // (one feature per thread: a small batch is all latency)
    p.pieces = F;
    const unsigned grid = (unsigned)std::min<int64_t>((lines * p.pieces + 255) / 256, 8ll * f->num_sms);
    if (tiled) tb::tb_rank_rows<1, tb::kRankTiles, false><<<grid, 256, 0, stream>>>(p);
    else if (pair) tb::tb_rank_rows<1, tb::kRankPairs, false><<<grid, 256, 0, stream>>>(p);
    else tb::tb_rank_rows<1, tb::kRankRows, false><<<grid, 256, 0, stream>>>(p);
  }
  CUDA_TRY(cudaGetLastError());
  ++f->launches;
  return TBK_OK;
}

// How the ranking kernel's tables fit shared memory: the widest piece (features a thread ranks
// together) and then the most pieces per block whose tables fit; rank_width 0: not even one feature's.
void plan_rank_tables(tbk_forest *f) {
  const auto &q = f->rf;
  const int F = q.num_features, room = 185 * 1024; // (beside the ranking kernel's buffers)
  auto bytes = [&](int first, int end) { // tables of the features [first, end)
    size_t b = 0;
    for (int i = first; i < end; ++i)
      b += sizeof(tb::RankFeature) + (q.features[i].buckets + 1 + 7) / 8 * 16 + (q.features[i].n + 3) / 4 * 16;
    return b;
  };
  f->rank_width = 0;
  for (int w = F <= tb::kRankPairFeatures ? 4 : 8; w >= (rank_tiled(F) ? 8 : 1); w /= 2) {
    for (int pieces = (F + w - 1) / w; pieces >= 1; --pieces) {
      size_t most = 0;
      for (int first = 0; first < F; first += w * pieces) most = std::max(most, bytes(first, std::min(F, first + w * pieces)));
      if (most <= (size_t)room) {
        f->rank_width = w;
        f->rank_pieces = pieces;
        f->rank_smem = (int)most;
        return;
      }
    }
  }
}

// fixed: keys and partial sums go to this memory, in as many passes as that takes (tbk_predict_noalloc).
int run_rank(tbk_forest *f, Mode mode, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out, int32_t out_kind,
             float *d_partial, int32_t *d_leaf_ids, cudaStream_t stream, unsigned char *fixed = nullptr, size_t fixed_bytes = 0) {
  const auto &q = f->rf;
  const int S = rank_stride(q.num_features), W = std::max(1, q.num_classes);
  const int kmode = mode == kLeafIds ? tb::kRankLeafIds : q.num_classes > 0 ? tb::kRankClasses : tb::kRankSums;
  int64_t pass = std::min(n_rows, rank_rows_per_pass(f));
  RankPlan plan = plan_rank(f, pass, mode == kLeafIds);
  if (plan.chunks > 1) {
    pass = std::min<int64_t>(pass, (int64_t)tb::kRankArrivals * 64); // (units of at least 64 rows)
    plan = plan_rank(f, pass, mode == kLeafIds);
  }
  while (fixed && rank_workspace_bytes(f, plan, pass) > fixed_bytes) { // (128 rows always fit)
    pass = std::max<int64_t>(128, pass / 256 * 128);
    plan = plan_rank(f, pass, mode == kLeafIds);
  }
  const bool tiled = rank_tiled(q.num_features);
  if (tiled && plan.quads == 0) return fail(TBK_ERR_UNSUPPORTED, "no launch shape holds rank keys of %d features under trees of %d levels", q.num_features, q.max_depth);
  const int walkers = rank_walkers(f, plan, n_rows);
  f->last_plan = rank_launch_plan(plan, walkers);
  tbk_forest::Workspace *ws = nullptr;
  int rc = TBK_OK;
  if (fixed) CUDA_TRY(cudaMemsetAsync(fixed, 0, tb::kRankArrivalBytes, stream)); // (others write it too)
  else rc = workspace_acquire(f, stream, rank_workspace_bytes(f, plan, pass), &ws);
  if (rc) return rc;
  unsigned char *const mem = fixed ? fixed : ws->mem;
  unsigned char *keys = mem + tb::kRankArrivalBytes;
  const bool small = !tiled && plan.units == 1; // one unit of rows per block: the variant for small batches
  const int unit_rows = tiled ? 32 * plan.tiles : 4 * walkers;
  // rows of a small host batch travel with the launch
  const bool inlined = f->inline_rows && small && n_rows * q.num_features <= tb::kRankInline;
  const void *const kernel = tiled ? pick_rank_tiles_kernel(plan.tiles, tb::rank_bytes(q.num_features), mode == kLeafIds)
                                   : pick_rank_kernel(S, small, q.whole_compare != 0, inlined, kmode);
  rc = allow_smem(f, kernel);
  if (rc) return rc;
  tb::RankWalkInlineParams p;
  static_cast<tb::RankWalkParams &>(p) = tb::RankWalkParams{};
  p.node_plane = f->d_rnode;
  p.leaf_plane = reinterpret_cast<const uint32_t *>(f->d_rleaf);
  if (mode == kLeafIds) p.leaf_plane = reinterpret_cast<const uint32_t *>(f->d_rorig);
  p.groups = f->d_rgroups;
  p.tree_index = f->d_rtree_index;
  p.class_begin = f->d_rclass_begin;
  p.keys = keys;
  p.scratch = reinterpret_cast<float *>(keys + rank_key_bytes(f, pass));
  p.arrivals = reinterpret_cast<unsigned int *>(mem);
  p.num_trees = q.num_trees;
  p.num_groups = (int32_t)q.groups.size();
  p.groups_per_chunk = kmode == tb::kRankClasses ? 0 : plan.per_chunk;
  p.num_classes = q.num_classes;
  p.classes_per_chunk = kmode == tb::kRankClasses ? plan.per_chunk : 0;
  p.write_partial = mode == kPartial ? 1 : 0;
  p.out_kind = out_kind == TBK_OUT_I8 ? 1 : 0;
  p.transform = q.transform;
  p.initial_value = (float)q.initial_value;
  p.uniform_depth = f->uniform_depth;
  p.quads = plan.quads;
  p.tile_bytes = 32 * S;
  p.stages = plan.stages;
  p.stage_bytes = plan.stage_bytes;
  p.status = f->d_status;
  if (f->timing) CUDA_TRY(cudaEventRecord(f->ev0, stream));
  for (int64_t done = 0; done < n_rows; done += pass) {
    const int64_t n = std::min(pass, n_rows - done);
    const int64_t units = (n + unit_rows - 1) / unit_rows; // (chunks: at most four units to a block)
    const int64_t batches = std::min(units, plan.grid_x);
    // A couple of values per walker thread: the walk ranks its rows itself.  (Every chunk's blocks
    // read the rows again, which host memory is too slow for.)
    const int64_t block_rows = std::min<int64_t>(n, (int64_t)plan.units * unit_rows);
    const bool fused = !tiled && pass == n_rows && plan.units < tb::kRWBatchUnits && block_rows * q.num_features <= 32 * tb::kRankInside * walkers &&
                       (!f->inline_rows || inlined || plan.chunks == 1);
    if (fused) {
      p.ranking = rank_rows_params(f, d_rows, n, ld, nullptr);
      for (int64_t r = 0; inlined && r < n; ++r)
        std::memcpy(p.inline_rows + r * q.num_features, f->inline_rows + r * ld, (size_t)q.num_features * 4);
    } else {
      rc = launch_rank_rows(f, d_rows + done * ld, n, ld, reinterpret_cast<uint16_t *>(keys), stream);
      if (rc) return rc;
    }
    p.n_rows = n;
    p.partial = d_partial ? d_partial + done * W : nullptr;
    p.out = d_out ? static_cast<unsigned char *>(d_out) + done * (out_kind == TBK_OUT_I8 ? 1 : 4) : nullptr;
    p.leaf_ids = d_leaf_ids ? d_leaf_ids + done * q.num_trees : nullptr;
    p.skip_first_copy = f->expire_next_wait ? 1 : 0;
    p.wait_tries = f->expire_next_wait ? 2000u : 0u;
    f->expire_next_wait = false;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)batches, (unsigned)plan.chunks);
    cfg.blockDim = dim3(32u * (unsigned)(walkers + 2));
    cfg.dynamicSmemBytes = (size_t)plan.smem;
    cfg.stream = stream;
    // the walk starts its tree copies while the rows are still being ranked
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = fused ? 0 : 1;
    void *args[] = {&p}; // (of which a kernel takes its own type's bytes)
    CUDA_TRY(cudaLaunchKernelExC(&cfg, kernel, args));
    ++f->launches;
  }
  if (f->timing) {
    CUDA_TRY(cudaEventRecord(f->ev1, stream));
    f->ev_pending = true;
  }
  return ws ? workspace_release(f, ws, stream) : TBK_OK;
}

// ---------------------------------------------------------------------------
// Lane layout (lane_pack.h)

struct LanePlan {
  int tiles = 1, shares = 1, chunks = 1, smem = 0;
  int64_t grid_x = 1;
};

// Enough warps for 48 on every SM, where there are that many: row tiles first, then shares of the
// trees within a block (at least four trees each, or a class), then further chunks of them.  Batches
// that leave most warps' places empty even so are one chain of loads: fewer trees to a share, and
// the tiles go to as many SMs as there are (1146 rows, 25 trees of 13 levels: a call took 9.6 us
// with 9 blocks and 6 trees in turn, 6.0 with 36 blocks and 2 trees).
LanePlan plan_lanes(const tbk_forest *f, int64_t n_rows, bool leaf_ids) {
  const auto &pk = f->packed;
  const int64_t tiles = (n_rows + 31) / 32, wanted = std::max<int64_t>(1, 48ll * f->num_sms / tiles);
  const bool classes = pk.num_classes > 0 && !leaf_ids;
  const int64_t parts = classes ? pk.num_classes : std::max<int64_t>(1, pk.num_trees / 4);
  int64_t most = parts;
  if (!classes)
    for (int per = 2; per >= 1 && tiles * most < 16ll * f->num_sms; per /= 2) most = std::max<int64_t>(1, pk.num_trees / per);
  LanePlan p;
  while (p.shares < 16 && p.shares < wanted && 2 * p.shares <= most) p.shares *= 2;
  if (classes && p.shares < wanted) p.shares = (int)std::min<int64_t>({16, wanted, most}); // (a class each, where they fit)
  p.tiles = (int)std::min<int64_t>(std::max<int64_t>(1, tiles / f->num_sms), 16 / p.shares);
  auto bytes = [&] { return p.tiles * (pk.num_features + 1) * 128 + p.tiles * p.shares * 256; };
  while (p.tiles > 1 && bytes() > 48 * 1024) --p.tiles;
  p.smem = bytes();
  p.grid_x = (tiles + p.tiles - 1) / p.tiles;
  // (chunks of a multiclass forest take a part of every class each)
  const int64_t chunks = classes ? pk.num_trees / pk.num_classes / 4 : (parts >= 2 * p.shares ? most : parts) / p.shares;
  p.chunks = (int)std::min({(wanted + p.shares - 1) / p.shares, std::max<int64_t>(1, chunks), (int64_t)64});
  if (f->user.tree_chunks > 0 && !classes) p.chunks = (int)std::min<int64_t>(f->user.tree_chunks, std::max<int64_t>(1, pk.num_trees / p.shares));
  return p;
}

tb::LaunchPlan lane_launch_plan(const LanePlan &l) {
  tb::LaunchPlan plan;
  plan.row_warps = l.tiles;
  plan.tree_threads = l.shares;
  plan.chunks = l.chunks;
  plan.smem_bytes = l.smem;
  plan.threads = 32 * l.tiles * l.shares;
  plan.grid_x = l.grid_x;
  return plan;
}

// fixed: the partial sums go to this memory, whatever the number of chunks (tbk_predict_noalloc).
int run_lanes(tbk_forest *f, Mode mode, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out, int32_t out_kind,
              float *d_partial, int32_t *d_leaf_ids, cudaStream_t stream, float *fixed = nullptr, size_t fixed_floats = 0) {
  const auto &pk = f->packed;
  const int W = std::max(1, pk.num_classes);
  const bool classes = pk.num_classes > 0;
  // (a chunk of a host batch is walked in the shape of the whole batch, see run)
  LanePlan plan = plan_lanes(f, std::max(n_rows, f->host_batch_rows), mode == kLeafIds);
  if (fixed && classes) plan.chunks = (int)std::max<int64_t>(1, std::min<int64_t>(plan.chunks, (int64_t)fixed_floats / (n_rows * W)));
  plan.grid_x = ((n_rows + 31) / 32 + plan.tiles - 1) / plan.tiles;
  f->last_plan = lane_launch_plan(plan);
  const bool second_pass = fixed != nullptr || (mode != kLeafIds && plan.chunks > 1);
  float *partial = d_partial;
  tbk_forest::Workspace *ws = nullptr;
  if (fixed) {
    partial = fixed;
    if ((size_t)plan.chunks * n_rows * W > fixed_floats)
      return fail(TBK_ERR_UNSUPPORTED, "tbk_predict_noalloc: %lld rows x %d tree chunks x %d outputs need %zu partial sums, the fixed "
                  "scratch holds %zu; split the batch or use tbk_predict", (long long)n_rows, plan.chunks, W,
                  (size_t)plan.chunks * n_rows * W, fixed_floats);
  } else if (second_pass) {
    const int rc = partials_acquire(f, stream, (size_t)plan.chunks * n_rows * W, &partial, &ws);
    if (rc) return rc;
  }
  tb::LaneParams p{};
  p.nodes = f->d_lnodes;
  p.root = f->d_lroot;
  p.tree_index = f->d_ltree_index;
  p.orig_node = f->d_lorig;
  p.class_end = f->d_lclass_end;
  p.class_tree = f->d_lclass_tree;
  p.rows = d_rows;
  p.n_rows = n_rows;
  p.ld = ld;
  p.partial = partial;
  p.out = d_out;
  p.leaf_ids = d_leaf_ids;
  p.num_trees = pk.num_trees;
  p.num_features = pk.num_features;
  p.num_classes = pk.num_classes;
  p.transform = pk.transform;
  p.out_kind = out_kind == TBK_OUT_I8 ? 1 : 0;
  p.write_partial = mode == kPartial || second_pass ? 1 : 0;
  p.initial_value = (float)pk.initial_value;
  p.tiles = plan.tiles;
  p.shares = plan.shares;
  p.vec4_ok = (pk.num_features % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(d_rows) & 15) == 0) ? 1 : 0;
  using K = void (*)(const tb::LaneParams);
  const bool longer = (classes ? (f->lane_class_trees + plan.chunks - 1) / plan.chunks
                               : (pk.num_trees + plan.shares * plan.chunks - 1) / (plan.shares * plan.chunks)) > tb::kLaneShortChain;
  const K k = mode == kLeafIds ? (classes ? tb::tb_walk_lanes_kernel<true, true, false> : tb::tb_walk_lanes_kernel<false, true, false>)
              : classes        ? (longer ? tb::tb_walk_lanes_kernel<true, false, true> : tb::tb_walk_lanes_kernel<true, false, false>)
                               : (longer ? tb::tb_walk_lanes_kernel<false, false, true> : tb::tb_walk_lanes_kernel<false, false, false>);
  int rc = allow_smem(f, (const void *)k);
  if (rc) return rc;
  if (f->timing) CUDA_TRY(cudaEventRecord(f->ev0, stream));
  k<<<dim3((unsigned)plan.grid_x, (unsigned)plan.chunks), f->last_plan.threads, plan.smem, stream>>>(p);
  CUDA_TRY(cudaGetLastError());
  ++f->launches;
  if (second_pass) {
    const int tpb = 256;
    if (mode == kPartial)
      tb::tb_sum_partials_kernel<<<(unsigned)((n_rows * W + tpb - 1) / tpb), tpb, 0, stream>>>(partial, plan.chunks, n_rows * W, d_partial);
    else
      tb::tb_finalize_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, stream>>>(
          partial, plan.chunks, n_rows, W, pk.num_classes, (float)pk.initial_value, pk.transform, d_out, out_kind);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
  }
  if (f->timing) {
    CUDA_TRY(cudaEventRecord(f->ev1, stream));
    f->ev_pending = true;
  }
  return ws ? workspace_release(f, ws, stream) : TBK_OK;
}

// One prediction over device-resident rows.
int run(tbk_forest *f, Mode mode, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out,
        int32_t out_kind, float *d_partial, int32_t *d_leaf_ids, cudaStream_t stream) {
  const auto &pk = f->packed;
  if (n_rows < 0 || ld < pk.num_features) return fail(TBK_ERR_INVALID, "ld (%lld) is smaller than the row size (%d)", (long long)ld, pk.num_features);
  if (n_rows == 0) return TBK_OK;
  if (!d_rows) return fail(TBK_ERR_INVALID, "null input pointer");
  if (mode == kPredict) {
    if (!d_out) return fail(TBK_ERR_INVALID, "null output pointer");
    if (out_kind == TBK_OUT_I8 && pk.num_classes == 0) return fail(TBK_ERR_INVALID, "int8 output needs a multiclass forest");
    if (out_kind != TBK_OUT_F32 && out_kind != TBK_OUT_I8) return fail(TBK_ERR_INVALID, "unknown output kind %d", out_kind);
  }
  CUDA_TRY(cudaSetDevice(f->device));
  f->last_ran = 0;
  if (f->rank) return run_rank(f, mode, d_rows, n_rows, ld, d_out, out_kind, d_partial, d_leaf_ids, stream);
  if (f->lanes) return run_lanes(f, mode, d_rows, n_rows, ld, d_out, out_kind, d_partial, d_leaf_ids, stream);
  if (f->quant) return run_quant(f, mode, d_rows, n_rows, ld, d_out, out_kind, d_partial, d_leaf_ids, stream);
  if (f->deep) return run_deep(f, mode, d_rows, n_rows, ld, d_out, d_partial, d_leaf_ids, stream);

  tb::ForestShape shape{pk.num_features, pk.num_classes, (int64_t)pk.groups.size(), pk.max_group_bytes,
                        (int32_t)pk.lut.size(), pk.representation, pk.tile_size};
  tb::LaunchPlan plan;
  // (a chunk of a host batch is walked in the shape of the whole batch: its sums then have the
  // order, and so every bit, of the same batch in device memory)
  std::string why = tb::select_launch(shape, f->user, std::max(n_rows, f->host_batch_rows), f->max_smem_optin, f->num_sms,
                                      mode == kLeafIds, &plan, mode == kPartial);
  if (!why.empty()) return fail(TBK_ERR_UNSUPPORTED, "%s", why.c_str());
  const int64_t rows_per_block = (int64_t)plan.row_warps * 32 * plan.rows_per_lane;
  plan.grid_x = (n_rows + rows_per_block - 1) / rows_per_block;
  f->last_plan = plan;

  const int W = std::max(1, pk.num_classes);
  const bool need_partials = mode == kPartial || (mode == kPredict && plan.chunks > 1);
  float *partial_dst = nullptr;
  tbk_forest::Workspace *ws = nullptr;
  if (mode == kLeafIds) {
    int rc = ensure_orig(f);
    if (rc) return rc;
  } else if (need_partials) {
    if (mode == kPartial && plan.chunks == 1) {
      partial_dst = d_partial;
    } else {
      const int rc = partials_acquire(f, stream, (size_t)plan.chunks * n_rows * W, &partial_dst, &ws);
      if (rc) return rc;
    }
  }

  tb::WalkParams p{};
  p.blob = f->d_blob;
  p.groups = f->d_groups;
  p.tree_class = f->d_tree_class;
  p.tree_index = f->d_tree_index;
  p.orig_node = f->d_orig_node;
  p.orig_off = f->d_orig_off;
  p.lut = f->d_lut;
  p.lut_bytes = (int32_t)pk.lut.size();
  p.rows = d_rows;
  p.n_rows = n_rows;
  p.ld = ld;
  p.partial = partial_dst;
  p.out = d_out;
  p.out_kind = out_kind;
  p.write_partial = need_partials ? 1 : 0;
  p.leaf_ids = mode == kLeafIds ? d_leaf_ids : nullptr;
  p.num_trees = pk.num_trees;
  p.num_groups = (int32_t)pk.groups.size();
  p.groups_per_chunk = plan.groups_per_chunk;
  p.num_features = pk.num_features;
  p.num_classes = pk.num_classes;
  p.transform = pk.transform;
  p.initial_value = (float)pk.initial_value;
  p.row_warps = plan.row_warps;
  p.tree_threads = plan.tree_threads;
  p.stage_bytes = plan.staged ? plan.stage_bytes : 0;
  p.stages = plan.stages;
  p.vec4_ok = (pk.num_features % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(d_rows) & 15) == 0) ? 1 : 0;
  p.status = f->d_status;
  p.skip_first_copy = (f->expire_next_wait && plan.staged) ? 1 : 0;
  p.wait_limit = f->expire_next_wait ? 2000u : 0u;
  f->expire_next_wait = false;
  // the plan's shared-memory size has no class table when class sums live in registers
  if (plan.class_regs && (plan.chunks != 1 || mode == kPartial))
    return fail(TBK_ERR_UNSUPPORTED, "launch plan with register class sums needs a single tree chunk");
  p.class_regs = plan.class_regs;

  const tb::WalkKernel fn = pick_kernel(pk.representation, pk.tile_size, plan, pk.num_features, &f->last_ran);
  if (const int rc = allow_smem(f, (const void *)fn)) return rc;
  if (f->timing) CUDA_TRY(cudaEventRecord(f->ev0, stream));
  dim3 grid((unsigned)plan.grid_x, (unsigned)plan.chunks), block((unsigned)plan.threads);
  fn<<<grid, block, plan.smem_bytes, stream>>>(p);
  CUDA_TRY(cudaGetLastError());
  ++f->launches;
  if (mode == kPredict && plan.chunks > 1) {
    const int tpb = 256;
    tb::tb_finalize_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, stream>>>(
        partial_dst, plan.chunks, n_rows, W, pk.num_classes, (float)pk.initial_value, pk.transform, d_out, out_kind);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
  } else if (mode == kPartial && plan.chunks > 1) {
    const int tpb = 256;
    const long long total = n_rows * W;
    tb::tb_sum_partials_kernel<<<(unsigned)((total + tpb - 1) / tpb), tpb, 0, stream>>>(partial_dst, plan.chunks, total, d_partial);
    CUDA_TRY(cudaGetLastError());
    ++f->launches;
  }
  if (f->timing) {
    CUDA_TRY(cudaEventRecord(f->ev1, stream));
    f->ev_pending = true;
  }
  return ws ? workspace_release(f, ws, stream) : TBK_OK;
}

// (after a synchronisation with the forest's launches)
int check_status(tbk_forest *f) {
  volatile int32_t *word = f->h_status;
  const int32_t st = *word;
  if (st != 0) {
    *word = 0;
    return fail(TBK_ERR_DEVICE_WAIT, "a bounded wait on a bulk copy expired inside the %s kernel (status %d)",
                st == tb::kStatusRanking ? "ranking" : "walk", st);
  }
  return TBK_OK;
}

// Uploads the planes of a 16-bit-key layout (quant_pack.h / deep_pack.h) and fills the
// threshold keys on the device, so that thresholds and row values are quantised by the
// very same arithmetic.
int upload_key_planes(tbk_forest *f, const std::vector<uint32_t> &node, const std::vector<float> &leaf,
                      const std::vector<float> &exact, const std::vector<int32_t> &orig,
                      const std::vector<tb::QuantGroup> &groups, const std::vector<int32_t> &tree_index,
                      const std::vector<float> &lo, const std::vector<float> &scale, int num_features, bool wide) {
  const size_t n = node.size();
  static_assert(sizeof(tb::QuantGroup) == sizeof(tb::DevQuantGroup), "group metadata layout");
  uint32_t dmin = 0xffffffffu, dmax = 0;
  for (const auto &g : groups) {
    dmin = std::min(dmin, g.depth);
    dmax = std::max(dmax, g.depth);
  }
  f->uniform_depth = dmin == dmax ? (int)dmin : 0;
  CUDA_TRY(cudaMalloc(&f->d_qnode, n * 4));
  CUDA_TRY(cudaMalloc(&f->d_qleaf, n * 4));
  CUDA_TRY(cudaMalloc(&f->d_qexact, n * 4));
  CUDA_TRY(cudaMalloc(&f->d_qorig, n * 4));
  CUDA_TRY(cudaMalloc(&f->d_qgroups, groups.size() * sizeof(tb::QuantGroup)));
  CUDA_TRY(cudaMalloc(&f->d_qtree_index, tree_index.size() * 4));
  // lo / scale are read with 16-byte loads: pad to a multiple of 4 entries
  const size_t nf = ((size_t)num_features + 1 + 3) / 4 * 4;
  CUDA_TRY(cudaMalloc(&f->d_qlo, nf * 4));
  CUDA_TRY(cudaMalloc(&f->d_qscale, nf * 4));
  CUDA_TRY(cudaMemset(f->d_qlo, 0, nf * 4));
  CUDA_TRY(cudaMemset(f->d_qscale, 0, nf * 4));
  CUDA_TRY(cudaMalloc(&f->d_ties, 128));
  CUDA_TRY(cudaMemset(f->d_ties, 0, 128));
  CUDA_TRY(cudaMemcpy(f->d_qnode, node.data(), n * 4, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(f->d_qleaf, leaf.data(), n * 4, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(f->d_qexact, exact.data(), n * 4, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(f->d_qorig, orig.data(), n * 4, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(f->d_qgroups, groups.data(), groups.size() * sizeof(tb::QuantGroup), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(f->d_qtree_index, tree_index.data(), tree_index.size() * 4, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(f->d_qlo, lo.data(), lo.size() * 4, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(f->d_qscale, scale.data(), scale.size() * 4, cudaMemcpyHostToDevice));
  tb::tb_quant_fill_keys<<<(unsigned)((n + 255) / 256), 256>>>(f->d_qnode, f->d_qexact, f->d_qlo, f->d_qscale,
                                                             (unsigned long long)n, num_features, wide ? 1 : 0, tb::deep_feature_code(num_features, 1));
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaDeviceSynchronize());
  ++f->launches;
  return TBK_OK;
}

void free_pipeline(tbk_forest *f) {
  cudaFree(f->d_in[0]); // (one block)
  for (int i = 0; i < tbk_forest::kPipeSlots; ++i) {
    pinned_pool().give_back(f->h_pin[i], f->pin_capacity[i]);
    pinned_pool().give_back(f->h_res[i], f->res_capacity[i]);
    f->d_in[i] = f->d_res[i] = f->h_pin[i] = f->h_res[i] = nullptr;
  }
  f->pipe_bytes = f->pipe_rows = 0;
}

bool is_pinned(const void *ptr) {
  cudaPointerAttributes attr{};
  const bool pinned = cudaPointerGetAttributes(&attr, ptr) == cudaSuccess && attr.type == cudaMemoryTypeHost;
  cudaGetLastError();
  return pinned;
}

// Small host batches: everything but the walk itself is latency, so there are no copies to
// enqueue and wait for.  The rows go through one pinned buffer that a ranking kernel reads over
// PCIe (every value once) -- or, up to 256 values, with the launch itself; other kernels read rows
// more than once and get them copied.  Results are written to pinned memory by the kernel that
// computes them, over a value that no prediction has; the call ends when the last one has been
// overwritten, several microseconds before fences in the kernel or the stream's end would tell.
// The status word is mapped host memory as well.
constexpr size_t kSmallRows = (size_t)512 << 10, kSmallDirect = (size_t)128 << 10, kSmallResults = (size_t)512 << 10;
constexpr uint32_t kNoResult = 0x7fa5c3e1u; // as a float: a NaN that no arithmetic returns
constexpr uint8_t kNoClass = 0xff;          // (class ids are at most 126)
int predict_host_small(tbk_forest *f, const float *h_rows, int64_t n_rows, int64_t ld, void *h_out, int32_t out_kind) {
  const size_t bytes = ((size_t)(n_rows - 1) * ld + f->packed.num_features) * 4; // (nothing behind the last row's values)
  const bool classes = out_kind == TBK_OUT_I8;
  const size_t out_bytes = (size_t)n_rows * (classes ? 1 : 4);
  cudaStream_t stream = f->streams[0];
  const size_t results_at = (bytes + 255) / 256 * 256;
  if (f->small_capacity < results_at + out_bytes) {
    pinned_pool().give_back(f->h_small, f->small_capacity);
    f->small_capacity = 0;
    f->h_small = pinned_pool().take(results_at + out_bytes, &f->small_capacity);
    if (!f->h_small) return fail(TBK_ERR_CUDA, "no pinned memory for the batch");
    CUDA_TRY(cudaHostGetDevicePointer(&f->d_small, f->h_small, 0));
  }
  unsigned char *results = f->h_small + results_at;
  if (classes) std::memset(results, kNoClass, out_bytes);
  else std::fill_n(reinterpret_cast<uint32_t *>(results), n_rows, kNoResult);
  copy_past_caches(f->h_small, reinterpret_cast<const unsigned char *>(h_rows), bytes);
  const unsigned char *rows = f->d_small;
  if (!f->rank || bytes > kSmallDirect) {
    if (!f->d_small_in) CUDA_TRY(cudaMalloc(&f->d_small_in, kSmallRows));
    CUDA_TRY(cudaMemcpyAsync(f->d_small_in, f->h_small, bytes, cudaMemcpyHostToDevice, stream));
    rows = f->d_small_in;
  }
  f->inline_rows = h_rows;
  const int rc = run(f, kPredict, reinterpret_cast<const float *>(rows), n_rows, ld, f->d_small + results_at, out_kind, nullptr,
                     nullptr, stream);
  f->inline_rows = nullptr;
  bool idle = rc != TBK_OK;
  for (int64_t r = 0; r < n_rows && !idle; ++r)
    for (int spin = 1; !idle; ++spin) {
      if (classes ? reinterpret_cast<volatile uint8_t *>(results)[r] != kNoClass
                  : reinterpret_cast<volatile uint32_t *>(results)[r] != kNoResult)
        break;
      idle = spin % 1024 == 0 && cudaStreamQuery(stream) != cudaErrorNotReady; // done without it, or an error
    }
  if (idle) {
    const cudaError_t e = cudaStreamSynchronize(stream);
    if (rc != TBK_OK) return rc;
    if (e != cudaSuccess) return fail(TBK_ERR_CUDA, "cudaStreamSynchronize: %s", cudaGetErrorString(e));
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  std::memcpy(h_out, results, out_bytes);
  return check_status(f);
}

// Packs a forest; batch_hint: rows of the batches to come, 0 if that is not known.
int create_image(const tbk_forest_arrays *fa, const tbk_schedule *schedule, int32_t smem_limit, int64_t batch_hint, tbk_image **out);

// Few trees over rows of 326 to 511 features: ranking a row costs about as much as walking it through fp32
// tiles, and takes a launch of its own.  Measured with 4, 6 and 8 levels, 30 to 400 trees over 350, 400, 450 and 500
// features, 100 to 30000 rows, microseconds on rank keys against fp32 tiles: 30 trees of 8 levels x 400 features
// 10.3 / 10.3 at 300 rows, 14.4 / 10.3 at 3000, 22.6 / 17.3 at 10000, 41.9 / 41.0 at 30000; 100 trees x 500 features
// 18.5 / 12.3 at 3000 rows, 30.7 / 30.8 at 10000, 61.7 / 80.2 at 30000; 64 trees x 450 features (no 16-byte loads)
// 18.5 / 16.4 at 3000 rows, 24.6 / 28.7 at 10000.  Of 324 such shapes 79 were slower than on fp32 tiles by more than
// 3 %; with this rule 23 are, and 2 slower than on rank keys.  Without a hint, and below 700 rows, ranks.
bool few_trees(int num_features, int64_t num_trees, int max_depth, int64_t batch_hint) {
  if (batch_hint < 700) return false;
  if (num_features % 4 != 0) return batch_hint >= 1500 && batch_hint < 6000 && 8 * num_trees <= num_features;
  if (batch_hint < 6000) return 4 * num_trees <= num_features;
  if (batch_hint < 20000) return 6 * num_trees <= num_features;
  return 100 * num_trees * max_depth <= 65 * (int64_t)num_features;
}

// Rows of more than 511 features whose features have at most 255 distinct thresholds: one-byte ranks instead of rounded
// keys, where the batches to come are announced (without a hint the layout stays that of images made ahead of time).  Of
// 170 shapes (520 to 2018 features, 100 to 1500 trees of 6 to 8 levels, 1024 to 262144 rows) none is slower by more than 3 %; microseconds
// on rounded keys and on ranks: 300 trees of 6 levels x 520 features 34.9 / 11.8, 55.0 / 19.6, 241.5 / 85.1 for 1024, 8192 and 65536
// rows; 600 trees of 8 levels x 1600 features 40.5 / 14.8, 66.3 / 42.7, 282 / 263; 800 x 1750 394 / 294 and 1000 x 2000 370 / 355 at
// 65536 rows, 1422 / 1401 at 262144 (1076 / 1085 at 200000).  Preparation takes as long in a warm process (1000 trees of 8 levels x 2000
// features 13.9 / 13.4 ms, 400 x 1000 9.1 / 8.7, 100 of 6 levels x 520 2.1 / 2.8); a process's first forest up to 20 ms longer (95 MB for keys).
bool byte_ranks(int64_t batch_hint) { return batch_hint > 0; }

} // namespace

extern "C" {

const char *tbk_last_error(void) { return g_last_error.c_str(); }

int tbk_forest_create(const tbk_forest_arrays *fa, const tbk_schedule *schedule, int32_t device,
                      int64_t batch_hint, tbk_forest **out) {
  if (!out) return fail(TBK_ERR_INVALID, "null argument");
  *out = nullptr;
  int smem_limit = 0;
  CUDA_TRY(cudaSetDevice(device));
  CUDA_TRY(cudaDeviceGetAttribute(&smem_limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
  tbk_image *img = nullptr;
  int rc = create_image(fa, schedule, smem_limit, batch_hint, &img);
  if (rc != TBK_OK) return rc;
  rc = tbk_forest_create_from_image(img, schedule, device, batch_hint, out);
  tbk_image_free(img);
  return rc;
}

int tbk_image_create(const tbk_forest_arrays *fa, const tbk_schedule *schedule, int32_t smem_limit, tbk_image **out) {
  return create_image(fa, schedule, smem_limit, 0, out);
}

} // extern "C"

namespace {
int create_image(const tbk_forest_arrays *fa, const tbk_schedule *schedule, int32_t smem_limit, int64_t batch_hint, tbk_image **out) {
  if (!fa || !out) return fail(TBK_ERR_INVALID, "null argument");
  *out = nullptr;
  if (fa->num_trees <= 0 || !fa->tree_off || !fa->left || !fa->right || !fa->feat || !fa->thr)
    return fail(TBK_ERR_INVALID, "forest arrays are incomplete");
  tb::Forest host;
  const int64_t T = fa->num_trees, N = fa->tree_off[T];
  if (N <= 0) return fail(TBK_ERR_INVALID, "forest has no nodes");
  host.tree_off.assign(fa->tree_off, fa->tree_off + T + 1);
  host.left.assign(fa->left, fa->left + N);
  host.right.assign(fa->right, fa->right + N);
  host.feat.assign(fa->feat, fa->feat + N);
  host.thr.assign(fa->thr, fa->thr + N);
  if (fa->num_classes > 0) {
    if (!fa->class_id) return fail(TBK_ERR_INVALID, "multiclass forest without class ids");
    host.class_id.assign(fa->class_id, fa->class_id + T);
  }
  host.num_classes = fa->num_classes;
  host.transform = fa->transform;
  host.initial_value = fa->initial_value;
  host.num_features = fa->num_features;
  if (fa->num_classes > 0 && fa->num_classes > 127) return fail(TBK_ERR_UNSUPPORTED, "more than 127 classes");
  if (smem_limit <= 0) smem_limit = 227 * 1024;

  std::unique_ptr<tbk_image> img(new tbk_image());
  tb::PackedImage &im = img->im;
  if (schedule) im.user = *schedule;
  im.smem_limit = smem_limit;

  // ---- choose the layout
  const int bits = im.user.feature_bits;
  if (bits != 0 && bits != 16 && bits != 32) return fail(TBK_ERR_INVALID, "feature_bits must be 0, 16 or 32");
  int rep = im.user.representation;
  const int ts = im.user.tile_size <= 0 ? 1 : im.user.tile_size;
  im.requested_representation = rep;
  im.requested_tile_size = ts;
  im.requested_feature_bits = bits;
  // an fp32 tile of 32 rows (plus the sentinel column) must fit beside a little metadata
  const bool fp32_tile_fits = (int64_t)(host.num_features + 1) * 128 + 1024 <= smem_limit;
  {
    const std::string verr = tb::validate(host);
    if (!verr.empty()) return fail(TBK_ERR_INVALID, "%s", verr.c_str());
  }
  int max_depth = 0;
#pragma omp parallel for reduction(max : max_depth) schedule(dynamic, 64) num_threads(tb::pack_threads()) if (N > 1 << 15)
  for (int64_t t = 0; t < T; ++t) max_depth = std::max(max_depth, (int)tb::tree_depth(host, t));
  // narrow rows: the key tiles of at least four 32-row tiles fit beside the ring, so the batch
  // kernel applies; measured faster than the fp32 walk on single-output forests of up to 8 levels
  const bool batch_fits =
      (smem_limit - tb::kQBBarBytes - tb::kQBRingBytes) / tb::quant_batch_tile_bytes(host.num_features) >= 4;
  // (multiclass forests too: one walker set per class, arg-max or per-class sums in the leaf warps)
  bool want_quant = (bits == 16 && max_depth <= tb::kQuantMaxDepth && (host.num_classes == 0 || batch_fits)) ||
                    (bits == 0 && (rep == TBK_REP_AUTO || rep == TBK_REP_REORG) && ts == 1 && !fp32_tile_fits &&
                     host.num_classes == 0) ||
                    (bits == 0 && rep == TBK_REP_AUTO && ts == 1 && max_depth <= tb::kQuantMaxDepth &&
                     (batch_fits || (host.num_features > tb::kRankMaxFeatures && host.num_classes == 0)));
  // (rows too wide for rank keys: the one-tile kernel; on fp32 tiles of 32 rows, one per block, 98431 rows
  // of 1303 features took 3.3 ms)
  // rank keys: whatever the key kernels would take, over at most kRankMaxFeatures features
  const bool tiles_do = bits == 0 && !batch_fits && fp32_tile_fits && host.num_classes == 0 &&
                        few_trees(host.num_features, T, max_depth, batch_hint);
  const bool want_rank =
      want_quant || (bits == 0 && rep == TBK_REP_AUTO && ts == 1 && max_depth <= tb::kRankMaxDepth && !tiles_do);
  const bool bytes_do = !tb::rank_bytes(host.num_features) || (bits == 0 && byte_ranks(batch_hint));
  if (want_rank && bytes_do && host.num_features <= tb::kRankMaxByteFeatures && rank_fits(host.num_features, max_depth, smem_limit)) {
    if (tb::pack_rank(host, &im.rf).empty()) {
      im.kind = tb::PackedImage::kRank;
      im.user.representation = TBK_REP_REORG;
      *out = img.release();
      return TBK_OK;
    }
    im.rf = tb::RankForest(); // (a feature with too many distinct thresholds, for one)
  }
  if (want_quant) {
    // narrow rows (batch kernel): features with whole-number thresholds become lattice features
    std::string qerr = tb::pack_quant(host, &im.qf, batch_fits);
    // Whole-number thresholds that could not be put on a lattice (a feature with other
    // thresholds too, or wide rows) mean integer-valued features whose rows tie with thresholds
    // all the time (measured: one comparison in 16 on 4-bit features, the key walk then runs at
    // a quarter of the fp32 walk's rate): such forests keep fp32 tiles unless keys were asked for.
    if (qerr.empty() && bits == 0 && fp32_tile_fits && 2 * im.qf.whole_number_splits > im.qf.num_splits)
      qerr = "integer-valued features";
    if (qerr.empty() && !batch_fits && quant_smem_bytes(host.num_features) > smem_limit)
      qerr = "rows are too wide for the 16-bit key tile";
    if (qerr.empty() && im.qf.node_plane.size() >= (1ull << 32))
      qerr = "forest too large for the 16-bit key layout (2^32 plane elements)";
    if (!qerr.empty()) {
      if (bits == 16) return fail(TBK_ERR_UNSUPPORTED, "%s", qerr.c_str());
      want_quant = false;
      im.qf = tb::QuantForest();
    }
  }
  // ---- deep trees: whole-tree stages over a key tile (deep_pack.h); not chosen for forests
  // whose thresholds are mostly whole numbers on features that cannot be lattice features
  // (integer-valued features then tie on every equality)
  bool deep_ok = !want_quant && host.num_classes == 0 && ts == 1 && bits != 32 &&
                 (bits == 16 || im.user.representation == TBK_REP_AUTO);
  if (deep_ok && bits == 0 && max_depth > tb::kQuantMaxDepth) {
    std::vector<float> lo, scale; // a negative scale marks a lattice feature
    if (tb::quant_feature_ranges(host, tb::kKey15Span, &lo, &scale, true).empty()) {
      int64_t splits = 0, whole = 0;
#pragma omp parallel for reduction(+ : splits, whole) schedule(static) num_threads(tb::pack_threads())
      for (int64_t g = 0; g < host.num_nodes(); ++g)
        if (!host.is_leaf(g)) {
          ++splits;
          whole += host.thr[g] == std::floor(host.thr[g]) && !(scale[host.feat[g]] < 0.f) ? 1 : 0;
        }
      deep_ok = 2 * whole <= splits;
    }
  }
  if (deep_ok) {
    int rw = 0, slots = 0;
    const bool fits = max_depth > tb::kQuantMaxDepth && max_depth <= tb::kDeepMaxDepth &&
                      deep_plan(host.num_features, max_depth, smem_limit, &rw, &slots);
    if (fits) {
      std::string derr = tb::pack_deep(host, &im.df);
      if (derr.empty()) {
        im.kind = tb::PackedImage::kDeep;
        im.deep_row_warps = rw;
        im.deep_slots = slots;
        im.user.representation = TBK_REP_REORG;
        *out = img.release();
        return TBK_OK;
      }
      if (bits == 16) return fail(TBK_ERR_UNSUPPORTED, "%s", derr.c_str());
      im.df = tb::DeepForest();
    } else if (bits == 16) {
      return fail(TBK_ERR_UNSUPPORTED, "16-bit feature keys: neither key layout fits this forest (depth %d, %d features)",
                  max_depth, host.num_features);
    }
  }
  if (bits == 16 && !want_quant)
    return fail(TBK_ERR_UNSUPPORTED, "16-bit feature keys cover single-output forests of at most %d levels and multiclass "
                                     "forests of at most %d levels over narrow rows, tile size 1 "
                                     "(this forest: %d levels, %d classes, %d features, tile size %d)",
                tb::kDeepMaxDepth, tb::kQuantMaxDepth, max_depth, host.num_classes, host.num_features, ts);
  if (rep == TBK_REP_AUTO) rep = TBK_REP_SPARSE;
  if (want_quant) {
    im.kind = tb::PackedImage::kQuant;
    im.user.representation = TBK_REP_REORG;
    *out = img.release();
    return TBK_OK;
  }
  // trees deeper than the key layouts reach (or than a shared-memory stage of tree groups could
  // hold), layout left to the library: nodes in global memory, every lane at its own pace
  if (im.user.representation == TBK_REP_AUTO && bits == 0 && ts == 1 && max_depth > tb::kQuantMaxDepth &&
      im.user.cache_trees != 1 && (host.num_features + 1) * 128 <= 96 * 1024 && tb::pack_lanes(host, &im.lf).empty()) {
    im.kind = tb::PackedImage::kLanes;
    im.user.representation = rep;
    *out = img.release();
    return TBK_OK;
  }
  im.lf = tb::LaneForest();
  tb::PackOptions opt;
  opt.representation = rep;
  opt.tile_size = ts;
  im.user.representation = rep;
  std::string err = tb::pack_forest(host, opt, &im.packed);
  if (!err.empty()) return fail(TBK_ERR_INVALID, "%s", err.c_str());
  im.kind = tb::PackedImage::kGeneral;
  *out = img.release();
  return TBK_OK;
}

} // namespace

extern "C" {

int tbk_image_free(tbk_image *img) {
  delete img;
  return TBK_OK;
}

int tbk_image_serialize(const tbk_image *img, void *buffer, uint64_t capacity, uint64_t *size) {
  if (!img || !size) return fail(TBK_ERR_INVALID, "null argument");
  *size = tb::serialized_image_size(img->im);
  if (!buffer) return TBK_OK;
  if (capacity < *size) return fail(TBK_ERR_INVALID, "buffer of %llu bytes, the image needs %llu",
                                    (unsigned long long)capacity, (unsigned long long)*size);
  std::vector<uint8_t> bytes;
  tb::serialize_image(img->im, &bytes);
  std::memcpy(buffer, bytes.data(), bytes.size());
  return TBK_OK;
}

int tbk_image_deserialize(const void *buffer, uint64_t size, tbk_image **out) {
  if (!buffer || !out) return fail(TBK_ERR_INVALID, "null argument");
  *out = nullptr;
  std::unique_ptr<tbk_image> img(new tbk_image());
  const std::string err = tb::deserialize_image(static_cast<const uint8_t *>(buffer), size, &img->im);
  if (!err.empty()) return fail(TBK_ERR_IO, "%s", err.c_str());
  // (not every width below kRankMaxByteFeatures has a launch shape under every depth; an image made here has one)
  const tb::RankForest &q = img->im.rf;
  if (img->im.kind == tb::PackedImage::kRank && !rank_fits(q.num_features, q.max_depth, img->im.smem_limit))
    return fail(TBK_ERR_UNSUPPORTED, "packed image: no launch shape holds rank keys of %d features under trees of %d levels in %d bytes "
                                     "of shared memory", q.num_features, q.max_depth, img->im.smem_limit);
  *out = img.release();
  return TBK_OK;
}

int tbk_image_matches(const tbk_image *img, const tbk_schedule *schedule, int32_t smem_limit) {
  if (!img) return 0;
  tbk_schedule want{};
  if (schedule) want = *schedule;
  const tb::PackedImage &im = img->im;
  const int ts = want.tile_size <= 0 ? 1 : want.tile_size;
  if (smem_limit <= 0) smem_limit = 227 * 1024;
  return im.requested_representation == want.representation && im.requested_tile_size == ts &&
         im.requested_feature_bits == want.feature_bits && im.smem_limit == smem_limit;
}

int tbk_forest_create_from_image(const tbk_image *img, const tbk_schedule *schedule, int32_t device,
                                 int64_t batch_hint, tbk_forest **out) {
  if (!img || !out) return fail(TBK_ERR_INVALID, "null argument");
  *out = nullptr;
  const tb::PackedImage &im = img->im;
  auto *f = new tbk_forest();
  pinned_pool().attach();
  f->user = im.user;
  if (schedule) { // launch-shape requests of the caller; the layout is the image's
    f->user.rows_per_block = schedule->rows_per_block;
    f->user.rows_per_thread = schedule->rows_per_thread;
    f->user.tree_threads = schedule->tree_threads;
    f->user.tree_chunks = schedule->tree_chunks;
    f->user.cache_trees = schedule->cache_trees;
  }
  f->batch_hint = batch_hint;
  f->device = device;
  auto bail = [&](int rc) {
    tbk_forest_free(f);
    return rc;
  };
#define CUDA_TRY_F(expr)                                                                   \
  do {                                                                                     \
    cudaError_t e__ = (expr);                                                              \
    if (e__ != cudaSuccess)                                                                \
      return bail(fail(TBK_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e__)));    \
  } while (0)
  auto done = [&]() { // (calls may come on streams that nothing orders behind the uploads)
    if (const int rc = uploads_done()) return bail(rc);
    *out = f;
    return (int)TBK_OK;
  };
  CUDA_TRY_F(cudaSetDevice(device));
  CUDA_TRY_F(cudaDeviceGetAttribute(&f->max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
  CUDA_TRY_F(cudaDeviceGetAttribute(&f->num_sms, cudaDevAttrMultiProcessorCount, device));
  if (im.smem_limit > f->max_smem_optin)
    return bail(fail(TBK_ERR_UNSUPPORTED, "the packed image was laid out for %d bytes of shared memory per block, this device has %d",
                     im.smem_limit, f->max_smem_optin));
  f->h_status = pinned_pool().take_status();
  if (!f->h_status) return bail(fail(TBK_ERR_CUDA, "no pinned memory for the status word"));
  CUDA_TRY_F(cudaHostGetDevicePointer(&f->d_status, f->h_status, 0));
  CUDA_TRY_F(cudaEventCreate(&f->ev0));
  CUDA_TRY_F(cudaEventCreate(&f->ev1));

  if (im.kind == tb::PackedImage::kDeep) {
    f->df = im.df; // (metadata and planes; the planes' host copies are dropped after the upload)
    auto &q = f->df;
    f->deep = true;
    f->deep_row_warps = im.deep_row_warps;
    f->deep_slots = im.deep_slots;
    f->packed.representation = tb::kReorg;
    f->packed.tile_size = 1;
    f->packed.num_features = q.num_features;
    f->packed.transform = q.transform;
    f->packed.initial_value = q.initial_value;
    f->packed.num_trees = q.num_trees;
    f->packed.num_nodes = q.num_nodes;
    f->packed.max_depth = q.max_depth;
    int urc = upload_key_planes(f, q.node_plane, q.leaf_plane, q.exact_plane, q.orig_leaf, q.pairs, q.tree_index,
                                q.lo, q.scale, q.num_features, false);
    if (urc != TBK_OK) return bail(urc);
    // (where it costs no row warps: 150000 rows of 200 features, 600 trees of 12 levels, 10 of them instead of 12: 946 -> 1117 us)
    if (f->uniform_depth >= 9 && q.num_features <= tb::kDeepNarrowFeatures &&
        deep_staged_plan(q.num_features, f->uniform_depth, f->max_smem_optin, &f->deep_staged_warps, &f->deep_staged_slots) &&
        f->deep_staged_warps >= f->deep_row_warps) {
      const uint32_t half = deep_half_words(f->uniform_depth);
      const long long trees = 2ll * (long long)q.pairs.size(), threads = trees << (f->uniform_depth - 1);
      if (cudaMalloc(&f->d_qsplit, (size_t)trees * 4 * half * 4) != cudaSuccess) {
        cudaGetLastError(); // (no room for the planes a second time: leaf values are gathered)
        f->d_qsplit = nullptr;
      } else {
        tb::tb_deep_split<<<(unsigned)((threads + 255) / 256), 256>>>(f->d_qnode, f->d_qleaf, f->d_qsplit, trees, (uint32_t)f->uniform_depth,
                                                                      q.pairs[0].slots, half);
        CUDA_TRY_F(cudaGetLastError());
        ++f->launches;
      }
    }
    std::vector<uint32_t>().swap(q.node_plane);
    std::vector<float>().swap(q.leaf_plane);
    std::vector<float>().swap(q.exact_plane);
    std::vector<int32_t>().swap(q.orig_leaf);
    tb::LaunchPlan &pl = f->last_plan;
    pl.row_warps = f->deep_row_warps; pl.tree_threads = 1; pl.rows_per_lane = 1; pl.chunks = 1; pl.staged = 1; pl.cache_rows = 1;
    pl.stage_bytes = 4u * tb::deep_tree_words((uint32_t)std::max(q.max_depth, tb::kDeepMinDepth)); pl.smem_bytes = deep_smem_bytes(f); pl.threads = 32 * (f->deep_row_warps + 1);
    return done();
  }
  auto upload = [](auto **dst, const auto &v) { // (an empty vector gets a few bytes)
    const size_t bytes = v.size() * sizeof(v[0]);
    cudaError_t e = cudaMalloc((void **)dst, std::max<size_t>(16, bytes));
    if (e == cudaSuccess && bytes) e = cudaMemcpy((void *)*dst, v.data(), bytes, cudaMemcpyHostToDevice);
    return e;
  };
  if (im.kind == tb::PackedImage::kLanes) {
    const auto &q = im.lf;
    f->lanes = true;
    f->packed.representation = tb::kSparse;
    f->packed.tile_size = 1;
    f->packed.num_features = q.num_features;
    f->packed.num_classes = q.num_classes;
    f->packed.transform = q.transform;
    f->packed.initial_value = q.initial_value;
    f->packed.num_trees = q.num_trees;
    f->packed.num_nodes = q.num_nodes;
    f->packed.max_depth = q.max_depth;
    static_assert(sizeof(tb::LaneNode) == sizeof(uint2), "node layout");
    CUDA_TRY_F(upload(&f->d_lnodes, q.nodes));
    CUDA_TRY_F(upload(&f->d_lroot, q.root));
    CUDA_TRY_F(upload(&f->d_ltree_index, q.tree_index));
    CUDA_TRY_F(upload(&f->d_lorig, q.orig_node));
    CUDA_TRY_F(upload(&f->d_lclass_end, q.class_end));
    std::vector<uint32_t> class_tree; // (end of every class's trees)
    for (uint32_t end : q.class_end) class_tree.push_back((uint32_t)(std::lower_bound(q.root.begin(), q.root.end(), end) - q.root.begin()));
    for (size_t c = 0; c < class_tree.size(); ++c)
      f->lane_class_trees = std::max<int64_t>(f->lane_class_trees, class_tree[c] - (c ? class_tree[c - 1] : 0u));
    CUDA_TRY_F(upload(&f->d_lclass_tree, class_tree));
    f->last_plan = lane_launch_plan(plan_lanes(f, batch_hint > 0 ? batch_hint : 65536, false));
    return done();
  }
  if (im.kind == tb::PackedImage::kRank) {
    const auto &q = im.rf;
    f->rank = true;
    f->packed.representation = tb::kReorg;
    f->packed.tile_size = 1;
    f->packed.num_features = q.num_features;
    f->packed.num_classes = q.num_classes;
    f->packed.transform = q.transform;
    f->packed.initial_value = q.initial_value;
    f->packed.num_trees = q.num_trees;
    f->packed.num_nodes = q.num_nodes;
    f->packed.max_depth = q.max_depth;
    static_assert(sizeof(tb::RankFeature) == sizeof(tb::DevRankFeature) && sizeof(tb::RankFeature) == 32, "rank table layout");
    // one block of device memory; what is small goes there in one copy
    {
      struct Part { void **dst; const void *src; size_t bytes, at; };
      std::vector<Part> parts;
      size_t total = 0;
      auto part = [&](auto **dst, const auto &v) {
        parts.push_back({(void **)dst, v.data(), v.size() * sizeof(v[0]), total});
        total += (parts.back().bytes + 255) / 256 * 256 + 256; // (empty vectors get an address too)
      };
      const std::vector<unsigned long long> zeros(16, 0);
      part(&f->d_ties, zeros);
      part(&f->d_rgroups, q.groups);
      part(&f->d_rtree_index, q.tree_index);
      part(&f->d_rclass_begin, q.class_begin);
      part(&f->d_rfeatures, q.features);
      part(&f->d_rlut, q.lut);
      part(&f->d_rthr, q.thresholds);
      const size_t small = total;
      // (one request for shared memory holds a slab's table and the warps' buffers; narrower rows whose batches are announced as too small for slabs need none)
      tb::SlabTables slabs;
      const bool large = batch_hint <= 0 || tb::rank_bytes(q.num_features) || slab_batch(f, batch_hint, q.num_features);
      if (rank_tiled(q.num_features) && large && tb::make_slab_tables(q, (uint32_t)(f->max_smem_optin - tb::slab_smem_bytes(0)), &slabs)) {
        parts.push_back({(void **)&f->d_rslabs, slabs.words.get(), slabs.num_words * 4, total});
        total += (parts.back().bytes + 255) / 256 * 256;
        f->slab_bytes = slabs.bytes;
        f->slab_buckets = slabs.buckets;
        f->slab_steps = slabs.steps;
      }
      part(&f->d_rnode, q.node_plane);
      part(&f->d_rleaf, q.leaf_plane);
      part(&f->d_rorig, q.orig_leaf);
      CUDA_TRY_F(cudaMalloc(&f->d_rank_block, total));
      const bool together = total <= (size_t)1 << 20;
      std::vector<unsigned char> staging(together ? total : small);
      for (const Part &pt : parts) {
        *pt.dst = f->d_rank_block + pt.at;
        if (pt.at < staging.size()) {
          if (pt.bytes) std::memcpy(staging.data() + pt.at, pt.src, pt.bytes);
        } else {
          CUDA_TRY_F(cudaMemcpy(*pt.dst, pt.src, pt.bytes, cudaMemcpyHostToDevice));
        }
      }
      CUDA_TRY_F(cudaMemcpy(f->d_rank_block, staging.data(), staging.size(), cudaMemcpyHostToDevice));
    }
    // of the host copy only the sizes and the feature table stay
    f->rf.num_features = q.num_features;
    f->rf.num_classes = q.num_classes;
    f->rf.transform = q.transform;
    f->rf.initial_value = q.initial_value;
    f->rf.num_trees = q.num_trees;
    f->rf.num_nodes = q.num_nodes;
    f->rf.max_depth = q.max_depth;
    f->rf.lattice = q.lattice;
    f->rf.whole_compare = q.whole_compare;
    f->rf.groups = q.groups;
    f->uniform_depth = (int)q.groups[0].depth;
    for (const auto &g : q.groups)
      if ((int)g.depth != f->uniform_depth) f->uniform_depth = 0;
    f->rf.features = q.features;
    for (const auto &rf : q.features) f->rank_used += rf.n > 0;
    plan_rank_tables(f);
    const int64_t rows = std::min(batch_hint > 0 ? batch_hint : 65536, rank_rows_per_pass(f));
    const RankPlan plan = plan_rank(f, rows, false);
    f->last_plan = rank_launch_plan(plan, rank_walkers(f, plan, rows));
    if (batch_hint > 0) { // the batches to come are known: their workspace is laid out now
      tbk_forest::Workspace &w = f->workspace[0];
      const size_t bytes = rank_workspace_bytes(f, plan, rows);
      CUDA_TRY_F(cudaMalloc(&w.mem, bytes));
      CUDA_TRY_F(cudaMemset(w.mem, 0, tb::kRankArrivalBytes));
      w.bytes = bytes;
    }
    return done();
  }
  if (im.kind == tb::PackedImage::kQuant) {
    f->qf = im.qf;
    const auto &q = f->qf;
    f->quant = true;
    // metadata shared with the generic entry points
    f->packed.representation = tb::kReorg;
    f->packed.tile_size = 1;
    f->packed.num_features = q.num_features;
    f->packed.num_classes = q.num_classes;
    f->packed.transform = q.transform;
    f->packed.initial_value = q.initial_value;
    f->packed.num_trees = q.num_trees;
    f->packed.num_nodes = q.num_nodes;
    f->packed.max_depth = q.max_depth;
    int urc = upload_key_planes(f, q.node_plane, q.leaf_plane, q.exact_plane, q.orig_leaf, q.groups, q.tree_index,
                                q.lo, q.scale, q.num_features, true);
    if (urc != TBK_OK) return bail(urc);
    if (q.num_classes > 0) {
      // every class goes to one of the two walker sets, whichever has fewer groups so far;
      // within a set the groups keep their order, so its classes come in increasing order
      const size_t G = q.groups.size();
      std::vector<int32_t> lists(2 * G, 0);
      int32_t count[2] = {0, 0};
      for (size_t g = 0; g < G;) {
        size_t e = g;
        while (e < G && q.group_class[e] == q.group_class[g]) ++e;
        const int s = count[1] < count[0] ? 1 : 0;
        for (; g < e; ++g) lists[(size_t)s * G + count[s]++] = (int32_t)g;
      }
      f->qset_count[0] = count[0];
      f->qset_count[1] = count[1];
      CUDA_TRY_F(cudaMalloc(&f->d_qset_groups, lists.size() * 4));
      CUDA_TRY_F(cudaMemcpy(f->d_qset_groups, lists.data(), lists.size() * 4, cudaMemcpyHostToDevice));
      CUDA_TRY_F(cudaMalloc(&f->d_qgroup_class, G * 4));
      CUDA_TRY_F(cudaMemcpy(f->d_qgroup_class, q.group_class.data(), G * 4, cudaMemcpyHostToDevice));
    }
    // host copies of the big planes are no longer needed
    std::vector<uint32_t>().swap(f->qf.node_plane);
    std::vector<float>().swap(f->qf.leaf_plane);
    std::vector<float>().swap(f->qf.exact_plane);
    std::vector<int32_t>().swap(f->qf.orig_leaf);
    tb::LaunchPlan &pl = f->last_plan;
    pl.row_warps = 1; pl.tree_threads = tb::kQWalkers; pl.rows_per_lane = 1; pl.chunks = 1; pl.staged = 1; pl.cache_rows = 1;
    pl.stage_bytes = tb::kQPiece; pl.smem_bytes = quant_smem_bytes(q.num_features); pl.threads = tb::kQThreads;
    if (const int batch = quant_batch_tiles(f, q.num_features)) { // narrow rows: the batch kernel
      pl.row_warps = batch;
      pl.smem_bytes = tb::quant_batch_smem_bytes(q.num_features, batch);
      pl.threads = tb::kQBThreads;
    }
    return done();
  }

  f->packed = im.packed;
  const auto &p = f->packed;
  CUDA_TRY_F(cudaMalloc(&f->d_blob, std::max<size_t>(16, p.blob.size())));
  CUDA_TRY_F(cudaMemcpy(f->d_blob, p.blob.data(), p.blob.size(), cudaMemcpyHostToDevice));
  static_assert(sizeof(tb::GroupMeta) == sizeof(tb::DevGroupMeta), "group metadata layout");
  CUDA_TRY_F(cudaMalloc(&f->d_groups, p.groups.size() * sizeof(tb::GroupMeta)));
  CUDA_TRY_F(cudaMemcpy(f->d_groups, p.groups.data(), p.groups.size() * sizeof(tb::GroupMeta), cudaMemcpyHostToDevice));
  CUDA_TRY_F(cudaMalloc(&f->d_tree_class, p.tree_class.size() * 2));
  CUDA_TRY_F(cudaMemcpy(f->d_tree_class, p.tree_class.data(), p.tree_class.size() * 2, cudaMemcpyHostToDevice));
  CUDA_TRY_F(cudaMalloc(&f->d_tree_index, p.tree_index.size() * 4));
  CUDA_TRY_F(cudaMemcpy(f->d_tree_index, p.tree_index.data(), p.tree_index.size() * 4, cudaMemcpyHostToDevice));
  CUDA_TRY_F(cudaMalloc(&f->d_lut, std::max<size_t>(16, p.lut.size())));
  CUDA_TRY_F(cudaMemcpy(f->d_lut, p.lut.data(), p.lut.size(), cudaMemcpyHostToDevice));
  // the packed blob is only needed on the device from here on
  std::vector<uint8_t>().swap(f->packed.blob);
  // settle the plan for the hinted batch so that get_info can report it
  tb::ForestShape shape{p.num_features, p.num_classes, (int64_t)p.groups.size(), p.max_group_bytes,
                        (int32_t)p.lut.size(), p.representation, p.tile_size};
  std::string why = tb::select_launch(shape, f->user, batch_hint > 0 ? batch_hint : 65536, f->max_smem_optin,
                                      f->num_sms, false, &f->last_plan);
  if (!why.empty()) return bail(fail(TBK_ERR_UNSUPPORTED, "%s", why.c_str()));
  return done();
}

int tbk_forest_free(tbk_forest *f) {
  if (!f) return TBK_OK;
  cudaSetDevice(f->device);
  free_pipeline(f);
  for (cudaStream_t st : f->streams)
    if (st) cudaStreamDestroy(st);
  for (int i = 0; i < tbk_forest::kPipeSlots; ++i) {
    if (f->slot_done[i]) cudaEventDestroy(f->slot_done[i]);
    if (f->slot_read[i]) cudaEventDestroy(f->slot_read[i]);
  }
  cudaFree(f->d_blob);
  cudaFree(f->d_groups);
  cudaFree(f->d_tree_class);
  cudaFree(f->d_tree_index);
  cudaFree(f->d_orig_node);
  cudaFree(f->d_orig_off);
  cudaFree(f->d_lut);
  pinned_pool().give_back_status(f->h_status);
  pinned_pool().give_back(f->h_small, f->small_capacity);
  cudaFree(f->d_small_in);
  cudaFree(f->d_qnode);
  cudaFree(f->d_qleaf);
  cudaFree(f->d_qexact);
  cudaFree(f->d_qsplit);
  cudaFree(f->d_qorig);
  cudaFree(f->d_qgroups);
  cudaFree(f->d_qtree_index);
  cudaFree(f->d_qset_groups);
  cudaFree(f->d_qgroup_class);
  cudaFree(f->d_qlo);
  cudaFree(f->d_qscale);
  if (!f->rank) cudaFree(f->d_ties);
  cudaFree(f->d_rank_block);
  for (void *d : {(void *)f->d_lnodes, (void *)f->d_lroot, (void *)f->d_ltree_index, (void *)f->d_lorig, (void *)f->d_lclass_end, (void *)f->d_lclass_tree})
    cudaFree(d);
  for (auto &w : f->workspace) {
    cudaFree(w.mem);
    if (w.done) cudaEventDestroy(w.done);
  }
  for (auto &c : f->captured) cudaFree(c.memory.mem);
  if (f->ev0) cudaEventDestroy(f->ev0);
  if (f->ev1) cudaEventDestroy(f->ev1);
  delete f;
  pinned_pool().detach();
  return TBK_OK;
}

int tbk_forest_get_info(const tbk_forest *f, tbk_forest_info *info) {
  if (!f || !info) return fail(TBK_ERR_INVALID, "null argument");
  std::memset(info, 0, sizeof *info);
  const auto &p = f->packed;
  info->num_trees = p.num_trees;
  info->num_nodes = p.num_nodes;
  info->num_groups = f->lanes ? p.num_trees : f->rank ? (int64_t)f->rf.groups.size() : f->quant ? (int64_t)f->qf.groups.size() : f->deep ? (int64_t)f->df.pairs.size() : (int64_t)p.groups.size();
  info->packed_bytes = f->lanes ? 8 * p.num_nodes : f->rank ? (int64_t)(8 * (f->rf.groups.back().elem_off + (uint64_t)f->rf.groups.back().slots * tb::kRankCols)) :
                       f->deep ? (int64_t)(f->df.pairs.empty() ? 0 : 8 * (f->df.pairs.back().elem_off + 2ull * f->df.pairs.back().slots)
                                                                          + (f->d_qsplit ? 32 * f->df.pairs.size() * deep_half_words(f->uniform_depth) : 0)) :
                       f->quant ? (int64_t)(f->qf.groups.empty() ? 0 : 8 * (f->qf.groups.back().elem_off + (uint64_t)f->qf.groups.back().slots * tb::kQuantCols)) :
                       p.groups.empty() ? 0 : (int64_t)(p.groups.back().byte_off +
      (((uint64_t)p.groups.back().slots * tb::kGroupTrees * p.tile_bytes + 15) & ~15ull));
  info->max_depth = p.max_depth;
  info->num_features = p.num_features;
  info->num_classes = p.num_classes;
  info->transform = p.transform;
  info->device = f->device;
  const tb::LaunchPlan &pl = f->last_plan;
  info->schedule.representation = p.representation;
  info->schedule.tile_size = p.tile_size;
  info->schedule.rows_per_block = pl.rows_per_block ? pl.rows_per_block : pl.row_warps * 32 * pl.rows_per_lane;
  info->schedule.rows_per_thread = pl.rows_per_lane;
  info->schedule.tree_threads = pl.tree_threads;
  info->schedule.tree_chunks = pl.chunks;
  info->schedule.cache_trees = pl.staged ? 1 : 2;
  info->layout = f->rank ? TBK_LAYOUT_RANK_KEYS : f->quant ? TBK_LAYOUT_ROUNDED_KEYS : f->deep ? TBK_LAYOUT_DEEP_KEYS : f->lanes ? TBK_LAYOUT_LANES : TBK_LAYOUT_TILES;
  info->schedule.feature_bits = (f->rank || f->quant || f->deep) ? 16 : 32;
  info->staged = pl.staged;
  info->smem_bytes = pl.smem_bytes;
  info->threads_per_block = pl.threads;
  info->reserved[2] = f->last_ran;
  if (f->d_ties) {
    // (statistics; synchronises with the device)
    unsigned long long ties = 0;
    if (cudaMemcpy(&ties, f->d_ties, 8, cudaMemcpyDeviceToHost) == cudaSuccess) {
      info->reserved[0] = (int32_t)(ties & 0x7fffffff);
      info->reserved[1] = (int32_t)(ties >> 31);
    }
  }
  return TBK_OK;
}

int tbk_predict(tbk_forest *f, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out,
                int32_t out_kind, void *stream) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  std::lock_guard<std::mutex> lock(f->mu);
  return run(f, kPredict, d_rows, n_rows, ld, d_out, out_kind, nullptr, nullptr, (cudaStream_t)stream);
}

int tbk_predict_partial(tbk_forest *f, const float *d_rows, int64_t n_rows, int64_t ld, float *d_partial,
                        void *stream) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  if (!d_partial && n_rows > 0) return fail(TBK_ERR_INVALID, "null output pointer");
  std::lock_guard<std::mutex> lock(f->mu);
  return run(f, kPartial, d_rows, n_rows, ld, nullptr, TBK_OUT_F32, d_partial, nullptr, (cudaStream_t)stream);
}

int tbk_finalize(tbk_forest *f, const float *d_partial, int64_t n_rows, void *d_out, int32_t out_kind,
                 void *stream) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  if (n_rows == 0) return TBK_OK;
  if (!d_partial || !d_out) return fail(TBK_ERR_INVALID, "null pointer");
  const auto &p = f->packed;
  if (out_kind == TBK_OUT_I8 && p.num_classes == 0) return fail(TBK_ERR_INVALID, "int8 output needs a multiclass forest");
  std::lock_guard<std::mutex> lock(f->mu);
  CUDA_TRY(cudaSetDevice(f->device));
  const int tpb = 256;
  tb::tb_finalize_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, (cudaStream_t)stream>>>(
      d_partial, 1, n_rows, std::max(1, p.num_classes), p.num_classes, (float)p.initial_value, p.transform, d_out, out_kind);
  CUDA_TRY(cudaGetLastError());
  ++f->launches;
  return TBK_OK;
}

int tbk_predict_leaf_ids(tbk_forest *f, const float *d_rows, int64_t n_rows, int64_t ld,
                         int32_t *d_leaf_ids, void *stream) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  if (!d_leaf_ids && n_rows > 0) return fail(TBK_ERR_INVALID, "null output pointer");
  std::lock_guard<std::mutex> lock(f->mu);
  return run(f, kLeafIds, d_rows, n_rows, ld, nullptr, TBK_OUT_F32, nullptr, d_leaf_ids, (cudaStream_t)stream);
}

int tbk_predict_host(tbk_forest *f, const float *h_rows, int64_t n_rows, int64_t ld, void *h_out,
                     int32_t out_kind) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  if (n_rows == 0) return TBK_OK;
  if (!h_rows || !h_out) return fail(TBK_ERR_INVALID, "null pointer");
  if (n_rows < 0 || ld < f->packed.num_features)
    return fail(TBK_ERR_INVALID, "ld (%lld) is smaller than the row size (%d)", (long long)ld, f->packed.num_features);
  std::lock_guard<std::mutex> lock(f->mu);
  CUDA_TRY(cudaSetDevice(f->device));
  if (!f->streams[0]) {
    for (cudaStream_t &st : f->streams) CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    for (cudaEvent_t &e : f->slot_done) CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (cudaEvent_t &e : f->slot_read) CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  const size_t out_elt = out_kind == TBK_OUT_I8 ? 1 : 4, row_bytes = (size_t)ld * 4;
  const bool was_timing = f->timing;
  f->timing = false; // per-chunk launches overlap on two streams; event timing does not apply
  struct Restore { // (on every way out)
    tbk_forest *f;
    bool timing;
    ~Restore() {
      f->timing = timing;
      f->host_batch_rows = 0;
    }
  } restore{f, was_timing};
  f->host_batch_rows = n_rows;
  if ((size_t)n_rows * row_bytes <= kSmallRows && (size_t)n_rows * out_elt <= kSmallResults)
    return predict_host_small(f, h_rows, n_rows, ld, h_out, out_kind);

  // Chunks of about a twelfth of the batch, 4 to 32 MiB: small enough that filling and draining
  // the pipeline is a small part of the whole and that a staging slot stays in the cores' caches.
  size_t chunk_bytes = std::min<size_t>((size_t)32 << 20, std::max<size_t>((size_t)4 << 20, (size_t)n_rows * row_bytes / 12));
  const int64_t chunk = std::min<int64_t>(std::max<int64_t>(1024, (int64_t)(chunk_bytes / row_bytes) / 1024 * 1024), (n_rows + 1023) / 1024 * 1024);
  chunk_bytes = (size_t)chunk * row_bytes;
  const bool in_pinned = is_pinned(h_rows), out_pinned = is_pinned(h_out);
  if (f->pipe_bytes < chunk_bytes || f->pipe_rows < (size_t)chunk) {
    free_pipeline(f);
    const size_t in = (chunk_bytes + 255) / 256 * 256, res = (size_t)chunk * 4;
    CUDA_TRY(cudaMalloc(&f->d_in[0], tbk_forest::kPipeSlots * (in + res)));
    for (int i = 0; i < tbk_forest::kPipeSlots; ++i) {
      f->d_in[i] = f->d_in[0] + (size_t)i * in;
      f->d_res[i] = f->d_in[0] + tbk_forest::kPipeSlots * in + (size_t)i * res;
    }
    f->pipe_bytes = chunk_bytes;
    f->pipe_rows = (size_t)chunk;
  }
  for (int64_t i = 0; i < std::min<int64_t>(tbk_forest::kPipeSlots, (n_rows + chunk - 1) / chunk); ++i) {
    if (!in_pinned && !f->h_pin[i]) f->h_pin[i] = pinned_pool().take(f->pipe_bytes, &f->pin_capacity[i]);
    if (!out_pinned && !f->h_res[i]) f->h_res[i] = pinned_pool().take(f->pipe_rows * 4, &f->res_capacity[i]);
    if ((!in_pinned && !f->h_pin[i]) || (!out_pinned && !f->h_res[i])) return fail(TBK_ERR_CUDA, "no pinned memory for the batch");
  }
  unsigned char *out = static_cast<unsigned char *>(h_out);
  constexpr int NS = tbk_forest::kPipeSlots;
  const int64_t num_chunks = (n_rows + chunk - 1) / chunk;
  Stager *stager = nullptr;
  if (!in_pinned) {
    if (!f->stager) f->stager.reset(new Stager(std::max(0, std::min(6, tb::pack_threads() - 1))));
    stager = f->stager.get();
    stager->start(h_rows, ((size_t)(n_rows - 1) * ld + f->packed.num_features) * 4, f->h_pin, NS, chunk_bytes);
  }
  int rc = TBK_OK;
  int64_t copied = 0, collected = 0, issued = 0; // chunks whose rows have left their slot / whose results are out / in flight
  auto rows_of = [&](int64_t c) { return std::min<int64_t>(chunk, n_rows - c * chunk); };
  // Takes note of what the GPU has finished; wait: until the oldest chunk's results are there.
  auto advance = [&](bool wait) {
    while (copied < issued && cudaEventQuery(f->slot_read[copied % NS]) == cudaSuccess) {
      ++copied;
      if (stager) stager->allow(copied + NS - 1);
    }
    while (collected < issued) {
      const int s = (int)(collected % NS);
      const cudaError_t e = wait ? cudaEventSynchronize(f->slot_done[s]) : cudaEventQuery(f->slot_done[s]);
      if (e == cudaErrorNotReady) break;
      if (e != cudaSuccess && rc == TBK_OK) rc = fail(TBK_ERR_CUDA, "host pipeline: %s", cudaGetErrorString(e));
      if (!out_pinned && rc == TBK_OK)
        std::memcpy(out + (size_t)(collected * chunk) * out_elt, f->h_res[s], (size_t)rows_of(collected) * out_elt);
      ++collected;
      if (wait) break;
    }
  };
  for (int64_t c = 0; c < num_chunks && rc == TBK_OK; ++c) {
    const int s = (int)(c % NS);
    const int64_t n = rows_of(c);
    const size_t bytes = ((size_t)(n - 1) * ld + f->packed.num_features) * 4; // (nothing behind the last row's values)
    cudaStream_t stream = f->streams[s & 1];
    while (stager && !stager->ready(c) && rc == TBK_OK)
      if (!stager->copy_one()) advance(false);
    while (collected + NS <= c && rc == TBK_OK) advance(true); // the slot's results must be out
    if (rc != TBK_OK) break;
    const void *src = stager ? static_cast<const void *>(f->h_pin[s]) : h_rows + c * chunk * ld;
    cudaError_t e = cudaMemcpyAsync(f->d_in[s], src, bytes, cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) e = cudaEventRecord(f->slot_read[s], stream);
    if (e != cudaSuccess) {
      rc = fail(TBK_ERR_CUDA, "host-to-device copy: %s", cudaGetErrorString(e));
      break;
    }
    rc = run(f, kPredict, reinterpret_cast<const float *>(f->d_in[s]), n, ld, f->d_res[s], out_kind, nullptr, nullptr, stream);
    if (rc != TBK_OK) break;
    e = cudaMemcpyAsync(out_pinned ? out + (size_t)(c * chunk) * out_elt : f->h_res[s], f->d_res[s], (size_t)n * out_elt, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaEventRecord(f->slot_done[s], stream);
    if (e != cudaSuccess) {
      rc = fail(TBK_ERR_CUDA, "device-to-host copy: %s", cudaGetErrorString(e));
      break;
    }
    ++issued;
    advance(false);
  }
  if (stager) stager->finish();
  while (collected < issued && rc == TBK_OK) advance(true);
  for (cudaStream_t st : f->streams) {
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess && rc == TBK_OK) rc = fail(TBK_ERR_CUDA, "cudaStreamSynchronize: %s", cudaGetErrorString(e));
  }
  return rc != TBK_OK ? rc : check_status(f);
}

int tbk_set_timing(tbk_forest *f, int32_t enable) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  f->timing = enable != 0;
  f->ev_pending = false;
  return TBK_OK;
}

int64_t tbk_last_kernel_time_us(tbk_forest *f) {
  if (!f || !f->ev_pending) return -1;
  if (cudaEventSynchronize(f->ev1) != cudaSuccess) return -1;
  float ms = 0.f;
  if (cudaEventElapsedTime(&ms, f->ev0, f->ev1) != cudaSuccess) return -1;
  return (int64_t)(ms * 1000.0f + 0.5f);
}

int64_t tbk_launch_count(const tbk_forest *f) { return f ? f->launches : 0; }

int tbk_check_status(tbk_forest *f) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  CUDA_TRY(cudaSetDevice(f->device));
  CUDA_TRY(cudaDeviceSynchronize());
  return check_status(f);
}

int tbk_debug_expire_next_wait(tbk_forest *f) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  std::lock_guard<std::mutex> lock(f->mu);
  f->expire_next_wait = true;
  return TBK_OK;
}

} // extern "C"

// ---------------------------------------------------------------------------
// Prediction for callers that must not allocate.
//
// Some hosts of this library may not call cudaMalloc on the prediction path: a serving
// loop whose memory is fixed at start-up (a pool carved once, with nothing left over for
// the driver to hand out later), a latency-critical thread that cannot afford the implicit
// device synchronisation an allocation may bring, or an embedding runtime whose policy
// forbids device allocations outside its own allocator.  tbk_predict sizes its tree-chunk
// partial sums at run time and grows a cudaMalloc'ed buffer when a larger batch arrives;
// this variant runs the same two kernels (walk into per-chunk partials, then the
// atomic-free second pass) with the partials in a fixed array that is part of the loaded
// library image, so it never allocates or frees anything.
//
// The array lives on every GPU that loads the library, from load until the process exits
// (kNoAllocScratchFloats * 4 bytes = 8 MiB per GPU).  In host code its name is only a
// stand-in for the device object; the device address is looked up once per device with
// cudaGetSymbolAddress while that device is current, and that address is what the kernels
// receive.

namespace {

constexpr size_t kNoAllocScratchFloats = size_t(1) << 21; // 2 Mi floats = 8 MiB
static __device__ __align__(256) float g_noalloc_scratch[kNoAllocScratchFloats];

constexpr int kMaxDevices = 64;
float *g_noalloc_addr[kMaxDevices] = {};
std::mutex g_noalloc_mu;

// Device address of the scratch array on `device` (which must be current).
int noalloc_scratch_address(int device, float **out) {
  if (device < 0 || device >= kMaxDevices) return fail(TBK_ERR_INVALID, "device index %d out of range", device);
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_addr[device]) {
    float *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr), g_noalloc_scratch);
    if (e != cudaSuccess || !ptr)
      return fail(TBK_ERR_CUDA, "cudaGetSymbolAddress(scratch) failed on device %d: %s", device, cudaGetErrorString(e));
    g_noalloc_addr[device] = ptr;
  }
  *out = g_noalloc_addr[device];
  return TBK_OK;
}

} // namespace

extern "C" int tbk_predict_noalloc(tbk_forest *f, const float *d_rows, int64_t n_rows, int64_t ld, void *d_out,
                                   int32_t out_kind, void *stream_) {
  if (!f) return fail(TBK_ERR_INVALID, "null forest");
  std::lock_guard<std::mutex> lock(f->mu);
  const auto &pk = f->packed;
  // (of rounded keys and of one-byte ranks only rows that an fp32 tile could hold too)
  const bool tile_fits = (int64_t)(pk.num_features + 1) * 128 + 1024 <= f->max_smem_optin;
  const bool wide = f->quant && quant_batch_tiles(f, pk.num_features) == 0 && tile_fits;
  if ((f->quant && !wide) || f->deep || (f->rank && tb::rank_bytes(pk.num_features) && !tile_fits))
    return fail(TBK_ERR_UNSUPPORTED, "tbk_predict_noalloc does not cover the rounded 16-bit key layouts");
  if (n_rows < 0 || ld < pk.num_features) return fail(TBK_ERR_INVALID, "ld (%lld) is smaller than the row size (%d)", (long long)ld, pk.num_features);
  if (n_rows == 0) return TBK_OK;
  if (!d_rows || !d_out) return fail(TBK_ERR_INVALID, "null pointer");
  if (out_kind != TBK_OUT_F32 && out_kind != TBK_OUT_I8) return fail(TBK_ERR_INVALID, "unknown output kind %d", out_kind);
  if (out_kind == TBK_OUT_I8 && pk.num_classes == 0) return fail(TBK_ERR_INVALID, "int8 output needs a multiclass forest");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  CUDA_TRY(cudaSetDevice(f->device));
  float *scratch = nullptr;
  f->last_ran = 0;
  int rc = noalloc_scratch_address(f->device, &scratch);
  if (rc != TBK_OK) return rc;
  if (f->rank)
    return run_rank(f, kPredict, d_rows, n_rows, ld, d_out, out_kind, nullptr, nullptr, stream, reinterpret_cast<unsigned char *>(scratch),
                    kNoAllocScratchFloats * sizeof(float));
  if (f->quant)
    return run_quant(f, kPredict, d_rows, n_rows, ld, d_out, out_kind, nullptr, nullptr, stream, scratch, kNoAllocScratchFloats);
  if (f->lanes)
    return run_lanes(f, kPredict, d_rows, n_rows, ld, d_out, out_kind, nullptr, nullptr, stream, scratch, kNoAllocScratchFloats);

  tb::ForestShape shape{pk.num_features, pk.num_classes, (int64_t)pk.groups.size(), pk.max_group_bytes,
                        (int32_t)pk.lut.size(), pk.representation, pk.tile_size};
  tb::LaunchPlan plan;
  // this call always writes partial sums, so the plan must be one for partial output: its
  // shared memory then includes the per-warp class table of a multiclass forest
  std::string why = tb::select_launch(shape, f->user, n_rows, f->max_smem_optin, f->num_sms, false, &plan, true);
  if (!why.empty()) return fail(TBK_ERR_UNSUPPORTED, "%s", why.c_str());
  if (plan.class_regs)
    return fail(TBK_ERR_UNSUPPORTED, "tbk_predict_noalloc: launch plan keeps class sums in registers and cannot write partial sums");
  const int W = std::max(1, pk.num_classes);
  const size_t need = (size_t)plan.chunks * (size_t)n_rows * (size_t)W;
  if (need > kNoAllocScratchFloats)
    return fail(TBK_ERR_UNSUPPORTED,
                "tbk_predict_noalloc: %lld rows x %d tree chunks x %d outputs need %zu partial sums, the fixed scratch "
                "holds %zu; split the batch or use tbk_predict",
                (long long)n_rows, plan.chunks, W, need, kNoAllocScratchFloats);

  tb::WalkParams p{};
  p.blob = f->d_blob;
  p.groups = f->d_groups;
  p.tree_class = f->d_tree_class;
  p.tree_index = f->d_tree_index;
  p.lut = f->d_lut;
  p.lut_bytes = (int32_t)pk.lut.size();
  p.rows = d_rows;
  p.n_rows = n_rows;
  p.ld = ld;
  p.partial = scratch; // every (chunk, row, output) element is written by the walk: nothing to clear
  p.out = d_out;
  p.out_kind = out_kind;
  p.write_partial = 1;
  p.num_trees = pk.num_trees;
  p.num_groups = (int32_t)pk.groups.size();
  p.groups_per_chunk = plan.groups_per_chunk;
  p.num_features = pk.num_features;
  p.num_classes = pk.num_classes;
  p.transform = pk.transform;
  p.initial_value = (float)pk.initial_value;
  p.row_warps = plan.row_warps;
  p.tree_threads = plan.tree_threads;
  p.stage_bytes = plan.staged ? plan.stage_bytes : 0;
  p.stages = plan.stages;
  p.vec4_ok = (pk.num_features % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(d_rows) & 15) == 0) ? 1 : 0;
  p.status = f->d_status;
  p.class_regs = 0; // class sums go through the shared-memory table the plan has sized
  const tb::WalkKernel fn = pick_kernel(pk.representation, pk.tile_size, plan, pk.num_features, &f->last_ran);
  if (const int rc = allow_smem(f, (const void *)fn)) return rc;
  dim3 grid((unsigned)plan.grid_x, (unsigned)plan.chunks), block((unsigned)plan.threads);
  fn<<<grid, block, plan.smem_bytes, stream>>>(p);
  CUDA_TRY(cudaGetLastError());
  const int tpb = 256;
  tb::tb_finalize_kernel<<<(unsigned)((n_rows + tpb - 1) / tpb), tpb, 0, stream>>>(
      scratch, plan.chunks, n_rows, W, pk.num_classes, (float)pk.initial_value, pk.transform, d_out, out_kind);
  CUDA_TRY(cudaGetLastError());
  f->launches += 2;
  return TBK_OK;
}

// ---------------------------------------------------------------------------
// Host-only utilities (no device is touched).

extern "C" {

int tbk_host_layout_check(const tbk_forest_arrays *fa, const tbk_schedule *schedule, const float *rows,
                          int64_t n_rows, int64_t ld, int32_t *leaf_ids, float *sums,
                          tbk_forest_info *info) {
  if (!fa || fa->num_trees <= 0) return fail(TBK_ERR_INVALID, "null or empty forest");
  tb::Forest host;
  const int64_t T = fa->num_trees, N = fa->tree_off[T];
  host.tree_off.assign(fa->tree_off, fa->tree_off + T + 1);
  host.left.assign(fa->left, fa->left + N);
  host.right.assign(fa->right, fa->right + N);
  host.feat.assign(fa->feat, fa->feat + N);
  host.thr.assign(fa->thr, fa->thr + N);
  if (fa->num_classes > 0 && fa->class_id) host.class_id.assign(fa->class_id, fa->class_id + T);
  host.num_classes = fa->num_classes;
  host.transform = fa->transform;
  host.initial_value = fa->initial_value;
  host.num_features = fa->num_features;
  if (schedule && schedule->feature_bits == 16) {
    // the key layouts: groups of 32 trees up to 8 levels, whole-tree stages beyond
    int max_depth = 0;
    {
      const std::string verr = tb::validate(host);
      if (!verr.empty()) return fail(TBK_ERR_INVALID, "%s", verr.c_str());
      for (int64_t t = 0; t < T; ++t) max_depth = std::max(max_depth, (int)tb::tree_depth(host, t));
    }
    int64_t ties = 0, groups = 0, elems = 0;
    if (max_depth <= tb::kQuantMaxDepth) {
      tb::QuantForest q;
      // (lattice features where the rows are narrow enough for the batch kernel, as at upload)
      const bool narrow = (227 * 1024 - tb::kQBBarBytes - tb::kQBRingBytes) / tb::quant_batch_tile_bytes(host.num_features) >= 4;
      std::string qerr = tb::pack_quant(host, &q, narrow);
      if (!qerr.empty()) return fail(TBK_ERR_UNSUPPORTED, "%s", qerr.c_str());
      if (rows && n_rows > 0) {
        tb::walk_quant_on_host(q, rows, n_rows, ld, leaf_ids, sums, &ties);
        // forests over narrow rows are uploaded as rank keys: those planes must select the same leaves
        tb::RankForest r;
        if (leaf_ids && tb::pack_rank(host, &r).empty()) {
          std::vector<int32_t> again((size_t)n_rows * T);
          int64_t searched = 0;
          tb::walk_rank_on_host(r, rows, n_rows, ld, again.data(), nullptr, &searched);
          if (std::memcmp(again.data(), leaf_ids, again.size() * 4) != 0) return fail(TBK_ERR_INVALID, "rank keys and quantised keys select different leaves");
        }
      }
      groups = (int64_t)q.groups.size();
      elems = (int64_t)q.node_plane.size();
    } else {
      tb::DeepForest q;
      std::string qerr = tb::pack_deep(host, &q);
      if (!qerr.empty()) return fail(TBK_ERR_UNSUPPORTED, "%s", qerr.c_str());
      if (rows && n_rows > 0) tb::walk_deep_on_host(q, rows, n_rows, ld, leaf_ids, sums, &ties);
      groups = (int64_t)q.pairs.size();
      elems = (int64_t)q.node_plane.size();
    }
    if (info) {
      std::memset(info, 0, sizeof *info);
      info->num_trees = T;
      info->num_nodes = N;
      info->num_groups = groups;
      info->packed_bytes = elems * 8;
      info->max_depth = max_depth;
      info->num_features = host.num_features;
      info->transform = host.transform;
      info->schedule.representation = TBK_REP_REORG;
      info->schedule.tile_size = 1;
      info->schedule.feature_bits = 16;
      info->reserved[0] = (int32_t)std::min<int64_t>(ties, 0x7fffffff);
    }
    return TBK_OK;
  }
  tb::PackOptions opt;
  opt.representation = schedule && schedule->representation >= 0 ? schedule->representation : 0;
  opt.tile_size = schedule && schedule->tile_size > 0 ? schedule->tile_size : 1;
  tb::PackedForest packed;
  std::string err = tb::pack_forest(host, opt, &packed);
  if (!err.empty()) return fail(TBK_ERR_INVALID, "%s", err.c_str());
  if (info) {
    std::memset(info, 0, sizeof *info);
    info->num_trees = packed.num_trees;
    info->num_nodes = packed.num_nodes;
    info->num_groups = (int64_t)packed.groups.size();
    info->packed_bytes = (int64_t)packed.blob.size();
    info->max_depth = packed.max_depth;
    info->num_features = packed.num_features;
    info->num_classes = packed.num_classes;
    info->transform = packed.transform;
    info->schedule.representation = packed.representation;
    info->schedule.tile_size = packed.tile_size;
    info->reserved[0] = packed.num_shapes;
    info->reserved[1] = (int32_t)packed.lut.size();
    info->reserved[2] = (int32_t)std::min<uint64_t>(packed.max_group_bytes, 0x7fffffff);
  }
  if (rows && n_rows > 0) tb::walk_packed_on_host(packed, rows, n_rows, ld, leaf_ids, sums);
  return TBK_OK;
}

int tbk_plan_launch(int32_t num_features, int32_t num_classes, int64_t num_groups, int64_t max_group_bytes,
                    int32_t lut_bytes, const tbk_schedule *schedule, int64_t n_rows, int32_t smem_limit,
                    int32_t num_sms, int32_t partial_sums, tbk_forest_info *info) {
  if (!info) return fail(TBK_ERR_INVALID, "null argument");
  tbk_schedule user{};
  if (schedule) user = *schedule;
  tb::ForestShape shape{num_features, num_classes, num_groups, (uint64_t)max_group_bytes, lut_bytes,
                        user.representation, user.tile_size > 0 ? user.tile_size : 1};
  tb::LaunchPlan pl;
  std::string why = tb::select_launch(shape, user, n_rows, smem_limit, num_sms, false, &pl, partial_sums != 0);
  if (!why.empty()) return fail(TBK_ERR_UNSUPPORTED, "%s", why.c_str());
  std::memset(info, 0, sizeof *info);
  info->schedule = user;
  info->schedule.rows_per_block = pl.row_warps * 32 * pl.rows_per_lane;
  info->schedule.rows_per_thread = pl.rows_per_lane;
  info->schedule.tree_threads = pl.tree_threads;
  info->schedule.tree_chunks = pl.chunks;
  info->schedule.cache_trees = pl.staged ? 1 : 2;
  info->staged = pl.staged;
  info->smem_bytes = pl.smem_bytes;
  info->threads_per_block = pl.threads;
  info->reserved[0] = pl.cache_rows;
  info->reserved[1] = (int32_t)std::min<int64_t>(pl.grid_x, 0x7fffffff);
  info->reserved[2] = pl.groups_per_chunk;
  info->reserved[3] = pl.class_regs;
  return TBK_OK;
}

} // extern "C"
