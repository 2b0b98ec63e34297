// sk_runtime.h -- host-side state behind the opaque C ABI handles.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "sk_common.h"
#include "sk_launch.h"
#include "sketchlib_b200.h"

struct Scratch {
  void *ptr = nullptr;
  size_t bytes = 0;
};

// Context scratch slots (each a growable device buffer).
enum ScratchSlot : int {
  kSlotCounts = 0,        // per-CTA tile counts of the distance kernel
  kSlotOut = 1,           // dense result staging
  kSlotResult = 2,        // kNN / threshold results
  kSlotTemp = 3,          // temporaries (scan storage, unpacking, probes)
  kSlotSplitCounts = 4,   // counts of tiles split along k
  kSlotLaunchMeta = 5,    // job table, work list, control block
  kSlotStaging = 6,       // sketch words in the reference layout on their way in
  kSlotPackedRef = 7,     // packed arrays of the databases of one sk_query_db call
  kSlotPackedQuery = 8,
  kSlotCountsB = 9,       // count scratch of launches on the second compute stream
  kSlotSplitCountsB = 10,
  kSlotSketchCodes = 11,  // bases of one sketching batch, rewritten as base codes
  kSlotSketchSeqs = 12,   // sequence offsets of the batch
  kSlotSketchItems = 13,  // sketching work items
  kSlotSketchTables = 14, // rolling-hash tables per k
  kSlotSketchBins = 15,   // bin minima per (sample, k)
  kSlotSketchWords = 16,  // finished sketches, inverse minhashes, densify flags
  kSlotSketchTable = 17,  // k-mer count table of read sets
  kSlotCodes = 18,        // coded tiles (code_kernels.cu)
  kSlotSketchRows = 19,   // per-row state of the low count
  kSlotCount = 20
};

struct sk_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = true;
  cudaStream_t copy_stream = nullptr;   // copies overlapped with kernels (created on first use)
  cudaEvent_t ev_ready[2] = {};         // double buffer b holds data
  cudaEvent_t ev_free[2] = {};          // double buffer b may be overwritten
  cudaStream_t stream_b = nullptr;      // second compute stream (chunk launches alternate)
  cudaStream_t pack_stream = nullptr;   // high-priority stream for packing uploaded chunks
  std::vector<cudaEvent_t> ev_chunk;    // chunk c packed
  cudaStream_t d2h_stream = nullptr;    // result rows copied back while later chunks compute
  std::vector<cudaEvent_t> ev_out;      // chunk c's output rows written
  cudaEvent_t ev_join = nullptr;        // second compute stream done
  int64_t code_limit = 0;               // bytes of coded tiles (0: automatic, -1: none)
  size_t few_limit = sk::kFewQueriesBytes;   // bytes of the few-queries workspace
  int64_t mem_limit = 0;                // bytes a dense call may stage output in (0 = free memory)
  int sm_count = 0;
  std::string err;
  int *cancel_host = nullptr;   // mapped pinned word polled by the kernels
  int *cancel_dev = nullptr;
  sk::DevStatus *status_dev = nullptr;
  unsigned long long last_tiles = 0;
  int tile_cfg = 0;                               // forced tile shape (0 = automatic)
  int semantics = 0;                              // sk::Semantics of later calls
  std::map<std::pair<int, int>, int> tuning;      // (K, s64) -> shape id
  Scratch scratch[kSlotCount];                    // reusable device buffers
  void *noalloc_scratch = nullptr;                // device address of the static no-alloc buffer
  // Jaccard / log-Jaccard tables by count of uncorrected jobs, per union size
  // (64 * sketchsize64); allocated on first use, freed with the context
  std::map<int64_t, std::pair<float *, double *>> count_tables;
  std::mutex count_tables_mu;
  std::recursive_mutex mu;
  // Databases and random models keep their context alive: sk_ctx_destroy only
  // marks it, the last dependent handle to go frees it.
  int refs = 1;
  bool destroyed = false;
};

struct sk_db {
  sk_ctx *ctx = nullptr;
  int64_t n = 0;
  int32_t K = 0, s64 = 0, bbits = 0;
  std::vector<int32_t> kmers;
  int32_t ng = 0;                 // granules in the packed array (padded samples / 64)
  uint32_t *packed = nullptr;     // [K][2*s64][ng][14][64]
  bool own_packed = true;         // false: the array is context scratch
  uint16_t *cluster = nullptr;    // [ng*64] random-match cluster ids
  int32_t max_cluster = 0;        // the largest of them
  std::vector<uint64_t> seq_len;  // per-sample sequence lengths
  double *jv = nullptr;           // [K][ng*64] equal-base factors
  int jv_rc = -1;
  float *jgpu = nullptr;          // [K] equal-base chances of the reference GPU path
  int jgpu_rc = -1;
};

struct sk_random {
  sk_ctx *ctx = nullptr;
  int mode = 0;
  int use_rc = 1;
  std::vector<int32_t> kmers;
  int n_clusters = 0;
  float *table = nullptr;         // [K][C][C]
  std::vector<float> centroids;   // [C][4] base-composition centroids (may be empty)
};

struct sk_sparse {
  std::vector<int64_t> i, j;
  std::vector<float> d;
};

namespace sk {

// Launches of the persistent distance kernel that share a tile shape and one
// meta buffer: the job table, and per launch its work list, split tiles and
// (coded launches) the row blocks to encode first.
struct Plan {
  struct Code {                // one range of row blocks of one job
    int job;
    CodeTask task;             // pointers are filled in when the buffers are known
    size_t words_off, lists_off, planes_off;   // in the launch's code buffer
    size_t chunk0;             // first entry in chunks
    size_t values;             // entry in values
  };
  struct Values {              // bin values of one column database
    const uint32_t *packed;
    int32_t kb, ng;
    size_t off;                // in the value area, after the code buffers
  };
  struct Sub {
    size_t item0 = 0, n_items = 0, split0 = 0;
    int32_t n_splits = 0;
    int32_t split_slots = 0;   // largest count-slot need of its split tiles
    bool wide = false;         // some job needs the wide kernel instance
    int code_buf = 0;          // which of the plan's two code buffers it uses
    size_t code_bytes = 0;
    std::vector<Code> codes;   // empty: a plain launch
    size_t values0 = 0, n_values = 0;   // value tasks to run first
  };
  const TileConfig *cfg = nullptr;
  int grid = 0;                // resident CTAs
  int sm_count = 0;
  int32_t k_slots = 1;
  size_t code_budget = 0;      // bytes of one launch's codes
  std::vector<JobParams> jobs;
  std::vector<WorkItem> items;
  std::vector<SplitTile> splits;
  std::vector<int4> chunks;
  std::vector<Values> values;
  bool values_by_caller = false;   // the caller queues the value tasks itself
  std::vector<Sub> subs;

  sk_status start(sk_ctx *ctx, const TileConfig &c, size_t budget);
  int add_job(const JobParams &jp);
  void add_tile(int job, int64_t tile);
  // The tiles of row tiles [rt0, rt1) and column tiles [ct0, ct1), coded, in
  // as many launches as the budget asks for.
  void add_coded(const JobParams &jp, int32_t rt0, int32_t rt1, int32_t ct0, int32_t ct1,
                 int code_buf);
  bool can_code(const JobParams &jp) const;
  void close_launch();         // ends the current launch
  bool open_empty() const { return items.size() == closed_items_; }
  size_t split_bytes() const;
  size_t code_stride() const;  // bytes of one code buffer
  size_t code_bytes() const;   // of the whole plan: code buffers and values
  size_t value_bytes_total() const { return value_bytes_; }

 private:
  int64_t choose_splits(size_t begin);
  void split_tail(size_t begin, Sub &sub);
  void add_piece(const JobParams &jp, int32_t rb0, int32_t rb1, int32_t cg0, int32_t cg1,
                 bool self, int code_buf);
  size_t closed_items_ = 0, closed_values_ = 0, value_bytes_ = 0;
  Sub open_;
};

struct MetaLayout {
  size_t items_off = 0, splits_off = 0, chunks_off = 0, ctrl_off = 0, ctrl_bytes = 0, bytes = 0;
};
MetaLayout meta_layout(size_t n_jobs, size_t n_items, size_t n_splits, size_t n_chunks,
                       size_t n_subs);

struct LaunchBuffers {
  void *meta = nullptr, *cta = nullptr, *split = nullptr, *codes = nullptr;
  char *values = nullptr;      // the value area of `codes`
  void *ctrl = nullptr;
  size_t ctrl_bytes = 0;
  LaunchParams lp{};
};

class DeviceGuard {
 public:
  explicit DeviceGuard(int dev);
  ~DeviceGuard();
  DeviceGuard(const DeviceGuard &) = delete;
  DeviceGuard &operator=(const DeviceGuard &) = delete;

 private:
  int prev_ = 0;
};

sk_status fail(sk_ctx *ctx, sk_status st, const char *fmt, ...);
void ctx_retain(sk_ctx *ctx);
void ctx_release(sk_ctx *ctx);
sk_status cuda_fail(sk_ctx *ctx, cudaError_t e, const char *what);
bool release_codes(sk_ctx *ctx);
cudaError_t device_alloc(sk_ctx *ctx, void **p, size_t bytes);
template <class T>
cudaError_t device_alloc(sk_ctx *ctx, T **p, size_t bytes) {
  return device_alloc(ctx, reinterpret_cast<void **>(p), bytes);
}
sk_status scratch(sk_ctx *ctx, int slot, size_t bytes, void **out);
sk_status begin_call(sk_ctx *ctx);
sk_status finish_call(sk_ctx *ctx);
const TileConfig *choose_config(sk_ctx *ctx, int K, int s64);
void plan_tiles(JobParams &jp, const TileConfig &cfg);
sk_status build_job(sk_ctx *ctx, const sk_db *ref, const sk_db *query, const sk_random *random,
                    int out_mode, int out_col, void *d_out, const TileConfig **cfg_out,
                    JobParams *jp);
bool few_queries(const sk_ctx *ctx, const JobParams &jp);
int64_t query_rows(sk_ctx *ctx, const sk_db *ref, int64_t n_query);
sk_status launch_job(sk_ctx *ctx, const JobParams &jp, const TileConfig &cfg);
// Points a job without random-match correction at the context's Jaccard /
// log-Jaccard tables by count for its union size, built on first use (one
// allocation and a small kernel, then a wait on the context stream); alloc
// false: only tables that already exist are used.  Corrected jobs, the
// reference GPU semantics, count output and sketches counted in chunks are
// left as they are (their epilogue computes per pair): per-entry tables for
// a Monte Carlo table measured no faster (20.69 against 20.71 ms at 4,096
// samples).
sk_status attach_count_tables(sk_ctx *ctx, JobParams *jp, bool alloc = true);
int32_t tail_block_parts(const JobParams &jp, int64_t r, int grid);
void tail_bounds(const JobParams &jp, int grid, int64_t *slots, int64_t *items);
bool use_codes(int64_t n_rows, int64_t n_cols, int32_t n_kmers, int32_t nb, bool self);
size_t code_bytes_wanted(const JobParams &jp);
size_t job_value_bytes(const JobParams &jp);
size_t code_reserve(sk_ctx *ctx, size_t values, size_t codes);
void code_wants(const std::vector<JobParams> &jobs, const TileConfig &cfg, size_t *values,
                size_t *codes);
size_t code_budget_for(sk_ctx *ctx, const std::vector<JobParams> &jobs, const TileConfig &cfg);
sk_status plan_with_codes(sk_ctx *ctx, const std::vector<JobParams> &jobs, const TileConfig &cfg,
                          const std::function<sk_status(size_t)> &make);
double padded_pairs(const TileConfig &cfg, int64_t n_ref, int64_t n_query);
sk_status db_alloc(sk_ctx *ctx, int64_t n, const int32_t *kmers, int32_t K, int32_t s64,
                   int32_t bbits, sk_db **out, int packed_slot = -1);
void db_free(sk_db *db);
sk_status make_plan(sk_ctx *ctx, const std::vector<JobParams> &jobs, const TileConfig &cfg,
                    size_t code_budget, Plan &plan);
sk_status upload_plan(sk_ctx *ctx, Plan &plan, LaunchBuffers &buf, bool owned);
sk_status reset_plan(sk_ctx *ctx, const LaunchBuffers &buf);
sk_status enqueue_launch(sk_ctx *ctx, const Plan &plan, const LaunchBuffers &buf, size_t i,
                         cudaStream_t stream);
sk_status enqueue_plan(sk_ctx *ctx, const Plan &plan, const LaunchBuffers &buf);
int resident_grid(sk_ctx *ctx, const TileConfig &cfg);
sk_status dense_to_device(sk_ctx *ctx, const sk_db *ref, const sk_db *query,
                          const sk_random *random, int out_mode, int out_col, void *d_out);
int64_t n_pairs(const sk_db *ref, const sk_db *query);
sk_status ensure_jv(sk_ctx *ctx, sk_db *db, int use_rc);
std::vector<double> equal_base_factors(const sk_db *db, int use_rc);
std::vector<float> equal_base_gpu(const sk_db *db, int use_rc);
sk_status ensure_copy_stream(sk_ctx *ctx);
size_t dense_budget(sk_ctx *ctx);
sk_status dense_blocked_to_host(sk_ctx *ctx, const sk_db *ref, const sk_db *query,
                                const sk_random *random, int out_mode, void *out, size_t budget);
size_t out_bytes(int out_mode, int64_t pairs, int K);

}  // namespace sk
