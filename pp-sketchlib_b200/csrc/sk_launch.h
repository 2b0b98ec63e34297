// sk_launch.h -- host-side declarations of the kernel launchers.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "sk_common.h"

namespace sk {

// One compiled instance of the tiled distance kernel.
struct TileConfig {
  int id;
  int tile_rows, tile_cols;      // CTA tile (rows x cols of pairs)
  int thread_rows, thread_cols;  // per-thread register block
  int max_kmers;                 // largest K the instance handles
  int stages;                    // pipeline depth
  int smem_bytes;
  cudaError_t (*launch)(const LaunchParams &, int grid, cudaStream_t);
  int (*blocks_per_sm)();        // resident CTAs per SM at this shape's shared memory
};

int tile_config_count();
const TileConfig *tile_config(int id);
// The 64 x 64 shape (8 x 4 pairs per thread, three CTAs per SM) used where
// 128 x 128 tiles would be mostly padding.
constexpr int kSmallTileConfig = 6;
// The shape with a coded instance.
constexpr int kCodedConfig = 1;
// Bytes of count scratch per slot (one per CTA, one per split tile).
inline size_t count_slot_bytes(const TileConfig &cfg, int k_slots) {
  return static_cast<size_t>(k_slots) * cfg.tile_rows * cfg.tile_cols * 2;
}

// aux_kernels.cu: lets `kernel` be launched with `bytes` of dynamic shared
// memory.  The limit belongs to the process, not to a context, so it is only
// ever raised: a launch of another thread keeps the size it asked for.
cudaError_t raise_smem_limit(const void *kernel, size_t bytes);
template <class... A>
cudaError_t raise_smem_limit(void (*kernel)(A...), size_t bytes) {
  return raise_smem_limit(reinterpret_cast<const void *>(kernel), bytes);
}

// code_kernels.cu: bin values of granules g0 .. g0 + n_g - 1 of a packed array
// of ng granules; the row and column encoders of one task.
cudaError_t prepare_code_kernels();
cudaError_t launch_code_values(const uint32_t *packed, int32_t kb, int32_t ng, int32_t g0,
                               int32_t n_g, uint32_t *values, int sm_count, cudaStream_t stream);
cudaError_t launch_codes(const CodeTask &t, int sm_count, cudaStream_t stream);

// query_kernel.cu: a narrow query job of at most kFewQueries rows.  `parts` is a
// workspace of `bytes`: few_queries_bytes() holds every reference's counts, or as
// many as fit `limit` (one CTA's at least), which are then taken part by part.
constexpr int kFewQueries = 128;
constexpr size_t kFewQueriesBytes = size_t(128) << 20;   // the limit of a context
int64_t few_queries_rows(int64_t n);   // rows computed for n queries, padding included
size_t few_queries_bytes(const JobParams &jp, int sm_count, size_t limit);
cudaError_t launch_few_queries(const JobParams &jp, uint16_t *parts, size_t bytes, DevStatus *status,
                               const volatile int *cancel, int sm_count, cudaStream_t stream);

// aux_kernels.cu
cudaError_t launch_pack(const uint64_t *words, int64_t n, int32_t n_kmers, int32_t s64,
                        int32_t ng, uint32_t *packed, cudaStream_t stream);
// Packs n samples (reference layout at `words`) into granules g0 .. g0+ng-1 of
// a packed array of ng_total granules.
cudaError_t launch_pack_range(const uint64_t *words, int64_t n, int32_t n_kmers, int32_t s64,
                              int32_t ng, int32_t g0, int32_t ng_total, uint32_t *packed,
                              cudaStream_t stream);
cudaError_t launch_unpack(const uint32_t *packed, int64_t n, int32_t n_kmers, int32_t s64,
                          int32_t ng, uint64_t *words, cudaStream_t stream);
cudaError_t launch_synth(const int32_t *parent, const uint32_t *thresh, int64_t n,
                         int32_t n_kmers, int32_t s64, uint64_t seed, uint64_t *words,
                         cudaStream_t stream);
// kNN over a condensed self column, or over dense rows.  Lists of at most
// kKnnListMax entries are kept per thread in shared memory, longer ones come from
// a radix select and a bitonic sort per row: the select costs its passes over the
// row whatever kNN is, the lists grow with kNN.  Lists and select, self calls in
// ms: 12,007 samples 4.7 and 5.9 with 1 neighbour, 5.5 and 6.1 with 16, 9.8 and
// 6.8 with 48, 65 and 16 with 200; 6,007 samples 1.3 and 1.6, 1.75 and 1.75, 3.2
// and 2.0, 19 and 2.9 (264 and 15 with 800).  100 rows of 30,011 references: 0.29
// and 0.30, 0.32 and 0.30, 0.48 and 0.31, 2.9 and 0.32.
constexpr int kKnnListMax = 16;
cudaError_t launch_knn_self(const float *col_vals, int64_t n, int32_t knn, int32_t jaccard,
                            int64_t *j_out, float *d_out, cudaStream_t stream);
cudaError_t launch_knn_rows(const float *vals, int64_t n_rows, int64_t n_cols, int32_t knn,
                            int64_t diag0, int32_t jaccard, int64_t *j_out, float *d_out,
                            cudaStream_t stream);
// Jaccard / log-Jaccard by intersection count 0 .. n-1 for jobs without
// random-match correction (JobParams::jtab / ltab).
cudaError_t launch_count_tables(double union_bits, int64_t n, float *jtab, double *ltab,
                                cudaStream_t stream);
cudaError_t launch_threshold_count(const float *vals, int64_t n, int32_t stride, int32_t col,
                                   float cutoff, int64_t *row_counts, cudaStream_t stream);
cudaError_t launch_threshold_fill(const float *vals, int64_t n, int32_t stride, int32_t col,
                                  float cutoff, const int64_t *row_offsets, int64_t *i_out,
                                  int64_t *j_out, float *d_out, cudaStream_t stream);
cudaError_t exclusive_scan_i64(const int64_t *in, int64_t *out, int64_t n, void *tmp,
                               size_t *tmp_bytes, cudaStream_t stream);
cudaError_t launch_long_to_square(const float *rr, int64_t n_rr, const float *qr,
                                  const float *qq, int64_t n_qq, float *square,
                                  cudaStream_t stream);
cudaError_t launch_square_to_long(const float *square, int64_t n, float *long_out,
                                  cudaStream_t stream);

}  // namespace sk
