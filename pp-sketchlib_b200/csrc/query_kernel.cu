// query_kernel.cu -- distances of a few queries against every reference.
//
// A 64-row tile of the distance kernel computes 64 rows whatever it holds, so
// one query against 30,011 references (K = 10, 156 words) took 6.3 ms, most of
// it padding; what the call cannot do without is one read of the references,
// 0.8 ms.  Here a thread owns four references (one 128-bit load per bit plane,
// straight from the packed stripes) and compares them with every query; the query
// words are broadcast from shared memory.  From 8 queries up a thread holds the 14
// planes of a block; for fewer the compiler holds a few at a time (32 registers
// for one query) and twice the warps keep as many loads in flight.  HBM-bound up
// to about 12 queries (14 LOP3 per query and 32 bins against 56 bytes), LOP3-bound
// above.
//
// The blocks of each k are cut into ranges so that a small reference set still
// fills the device; a range's counts go to a uint16 array [k][range][query]
// [reference], and a second kernel adds the ranges up and finishes the pairs,
// one per thread.  The array is bounded; more references than it holds the counts
// of are taken a part at a time.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "sk_device.cuh"
#include "sk_launch.h"

namespace sk {

namespace {

constexpr int kThreads = 128;
constexpr int kCols = 4 * kThreads;      // references per CTA
constexpr int kTileBlocks = 16;          // blocks whose query words are staged at a time
constexpr int kFinishPairs = 128;

template <int NQ>
__global__ void __launch_bounds__(kThreads)
few_queries_kernel(const JobParams jp, int groups, int ranges, uint16_t *__restrict__ parts, int64_t ldc,
                   DevStatus *status, const volatile int *cancel) {
  __shared__ __align__(16) uint32_t qw[kTileBlocks * kBbits * NQ];
  __shared__ int s_stop;
  if (threadIdx.x == 0) s_stop = poll_cancelled(status, cancel) ? 1 : 0;
  __syncthreads();
  if (s_stop) return;
  const int range = blockIdx.y % ranges, k = blockIdx.y / ranges;
  const int q0 = (blockIdx.x % groups) * NQ;   // this CTA's queries: q0 .. q0 + NQ - 1
  const int b0 = static_cast<int>(static_cast<int64_t>(jp.nb) * range / ranges);
  const int b1 = static_cast<int>(static_cast<int64_t>(jp.nb) * (range + 1) / ranges);
  const int64_t col = static_cast<int64_t>(blockIdx.x / groups) * kCols + 4 * threadIdx.x;
  const bool active = col < ldc;
  const uint32_t *src = jp.col_words + (col / kGranule) * kStripeWords + col % kGranule;
  const int64_t stride = static_cast<int64_t>(jp.ng_cols) * kStripeWords;   // words per block
  const uint32_t one = jp.one, hi_one = one << 16;
  uint32_t cnt[NQ][2];   // references 0, 1 and 2, 3 as 16-bit halves (at most 65,472)
#pragma unroll
  for (int q = 0; q < NQ; ++q) cnt[q][0] = cnt[q][1] = 0;
  for (int t0 = b0; t0 < b1; t0 += kTileBlocks) {
    const int nt = min(kTileBlocks, b1 - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < nt * kBbits * NQ; i += kThreads) {
      const int q = i % NQ, pl = i / NQ % kBbits, b = i / (NQ * kBbits);
      // queries past the last repeat it: the array holds them, their counts are not used
      const int64_t kb = static_cast<int64_t>(k) * jp.nb + t0 + b;
      const int row = min(q0 + q, static_cast<int>(jp.n_rows) - 1);
      qw[i] = jp.row_words[(kb * jp.ng_rows + row / kGranule) * kStripeWords + pl * kGranule +
                           row % kGranule];
    }
    __syncthreads();
    if (!active) continue;
    for (int b = 0; b < nt; ++b) {
      const uint32_t *p = src + (static_cast<int64_t>(k) * jp.nb + t0 + b) * stride;
      uint4 c[kBbits];
#pragma unroll
      for (int pl = 0; pl < kBbits; ++pl)
        c[pl] = __ldg(reinterpret_cast<const uint4 *>(p + pl * kGranule));
      const uint32_t *w = qw + b * kBbits * NQ;
      constexpr int G = NQ < 4 ? NQ : 4;   // queries compared at a time
#pragma unroll
      for (int g = 0; g < NQ; g += G) {
        uint32_t acc[G][4];
#pragma unroll
        for (int pl = 0; pl < kBbits; ++pl) {
          uint32_t qv[G];
          if constexpr (G == 4) {
            const uint4 v = *reinterpret_cast<const uint4 *>(w + pl * NQ + g);
            qv[0] = v.x; qv[1] = v.y; qv[2] = v.z; qv[3] = v.w;
          } else {
#pragma unroll
            for (int i = 0; i < G; ++i) qv[i] = w[pl * NQ + g + i];
          }
          const uint32_t cv[4] = {c[pl].x, c[pl].y, c[pl].z, c[pl].w};
#pragma unroll
          for (int i = 0; i < G; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              acc[i][j] = pl == 0 ? lop_eq(qv[i], cv[j]) : lop_eq_and(acc[i][j], qv[i], cv[j]);
        }
#pragma unroll
        for (int i = 0; i < G; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            cnt[g + i][h] = mad_u32(__popc(acc[i][2 * h + 1]), hi_one,
                                    mad_u32(__popc(acc[i][2 * h]), one, cnt[g + i][h]));
      }
    }
  }
  if (!active) return;
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    if (q0 + q < jp.n_rows)
      *reinterpret_cast<uint2 *>(
          parts + (static_cast<int64_t>(blockIdx.y) * jp.n_rows + q0 + q) * ldc + col) =
          make_uint2(cnt[q][0], cnt[q][1]);
}

// Pairs of query blockIdx.y with 128 references: a thread adds up the ranges
// of 8 references at every eighth k (128-bit loads), then finishes one pair.
__global__ void __launch_bounds__(kFinishPairs)
few_queries_finish_kernel(const JobParams jp, int ranges, const uint16_t *__restrict__ parts,
                          int64_t col_begin, int64_t ldc, const DevStatus *status) {
  __shared__ __align__(16) uint16_t sums[kNarrowKmers * kFinishPairs];
  if (reinterpret_cast<const volatile DevStatus *>(status)->error != 0) return;
  const int64_t gi = blockIdx.y, col0 = static_cast<int64_t>(blockIdx.x) * kFinishPairs;
  const int g = threadIdx.x % (kFinishPairs / 8);
  for (int k = threadIdx.x / (kFinishPairs / 8); k < jp.n_kmers; k += 8) {
    uint4 c = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 8
    for (int r = 0; r < ranges; ++r) {
      const uint4 v = *reinterpret_cast<const uint4 *>(
          parts + ((static_cast<int64_t>(k) * ranges + r) * jp.n_rows + gi) * ldc + col0 + 8 * g);
      c.x += v.x; c.y += v.y; c.z += v.z; c.w += v.w;
    }
    *reinterpret_cast<uint4 *>(sums + k * kFinishPairs + 8 * g) = c;
  }
  __syncthreads();
  const int64_t gj = col_begin + col0 + threadIdx.x;
  if (gj < jp.n_cols) finish_pair_any<false>(jp, gi, gj, sums + threadIdx.x, kFinishPairs);
}

// Queries a CTA compares and CTAs per reference range.  A group of up to 8
// costs little more than reading the references, 12 and 16 are LOP3-bound;
// 32 at once hold too few warps (3.76 ms for 32 queries against 30,011
// references, K = 10; two groups of 16: 2.8).
struct Groups {
  int nq, groups;
};
Groups query_groups(int64_t n) {
  for (int nq : {1, 2, 4, 8})
    if (n <= nq) return {nq, 1};
  const int by12 = static_cast<int>((n + 11) / 12), by16 = static_cast<int>((n + 15) / 16);
  return by12 * 12 < by16 * 16 ? Groups{12, by12} : Groups{16, by16};
}

// Block ranges per k over n references: enough CTAs for eight per SM, of at
// least eight blocks.
int query_ranges(const JobParams &jp, int64_t n, int sm_count) {
  const int64_t ctas = (n + kCols - 1) / kCols * query_groups(jp.n_rows).groups * jp.n_kmers;
  const int64_t want = (8 * static_cast<int64_t>(sm_count) + ctas - 1) / ctas;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(want, jp.nb / 8)));
}

int64_t padded_cols(int64_t n) { return (n + kFinishPairs - 1) / kFinishPairs * kFinishPairs; }

// Bytes of the counts of n references in `ranges` block ranges per k.
size_t parts_bytes(const JobParams &jp, int64_t n, int ranges) {
  return static_cast<size_t>(ranges) * jp.n_kmers * jp.n_rows * padded_cols(n) * 2;
}

}  // namespace

int64_t few_queries_rows(int64_t n) {
  const Groups g = query_groups(n);
  return static_cast<int64_t>(g.nq) * g.groups;
}

size_t few_queries_bytes(const JobParams &jp, int sm_count, size_t limit) {
  const size_t all = parts_bytes(jp, jp.n_cols, query_ranges(jp, jp.n_cols, sm_count));
  return std::min(all, std::max(limit, parts_bytes(jp, std::min<int64_t>(jp.n_cols, kCols), 1)));
}

cudaError_t launch_few_queries(const JobParams &jp, uint16_t *parts, size_t bytes, DevStatus *status,
                               const volatile int *cancel, int sm_count, cudaStream_t stream) {
  const Groups g = query_groups(jp.n_rows);
  // as many references at a time as their counts fit the workspace, in steps of
  // what a CTA takes
  int64_t step = jp.n_cols;
  int ranges = query_ranges(jp, step, sm_count);
  auto fits = [&] { return parts_bytes(jp, step, ranges) <= bytes; };
  while (!fits() && step > kCols) {
    step = (step / 2 + kCols - 1) / kCols * kCols;
    ranges = query_ranges(jp, step, sm_count);
  }
  while (!fits() && ranges > 1) --ranges;
  for (int64_t c0 = 0; c0 < jp.n_cols; c0 += step) {
    const int64_t n = std::min(step, jp.n_cols - c0), ldc = padded_cols(n);
    JobParams part = jp;   // whose columns begin at c0, a whole number of granules
    part.col_words += c0 / kGranule * kStripeWords;
    // a range's groups are neighbours, so that they share its references in L2
    const dim3 grid(static_cast<unsigned int>((n + kCols - 1) / kCols * g.groups),
                    static_cast<unsigned int>(jp.n_kmers * ranges));
#define SK_FEW(N)                                                                                \
  few_queries_kernel<N><<<grid, kThreads, 0, stream>>>(part, g.groups, ranges, parts, ldc, status, \
                                                       cancel)
    switch (g.nq) {
      case 1: SK_FEW(1); break;
      case 2: SK_FEW(2); break;
      case 4: SK_FEW(4); break;
      case 8: SK_FEW(8); break;
      case 12: SK_FEW(12); break;
      default: SK_FEW(16); break;
    }
#undef SK_FEW
    const dim3 finish(static_cast<unsigned int>(ldc / kFinishPairs), static_cast<unsigned int>(jp.n_rows));
    few_queries_finish_kernel<<<finish, kFinishPairs, 0, stream>>>(jp, ranges, parts, c0, ldc, status);
  }
  return cudaGetLastError();
}

}  // namespace sk
