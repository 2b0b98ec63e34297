// code_kernels.cu -- bin values rewritten as short codes, one dictionary per
// block of 128 rows, for the distance kernel's coded instance.
//
// Two bins match when their 14-bit values are equal, and only a tile's row
// values matter to it: a column value that no row of the tile holds matches
// nothing, whatever it is.  So each bin of a block of 128 rows gets a
// dictionary of its distinct values (codes 1 .. D, D <= 128), rows and columns
// are rewritten as codes (0: not in the dictionary), and the distance kernel
// compares ceil(log2(D + 1)) <= 8 bit planes instead of 14 (10.0 ms instead of
// 18.9 at 4,096 samples, K = 8, 156 words; encoding takes 4.1).  Equality of
// codes is equality of values, so the counts are the same integers.  D depends on
// the data (about 60 .. 80 of 128 rows on random trees: 7 planes; 40 .. 60 in
// clades: 6), its bound does not.
//
//   code_values   the packed stripes as bin values, once per call;
//   code_rows     per (row block, k, 32-bin block): the dictionaries, the
//                 rows' codes, the number of planes;
//   code_columns  the columns' codes, by table lookup.
//
// Layout, per row block rb and block kb = k * nb + block: a row of 128-sample
// groups, the block's own rows first, then the columns; a group is
// [8 planes][128 samples] uint32 (4 KB), of which the first `planes[rb][kb]`
// are written and read.  Bit 8 b + q of a plane word is bin (4 q + b) of the
// block in the order transpose_planes leaves them; rows and columns go through
// the same steps, so the order does not matter to a count.
#include <cuda_runtime.h>

#include <cstdint>

#include "sk_device.cuh"
#include "sk_launch.h"

namespace sk {

namespace {

constexpr int kTableBytes = 1 << kBbits;   // one byte per bin value
constexpr int kPassBins = 4;               // bins per pass of the row encoder: 8 passes per block
constexpr int kRowThreads = kCodeGroup;    // one row per thread
constexpr int kLookupThreads = kCodeChunkGroups * 32;
constexpr int kTableWarps = 4;             // (bin, row block) of a pass each
constexpr int kColThreads = kLookupThreads + 32 * kTableWarps;   // and four table warps: 512 x 112 + 128 x 32 registers
constexpr int kColSamples = 4;             // columns per thread
constexpr int kPairTableBytes = 2 * kTableBytes + 16;   // 2-byte entries, one spare
constexpr int kTableSets = 3;              // passes the table warps may be ahead
// the sets of two tables, two buffers of two dictionary lists
constexpr int kColTableBytes = 2 * kTableSets * kPairTableBytes + 2 * 2 * kCodeListWords * 2;
constexpr uint64_t kListWaitNs = 2000000000ull;   // 2 s bounded wait
constexpr int kValueThreads = 256;

// (a & m) | (b & ~m): one LOP3.
__device__ __forceinline__ uint32_t bit_select(uint32_t a, uint32_t b, uint32_t m) {
  return (a & m) | (b & ~m);
}

// Exchanges the off-diagonal s x s blocks of a 2s x 2s bit matrix whose row r
// is bits of a and row r + s bits of c: two shifts and two LOP3s.
__device__ __forceinline__ void butterfly(uint32_t &a, uint32_t &c, int s, uint32_t m) {
  const uint32_t x = bit_select(a, c << s, m);
  c = bit_select(a >> s, c, m);
  a = x;
}

// 14 plane words of one sample (bit i: bin i) -> 16 words of two 16-bit bin
// values each (word j: bin j in the low half, bin j + 16 in the high half): a
// 16 x 16 bit transpose in both halves at once.
__device__ __forceinline__ void transpose_planes(uint32_t (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t a = w[i], c = w[i + 8];
    w[i] = __byte_perm(a, c, 0x6240);
    w[i + 8] = __byte_perm(a, c, 0x7351);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if ((i & 4) == 0) butterfly(w[i], w[i + 4], 4, 0x0F0F0F0Fu);
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if ((i & 2) == 0) butterfly(w[i], w[i + 2], 2, 0x33333333u);
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if ((i & 1) == 0) butterfly(w[i], w[i + 1], 1, 0x55555555u);
}

// 8 words of four one-byte codes (word q: the codes of pass q) -> 8 plane
// words: an 8 x 8 bit transpose in each byte.
__device__ __forceinline__ void transpose_codes(uint32_t (&a)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((i & 4) == 0) butterfly(a[i], a[i + 4], 4, 0x0F0F0F0Fu);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((i & 2) == 0) butterfly(a[i], a[i + 2], 2, 0x33333333u);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((i & 1) == 0) butterfly(a[i], a[i + 1], 1, 0x55555555u);
}

// The value of bin b of pass q (two words hold a pass's four bins).
template <int B>
__device__ __forceinline__ uint32_t pass_value(uint32_t w0, uint32_t w1) {
  const uint32_t w = B < 2 ? w0 : w1;
  return (B & 1) ? w >> 16 : w & 0xFFFFu;
}

__device__ __forceinline__ bool cancelled(const DevStatus *status) {
  return (reinterpret_cast<const volatile DevStatus *>(status)->error & 2u) != 0;
}

// One CTA per (kb, row block).  Per pass of four bins, each row writes its
// index at its value's entry of the bin's table; the row found there
// afterwards stands for the value.  The standing rows are numbered by ballots,
// put value and code into the dictionary, and every row reads its code back.
// The tables need no clearing: only entries written in the pass are read.
// Bound by the barriers between those steps (four per pass); three CTAs per SM
// overlap them.
__global__ void __launch_bounds__(kRowThreads, 3)
code_rows_kernel(const CodeTask t) {
  extern __shared__ unsigned char row_tables[];   // [kPassBins][kTableBytes]
  __shared__ int warp_count[kRowThreads / 32][kPassBins];
  if (__syncthreads_or(cancelled(t.status))) return;   // all of the CTA or none
  const int row = threadIdx.x, warp = row >> 5, lane = row & 31;
  const int64_t items = static_cast<int64_t>(t.kb) * t.n_rb;
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const int rb = static_cast<int>(item % t.n_rb);
    const int kb = static_cast<int>(item / t.n_rb);
    // rows past the last sample repeat it, so they add no value of their own
    int64_t s = static_cast<int64_t>(t.layout.rb0 + rb) * kCodeGroup + row;
    if (s >= t.n_rows) s = t.n_rows - 1;
    const uint32_t *src = t.row_words +
                          (static_cast<int64_t>(kb) * t.ng_rows + s / kGranule) * kStripeWords +
                          s % kGranule;
    uint32_t w[16];
#pragma unroll
    for (int p = 0; p < kBbits; ++p) w[p] = src[p * kGranule];
    w[14] = w[15] = 0;
    transpose_planes(w);
    uint16_t *list = t.lists + (static_cast<int64_t>(rb) * t.kb + kb) * kCodeListWords;
    uint32_t code[8];
    int most = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t v[kPassBins] = {
          pass_value<0>(w[2 * q], w[2 * q + 1]), pass_value<1>(w[2 * q], w[2 * q + 1]),
          pass_value<2>(w[2 * q], w[2 * q + 1]), pass_value<3>(w[2 * q], w[2 * q + 1])};
#pragma unroll
      for (int b = 0; b < kPassBins; ++b)
        row_tables[b * kTableBytes + v[b]] = static_cast<unsigned char>(row);
      __syncthreads();
      bool mine[kPassBins];
      uint32_t own[kPassBins];   // a standing row's code
      unsigned int bal[kPassBins];
#pragma unroll
      for (int b = 0; b < kPassBins; ++b) {
        mine[b] = row_tables[b * kTableBytes + v[b]] == row;
        bal[b] = __ballot_sync(0xffffffffu, mine[b]);
        if (lane == b) warp_count[warp][b] = __popc(bal[b]);
      }
      __syncthreads();
#pragma unroll
      for (int b = 0; b < kPassBins; ++b) {
        int before = 0, total = 0;
#pragma unroll
        for (int u = 0; u < kRowThreads / 32; ++u) {
          const int n = warp_count[u][b];
          before += u < warp ? n : 0;
          total += n;
        }
        most = max(most, total);
        uint16_t *l = list + (q * kPassBins + b) * kCodeGroup;   // word 2q + b / 2, half b % 2
        if (mine[b]) {
          const int rank = before + __popc(bal[b] & ((1u << lane) - 1u));
          own[b] = rank + 1;
          row_tables[b * kTableBytes + v[b]] = static_cast<unsigned char>(rank + 1);
          l[rank] = static_cast<uint16_t>(v[b]);
        }
        if (row >= total) l[row] = kCodeNoValue;
      }
      __syncthreads();
      uint32_t c = 0;
#pragma unroll
      for (int b = 0; b < kPassBins; ++b)
        c |= (mine[b] ? own[b] : static_cast<uint32_t>(row_tables[b * kTableBytes + v[b]])) << (8 * b);
      code[q] = c;
      __syncthreads();
    }
    transpose_codes(code);
    // every thread counted the same totals; planes 4 .. 8 are compiled in the
    // distance kernel
    const int planes = max(kCodeMinPlanes, 32 - __clz(most));
    uint32_t *dst = t.words + code_stripe(t.layout, t.kb, t.layout.rb0 + rb, kb, 0) + row;
    // all planes: a pair of blocks reads as many as its larger dictionary has
#pragma unroll
    for (int p = 0; p < kCodeMaxPlanes; ++p) dst[p * kCodeGroup] = code[p];
    if (row == 0) t.planes[static_cast<int64_t>(rb) * t.kb + kb] = static_cast<uint8_t>(planes);
  }
}

// Packed stripes -> bin values, [kb][16 words][padded samples]: word j of a
// sample holds its bins j and j + 16 of the block in the order
// transpose_planes leaves them, doubled (offsets of 2-byte table entries).  The transpose is paid once per database
// instead of once per row block (32 times at 4,096 samples).  HBM-bound: 56
// bytes read and 64 written per sample and block.
__global__ void __launch_bounds__(kValueThreads)
code_values_kernel(const uint32_t *__restrict__ packed, int32_t kb, int32_t ng, int32_t g0,
                   int32_t n_g, uint32_t *__restrict__ values) {
  const int64_t total = static_cast<int64_t>(kb) * n_g * kGranule;
  const int64_t ld = static_cast<int64_t>(ng) * kGranule;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kValueThreads) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * kValueThreads) {
    const int64_t r = i / kGranule;
    const int64_t k = r / n_g, g = g0 + r % n_g;
    const int lane = static_cast<int>(i % kGranule);
    const uint32_t *src = packed + (k * ng + g) * kStripeWords + lane;
    uint32_t w[16];
#pragma unroll
    for (int p = 0; p < kBbits; ++p) w[p] = src[p * kGranule];
    w[14] = w[15] = 0;
    transpose_planes(w);
    uint32_t *dst = values + k * 16 * ld + g * kGranule + lane;
#pragma unroll
    for (int j = 0; j < 16; ++j) dst[j * ld] = w[j] << 1;   // 14-bit values: no carry between halves
  }
}

// One CTA per (kb, two neighbouring row blocks, range of up to
// kCodeChunkGroups column groups) at a time.  16 warps look columns up, four
// consecutive columns per thread: a pass takes one value word (two bins) of
// each, from tables indexed by the 14-bit value whose 16-bit entries hold the
// codes of both row blocks.  Four more warps clear and fill the tables of the
// passes ahead, one (bin, row block) each from the dictionary lists, which come
// by bulk copy an item ahead.  Three sets of tables, each with an mbarrier for
// "filled" and one for "read": no warp waits for the slowest of a pass, and one
// that transposes and stores the codes of an item does so while others look up
// the next.  A lookup's 32 lanes fall on random banks (3.2 cycles of the
// shared-memory pipe per warp), the bound of a full range.
//
// What held earlier forms back, at 4,096 samples (K = 8, 156 words): one row
// block per lookup, loads one pass ahead of their use (a pass then lasts one
// memory latency): 6.6 ms; list entries loaded by the lookup warps that also
// filled the tables, all passes unrolled (instruction fetch): 4.5 to 5.1 ms; two
// sets of tables and a barrier of the CTA per pass: 3.59 ms (8,000 samples 14.6
// ms, 300 queries against 20,011 3.31).  As it stands 2.92 ms (10.2, 2.53), about
// half of the shared-memory pipe's time.  The next item's lines prefetched to L2,
// which helped few row blocks at a barrier per pass, costs since (2.63 for 2.53,
// 3.00 for 2.91); loads 8 words ahead instead of 4 spill (3.60).
__global__ void __launch_bounds__(kColThreads, 1) code_columns_kernel(const CodeTask t) {
  extern __shared__ __align__(128) unsigned char tables[];   // [kTableSets][2 bins] tables
  // dictionary lists of the current and the next item: [2][2 row blocks]
  uint16_t *lists = reinterpret_cast<uint16_t *>(tables + 2 * kTableSets * kPairTableBytes);
  __shared__ __align__(8) uint64_t list_bar[2];
  __shared__ __align__(8) uint64_t filled[kTableSets], read[kTableSets];
  if (__syncthreads_or(cancelled(t.status))) return;   // all of the CTA or none
  const int tid = threadIdx.x, lane = tid & 31;
  for (int i = tid; i < 2 * kTableSets * kPairTableBytes / 16; i += kColThreads)
    reinterpret_cast<uint4 *>(tables)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    mbar_init(&list_bar[0], 1);
    mbar_init(&list_bar[1], 1);
    for (int i = 0; i < kTableSets; ++i) {
      mbar_init(&filled[i], kTableWarps);
      mbar_init(&read[i], kLookupThreads / 32);
    }
    fence_mbar_init();
  }
  // the work items, (kb, chunk) in steps of the grid; a chunk names the first
  // of two row blocks of the range and its first and end column group
  const int step_kb = gridDim.x / t.n_chunks, step_c = gridDim.x % t.n_chunks;
  int kb = blockIdx.x / t.n_chunks, ci = blockIdx.x % t.n_chunks;
  auto advance = [&](int &k, int &c) {
    k += step_kb;
    c += step_c;
    if (c >= t.n_chunks) {
      c -= t.n_chunks;
      ++k;
    }
    return k < t.kb;
  };
  int4 chunk = t.chunks[ci];
  __syncthreads();

  if (tid >= kLookupThreads) {
    // ------------------------------------------------------------ table warps
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    const int role = (tid - kLookupThreads) >> 5, bin = role & 1, block = role >> 1;
    auto fetch = [&](const int4 &c, int k, int b) {   // starts the copy of an item's lists
      const int n = min(2, t.n_rb - c.x);
      mbar_arrive_expect_tx(&list_bar[b], n * kCodeListWords * 2);
      for (int r = 0; r < n; ++r)
        bulk_g2s(lists + (b * 2 + r) * kCodeListWords,
                 t.lists + (static_cast<int64_t>(c.x + r) * t.kb + k) * kCodeListWords,
                 kCodeListWords * 2, &list_bar[b]);
    };
    // a list that never lands, or a set never given back, is recorded, once;
    // what is there instead is still in range.  No list is fetched after that,
    // and those in flight land (or their wait runs out again) before the CTA's
    // shared memory goes away.
    bool waits = true;
    auto wait = [&](uint64_t *bar, uint32_t parity) {
      if (waits && !mbar_wait_bounded(bar, parity, kListWaitNs)) {
        waits = false;
        atomicOr(&t.status->error, 1u);
        t.status->where = 3;
      }
    };
    // this lane's four values of the pass's bin; none where the row block ends
    auto entries = [&](const int4 &c, int b, int pass) {
      if (c.x + block >= t.n_rb) return make_uint2(~0u, ~0u);
      return reinterpret_cast<const uint2 *>(lists + (b * 2 + block) * kCodeListWords +
                                             (2 * pass + bin) * kCodeGroup)[lane];
    };
    // unused values go to the spare entry behind the table
    auto put = [&](int set, uint2 vals, int code) {
      unsigned char *tab = tables + (set * 2 + bin) * kPairTableBytes + block;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t v = ((e < 2 ? vals.x : vals.y) >> (16 * (e & 1))) & 0xFFFFu;
        tab[2 * min(v, static_cast<uint32_t>(kTableBytes))] =
            static_cast<unsigned char>(code < 0 ? 0 : code + e);
      }
    };
    const int code = 4 * lane + 1;
    int b = 0;                    // list buffer of the current item
    uint32_t list_phase[2] = {0, 0};
    int set = 0;
    uint32_t phase = 1;           // a new set's first wait passes
    uint2 held[kTableSets];       // the sets' entries, the set to fill next first
#pragma unroll
    for (int i = 0; i < kTableSets; ++i) held[i] = make_uint2(~0u, ~0u);
    if (role == 0 && lane == 0) fetch(chunk, kb, 0);
    while (true) {
      int next_kb = kb, next_ci = ci;
      const bool more = advance(next_kb, next_ci);
      const int4 next = t.chunks[more ? next_ci : ci];
      // every table warp is done with the other buffer
      asm volatile("bar.sync 1, %0;" ::"n"(kTableWarps * 32) : "memory");
      if (more && waits && role == 0 && lane == 0) fetch(next, next_kb, b ^ 1);
      wait(&list_bar[b], list_phase[b]);
      if (waits) list_phase[b] ^= 1u;
#pragma unroll 1
      for (int pass = 0; pass < 16; ++pass) {
        const uint2 vals = entries(chunk, b, pass);
        wait(&read[set], phase);
        put(set, held[0], -1);
        __syncwarp();
        put(set, vals, code);
        __syncwarp();
        if (lane == 0) mbar_arrive(&filled[set]);
#pragma unroll
        for (int i = 0; i + 1 < kTableSets; ++i) held[i] = held[i + 1];
        held[kTableSets - 1] = vals;
        if (++set == kTableSets) {
          set = 0;
          phase ^= 1u;
        }
      }
      if (!more) {
        if (!waits && role == 0 && lane == 0)
          for (int i = 0; i < 2; ++i) mbar_wait_bounded(&list_bar[i], list_phase[i], kListWaitNs);
        return;
      }
      kb = next_kb;
      ci = next_ci;
      chunk = next;
      b ^= 1;
    }
  }

  // -------------------------------------------------------------- lookup warps
  asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
  const int64_t ld4 = static_cast<int64_t>(t.ng_cols) * (kGranule / 4);   // uint4 per value word
  // this thread's value words of an item; active: it has columns there
  auto values_of = [&](const int4 &c, int k, bool &active) {
    const int64_t s = static_cast<int64_t>(c.y) * kCodeGroup + tid * kColSamples;
    active = s < static_cast<int64_t>(c.z) * kCodeGroup;
    return reinterpret_cast<const uint4 *>(t.col_values) + static_cast<int64_t>(k) * 16 * ld4 +
           (active ? s / 4 : 0);
  };
  bool active;
  const uint4 *val = values_of(chunk, kb, active);
  uint4 w[4] = {};   // value words j .. j + 3
  if (active) {
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = val[j * ld4];
  }
  int set = 0;
  uint32_t phase = 0;
  bool waits = true;
  while (true) {
    int next_kb = kb, next_ci = ci;
    const bool more = advance(next_kb, next_ci);
    const int4 next = t.chunks[more ? next_ci : ci];
    bool next_active;
    const uint4 *next_val = values_of(next, more ? next_kb : kb, next_active);
    // planes of the pair of blocks kb belongs to (the count per row block is even)
    uint32_t pair_planes[2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
      pair_planes[r] = reinterpret_cast<const uint16_t *>(
          t.planes)[(static_cast<int64_t>(min(chunk.x + r, t.n_rb - 1)) * t.kb + kb) / 2];
    uint32_t code[2][kColSamples][8];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint4 v = w[j & 3];
      if (j < 12) {
        if (active) w[j & 3] = val[(j + 4) * ld4];
      } else if (more && next_active) {
        w[j & 3] = next_val[(j - 12) * ld4];
      }
      if (waits && !mbar_wait_bounded(&filled[set], phase, kListWaitNs)) {
        waits = false;
        atomicOr(&t.status->error, 1u);
        t.status->where = 4;
      }
      if (active) {
        const unsigned char *tab = tables + set * 2 * kPairTableBytes;
        const uint32_t vv[kColSamples] = {v.x, v.y, v.z, v.w};   // entry offsets: 2 x value
#pragma unroll
        for (int i = 0; i < kColSamples; ++i) {
          const uint32_t c0 = *reinterpret_cast<const uint16_t *>(tab + (vv[i] & 0xFFFFu));
          const uint32_t c1 =
              *reinterpret_cast<const uint16_t *>(tab + kPairTableBytes + (vv[i] >> 16));
          // bytes: first block's codes of the two bins, second block's
          const uint32_t both = __byte_perm(c0, c1, 0x5140);
          if (j & 1) {
            const uint32_t even = code[0][i][j >> 1];
            code[0][i][j >> 1] = __byte_perm(even, both, 0x5410);
            code[1][i][j >> 1] = __byte_perm(even, both, 0x7632);
          } else {
            code[0][i][j >> 1] = both;
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&read[set]);
      if (++set == kTableSets) {
        set = 0;
        phase ^= 1u;
      }
    }
    if (active) {
      const int64_t s = static_cast<int64_t>(chunk.y) * kCodeGroup + tid * kColSamples;
      const int32_t cg = static_cast<int32_t>(s / kCodeGroup);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int local = chunk.x + r, rb = t.layout.rb0 + local;
        // the second row block may not exist, or start one group later
        if (local < t.n_rb && cg >= code_first_group(t.layout, rb)) {
#pragma unroll
          for (int i = 0; i < kColSamples; ++i) transpose_codes(code[r][i]);
          const int planes = static_cast<int>(max(pair_planes[r] & 0xFFu, pair_planes[r] >> 8));
          uint32_t *dst = t.words +
                          code_stripe(t.layout, t.kb, rb, kb,
                                      1 + cg - code_first_group(t.layout, rb)) +
                          s % kCodeGroup;
#pragma unroll
          for (int p = 0; p < kCodeMaxPlanes; ++p)
            if (p < planes)
              *reinterpret_cast<uint4 *>(dst + p * kCodeGroup) =
                  make_uint4(code[r][0][p], code[r][1][p], code[r][2][p], code[r][3][p]);
        }
      }
    }
    if (!more) return;
    kb = next_kb;
    ci = next_ci;
    chunk = next;
    val = next_val;
    active = next_active;
  }
}

}  // namespace

cudaError_t prepare_code_kernels() {
  const cudaError_t e = raise_smem_limit(code_rows_kernel, kPassBins * kTableBytes);
  return e == cudaSuccess ? raise_smem_limit(code_columns_kernel, kColTableBytes) : e;
}

cudaError_t launch_code_values(const uint32_t *packed, int32_t kb, int32_t ng, int32_t g0,
                               int32_t n_g, uint32_t *values, int sm_count, cudaStream_t stream) {
  const int64_t blocks =
      (static_cast<int64_t>(kb) * n_g * kGranule + kValueThreads - 1) / kValueThreads;
  const int grid = static_cast<int>(blocks < 8 * sm_count ? blocks : 8 * sm_count);
  code_values_kernel<<<grid, kValueThreads, 0, stream>>>(packed, kb, ng, g0, n_g, values);
  return cudaGetLastError();
}

cudaError_t launch_codes(const CodeTask &t, int sm_count, cudaStream_t stream) {
  cudaError_t e = prepare_code_kernels();
  if (e != cudaSuccess) return e;
  const int64_t row_items = static_cast<int64_t>(t.kb) * t.n_rb;
  const int64_t col_items = static_cast<int64_t>(t.kb) * t.n_chunks;
  const int64_t g1 = row_items < 3 * sm_count ? row_items : 3 * sm_count;
  const int64_t g2 = col_items < sm_count ? col_items : sm_count;
  code_rows_kernel<<<static_cast<int>(g1), kRowThreads, kPassBins * kTableBytes, stream>>>(t);
  code_columns_kernel<<<static_cast<int>(g2), kColThreads, kColTableBytes, stream>>>(t);
  return cudaGetLastError();
}

}  // namespace sk
