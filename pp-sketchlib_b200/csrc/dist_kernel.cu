// dist_kernel.cu -- the fused bit-sliced MinHash distance kernel for sm_100a.
//
// A persistent kernel: every CTA pulls work items (job, tile, k range) from a
// device queue, so one launch can serve one all-vs-all, one query batch or a
// whole batch of unrelated databases of different sizes, k sets and sketch
// widths.  One thread of a producer warp stages, step by step, the bit planes
// of the tile's row and column samples into shared memory with bulk copies (TMA
// engine, mbarrier completion) and records each step in a per-stage descriptor.
// The other warps consume: each thread intersects a TQ x TR register block of
// pairs
//     acc = AND over planes of ~(row_word ^ col_word)   (one LOP3 per plane)
//     count += popc(acc)                                 (POPC + IMAD)
// which is calc_intersize (src/dist/dist.cpp:50-78) for 32 bins at a time,
// counts itself off the stage, parks its per-k counts in L2-resident scratch,
// and after a whole tile's last k turns its own pairs into random-corrected
// Jaccards and the log-linear core/accessory fit, written straight to the long
// form.  Tiles cut into several items are finished by a second kernel.
//
// The planes are the 14 of the packed database (2 blocks per step), or the 4 to
// 8 of dictionary codes (code_kernels.cu; 8 blocks per step, compared in pairs
// of blocks so that one block's popcounts overlap the other's LOP3s).  Bound by
// the LOP3 rate: 4,096 samples at K = 8, 156 words, 128 x 128 tiles: 14 planes
// 18.9 ms (0.84 of it), 7 planes 10.4 ms (0.79).
//
// Replaces calculate_dists (src/gpu/dist.cu:164-317): one thread per pair with
// strided 8-byte global loads there; register-blocked tiles over staged
// stripes here.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>

#include "sk_device.cuh"
#include "sk_launch.h"

namespace sk {

constexpr int kBlocksPerStage = 2;   // 32-bin blocks per pipeline stage
constexpr int kCodedBlocks = 8;      // the same for coded tiles, whose blocks are half as large
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s bounded waits

// Per-stage step descriptor written by the producer before it arms the stage.
struct StepMeta {
  int32_t job;
  int32_t ti, tj;     // tile coordinates within the job
  int32_t kidx;       // count slot of this step: k-mer index x nchunk + chunk
  int32_t flags;      // kStepEnd / kStepLastOfK (last step of a count slot) / kStepLastOfItem
  int32_t split;      // split slot of the item, -1 for whole tiles
  uint32_t planes;    // coded: bit planes of the step's blocks, one byte each (0: no block)
};
constexpr int32_t kStepEnd = 1, kStepLastOfK = 2, kStepLastOfItem = 4;

template <int QT, int RT, int TQ, int TR, int STAGES, bool CODED>
struct TileShape {
  static constexpr int kThreads = (QT / TQ) * (RT / TR);   // consumers
  // 16 consumer warps leave 96 registers a thread once a producer warp joins
  // them (five warps on one sub-partition), too few for the pair block, so
  // that shape launches a whole producer warpgroup and the consumers take
  // over the registers it does not need: 512 x 112 + 128 x 32 = 640 x 96.
  static constexpr bool kSplitRegs = kThreads == 512;
  static constexpr int kBlockThreads = kThreads + (kSplitRegs ? 128 : 32);   // and the producer
  static constexpr int kPairsPerThread = TQ * TR;
  static constexpr int kQG = QT / kGranule;
  static constexpr int kRG = RT / kGranule;
  static constexpr int kStageQWords =
      CODED ? kCodedBlocks * kCodeStripeWords : kBlocksPerStage * kQG * kStripeWords;
  static constexpr int kStageRWords =
      CODED ? kCodedBlocks * kCodeStripeWords : kBlocksPerStage * kRG * kStripeWords;
  static constexpr int kStageBytes = (kStageQWords + kStageRWords) * 4;
  static constexpr int kSmemBytes = STAGES * kStageBytes;
  static_assert(QT % kGranule == 0 && RT % kGranule == 0, "tiles are whole granules");
  static_assert(kGranule % TQ == 0 && kGranule % TR == 0, "thread blocks stay in a granule");
  static_assert(TQ % 4 == 0 && TR % 4 == 0, "128-bit shared loads");
  static_assert(kPairsPerThread % 8 == 0, "counts are stored as 16-byte groups");
  static_assert(QT % RT == 0, "triangular map needs tile_rows multiple of tile_cols");
  static_assert(STAGES >= 2, "the producer runs ahead of the consumers");
  static_assert(kThreads % 32 == 0, "whole warps");
  static_assert(!CODED || (QT == kCodeGroup && RT == kCodeGroup), "a coded tile is one group by one");
};

// Adds one 32-bin block's matches of a thread's TQ x TR pairs to its counts:
// the block's PLANES bit planes of the rows at qb and the columns at rb, LD
// words from one plane to the next.  Counts of columns 2c and 2c + 1 share a
// register; one and hi_one are 1 and 1 << 16 at run time.
template <int TQ, int TR, int PLANES, int LD>
__device__ __forceinline__ void count_block(const uint32_t *qb, const uint32_t *rb, uint32_t one,
                                            uint32_t hi_one, uint32_t (&cnt)[TQ][TR / 2]) {
  uint32_t acc[TQ][TR];
#pragma unroll
  for (int pl = 0; pl < PLANES; ++pl) {
    uint32_t qv[TQ], rv[TR];
    // column words before row words: measured 0.3% faster than the reverse
#pragma unroll
    for (int j = 0; j < TR; j += 4) {
      const uint4 v = *reinterpret_cast<const uint4 *>(rb + pl * LD + j);
      rv[j] = v.x; rv[j + 1] = v.y; rv[j + 2] = v.z; rv[j + 3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < TQ; i += 4) {
      const uint4 v = *reinterpret_cast<const uint4 *>(qb + pl * LD + i);
      qv[i] = v.x; qv[i + 1] = v.y; qv[i + 2] = v.z; qv[i + 3] = v.w;
    }
    // column-major issue order: measured 0.5% faster than row-major
#pragma unroll
    for (int j = 0; j < TR; ++j)
#pragma unroll
      for (int i = 0; i < TQ; ++i)
        acc[i][j] = pl == 0 ? lop_eq(qv[i], rv[j]) : lop_eq_and(acc[i][j], qv[i], rv[j]);
  }
#pragma unroll
  for (int i = 0; i < TQ; ++i)
#pragma unroll
    for (int j = 0; j < TR / 2; ++j)
      cnt[i][j] = mad_u32(__popc(acc[i][2 * j + 1]), hi_one,
                          mad_u32(__popc(acc[i][2 * j]), one, cnt[i][j]));
}

// Two blocks of coded tiles with as many planes, so that the popcounts of the
// first overlap the LOP3s of the second.
template <int TQ, int TR, int PLANES>
__device__ __forceinline__ void count_pair(const uint32_t *qb, const uint32_t *rb, uint32_t one,
                                           uint32_t hi_one, uint32_t (&cnt)[TQ][TR / 2]) {
  count_block<TQ, TR, PLANES, kCodeGroup>(qb, rb, one, hi_one, cnt);
  count_block<TQ, TR, PLANES, kCodeGroup>(qb + kCodeStripeWords, rb + kCodeStripeWords, one, hi_one,
                                          cnt);
}

// Count scratch layout (per CTA slot, and per split slot): [k][threads][pairs
// per thread] uint16; a thread writes and reads back only its own entries.
// WIDE: the instance for jobs with more than kNarrowKmers k-mer lengths or
// sketches counted in chunks (one count slot per chunk of kMaxChunkBlocks
// blocks); the narrow instance keeps one slot per k and the unrolled
// epilogues, whose code size the hot loop is sensitive to.
// CODED: the narrow instance over the tiles' codes (code_kernels.cu): 4 to 8
// planes per block instead of 14, the number given per block.
template <int QT, int RT, int TQ, int TR, int STAGES, int MINB, bool WIDE, bool CODED>
__global__ void __launch_bounds__(TileShape<QT, RT, TQ, TR, STAGES, CODED>::kBlockThreads, MINB)
    dist_items_kernel(const LaunchParams lp) {
  using S = TileShape<QT, RT, TQ, TR, STAGES, CODED>;
  static_assert(!(WIDE && CODED), "wide jobs are not coded");
  constexpr int kStep = CODED ? kCodedBlocks : kBlocksPerStage;   // blocks per step
  constexpr int NT = S::kThreads;
  constexpr int PT = S::kPairsPerThread;
  constexpr int TCOLS = RT / TR;

  extern __shared__ __align__(128) unsigned char smem[];
  uint32_t *sq = reinterpret_cast<uint32_t *>(smem);
  uint32_t *sr = sq + STAGES * S::kStageQWords;
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES];
  __shared__ StepMeta meta[STAGES];
  __shared__ volatile int s_abort;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], NT / 32);
    }
    fence_mbar_init();
    s_abort = 0;
  }
  __syncthreads();

  // ---------------------------------------------------------------- producer
  // One thread of its own warp keeps STAGES steps in flight: it waits until
  // every consumer warp has left a stage, then issues the copies of the step
  // STAGES later.  When a consumer warp did this in turn it waited for the
  // slowest warp of the step while its scheduler ran one warp short, about 5%
  // of a launch over coded tiles.
  if (warp >= NT / 32) {
    if constexpr (S::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (tid != NT) return;
    const uint32_t *rows = nullptr, *cols = nullptr;
    const uint8_t *planes_of = nullptr;   // coded: planes of the row block's blocks
    int64_t kb_stride = 0;                // coded: words from one block to the next
    int32_t job = 0, ti = 0, tj = 0, k = 0, k1 = 0, split = -1, nb = 0, ngr = 0, ngc = 0;
    int32_t b0 = 0, bstart = 0, bend = 0, bpart = 0, nbpart = 1;   // block range of each k
    int32_t slot = 0, slot_end = 0, chunk_nb = 0;   // WIDE: count slot, its last block + 1
    bool have = false;
    uint32_t armed = 0;   // steps whose copies were issued
    int s = 0;
    uint32_t parity = 1;  // of the phase in which the consumers leave the stage (first: none)
    for (uint32_t t = 0;; ++t) {
      if (t >= STAGES && !mbar_wait_bounded(&empty_bar[s], parity, kWaitLimitNs)) {
        s_abort = 1;
        atomicOr(&lp.status->error, 1u);
        lp.status->where = 2;
      }
      if (s_abort != 0) {
        // some wait ran out: the consumers leave by themselves; nothing more is
        // issued, and the copies in flight land (or their wait runs out) before
        // the CTA's shared memory goes away
        for (uint32_t u = armed > STAGES ? armed - STAGES : 0; u < armed; ++u)
          mbar_wait_bounded(&full_bar[u % STAGES], (u / STAGES) & 1u, kWaitLimitNs);
        return;
      }
      if (!have) {
        const bool cancelled = poll_cancelled(lp.status, lp.cancel);
        const unsigned long long idx = cancelled ? ~0ull : atomicAdd(lp.item_counter, 1ull);
        if (idx >= static_cast<unsigned long long>(lp.n_items)) {
          meta[s].flags = kStepEnd;
          mbar_arrive(&full_bar[s]);   // completes the phase without data
          return;
        }
        const WorkItem it = lp.items[idx];
        const JobParams &jp = lp.jobs[it.job];
        job = it.job;
        tile_coords(jp, it.tile, ti, tj);
        k = it.k0;
        k1 = it.k1;
        split = it.split;
        nb = jp.nb;
        bstart = it.b1 ? it.b0 : 0;
        bend = it.b1 ? it.b1 : jp.nb;
        bpart = it.bpart;
        nbpart = it.nbpart > 1 ? it.nbpart : 1;
        b0 = WIDE ? 0 : bstart;
        if constexpr (CODED) {
          const int32_t KB = jp.n_kmers * jp.nb;
          rows = jp.code_words + code_stripe(jp.code, KB, ti, 0, 0);
          cols = jp.code_words + code_stripe(jp.code, KB, ti, 0, 1 + tj - code_first_group(jp.code, ti));
          kb_stride = static_cast<int64_t>(code_groups(jp.code, ti)) * kCodeStripeWords;
          planes_of = jp.code_planes + static_cast<int64_t>(ti - jp.code.rb0) * KB;
        } else {
          rows = jp.row_words;
          cols = jp.col_words;
          ngr = jp.ng_rows;
          ngc = jp.ng_cols;
        }
        if constexpr (WIDE) {
          slot = it.k0 * jp.nchunk;
          chunk_nb = jp.chunk_nb;
          slot_end = jp.chunk_nb;   // chunk_nb == nb when one slot holds a whole k
        }
        have = true;
        atomicAdd(&lp.status->tiles_done, 1ull);
      }
      // slot ends fall on step boundaries (chunk_nb and nb are even); a coded
      // step may end a slot with fewer blocks
      const bool last_of_slot = WIDE ? b0 + kStep >= slot_end : b0 + kStep >= bend;
      const bool last_of_k = WIDE ? last_of_slot && slot_end >= nb : last_of_slot;
      const bool last_of_item = last_of_k && k + 1 >= k1;
      StepMeta &m = meta[s];
      m.job = job;
      m.ti = ti;
      m.tj = tj;
      m.kidx = WIDE ? slot : k * nbpart + bpart;
      m.flags = (last_of_slot ? kStepLastOfK : 0) | (last_of_item ? kStepLastOfItem : 0);
      m.split = split;
      if constexpr (CODED) {
        const int32_t kb = k * nb + b0;   // even: steps and block ranges are pairs of blocks
        const int n = min(kStep, bend - b0) / 2;
        uint32_t planes = 0, bytes = 0;
        for (int b = 0; b < n; ++b) {
          // a pair of blocks compares the planes of its larger dictionary,
          // clamped to what the stage holds and the kernel compares
          const uint32_t two = __ldg(reinterpret_cast<const uint16_t *>(planes_of + kb) + b);
          const uint32_t p = min(max(max(two & 0xFFu, two >> 8), static_cast<uint32_t>(kCodeMinPlanes)),
                                 static_cast<uint32_t>(kCodeMaxPlanes));
          planes |= p << (8 * b);
          bytes += 4 * p * kCodeGroup * 4;
        }
        m.planes = planes;
        mbar_arrive_expect_tx(&full_bar[s], bytes);
        for (int b = 0; b < 2 * n; ++b) {
          const uint32_t len = ((planes >> (8 * (b / 2))) & 0xFFu) * kCodeGroup * 4;
          const int64_t off = (kb + b) * kb_stride;
          bulk_g2s(sq + (s * kStep + b) * kCodeStripeWords, rows + off, len, &full_bar[s]);
          bulk_g2s(sr + (s * kStep + b) * kCodeStripeWords, cols + off, len, &full_bar[s]);
        }
      } else {
        mbar_arrive_expect_tx(&full_bar[s], S::kStageBytes);
#pragma unroll
        for (int b = 0; b < kBlocksPerStage; ++b) {
          const int64_t blk = static_cast<int64_t>(k) * nb + b0 + b;
          const uint32_t *src_q =
              rows + ((blk * ngr) + static_cast<int64_t>(ti) * S::kQG) * kStripeWords;
          const uint32_t *src_r =
              cols + ((blk * ngc) + static_cast<int64_t>(tj) * S::kRG) * kStripeWords;
          bulk_g2s(sq + (s * kBlocksPerStage + b) * S::kQG * kStripeWords, src_q,
                   S::kQG * kStripeBytes, &full_bar[s]);
          bulk_g2s(sr + (s * kBlocksPerStage + b) * S::kRG * kStripeWords, src_r,
                   S::kRG * kStripeBytes, &full_bar[s]);
        }
      }
      armed = t + 1;
      b0 += kStep;
      if constexpr (WIDE) {
        if (last_of_slot) {
          ++slot;
          if (last_of_k) {
            b0 = 0;
            ++k;
            slot_end = chunk_nb;
            if (last_of_item) have = false;
          } else {
            slot_end = min(slot_end + chunk_nb, nb);
          }
        }
      } else if (last_of_k) {
        b0 = bstart;
        ++k;
        if (last_of_item) have = false;
      }
      if (++s == STAGES) {
        s = 0;
        parity ^= 1u;
      }
    }
  }

  // ---------------------------------------------------------------- consumers
  // Counts of one k for columns 2c and 2c + 1 share a register (low / high
  // 16 bits): at most 64 * sketchsize64 <= 65,472 per k, so the low half never
  // carries.  `one` is 1 at run time, which keeps the count multiply-adds on
  // the FMA pipe and the ALU free for the LOP3s.
  if constexpr (S::kSplitRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
  const int tq = tid / TCOLS;
  const int tr = tid % TCOLS;
  const int row0 = tq * TQ;   // first tile row of this thread
  const int col0 = tr * TR;   // first tile column of this thread
  const int64_t slot_k_stride = static_cast<int64_t>(NT) * PT;      // uint16 between k slots
  const int64_t split_size = slot_k_stride * lp.split_slots;
  uint16_t *my_counts = lp.cta_scratch + blockIdx.x * slot_k_stride * lp.k_slots +
                        static_cast<int64_t>(tid) * PT;
  const uint32_t one = lp.jobs[0].one;
  const uint32_t hi_one = one << 16;
  uint32_t cnt[TQ][TR / 2];
#pragma unroll
  for (int i = 0; i < TQ; ++i)
#pragma unroll
    for (int j = 0; j < TR / 2; ++j) cnt[i][j] = 0;

  int s = 0;              // stage of the step
  uint32_t parity = 0;    // phase parity of the step on that stage
  while (true) {
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full_bar[s], parity, kWaitLimitNs))) {
      // a stage never landed: record it and leave; the producer's wait for
      // this warp runs out, or it sees the flag, and ends too
      s_abort = 1;
      atomicOr(&lp.status->error, 1u);
      lp.status->where = 1;
      return;
    }
    const StepMeta m = meta[s];
    if (m.flags & kStepEnd) break;

    if constexpr (CODED) {
      const uint32_t *qb = sq + s * kStep * kCodeStripeWords + row0;
      const uint32_t *rb = sr + s * kStep * kCodeStripeWords + col0;
#pragma unroll 1
      for (uint32_t planes = m.planes; planes != 0; planes >>= 8) {
        switch (planes & 0xFFu) {   // the same for every thread
          case 4: count_pair<TQ, TR, 4>(qb, rb, one, hi_one, cnt); break;
          case 5: count_pair<TQ, TR, 5>(qb, rb, one, hi_one, cnt); break;
          case 6: count_pair<TQ, TR, 6>(qb, rb, one, hi_one, cnt); break;
          case 7: count_pair<TQ, TR, 7>(qb, rb, one, hi_one, cnt); break;
          default: count_pair<TQ, TR, 8>(qb, rb, one, hi_one, cnt); break;
        }
        qb += 2 * kCodeStripeWords;
        rb += 2 * kCodeStripeWords;
      }
    } else {
#pragma unroll
      for (int b = 0; b < kBlocksPerStage; ++b) {
        const uint32_t *qb = sq + (s * kBlocksPerStage + b) * S::kQG * kStripeWords +
                             (row0 / kGranule) * kStripeWords + (row0 % kGranule);
        const uint32_t *rb = sr + (s * kBlocksPerStage + b) * S::kRG * kStripeWords +
                             (col0 / kGranule) * kStripeWords + (col0 % kGranule);
        count_block<TQ, TR, kBbits, kGranule>(qb, rb, one, hi_one, cnt);
      }
    }

    // this warp has read the stage: the producer refills it once all have
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty_bar[s]);
    if (++s == STAGES) {
      s = 0;
      parity ^= 1u;
    }

    if (m.flags & kStepLastOfK) {
      // counts of count slot m.kidx done: park them (own slot or split slot)
      uint16_t *base = m.split >= 0
                           ? lp.split_scratch + m.split * split_size + static_cast<int64_t>(tid) * PT
                           : my_counts;
      // pair q = i * TR + j is uint16 q of the slot: word q / 2 = cnt[i][j / 2]
      uint4 *dst = reinterpret_cast<uint4 *>(base + m.kidx * slot_k_stride);
      constexpr int CW = TR / 2;
#pragma unroll
      for (int w = 0; w < PT / 8; ++w)
        dst[w] = make_uint4(cnt[(4 * w) / CW][(4 * w) % CW], cnt[(4 * w + 1) / CW][(4 * w + 1) % CW],
                            cnt[(4 * w + 2) / CW][(4 * w + 2) % CW],
                            cnt[(4 * w + 3) / CW][(4 * w + 3) % CW]);
#pragma unroll
      for (int i = 0; i < TQ; ++i)
#pragma unroll
        for (int j = 0; j < TR / 2; ++j) cnt[i][j] = 0;
    }

    if ((m.flags & kStepLastOfItem) && m.split < 0) {
      const JobParams &jp = lp.jobs[m.job];
      const int64_t gi0 = static_cast<int64_t>(m.ti) * QT + row0;
      const int64_t gj0 = static_cast<int64_t>(m.tj) * RT + col0;
#pragma unroll 1
      for (int q = 0; q < PT; ++q) {
        const int64_t gi = gi0 + q / TR;
        const int64_t gj = gj0 + q % TR;
        if (pair_valid(jp, gi, gj))
          finish_pair_any<WIDE, CODED>(jp, gi, gj, my_counts + q, static_cast<int>(slot_k_stride));
      }
    }
  }
}

// The epilogue of the split tiles, one thread per pair over every SM.
//
// A split tile's counts lie in its slot by block range.  A CTA first adds up
// the ranges of its 128 pairs: a thread owns 8 neighbouring pairs (one 128-bit
// load per range; two 16-bit counts per word never carry, their sums fit 16
// bits) at every eighth k, so a tile cut into hundreds of ranges keeps enough
// loads in flight.  The sums go to shared memory, where finish_pair_any reads
// them.  A pair's arithmetic is a chain of about 575 FP64 instructions: finished
// inside the distance kernel by the last part's CTA, 32 pairs per thread one
// after another, it held a single CTA for about 300 us at the end of a launch.
// Wide jobs (one slot per chunk, no block ranges) are read where they lie.
constexpr int kFinishPairs = 128;   // threads = pairs per CTA

template <int QT, int RT, int TQ, int TR, bool WIDE>
__global__ void __launch_bounds__(kFinishPairs) finish_splits_kernel(const LaunchParams lp) {
  constexpr int PT = TQ * TR;
  constexpr int TCOLS = RT / TR;
  constexpr int kStride = QT * RT;   // uint16 between count slots
  constexpr int kGroups = kStride / kFinishPairs;
  __shared__ __align__(16) uint16_t sums[WIDE ? 8 : kNarrowKmers * kFinishPairs];
  __shared__ int32_t s_ti, s_tj;
  // an item that was cancelled or timed out parked nothing: its slot holds
  // another launch's counts
  if (*reinterpret_cast<const volatile unsigned int *>(&lp.status->error) != 0) return;
  const int split = blockIdx.x / kGroups;
  const int p0 = (blockIdx.x % kGroups) * kFinishPairs;   // first pair within the tile
  const SplitTile st = lp.splits[split];
  const JobParams &jp = lp.jobs[st.job];
  if (threadIdx.x == 0) {
    int32_t ti, tj;
    tile_coords(jp, st.tile, ti, tj);
    s_ti = ti;
    s_tj = tj;
  }
  const uint16_t *src =
      lp.split_scratch + static_cast<int64_t>(split) * lp.split_slots * kStride + p0;
  if constexpr (!WIDE) {
    const int g = threadIdx.x % (kFinishPairs / 8);
    for (int k = threadIdx.x / (kFinishPairs / 8); k < jp.n_kmers; k += 8) {
      const uint16_t *s = src + static_cast<int64_t>(k) * st.nbpart * kStride + 8 * g;
      uint4 c = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 8
      for (int b = 0; b < st.nbpart; ++b) {
        const uint4 v = *reinterpret_cast<const uint4 *>(s + static_cast<int64_t>(b) * kStride);
        c.x += v.x; c.y += v.y; c.z += v.z; c.w += v.w;
      }
      *reinterpret_cast<uint4 *>(sums + k * kFinishPairs + 8 * g) = c;
    }
  }
  __syncthreads();
  const int p = p0 + threadIdx.x;
  const int owner = p / PT, q = p % PT;
  const int64_t gi = static_cast<int64_t>(s_ti) * QT + owner / TCOLS * TQ + q / TR;
  const int64_t gj = static_cast<int64_t>(s_tj) * RT + owner % TCOLS * TR + q % TR;
  if (!pair_valid(jp, gi, gj)) return;
  if constexpr (WIDE) finish_pair_any<true>(jp, gi, gj, src + threadIdx.x, kStride);
  else finish_pair_any<false>(jp, gi, gj, sums + threadIdx.x, kFinishPairs);
}

// ------------------------------------------------------------ config registry

namespace {

// Raises the instance's dynamic shared memory limit once (before any launch,
// so never inside a stream capture).
template <int QT, int RT, int TQ, int TR, int STAGES, int MINB, bool WIDE, bool CODED>
cudaError_t ensure_smem_attr() {
  using S = TileShape<QT, RT, TQ, TR, STAGES, CODED>;
  static cudaError_t status = cudaFuncSetAttribute(
      dist_items_kernel<QT, RT, TQ, TR, STAGES, MINB, WIDE, CODED>,
      cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmemBytes);
  return status;
}

template <int QT, int RT, int TQ, int TR, int STAGES, int MINB, bool WIDE, bool CODED>
cudaError_t launch_one(const LaunchParams &lp, int grid, cudaStream_t stream) {
  using S = TileShape<QT, RT, TQ, TR, STAGES, CODED>;
  cudaError_t e = ensure_smem_attr<QT, RT, TQ, TR, STAGES, MINB, WIDE, CODED>();
  if (e != cudaSuccess) return e;
  dist_items_kernel<QT, RT, TQ, TR, STAGES, MINB, WIDE, CODED>
      <<<grid, S::kBlockThreads, S::kSmemBytes, stream>>>(lp);
  if (lp.n_splits > 0)
    finish_splits_kernel<QT, RT, TQ, TR, WIDE>
        <<<lp.n_splits * (QT * RT / kFinishPairs), kFinishPairs, 0, stream>>>(lp);
  return cudaGetLastError();
}

// Coded tiles are 128 x 128, with one instance.
constexpr int kCodedStages = 3;   // of 64 KB
constexpr bool has_coded(int QT, int RT, int TQ, int TR) {
  return QT == kCodeGroup && RT == kCodeGroup && TQ == 8 && TR == 4;
}

template <int QT, int RT, int TQ, int TR, int STAGES, int MINB>
cudaError_t launch_cfg(const LaunchParams &lp, int grid, cudaStream_t stream) {
  if constexpr (has_coded(QT, RT, TQ, TR)) {
    if (lp.coded) return launch_one<QT, RT, TQ, TR, kCodedStages, MINB, false, true>(lp, grid, stream);
  } else if (lp.coded) {
    return cudaErrorInvalidValue;
  }
  if (lp.wide) return launch_one<QT, RT, TQ, TR, STAGES, MINB, true, false>(lp, grid, stream);
  return launch_one<QT, RT, TQ, TR, STAGES, MINB, false, false>(lp, grid, stream);
}

template <int QT, int RT, int TQ, int TR, int STAGES, int MINB, bool WIDE, bool CODED>
int occupancy_one() {
  using S = TileShape<QT, RT, TQ, TR, STAGES, CODED>;
  if (ensure_smem_attr<QT, RT, TQ, TR, STAGES, MINB, WIDE, CODED>() != cudaSuccess) return 0;
  int blocks = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &blocks, dist_items_kernel<QT, RT, TQ, TR, STAGES, MINB, WIDE, CODED>, S::kBlockThreads,
          S::kSmemBytes) != cudaSuccess)
    return 0;
  return blocks;
}

// Resident CTAs per SM of every instance (a grid sized by it suits them all).
template <int QT, int RT, int TQ, int TR, int STAGES, int MINB>
int occupancy_cfg() {
  int n = std::min(occupancy_one<QT, RT, TQ, TR, STAGES, MINB, false, false>(),
                   occupancy_one<QT, RT, TQ, TR, STAGES, MINB, true, false>());
  if constexpr (has_coded(QT, RT, TQ, TR))
    n = std::min(n, occupancy_one<QT, RT, TQ, TR, kCodedStages, MINB, false, true>());
  return n;
}

template <int QT, int RT, int TQ, int TR, int STAGES, int MINB>
constexpr TileConfig make_cfg(int id) {
  return TileConfig{id,
                    QT,
                    RT,
                    TQ,
                    TR,
                    kMaxKmers,
                    STAGES,
                    TileShape<QT, RT, TQ, TR, STAGES, false>::kSmemBytes,
                    &launch_cfg<QT, RT, TQ, TR, STAGES, MINB>,
                    &occupancy_cfg<QT, RT, TQ, TR, STAGES, MINB>};
}

const TileConfig kConfigs[] = {
    make_cfg<128, 128, 8, 4, 4, 1>(1),  // default: 512 threads, 16 warps, one CTA per SM
    make_cfg<128, 64, 8, 4, 4, 2>(2),   // 256 threads, two CTAs per SM
    make_cfg<64, 64, 4, 4, 4, 2>(3),    // small tiles, 16 pairs per thread
    make_cfg<128, 128, 8, 8, 4, 1>(4),  // 256 threads, 64 pairs per thread
    make_cfg<128, 64, 4, 8, 4, 2>(5),   // transposed thread block
    make_cfg<64, 64, 8, 4, 4, 3>(6),    // 128 threads, three CTAs per SM
};

}  // namespace

int tile_config_count() { return static_cast<int>(sizeof(kConfigs) / sizeof(kConfigs[0])); }

const TileConfig *tile_config(int id) {
  for (const TileConfig &c : kConfigs)
    if (c.id == id) return &c;
  return nullptr;
}

}  // namespace sk
