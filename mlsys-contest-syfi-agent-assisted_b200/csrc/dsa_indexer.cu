// DSA top-k indexer (definition dsa_topk_indexer_fp8_h64_d128_topk2048_ps64), the sibling operator of the MoE
// layer that shares its building blocks: FP8 scoring on the tensor cores and a selection of the best tokens.
//
// Replaces the reference's score_kernel (dsa_indexer/solution/cuda/dsa_topk_indexer.cu:78-250: e4m3 unpacked
// to bf16 in shared memory, wmma 16x16x16) and topk_kernel_radix (:251-395: one 8-bit histogram, tokens of the
// threshold byte in arbitrary order), and computes what the definition's configured entry point computes
// (dsa_indexer/solution/python/dsa_topk_indexer.py:64-112, pure torch):
//     score[t] = sum_h weights[b, h] * relu(q[b, h, :] . (k8[t, :] * kscale[t])),   best 2048 tokens, best first.
//
//   score kernel : one CTA per (sequence, run of 128 to 1024 tokens), 128 tokens = two cache pages per MMA, key tiles and
//                  accumulators double-buffered.  The pages' 64 x 128 e4m3 bytes are
//                  contiguous in the cache (a page is 64 rows of 128 bytes followed by 64 f32 scales = 66 rows of
//                  128 bytes), so one tensor map over the cache as rows of 128 bytes fetches a page with one TMA
//                  box; the query's 64 heads are a second box.  tcgen05.mma kind::f8f6f4, M = 128 tokens,
//                  N = 64 heads, K = 128 in four steps, accumulator in tensor memory; the raw e4m3 products are
//                  exact, so the token's scale is applied once, after the sum over K.  Each thread then owns a
//                  token: relu, times the head weight, summed over the 64 heads in head order.
//   select kernel: a counting sort by value over a cluster of CTAs per sequence (best first, ties by position), with an
//                  exact radix select over the cluster and a bitonic sort for score distributions that it does not
//                  separate.
// Every wait is bounded; a failure is recorded in the status word the host entry point reads back.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <mutex>

#include "../../include/syfi_dsa.h"
#include "dsa_bins.h"
#include "moe_internal.h"
#include "ptx.cuh"

namespace syfi {

namespace {

namespace cg = cooperative_groups;

constexpr int kHeads = 64;
constexpr int kDim = 128;
constexpr int kPage = 64;
constexpr int kPageRows = 66;                 // 128-byte rows per cache page: 64 key rows + 2 rows of scales
constexpr int kPageBytes = kPageRows * 128;   // 8448
constexpr int kKeep = SYFI_DSA_TOPK;          // tokens kept per sequence
constexpr int kTokTile = 128;                 // tokens per MMA: two cache pages
constexpr int kMaxTilesPerCta = 8;            // a score CTA walks up to 1024 tokens of one sequence
constexpr int kScoreThreads = 160;            // four epilogue warps (one tensor-memory lane quarter each) + a producer / MMA warp
constexpr int kScoreStages = 2;
constexpr int kScoreSmem = 1024 + kScoreStages * kTokTile * kDim + kHeads * kDim;   // slack + key tiles + query tile
constexpr int kSelectThreads = 1024;
constexpr int kMaxCluster = 8;                // select CTAs that share a sequence
constexpr long long kWaitLimit = 1ll << 31;   // SM clocks (about a second)
constexpr int kStatusScoreTimeout = 201;

// Score kernel: CTA (x, b) scores the x-th run of tiles_per_cta * 128 tokens of sequence b, 128 at a time, through a two-deep
// ring of key tiles in shared memory and two accumulators in tensor memory: while the four epilogue warps turn
// tile i into scores, the tensor core works on tile i + 1 and TMA fetches tile i + 2.
__global__ void __launch_bounds__(kScoreThreads)
dsa_score_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const uint8_t* __restrict__ cache, const float* __restrict__ weights,
                 const int32_t* __restrict__ seq_lens, const int32_t* __restrict__ block_table, int max_pages,
                 float* __restrict__ scores, int max_ls, int tiles_per_cta, uint2* __restrict__ ranges, int* __restrict__ status,
                 long long wait_limit) {
  const int b = blockIdx.y, t_begin = blockIdx.x * tiles_per_cta * kTokTile;
  pdl_wait();                                  // the selection of the call before reads the scores written here
  pdl_trigger();
  const int n = min(seq_lens[b], max_ls);
  if (t_begin >= n) return;                    // the whole CTA leaves before any barrier or allocation
  const int tiles = min(tiles_per_cta, (n - t_begin + kTokTile - 1) / kTokTile);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* s_k = smem;                                     // [2 stages][128 tokens][128 B], 128-byte swizzle
  uint8_t* s_q = smem + kScoreStages * kTokTile * kDim;    // [64 heads][128 B]
  __shared__ uint64_t full[kScoreStages], empty[kScoreStages], tfull[kScoreStages], tempty[kScoreStages], qfull, idle;
  __shared__ uint32_t s_tmem;
  __shared__ float s_w[kHeads];
  __shared__ int s_page[2 * kMaxTilesPerCta];
  __shared__ volatile int s_abort;
  __shared__ uint2 s_range[4];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < kHeads) s_w[tid] = weights[b * kHeads + tid];
  if (tid < 2 * tiles)
    s_page[tid] = (t_begin + tid * kPage < n) ? block_table[b * max_pages + t_begin / kPage + tid] : -1;
  if (tid == 0) {
    for (int i = 0; i < kScoreStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);                // one arrival per epilogue warp
    }
    mbar_init(&qfull, 1);
    mbar_init(&idle, 1);
    s_abort = 0;
    fence_barrier_init();
  }
  if (warp == 4) {
    tmem_alloc(&s_tmem, kScoreStages * kHeads);            // two accumulators of 64 columns
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = s_tmem;

  int loaded = 0;                              // key tiles that the producer has asked for
  if (warp == 4) {
    if (lane == 0) {
      // ---------------------------------------------------------- producer and MMA issuer (one thread)
      const uint64_t pol = l2_policy_evict_first();        // the cache is streamed once
      auto load_tile = [&](int i) {
        const int st = i % kScoreStages;
        const int pages = s_page[2 * i + 1] >= 0 ? 2 : 1;
        mbar_arrive_expect_tx(&full[st], pages * kPage * kDim);
        for (int p = 0; p < pages; ++p)
          tma_load_2d(s_k + st * kTokTile * kDim + p * kPage * kDim, &tm_k, &full[st], 0, s_page[2 * i + p] * kPageRows, pol);
        loaded = i + 1;
      };
      mbar_arrive_expect_tx(&qfull, kHeads * kDim);
      tma_load_2d(s_q, &tm_q, &qfull, 0, b * kHeads, l2_policy_evict_last());
      load_tile(0);
      if (tiles > 1) load_tile(1);
      bool alive = mbar_wait_bounded(&qfull, 0, &s_abort, kStatusScoreTimeout, wait_limit);
      const uint64_t b0 = umma_smem_desc_sw128(smem_u32(s_q));
      const uint32_t idesc = umma_idesc_e4m3_m128(kHeads);
      for (int i = 0; i < tiles && alive; ++i) {
        const int st = i % kScoreStages;
        const uint32_t ph = (i / kScoreStages) & 1u;
        if (!mbar_wait_bounded(&full[st], ph, &s_abort, kStatusScoreTimeout, wait_limit)) break;
        if (!mbar_wait_bounded(&tempty[st], ph ^ 1u, &s_abort, kStatusScoreTimeout, wait_limit)) break;
        tc_fence_after();
        const uint64_t a0 = umma_smem_desc_sw128(smem_u32(s_k + st * kTokTile * kDim));
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) umma_f8(tmem_base + st * kHeads, a0 + 2 * k4, b0 + 2 * k4, idesc, k4 > 0 ? 1u : 0u);
        umma_commit(&empty[st]);               // the key tile may be overwritten once these MMAs have read it
        umma_commit(&tfull[st]);
        if (i + kScoreStages < tiles) {
          if (!mbar_wait_bounded(&empty[st], ph, &s_abort, kStatusScoreTimeout, wait_limit)) break;
          load_tile(i + kScoreStages);
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue: thread = token lane of the tile
    const int tl = tid;                        // 0..127
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    uint32_t low = 0xffffffffu, high = 0u;     // range of this thread's scores, for the selection's bins
    bool alive = true;
    for (int i = 0; i < tiles; ++i) {
      const int st = i % kScoreStages;
      const uint32_t ph = (i / kScoreStages) & 1u;
      const int t = t_begin + i * kTokTile + tl;
      const int page = s_page[2 * i + (tl >> 6)];
      const bool valid = t < n && page >= 0;
      // the token's scale sits behind the page's 64 x 128 key bytes; requested before the wait
      const float scale = valid ? __ldg(reinterpret_cast<const float*>(cache + static_cast<size_t>(page) * kPageBytes +
                                                                       kPage * kDim + (tl & (kPage - 1)) * 4))
                                : 0.0f;
      mbar_wait_or_clear(alive, &tfull[st], ph, &s_abort, kStatusScoreTimeout, wait_limit);   // (failed: the rest of the run has no scores)
      tc_fence_after();
      float acc = 0.0f;
#pragma unroll
      for (int c = 0; c < kHeads / 16; ++c) {
        uint32_t r[16];
        tmem_ld16(lane_addr + st * kHeads + c * 16, r);
        tmem_ld_wait_for(r);
        if (c == kHeads / 16 - 1) {            // the accumulator is in registers: hand it back
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[st]);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) acc = fmaf(s_w[c * 16 + j], fmaxf(__uint_as_float(r[j]) * scale, 0.0f), acc);
      }
      // no page here: below every score and outside the range, so that the selection never meets what an earlier call left
      const bool scored = valid && alive;
      if (t < n) scores[static_cast<size_t>(b) * max_ls + t] = scored ? acc : -INFINITY;
      if (scored) {
        low = min(low, score_key(acc));
        high = max(high, score_key(acc));
      }
    }
    low = __reduce_min_sync(0xffffffffu, low);
    high = __reduce_max_sync(0xffffffffu, high);
    if (lane == 0) s_range[warp] = make_uint2(low, high);
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    uint2 r = s_range[0];
    for (int w = 1; w < 4; ++w) r = make_uint2(min(r.x, s_range[w].x), max(r.y, s_range[w].y));
    ranges[static_cast<size_t>(b) * gridDim.x + blockIdx.x] = r;
  }
  if (s_abort != 0) {
    // A role gave up: copies and MMAs may still be on their way, which otherwise the epilogue has waited for.
    if (tid == 4 * 32) {
      mbar_wait_landed(&qfull, 0);
      for (int i = max(loaded - kScoreStages, 0); i < loaded; ++i) mbar_wait_landed(&full[i % kScoreStages], (i / kScoreStages) & 1);
      umma_commit(&idle);
      mbar_wait_landed(&idle, 0);
    }
    __syncthreads();
  }
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kScoreStages * kHeads);
  }
  if (tid == 0 && s_abort != 0) atomicExch(status, s_abort);
}

// The best k = min(2048, n) of a sequence's n items, best first, left in the first CTA's s_item[0 .. 2047] (zeros behind
// them); all `ctas` CTAs that share the sequence call it, each for its own items.  An item is (order-preserving key of the
// score << 32) | ~position, so items are distinct, "larger" means "better score, then lower position", and the cut is one
// exact item value: an 8-pass radix select over the 64 bits (one byte per pass, a histogram in shared memory, the top
// bytes' through warp-aggregated increments, since most scores of a sequence share those), a compaction of the items at
// or above the cut, and in the first CTA a bitonic sort.  In a pass every CTA counts its own items, and all of them sum
// the CTAs' 256 counts and so come to the same byte; two histograms in turn need one cluster barrier per pass.
// get(j) returns the calling thread's j-th item, 0 where it has none; j < N, or any j, with per_thread of them, where N is 0.
template <int N, typename Get>
__device__ __forceinline__ void select_best(Get get, int per_thread, int k, int ctas, int rank, unsigned long long* s_item,
                                            unsigned long long* s_swap, int* s_arrived, int (*s_hist)[256], int* s_misc) {
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31;
  auto each = [&](auto f) {
    if constexpr (N > 0) {
#pragma unroll
      for (int j = 0; j < N; ++j) f(get(j));
    } else {
      for (int j0 = 0; j0 < per_thread; j0 += 4) {      // four loads in flight
        unsigned long long it[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) it[j] = get(j0 + j);
#pragma unroll
        for (int j = 0; j < 4; ++j) f(it[j]);
      }
    }
  };
  unsigned long long prefix = 0ull, mask = 0ull;
  int want = k;
  for (int shift = 56; shift >= 0; shift -= 8) {
    int* const hist = s_hist[(shift >> 3) & 1];
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    each([&](unsigned long long it) {
      const int bin = (it != 0ull && (it & mask) == prefix) ? static_cast<int>((it >> shift) & 255ull) : 256;
      if (shift >= 48) {      // sign and exponent: a handful of values, so the warp adds up its lanes first
        const unsigned peers = __match_any_sync(0xffffffffu, bin);
        if (bin < 256 && lane == __ffs(peers) - 1) atomicAdd(&hist[bin], __popc(peers));
      } else if (bin < 256) { // mantissa and position bytes: spread out, and fewer items match the prefix each pass
        atomicAdd(&hist[bin], 1);
      }
    });
    if (ctas > 1) cluster.sync();
    else __syncthreads();
    // the byte value at which the count from the top reaches `want`: thread t < 256 owns value 255 - t, an
    // inclusive scan in thread order counts the items with that byte or a larger one
    int h = 0, incl = 0;
    if (tid < 256) {
      if (ctas > 1) {
#pragma unroll
        for (int c = 0; c < kMaxCluster; ++c)
          if (c < ctas) h += cluster.map_shared_rank(hist, c)[255 - tid];
      } else {
        h = hist[255 - tid];
      }
      incl = h;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
      }
      if (lane == 31) s_misc[4 + (tid >> 5)] = incl;
    }
    __syncthreads();
    if (tid < 256) {
      for (int w = 0; w < (tid >> 5); ++w) incl += s_misc[4 + w];
      if (incl >= want && incl - h < want) {
        s_misc[0] = 255 - tid;
        s_misc[1] = incl - h;
        s_misc[3] = h;
      }
    }
    __syncthreads();
    prefix |= static_cast<unsigned long long>(s_misc[0]) << shift;
    mask |= 255ull << shift;
    want -= s_misc[1];
    const bool all_taken = s_misc[3] == want;   // every item that still matches the prefix is wanted: no more passes
    __syncthreads();
    if (all_taken) break;
  }
  const unsigned long long cut = prefix;       // the k-th best item (its leading bytes, when the passes stopped early)
  if (tid == 0) s_misc[2] = 0;
  __syncthreads();
  each([&](unsigned long long it) {            // one counter increment per warp and round, not per winner
    const bool win = it != 0ull && it >= cut;
    const unsigned winners = __ballot_sync(0xffffffffu, win);
    int base = 0;
    if (lane == 0 && winners != 0u) base = atomicAdd(&s_misc[2], __popc(winners));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (win) s_item[base + __popc(winners & ((1u << lane) - 1u))] = it;
  });
  __syncthreads();
  unsigned long long *buf = s_swap, *other = s_item;
  if (ctas > 1) {                              // every CTA's winners in one piece to the first one
    const int own = s_misc[2];
    if (tid == 0) s_misc[0] = atomicAdd(cluster.map_shared_rank(s_arrived, 0), own);
    __syncthreads();
    unsigned long long* to = cluster.map_shared_rank(s_swap, 0) + s_misc[0];
    for (int i = tid; i < own; i += kSelectThreads) to[i] = s_item[i];
    cluster.sync();
    if (rank != 0) return;
    buf = s_item;
    other = s_swap;
  }
  for (int i = k + tid; i < kKeep; i += kSelectThreads) other[i] = 0ull;
  __syncthreads();
  // Bitonic sort, descending, two adjacent items per thread in registers.  A compare-exchange at distance d pairs
  // item i with item i ^ d: d = 1 is inside the thread, d = 2 .. 32 pairs this thread with lane ^ (d / 2) of its
  // warp (shuffles, no barrier), d >= 64 goes through shared memory (two buffers in turn: one barrier per stage,
  // 15 stages instead of 66 barriers).  The first of a pair keeps the larger item where the block of `size`
  // items it lies in is sorted downwards ((i & size) == 0), the smaller one otherwise.
  unsigned long long e0 = other[2 * tid], e1 = other[2 * tid + 1];
  auto pick = [](unsigned long long a, unsigned long long c, bool keep_max) {
    return keep_max ? (a > c ? a : c) : (a < c ? a : c);
  };
  for (int size = 2; size <= kKeep; size <<= 1) {
    const bool desc = ((2 * tid) & size) == 0;
    for (int stride = size >> 1; stride >= 64; stride >>= 1) {
      buf[2 * tid] = e0;
      buf[2 * tid + 1] = e1;
      __syncthreads();
      const int half = stride >> 1;
      const int pt = tid ^ half;
      const bool keep_max = ((tid & half) == 0) == desc;
      e0 = pick(e0, buf[2 * pt], keep_max);
      e1 = pick(e1, buf[2 * pt + 1], keep_max);
      unsigned long long* t = buf; buf = other; other = t;
    }
    for (int stride = (size >> 1) < 32 ? (size >> 1) : 32; stride >= 2; stride >>= 1) {
      const int half = stride >> 1;
      const bool keep_max = ((tid & half) == 0) == desc;
      e0 = pick(e0, __shfl_xor_sync(0xffffffffu, e0, half), keep_max);
      e1 = pick(e1, __shfl_xor_sync(0xffffffffu, e1, half), keep_max);
    }
    const unsigned long long hi = e0 > e1 ? e0 : e1, lo = e0 > e1 ? e1 : e0;
    e0 = desc ? hi : lo;
    e1 = desc ? lo : hi;
  }
  __syncthreads();                             // every reader of either buffer is through
  s_item[2 * tid] = e0;
  s_item[2 * tid + 1] = e1;
  __syncthreads();
}

constexpr int kMaxInBin = 512;     // most items a bin at or above the cut may hold, see dsa_select_kernel
constexpr int kMaxListed = kKeep + kMaxInBin;
constexpr int kTablePages = 2048;  // block-table entries kept in shared memory
constexpr int kSelectSmem = 2 * kMaxListed * 8 + kBins * 4 + kTablePages * 4;
static_assert(kMaxListed * 8 >= kBins * 4 && kKeep * 8 <= kBins * 4, "aliases of the selection's buffers");

// Selection and sort in one pass over the scores: a counting sort by value.  A cluster of CTAs shares a sequence, CTA r
// takes every gridDim.x-th block of 1024 positions (PER blocks at most, kept in registers; PER = 0: any number, read
// again in both sweeps).
//   1. the range of the sequence's scores (the score kernel left one per run of tokens) is cut into 4096 equal bins;
//   2. histogram of the bins per CTA, summed over the cluster slice by slice (each CTA a share of the bins: distributed
//      shared memory moves about 16 bytes per clock and CTA, and the first CTA fetching all of it took 3.7 us) into the
//      first CTA;
//   3. the first CTA sums the counts from the top: every bin gets the rank of its first item, and the bin in which the
//      count reaches 2048 is the cut;
//   4. every item of the cut bin or a higher one goes to the first CTA (the others collect theirs and send them in one
//      piece: an atomic on a remote cursor per item took 3 us), which groups them by bin, each at its bin's cursor;
//   5. an item's final rank is its bin's first rank plus the number of larger items in the bin (a handful), so the
//      2048 best are written best first without a sorting network.
// The kernel is a chain of short steps between barriers, so what counts is their number: an eight-pass radix select and
// a 66-stage bitonic sort per 16384 positions, then the same again over the chunks' candidates, took 25 us for three
// short sequences and 22 + 32 us for 32 sequences of 65536 tokens; this one takes about 6 us and
// 16 us (the latter under ncu, with cold caches).
// Where the bins do not separate the scores (a bin at or above the cut holds more than kMaxInBin items: ties, or
// outliers that stretch the range; infinities and NaNs), the cluster selects by radix instead, see select_best: us per
// call, separable scores / one outlier per sequence / the same with the first CTA alone on the whole sequence:
// 1 sequence of 65536 tokens 19 / 39 / 124, 32 of them 58 / 87 / 177, 1 of 262144 35 / 93 / 475, of 1048576 78 / 244 / 1700.
// Both orders are exact: by score key, then by position.
// PER = 0 keeps to 32 registers, so that two CTAs fit an SM: 32 sequences of 140000 tokens take 113 us per call, 130 with
// the 56 registers the compiler takes when it may.
template <int PER, bool CLUSTER>
__global__ void __launch_bounds__(kSelectThreads, PER == 0 ? 2 : 1)
dsa_select_kernel(const float* __restrict__ scores, const uint2* __restrict__ ranges, int runs, int run_len, int max_ls,
                  const int32_t* __restrict__ seq_lens, const int32_t* __restrict__ block_table, int max_pages,
                  int32_t* __restrict__ out) {
  extern __shared__ int4 s_dyn[];
  int4* s_hist4 = s_dyn;                                            // [kBins] counts; later the items that arrive
  int* s_hist = reinterpret_cast<int*>(s_hist4);
  unsigned long long* s_in = reinterpret_cast<unsigned long long*>(s_hist4);
  unsigned long long* s_item = s_in + kMaxListed;                   // [kMaxListed] items grouped by bin
  int4* s_cursor4 = reinterpret_cast<int4*>(s_item + kMaxListed);   // [kBins] counts of the sequence, then cursors
  int* s_cursor = reinterpret_cast<int*>(s_cursor4);
  int* s_table = s_cursor + kBins;                                  // [kTablePages] start of the sequence's block table
  __shared__ int s_scan[32];
  __shared__ int s_cut[3];              // cut bin (-1: the bins do not separate the scores), candidate, items at or above it
  __shared__ int s_own, s_base;         // items this CTA has collected, their place in the first CTA's s_in
  __shared__ int s_arrived;             // first CTA: items in s_in
  __shared__ int s_radix[2][256], s_misc[12];
  cg::cluster_group cluster = cg::this_cluster();
  const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = CLUSTER ? static_cast<int>(blockIdx.x) : 0;
  s_hist4[tid] = make_int4(0, 0, 0, 0);
  if (tid == 0) { s_own = 0; s_arrived = 0; }
  pdl_wait();
  pdl_trigger();
  const int n = min(seq_lens[b], max_ls);
  int32_t* o = out + static_cast<size_t>(b) * kKeep;
  if (n <= 0) {                         // the same for every CTA of the cluster
    if (rank == 0)
      for (int i = tid; i < kKeep; i += kSelectThreads) o[i] = -1;
    return;
  }
  // a sequence that fits one CTA's registers is finished by the first CTA, without the cluster's barriers
  const bool joint = CLUSTER && n > (PER > 0 ? PER : 8) * kSelectThreads;
  const int ctas = joint ? static_cast<int>(gridDim.x) : 1;
  if (rank >= ctas) return;
  const int k = min(kKeep, n);
  const float* sc = scores + static_cast<size_t>(b) * max_ls;
  const int32_t* table = block_table + static_cast<size_t>(b) * max_pages;
  const int first = rank * kSelectThreads + tid, step = ctas * kSelectThreads;
  float mine[PER > 0 ? PER : 1];
  // f(score, position) for each of this thread's positions
  auto sweep = [&](auto f) {
    if constexpr (PER > 0) {
#pragma unroll
      for (int j = 0; j < PER; ++j)
        if (first + j * step < n) f(mine[j], first + j * step);
    } else {
      for (int i = first; i < n; i += step) f(__ldg(sc + i), i);
    }
  };
  if constexpr (PER > 0) {
#pragma unroll
    for (int j = 0; j < PER; ++j) mine[j] = first + j * step < n ? __ldg(sc + first + j * step) : 0.0f;
  }

  if (rank == 0)
    for (int i = tid; i < kTablePages && i * kPage < n; i += kSelectThreads) s_table[i] = table[i];

  // 1. range (every warp for itself: no barrier)
  uint32_t low = 0xffffffffu, high = 0u;
  for (int i = lane; i * run_len < n; i += 32) {
    const uint2 r = ranges[static_cast<size_t>(b) * runs + i];
    low = min(low, r.x);
    high = max(high, r.y);
  }
  const float lowest = key_score(__reduce_min_sync(0xffffffffu, low));
  const float range = key_score(__reduce_max_sync(0xffffffffu, high)) - lowest;
  const float scale = static_cast<float>(kBins - 1) / range;
  // NaNs and infinities make the range, ties and tiny ranges the scale useless
  const bool binned = range > 0.0f && range <= 3.0e38f && scale <= 3.0e38f;
  __syncthreads();

  // 2. histogram
  if (binned) sweep([&](float s, int) { atomicAdd(&s_hist[score_bin(s, lowest, scale)], 1); });
  if (joint) {
    cluster.sync();
    const int quads = kBins / 4 / ctas;   // cluster sizes are powers of two
    if (tid < quads) {
      const int i = rank * quads + tid;
      int4 r[kMaxCluster];
#pragma unroll
      for (int c = 0; c < kMaxCluster; ++c)
        r[c] = c < ctas ? cluster.map_shared_rank(s_hist4, c)[i] : make_int4(0, 0, 0, 0);
#pragma unroll
      for (int c = 1; c < kMaxCluster; ++c) {
        r[0].x += r[c].x; r[0].y += r[c].y; r[0].z += r[c].z; r[0].w += r[c].w;
      }
      cluster.map_shared_rank(s_cursor4, 0)[i] = r[0];
    }
    cluster.sync();
  } else {
    __syncthreads();
  }

  // 3. first rank of every bin, and the cut; thread t has bins 4 t .. 4 t + 3 counted from the top
  if (rank == 0) {
    static_assert(kBins == 4 * kSelectThreads, "four bins per thread");
    const int quad = kSelectThreads - 1 - tid;
    const int4 q = joint ? s_cursor4[quad] : s_hist4[quad];
    const int h[4] = {q.w, q.z, q.y, q.x}, sum = q.x + q.y + q.z + q.w;
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += up;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    int at = __reduce_add_sync(0xffffffffu, lane < warp ? s_scan[lane] : 0) + incl - sum;   // items above this thread's bins
    bool crowded = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int bin = 4 * quad + 3 - j;
      s_cursor[bin] = at;
      crowded |= at < k && h[j] > kMaxInBin;
      if (at < k && at + h[j] >= k) { s_cut[1] = bin; s_cut[2] = at + h[j]; }
      at += h[j];
    }
    crowded = __syncthreads_or(crowded);
    if (tid == 0) s_cut[0] = binned && !crowded ? s_cut[1] : -1;
  }
  int cut;
  if (joint) {
    cluster.sync();
    cut = cluster.map_shared_rank(s_cut, 0)[0];
  } else {
    __syncthreads();
    cut = s_cut[0];
  }

  auto item_of = [](float s, int i) {
    return (static_cast<unsigned long long>(score_key(s)) << 32) | static_cast<uint32_t>(~i);
  };
  auto token = [&](unsigned long long item) {
    const int pos = static_cast<int>(~static_cast<uint32_t>(item)), page = pos / kPage;
    const int cache_page = page < kTablePages ? s_table[page] : table[page];
    return cache_page < 0 ? -1 : cache_page * kPage + pos % kPage;
  };
  if (cut < 0) {
    select_best<PER>([&](int j) {
      const int i = first + j * step;
      return i < n ? item_of(PER > 0 ? mine[PER > 0 ? j : 0] : __ldg(sc + i), i) : 0ull;
    }, (n + step - 1) / step, k, ctas, rank, s_item, reinterpret_cast<unsigned long long*>(s_cursor), &s_arrived, s_radix, s_misc);
    if (rank != 0) return;
    for (int i = tid; i < kKeep; i += kSelectThreads) o[i] = i < k ? token(s_item[i]) : -1;
    return;
  }

  // 4. the items at or above the cut bin, grouped by bin
  auto bin_of = [&](unsigned long long it) { return score_bin(key_score(static_cast<uint32_t>(it >> 32)), lowest, scale); };
  if (rank == 0) {
    sweep([&](float s, int i) {
      const int bin = score_bin(s, lowest, scale);
      if (bin >= cut) s_item[atomicAdd(&s_cursor[bin], 1)] = item_of(s, i);
    });
  } else {
    sweep([&](float s, int i) {
      if (score_bin(s, lowest, scale) >= cut) s_item[atomicAdd(&s_own, 1)] = item_of(s, i);
    });
    __syncthreads();
    if (tid == 0 && s_own > 0) s_base = atomicAdd(cluster.map_shared_rank(&s_arrived, 0), s_own);
    __syncthreads();
    unsigned long long* in = cluster.map_shared_rank(s_in, 0) + s_base;
    for (int i = tid; i < s_own; i += kSelectThreads) in[i] = s_item[i];
  }
  if (joint) cluster.sync();     // also keeps the first CTA's shared memory until the others are through with it
  else __syncthreads();
  if (rank != 0) return;

  if (joint) {
    for (int i = tid; i < s_arrived; i += kSelectThreads) {
      const unsigned long long it = s_in[i];
      s_item[atomicAdd(&s_cursor[bin_of(it)], 1)] = it;
    }
    __syncthreads();
  }
  // 5. a bin's cursor now stands at the first rank of the next lower bin
  for (int i = tid; i < s_cut[2]; i += kSelectThreads) {
    const unsigned long long it = s_item[i];
    const int bin = bin_of(it), end = s_cursor[bin];
    int at = bin == kBins - 1 ? 0 : s_cursor[bin + 1];
    int final_rank = at;
#pragma unroll 4
    for (; at < end; ++at) final_rank += s_item[at] > it;
    if (final_rank < k) o[final_rank] = token(it);
  }
  for (int i = k + tid; i < kKeep; i += kSelectThreads) o[i] = -1;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

typedef CUresult (*IsCapturingFn)(CUstream, CUstreamCaptureStatus*);
typedef CUresult (*StreamIdFn)(CUstream, unsigned long long*);

// Driver functions without a link to libcuda.  (The runtime has the two on streams as well; it takes 40 ns for each instead
// of 11, and a short batch is bound by the host's part of the call.)
struct Driver {
  EncodeTiledFn encode_tiled = nullptr;
  IsCapturingFn is_capturing = nullptr;
  StreamIdFn stream_id = nullptr;
};

template <typename Fn>
void driver_fn(const char* name, Fn* fn) {
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
    *fn = reinterpret_cast<Fn>(p);
}

const Driver& driver() {
  static Driver d;
  static std::once_flag once;
  std::call_once(once, [] {
    driver_fn("cuTensorMapEncodeTiled", &d.encode_tiled);
    driver_fn("cuStreamIsCapturing", &d.is_capturing);
    driver_fn("cuStreamGetId", &d.stream_id);
  });
  return d;
}

// rows of 128 bytes, boxes of 64 rows, 128-byte swizzle
bool rows128_map(CUtensorMap* m, const void* base, uint64_t rows) {
  const EncodeTiledFn fn = driver().encode_tiled;
  if (!fn) return false;
  const cuuint64_t dims[2] = {128, rows};
  const cuuint64_t strides[1] = {128};
  const cuuint32_t box[2] = {128, 64};
  const cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int PER, bool CLUSTER>
cudaError_t launch_select_as(int ctas, const float* scores, const uint2* ranges, int runs, int run_len,
                             int max_ls, const int32_t* seq_lens, const int32_t* block_table, int batch, int max_pages,
                             int32_t* out, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, batch);
  cfg.blockDim = dim3(kSelectThreads);
  cfg.dynamicSmemBytes = kSelectSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = ctas;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CLUSTER ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, dsa_select_kernel<PER, CLUSTER>, scores, ranges, runs, run_len, max_ls, seq_lens,
                            block_table, max_pages, out);
}

// CTAs per sequence by the table's width and the batch.  8192 positions per CTA (eight per thread in registers) while
// that gives at most one CTA per SM, else 16384: clusters of eight with two CTAs on every SM do not all find room at
// once (32 sequences of 65536 tokens: 72 us per call with eight CTAs each, 63 us with four).  Beyond 131072
// positions the scores are read again (from L2) in each sweep.
cudaError_t launch_select(const float* scores, const uint2* ranges, int runs, int run_len, int max_ls,
                          const int32_t* seq_lens, const int32_t* block_table, int batch, int max_pages, int32_t* out,
                          int num_sms, cudaStream_t st) {
  auto run = [&](auto* launch, int ctas) {
    return launch(ctas, scores, ranges, runs, run_len, max_ls, seq_lens, block_table, batch, max_pages, out, st);
  };
  auto ctas_for = [&](int positions) {
    int ctas = 1;
    while (ctas < kMaxCluster && static_cast<int64_t>(ctas) * positions < max_ls) ctas *= 2;
    return ctas;
  };
  const int c8 = ctas_for(8 * kSelectThreads), c16 = ctas_for(16 * kSelectThreads);
  if (c8 == 1) return run(launch_select_as<8, false>, 1);
  if (static_cast<int64_t>(c16) * 16 * kSelectThreads < max_ls) return run(launch_select_as<0, true>, kMaxCluster);
  if (c8 * 8 * kSelectThreads >= max_ls && static_cast<int64_t>(batch) * c8 <= num_sms) return run(launch_select_as<8, true>, c8);
  return c16 == 1 ? run(launch_select_as<16, false>, 1) : run(launch_select_as<16, true>, c16);
}

// The scores of every token of every sequence with their ranges, one buffer per stream: calls on one stream follow each
// other, calls on two may run at the same time.  A stream is known by its id, which is never given out twice (a handle
// may be, after the stream was destroyed); a stream that is being captured cannot be asked for it and is known by its
// handle.
struct Scratch {
  cudaStream_t handle = nullptr;
  unsigned long long id = 0; // 0: not known yet
  uint64_t last_use = 0;     // 0: free
  float* scores = nullptr;
  size_t floats = 0;
  bool captured = false;     // a graph may use it
};
constexpr int kMaxScratch = 8;   // streams of a device that hold one at a time; the next one takes over the least recently used

struct Device {
  Scratch scratch[kMaxScratch];
  uint64_t calls = 0;
  int* status = nullptr;
  long long next_wait_limit = 0;   // syfi_dsa_debug_wait_limit: applies to the next call, then clears itself
  bool checked = false;
  int num_sms = 0;
};
std::mutex g_mu;
Device g_devices[64];

int fail(int code, const char* msg) { return set_last_error(code, msg); }

// Allocation must not end a capture that is going on, on this stream or another.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The stream's buffer of at least `need` floats; null with the error code in *rc when there is none.
Scratch* scratch_of(Device& d, cudaStream_t st, size_t need, int* rc) {
  const Driver& drv = driver();
  CUstreamCaptureStatus capture = CU_STREAM_CAPTURE_STATUS_NONE;
  unsigned long long id = 0;
  bool known = drv.is_capturing && drv.stream_id;
  if (known && drv.is_capturing(st, &capture) != CUDA_SUCCESS) capture = CU_STREAM_CAPTURE_STATUS_NONE;   // the default stream beside a capture: the launch will say so
  const bool capturing = capture != CU_STREAM_CAPTURE_STATUS_NONE;
  if (known && !capturing) known = drv.stream_id(st, &id) == CUDA_SUCCESS;
  if (!known) {
    *rc = fail(SYFI_DSA_ERR_CUDA, "not a stream of the current device");
    return nullptr;
  }
  // The stream's own; of two (below) the larger.
  Scratch *s = nullptr, *spare = nullptr;
  for (Scratch& c : d.scratch) {
    if (c.last_use == 0) spare = &c;
    else if ((capturing || c.id == 0 ? c.handle == st : c.id == id) && (!s || c.floats > s->floats)) s = &c;
  }
  if (s && s->floats < need && (capturing || s->captured) && spare) s = nullptr;   // a graph keeps the small one
  if (capturing && !spare && (!s || s->floats < need)) {
    // Nothing may wait now, so nothing can be freed: whichever is large enough, as if the two streams were one.
    s = nullptr;
    for (Scratch& c : d.scratch)
      if (c.floats >= need && (!s || c.last_use < s->last_use)) s = &c;
    if (!s) *rc = fail(SYFI_DSA_ERR_CUDA, "no scratch buffer is large enough, and none can be had during a capture");
    else s->captured = true;
    return s;
  }
  if (!s) {
    s = spare;
    if (!s) {   // the one that was not used for longest, of those that no graph needs, if there is one
      for (Scratch& c : d.scratch)
        if (!s || (c.captured != s->captured ? s->captured : c.last_use < s->last_use)) s = &c;
      if (cudaDeviceSynchronize() != cudaSuccess) {
        *rc = fail(SYFI_DSA_ERR_CUDA, "device synchronisation failed");
        return nullptr;
      }
    }
    s->handle = st;
    s->id = 0;
    s->captured = false;
  }
  if (need > s->floats) {
    if (s->scores) {
      if (cudaDeviceSynchronize() != cudaSuccess) {
        *rc = fail(SYFI_DSA_ERR_CUDA, "device synchronisation failed");
        return nullptr;
      }
      cudaFree(s->scores);
    }
    s->scores = nullptr;
    s->floats = 0;
    RelaxedCapture relaxed;
    if (cudaMalloc(&s->scores, need * sizeof(float)) != cudaSuccess) {
      s->last_use = 0;
      *rc = fail(SYFI_DSA_ERR_CUDA, "out of device memory for the scores");
      return nullptr;
    }
    s->floats = need;
  }
  if (id != 0) s->id = id;
  if (capturing) s->captured = true;
  s->last_use = ++d.calls;
  return s;
}

}  // namespace

}  // namespace syfi

using namespace syfi;

extern "C" int syfi_dsa_topk_indexer(const void* q_index_fp8, const void* k_index_cache_fp8, const float* weights,
                                     const int32_t* seq_lens, const int32_t* block_table, int32_t batch,
                                     int64_t num_pages, int32_t max_pages, int32_t* topk_indices, void* stream) {
  if (batch < 0 || batch > (1 << 20)) return fail(SYFI_DSA_ERR_INVALID, "batch out of range");
  if (batch == 0) return SYFI_DSA_OK;
  if (num_pages < 1 || num_pages > (1ll << 24)) return fail(SYFI_DSA_ERR_INVALID, "num_pages out of range");
  if (max_pages < 1 || max_pages > (1 << 20)) return fail(SYFI_DSA_ERR_INVALID, "max_pages (block table width) out of range");
  const void* ptrs[] = {q_index_fp8, k_index_cache_fp8, weights, seq_lens, block_table, topk_indices};
  for (const void* p : ptrs)
    if (!p || (reinterpret_cast<uintptr_t>(p) & 15u)) return fail(SYFI_DSA_ERR_INVALID, "a tensor argument is null or not 16-byte aligned");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(SYFI_DSA_ERR_CUDA, "no current CUDA device: this library has no CPU path");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int max_ls = max_pages * kPage;
  std::lock_guard<std::mutex> lock(g_mu);
  Device& d = g_devices[dev];
  if (!d.checked) {     // once per device: the attribute queries cost more than the kernels
    int major = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess || major != 10 ||
        cudaDeviceGetAttribute(&d.num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return fail(SYFI_DSA_ERR_CUDA, "this library is built for sm_100a (B200) only");
    d.checked = true;
  }
  // scores, and a score range per 128 tokens at most (a multiple of 64 floats before it)
  const size_t n_scores = static_cast<size_t>(batch) * max_ls;
  const size_t need = n_scores + 2 * static_cast<size_t>(batch) * ((max_ls + kTokTile - 1) / kTokTile);
  int rc = SYFI_DSA_OK;
  Scratch* const s = scratch_of(d, st, need, &rc);
  if (!s) return rc;
  if (!d.status) {
    if (cudaMalloc(&d.status, 16) != cudaSuccess) return fail(SYFI_DSA_ERR_CUDA, "out of device memory");
    cudaMemset(d.status, 0, 16);
    auto raise = [](auto* kernel, int bytes) {
      return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
    };
    if (!raise(dsa_score_kernel, kScoreSmem) || !raise(dsa_select_kernel<8, false>, kSelectSmem) ||
        !raise(dsa_select_kernel<8, true>, kSelectSmem) || !raise(dsa_select_kernel<16, true>, kSelectSmem) ||
        !raise(dsa_select_kernel<16, false>, kSelectSmem) || !raise(dsa_select_kernel<0, true>, kSelectSmem))
      return fail(SYFI_DSA_ERR_CUDA, "cannot raise the shared-memory limit of the indexer's kernels");
  }
  const long long wait_limit = d.next_wait_limit > 0 ? d.next_wait_limit : kWaitLimit;
  d.next_wait_limit = 0;
  CUtensorMap tm_q, tm_k;
  if (!rows128_map(&tm_q, q_index_fp8, static_cast<uint64_t>(batch) * kHeads) ||
      !rows128_map(&tm_k, k_index_cache_fp8, static_cast<uint64_t>(num_pages) * kPageRows))
    return fail(SYFI_DSA_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  // Tiles per score CTA: as few as keep a few waves of CTAs (four to five fit an SM) in flight by the table's width;
  // a short table is a matter of latency, where each tile more in a CTA's chain is about half a microsecond.
  const int64_t tiles = static_cast<int64_t>(batch) * ((max_ls + kTokTile - 1) / kTokTile);
  // us per call with 1 / 2 / 4 / 8 tiles: 8 sequences (4096 tiles) 38.4 / 26.8 / 23.7 / 24.7, 24 (6144) 42.3 / 28.5 / 23.3 /
  // 24.2, 16 (8192) 63.9 / 44.0 / 37.8 / 37.5, 40 (20480) 114.7 / 66.2 / 46.0 / 40.0.
  const int per_cta = tiles <= 1024 ? 1 : tiles <= 2048 ? 2 : tiles <= 12288 ? 4 : kMaxTilesPerCta;
  const int runs = (max_ls + per_cta * kTokTile - 1) / (per_cta * kTokTile);
  uint2* ranges = reinterpret_cast<uint2*>(s->scores + n_scores);
  if (launch_dependent(dsa_score_kernel, dim3(runs, batch), dim3(kScoreThreads), kScoreSmem, st, tm_q, tm_k,
                       static_cast<const uint8_t*>(k_index_cache_fp8), weights, seq_lens, block_table, max_pages,
                       s->scores, max_ls, per_cta, ranges, d.status, wait_limit) != cudaSuccess)
    return fail(SYFI_DSA_ERR_CUDA, "score kernel launch failed");
  if (launch_select(s->scores, ranges, runs, per_cta * kTokTile, max_ls, seq_lens, block_table, batch, max_pages,
                    topk_indices, d.num_sms, st) != cudaSuccess)
    return fail(SYFI_DSA_ERR_CUDA, "select kernel launch failed");
  return SYFI_DSA_OK;
}

// Test hook for the bounded waits, no part of the interface: a wait of the next call's score kernel on the current device may
// take this many SM clocks (0: the normal limit).
extern "C" int syfi_dsa_debug_wait_limit(int64_t clocks) {
  if (clocks < 0) return fail(SYFI_DSA_ERR_INVALID, "a wait limit must not be negative");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(SYFI_DSA_ERR_CUDA, "no current CUDA device");
  std::lock_guard<std::mutex> lock(g_mu);
  g_devices[dev].next_wait_limit = clocks;
  return SYFI_DSA_OK;
}

extern "C" int syfi_dsa_check(void* stream) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(SYFI_DSA_ERR_CUDA, "no current CUDA device");
  if (cudaStreamSynchronize(static_cast<cudaStream_t>(stream)) != cudaSuccess)
    return fail(SYFI_DSA_ERR_CUDA, "stream synchronisation failed");
  std::lock_guard<std::mutex> lock(g_mu);
  Device& d = g_devices[dev];
  if (!d.status) return SYFI_DSA_OK;
  int status = 0;
  if (cudaMemcpy(&status, d.status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return fail(SYFI_DSA_ERR_CUDA, "cannot read the status word");
  if (status != 0) {
    cudaMemset(d.status, 0, sizeof(int));
    char msg[128];
    snprintf(msg, sizeof(msg), "a kernel reported status %d (201: a bounded wait in the score kernel ran out)", status);
    return fail(SYFI_DSA_ERR_DEVICE, msg);
  }
  return SYFI_DSA_OK;
}
