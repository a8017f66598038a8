// Work list of the varlen tile scheduler.
//
// In packed (cu_seqlens) mode the attention kernels do not launch a rectangular grid of
// ceil(max_seqlen / 128) tiles per sequence and let the tiles past a short sequence's end exit;
// they work through a compact list of (sequence, tile) items, built on the device from cu_seqlens by
// the single-CTA kernel below with no host synchronisation:
//
//   * an item is one 128-row tile on the list's "own" side (query tiles for the forward, key
//     tiles for the backward); its cost is the number of 128-row steps on the other side;
//   * items are ordered most expensive first (sequences bucketed by their step count). Inspected on
//     its own the list has the ragged last tile of every sequence -- fewer live rows, trimmed inner
//     work -- after all full tiles; the attention calls build it with the ragged tiles at the end of
//     their own cost class (`merged`): a ragged tile of a long sequence is still long work, and at the
//     end of the list it started when everything else was finished. Persistent CTAs take the units
//     (entry x head) in list order from a counter (the first entry's reserved word, zero when the
//     list is new), so long units start first, short ones fill the gaps, and ragged visible-token
//     counts do not leave SMs idle. One 2000-token sequence among thirty 200-token ones, 12 heads:
//     forward 44.6 us with one CTA per unit and 51.6 with units dealt out by position, 35.3 from the
//     counter; whole backward 90.7 (dealt out) and 84.3 us;
//   * rows of the packed buffer past the last sequence (a caller may pack into a buffer of fixed
//     capacity to avoid a device-to-host sync) form one more pseudo-sequence, index `batch`, that
//     owns rows [cu_seqlens[batch], total) and has nothing on the other side: its items make the
//     kernels write zeros there, so every row of every output is defined;
//   * the backward's list may have runs (SchedRuns): one item for all key tiles of a sequence, for one CTA per head;
//   * the list has a host-known capacity of floor(total / 128) + batch + 1 entries; unused entries
//     have seq = -1 and end a CTA's work;
//   * an entry carries the sequence's offsets and lengths on both sides, so a CTA learns all it
//     needs about its work from one 32-byte read instead of a chain of dependent loads.
//
// The same kernel validates the packing it reads: offsets non-negative and non-decreasing, every
// length <= max_seqlen (the caller's bound sizes tensor maps and grids), last offset <= total
// tokens. On a violation it writes kStatusBadSeqlens to the status word and leaves the whole list
// empty, so the attention kernel does nothing instead of reading out of bounds.
//
// The reference's ragged consumer that this serves is the per-image eval loop of
// src/nanobrain/model.py:254-270 and the per-sample visible counts of model.py:186-199.
#pragma once

#include "ptx.cuh"

namespace nb {

// One work item; mirrors nb_attn_sched_item in include/nb_attn.h.
struct __align__(16) SchedItem {
  int32_t seq;          // sequence index; `batch` = the rows past the last sequence; -1 = unused entry
  int32_t tile;         // 128-row tile on the own side; -1: all of them (see SchedRuns)
  int32_t own_begin;    // first packed row of the sequence on the own side
  int32_t own_len;      // its length there
  int32_t other_begin;  // the same on the side the item's inner loop walks
  int32_t other_len;
  int32_t reserved[2];  // zero in a new list; the first entry's count the units taken and the CTAs done
};
static_assert(sizeof(SchedItem) == 32, "two 16-byte loads");

// Reads one entry with two 16-byte loads (one memory round trip).
__device__ __forceinline__ SchedItem sched_load(const SchedItem* items, uint32_t idx) {
  const int4* src = reinterpret_cast<const int4*>(items + idx);
  const int4 a = src[0], b = src[1];
  SchedItem it;
  it.seq = a.x, it.tile = a.y, it.own_begin = a.z, it.own_len = a.w;
  it.other_begin = b.x, it.other_len = b.y, it.reserved[0] = 0, it.reserved[1] = 0;
  return it;
}

// Takes the next unit of a list.
__device__ __forceinline__ uint32_t sched_next(const SchedItem* items) {
  return uint32_t(atomicAdd(const_cast<int32_t*>(&items[0].reserved[0]), 1));
}

// A CTA takes no more units. The last of `ctas` leaves the list as it was when new, for the next launch.
__device__ __forceinline__ void sched_leave(const SchedItem* items, uint32_t ctas) {
  int32_t* words = const_cast<int32_t*>(items[0].reserved);
  if (uint32_t(atomicAdd(words + 1, 1)) == ctas - 1) words[0] = words[1] = 0;
}

constexpr int kSchedThreads = 1024;
constexpr int kSchedBuckets = 1024;  // step counts >= kSchedBuckets - 1 share the first bucket
constexpr int kSchedTile = 128;

// Upper bound of the number of items of a packing with `total` tokens in `batch` sequences (plus
// the pseudo-sequence of the unused rows at the end).
__host__ __device__ inline int64_t sched_capacity(int64_t total, int32_t batch) {
  return total / kSchedTile + batch + 1;
}

struct SchedParams {
  const int32_t* cu_own;    // offsets on the side whose tiles become items
  const int32_t* cu_other;  // offsets on the side an item's inner loop walks
  int32_t batch;
  int32_t max_own, max_other;
  int64_t total_own, total_other;
  SchedItem* items;  // [n_items]
  int32_t n_items;  // capacity, >= sched_capacity(total_own, batch)
  int32_t* status;
  int32_t merged;  // ragged tiles at the end of their cost class instead of after all full tiles
  // Runs (see SchedRuns) have at most this many tiles on the other side. -1: no sequence has more than one tile on the
  // own side.
  int32_t run_tiles;
  int32_t heads, sms;
  int32_t* rest;  // where the list of the sequences that are no runs goes
};

// Exclusive prefix sum over one value per thread of a block of kThreads threads (returns the
// exclusive prefix and writes the grand total to *total). `scratch` holds 32 ints.
template <int kThreads>
__device__ __forceinline__ int block_exclusive_scan(int v, int* scratch, int* total) {
  static_assert(kThreads % 32 == 0 && kThreads <= 1024, "whole warps");
  constexpr int kWarps = kThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += up;
  }
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < kWarps ? scratch[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += up;
    }
    scratch[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  const int warp_prefix = warp > 0 ? scratch[warp - 1] : 0;
  *total = scratch[31];
  __syncthreads();  // scratch may be reused
  return warp_prefix + incl - v;
}

// Does this kernel's part of one sequence: lengths, validity, bucket.
struct SchedSeq {
  int full;    // full tiles on the own side
  int ragged;  // 1 if a partial last tile exists
  int bucket;  // 0 = most expensive
  bool ok;
  bool run;  // one item stands for all tiles
  int own_begin, own_len, other_begin, other_len;
};

// Which sequences are runs: one item, all of whose tiles the CTA that takes it works off one after the other.
// A sequence with something on both sides is one if it has a single tile on the own side, or if its
// index is below `below`, it has at most run_tiles tiles on the other side and a cost (steps of all its tiles) of at
// most max_cost. below = -1: there are none.
struct SchedRuns {
  int below, max_cost;
};
__host__ __device__ inline int sched_tiles(int len) { return len / kSchedTile + (len % kSchedTile != 0); }
// Steps of the sequence as a run; 0 if it is none.
__host__ __device__ inline int sched_run_cost(const SchedParams& p, const SchedSeq& s, int i, const SchedRuns& r) {
  if (r.below < 0 || !s.ok || s.own_len <= 0 || s.other_len <= 0) return 0;
  const int own = sched_tiles(s.own_len), other = sched_tiles(s.other_len);
  if (own == 1) return other;
  // (One tile on the other side that several own tiles add to: no step in between for an addition to complete.)
  if (i >= r.below || other > p.run_tiles || other == 1 || own > r.max_cost / other) return 0;
  return own * other;
}

__host__ __device__ inline SchedItem sched_item(const SchedSeq& s, int seq, int tile) {
  SchedItem it;
  it.seq = seq, it.tile = s.run ? -1 : tile;
  it.own_begin = s.own_begin, it.own_len = s.own_len, it.other_begin = s.other_begin, it.other_len = s.other_len;
  it.reserved[0] = it.reserved[1] = 0;
  return it;
}

__host__ __device__ inline SchedItem sched_no_item() {
  SchedItem it;
  it.seq = -1, it.tile = 0, it.own_begin = it.own_len = it.other_begin = it.other_len = 0;
  it.reserved[0] = it.reserved[1] = 0;
  return it;
}

// i in [0, batch]: i == batch is the pseudo-sequence of the rows past the last sequence.
__host__ __device__ inline int sched_bucket(int steps) {
  return kSchedBuckets - 1 - (steps < kSchedBuckets - 1 ? steps : kSchedBuckets - 1);
}
__host__ __device__ inline SchedSeq sched_classify(const SchedParams& p, int i) {
  SchedSeq s;
  s.run = false;
  int64_t len, steps_len;
  if (i == p.batch) {
    len = p.total_own - int64_t(p.cu_own[i]);
    steps_len = 0;
    s.ok = len >= 0;  // the last offset does not exceed the token count
    s.own_begin = p.cu_own[i];
    s.other_begin = 0;
  } else {
    const int64_t a = p.cu_own[i], b = p.cu_own[i + 1];
    const int64_t c = p.cu_other[i], d = p.cu_other[i + 1];
    len = b - a;
    steps_len = d - c;
    s.ok = a >= 0 && c >= 0 && len >= 0 && steps_len >= 0 && len <= p.max_own && steps_len <= p.max_other &&
           b <= p.total_own && d <= p.total_other;
    s.own_begin = int(a);
    s.other_begin = int(c);
  }
  s.own_len = int(len);
  s.other_len = int(steps_len);
  s.full = len > 0 ? int(len / kSchedTile) : 0;
  s.ragged = len > 0 && (len % kSchedTile) != 0;
  const int steps = steps_len > 0 ? int((steps_len + kSchedTile - 1) / kSchedTile) : 0;
  s.bucket = sched_bucket(steps);
  return s;
}
// The same with runs: a run is one full tile of the run's cost.
__host__ __device__ inline SchedSeq sched_classify(const SchedParams& p, int i, const SchedRuns& r) {
  SchedSeq s = sched_classify(p, i);
  if (const int cost = sched_run_cost(p, s, i, r)) s.run = true, s.full = 1, s.ragged = 0, s.bucket = sched_bucket(cost);
  return s;
}

// ---- runs ---------------------------------------------------------------------------------
constexpr int kSchedRunSeqs = 2048;  // packings of more sequences have no runs (their ends are kept in shared memory)

template <int kThreads>
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v, unsigned long long* scratch) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) v += scratch[w];
  __syncthreads();  // scratch may be reused
  return v;
}

struct SchedRunShared {
  unsigned long long sum[32];
  int scratch[32];
  int count, most, below, bad;
  int cost[kSchedRunSeqs];  // steps of the sequence as a run of several tiles, 0: it can be none
};

// The rule for this packing; every block that calls it comes to the same one. A run must not outlast a CTA's share of
// all steps, and what the runs leave of the work has to stay single tiles, which fill the gaps at the runs' end: the
// list's order, most expensive first, evens out what runs differ, but only to the cheapest one's cost. So runs fill
// whole rounds over the SMs, either rounds of the most expensive run's cost or rounds of the average cost with half an
// average run per SM left over, whichever is more. (32 sequences of 720..920 tokens and 12 heads: one round of 64 steps
// or two of 48 out of a share of 124, which is 2.5 % less time. Without the half run, 64 of them, five rounds of 48 out
// of 247: 4 % more.)
template <int kThreads>
__device__ __forceinline__ SchedRuns sched_runs(const SchedParams& p, SchedRunShared& sm) {
  if (threadIdx.x == 0) sm.count = sm.most = 0, sm.below = p.batch, sm.bad = 0;
  __syncthreads();
  unsigned long long steps = 0;
#pragma unroll 1
  for (int i = threadIdx.x; i <= p.batch; i += kThreads) {
    const SchedSeq s = sched_classify(p, i);
    if (!s.ok) sm.bad = 1;
    if (!s.ok || i == p.batch) continue;
    steps += (unsigned long long)sched_tiles(s.own_len) * unsigned(sched_tiles(s.other_len));
    sm.cost[i] = s.own_len > kSchedTile ? sched_run_cost(p, s, i, {p.batch, 0x7fffffff}) : 0;
  }
  steps = block_sum<kThreads>(steps, sm.sum);
  if (sm.bad) return {-1, 0};
  if (p.run_tiles < 0) return {0, 0};
  const unsigned long long share = steps * unsigned(p.heads) / unsigned(p.sms);
  const SchedRuns all = {p.batch, share < 0x7fffffffull ? int(share) : 0x7fffffff};
  unsigned long long total = 0;
  int count = 0, most = 0;
#pragma unroll 1
  for (int i = threadIdx.x; i < p.batch; i += kThreads) {
    const int cost = sm.cost[i];
    if (cost > 0 && cost <= all.max_cost) total += unsigned(cost), ++count, most = max(most, cost);
  }
  if (count > 0) atomicAdd(&sm.count, count), atomicMax(&sm.most, most);
  total = block_sum<kThreads>(total, sm.sum);
  if (sm.count == 0) return {0, 0};
  const unsigned long long average = (total + unsigned(sm.count) - 1) / unsigned(sm.count);
  unsigned long long rounds = share / average;
  if (rounds > 0 && share - rounds * average < average / 2) --rounds;
  const unsigned long long steps_per_sm = max(rounds * average, share / unsigned(sm.most) * unsigned(sm.most));
  const unsigned long long budget = steps_per_sm * unsigned(p.sms) / unsigned(p.heads);
  if (total <= budget) return all;
  unsigned long long before = 0;
#pragma unroll 1
  for (int base = 0; base < p.batch && before <= budget; base += kThreads) {
    const int i = base + threadIdx.x;
    int cost = i < p.batch ? sm.cost[i] : 0;
    if (cost > all.max_cost) cost = 0;
    int sum = 0;
    const int excl = block_exclusive_scan<kThreads>(cost, sm.scratch, &sum);
    if (cost > 0 && before + unsigned(excl) + unsigned(cost) > budget) atomicMin(&sm.below, i);
    before += unsigned(sum);
  }
  __syncthreads();
  return {sm.below, all.max_cost};
}

// The sequences that are no runs, as the epilogue reads them: word 0 counts the rows on the other side that
// belong to them; row x of these (in the order of the sequences) is row x + shift of the whole, shift from the first
// entry whose `end` exceeds x. One entry per sequence, the first one's with the rows before it, and one for the rows past
// the last one.
struct SchedRest {
  int end, shift;
};
__host__ __device__ inline size_t sched_rest_bytes(int32_t batch) { return 16 + (size_t(batch) + 1) * sizeof(SchedRest); }
template <int kThreads>
__device__ __forceinline__ void sched_write_rest(const SchedParams& p, const SchedRuns& r, SchedRunShared& sm) {
  SchedRest* rest = reinterpret_cast<SchedRest*>(p.rest + 4);
  int before = 0;
#pragma unroll 1
  for (int base = 0; base <= p.batch; base += kThreads) {
    const int i = base + threadIdx.x;
    int begin = 0, rows = 0;
    if (sm.bad) {  // not a packing: all rows
      rows = i == 0 ? int(p.total_other) : 0;
    } else if (i <= p.batch) {
      // (Rows before the first sequence are nobody's: the first entry has them, also in front of a run.)
      begin = i > 0 ? p.cu_other[i] : 0;
      rows = (i < p.batch ? p.cu_other[i + 1] : int(p.total_other)) - begin;
      if (sched_run_cost(p, sched_classify(p, i), i, r) > 0) rows = i > 0 ? 0 : p.cu_other[0];
    }
    int sum = 0;
    const int at = before + block_exclusive_scan<kThreads>(rows, sm.scratch, &sum);
    if (i <= p.batch) rest[i] = {at + rows, begin - at};
    before += sum;
  }
  if (threadIdx.x == 0) p.rest[0] = before;
}

// Shared-memory state of one list build.
struct SchedShared {
  int full_pos[kSchedBuckets];    // full tiles per bucket, then the bucket's write cursor
  int ragged_pos[kSchedBuckets];  // ragged tiles per bucket, then the bucket's write cursor
  int scratch[32];
  int bad;
};

// Builds the list with one block of kThreads threads (every thread of the block must call it).
template <int kThreads>
__device__ __forceinline__ void sched_build(const SchedParams& p, SchedShared& sm, const SchedRuns runs = {-1, 0}) {
  static_assert(kSchedBuckets % kThreads == 0, "each thread owns a run of consecutive buckets");
  constexpr int kPer = kSchedBuckets / kThreads;
  const int tid = threadIdx.x;
  for (int k = 0; k < kPer; ++k) {
    sm.full_pos[tid * kPer + k] = 0;
    sm.ragged_pos[tid * kPer + k] = 0;
  }
  if (tid == 0) sm.bad = 0;
  __syncthreads();

  for (int i = tid; i <= p.batch; i += kThreads) {
    const SchedSeq s = sched_classify(p, i, runs);
    if (!s.ok) {
      sm.bad = 1;
    } else {
      if (s.full) atomicAdd(&sm.full_pos[s.bucket], s.full);
      if (s.ragged) atomicAdd(&sm.ragged_pos[s.bucket], 1);
    }
  }
  __syncthreads();
  int my_full = 0, my_ragged = 0;
  for (int k = 0; k < kPer; ++k) {
    my_full += sm.full_pos[tid * kPer + k];
    my_ragged += sm.ragged_pos[tid * kPer + k];
  }
  int total_full = 0, total_ragged = 0;
  int full_at = block_exclusive_scan<kThreads>(p.merged ? my_full + my_ragged : my_full, sm.scratch, &total_full);
  int ragged_at = 0;
  if (!p.merged) ragged_at = block_exclusive_scan<kThreads>(my_ragged, sm.scratch, &total_ragged);
  const bool overflow = int64_t(total_full) + total_ragged > p.n_items;  // cannot happen for a valid packing
  if (sm.bad || overflow) {
    if (tid == 0 && p.status) atomicExch(p.status, (int)kStatusBadSeqlens);
    for (int i = tid; i < p.n_items; i += kThreads) p.items[i] = sched_no_item();
    return;
  }
  ragged_at += total_full;
  for (int k = 0; k < kPer; ++k) {
    const int nf = sm.full_pos[tid * kPer + k], nr = sm.ragged_pos[tid * kPer + k];
    sm.full_pos[tid * kPer + k] = full_at;
    full_at += nf;
    sm.ragged_pos[tid * kPer + k] = p.merged ? full_at : ragged_at;
    if (p.merged) full_at += nr;
    else ragged_at += nr;
  }
  __syncthreads();

  for (int i = tid; i <= p.batch; i += kThreads) {
    const SchedSeq s = sched_classify(p, i, runs);
    if (s.full) {
      const int at = atomicAdd(&sm.full_pos[s.bucket], s.full);
      for (int t = 0; t < s.full; ++t) p.items[at + t] = sched_item(s, i, t);
    }
    if (s.ragged) {
      const int at = atomicAdd(&sm.ragged_pos[s.bucket], 1);
      p.items[at] = sched_item(s, i, s.full);
    }
  }
  for (int i = total_full + total_ragged + tid; i < p.n_items; i += kThreads) p.items[i] = sched_no_item();
}

__global__ void __launch_bounds__(kSchedThreads) attn_sched_kernel(const SchedParams p) {
  __shared__ SchedShared sm;
  pdl_wait();  // cu_seqlens may come from the kernel right before this one
  pdl_launch_dependents();
  sched_build<kSchedThreads>(p, sm);
}

}  // namespace nb
