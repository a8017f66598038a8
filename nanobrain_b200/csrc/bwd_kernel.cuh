// Backward attention kernels (head_dim 64, bf16 tensors, fp32 accumulation):
//
//   attn_bwd_prologue_kernel : delta[row] = sum_d dO[row,d] * O[row,d] (warp-shuffle row dot) and
//                              clears the fp32 dQ accumulator. HBM-bound.
//   attn_bwd_kernel          : a work unit is one 128-row K/V tile of one (sequence, head), walked
//                              over the sequence's queries in 128-row steps. Everything is computed
//                              transposed (a tensor-memory lane is a key row; a compute thread holds
//                              four key rows x 16 query columns of a step):
//                                S^T  = K Q^T                       (A = K from tensor memory)
//                                dP^T = V dO^T                      (A = V from tensor memory)
//                                P^T  = exp2(S^T*scale_log2 - lse)  (recomputed from the saved LSE)
//                                dS^T = P^T o (dP^T - delta)
//                                dV  += P^T dO                      (A = P^T from tensor memory)
//                                dK  += dS^T Q                      (A = dS^T from tensor memory)
//                                dQ   = dS K                        (A = dS from shared memory)
//                              What bounds it: the SM's shared-memory port (operand reads of the MMAs,
//                              128 B per clock), the compute warps' dependent chain and the board's
//                              power limit (at 1 kW, on long sequences, the SMs run at 1.47-1.6 GHz of 1.965). So operands
//                              come from tensor memory wherever they can: K and V are copied there once
//                              per work unit (tcgen05.cp) and P^T and dS^T are written over the scores
//                              they came from; only dQ reads both operands from shared memory. Per step
//                              the port then carries 896 clocks of operand reads where A operands from
//                              shared memory need 1408.
//                              dQ tiles are added into the fp32 accumulator with TMA add-reductions
//                              because every K/V tile of a sequence contributes to every dQ row.
//                              CTAs are persistent (one per SM): each walks its share of the work
//                              units and the step pipeline runs on through the boundary between
//                              two units -- K is double-buffered, V is reloaded as soon as it
//                              has been copied into tensor memory, dV / dK leave through the drain
//                              warps while the next unit's first steps run -- so a unit's start-up
//                              and tail (a third of a CTA's life on ~800-token sequences) overlap
//                              its neighbours' steps.
//                              Warp roles (512 threads): warps 0-7 are two compute warpgroups that
//                              split the 128 query columns of a step (64 each); warps 8, 10, 11 are
//                              three MMA issuers (dV and the next S^T; dK and the next dP^T; dQ: one
//                              elected thread each, so that a wait of one does not hold back the
//                              others); warp 9 fetches the units, drives TMA and stages the steps'
//                              LSE/delta rows and control words; warps 12-15 drain the dQ tiles (one
//                              tensor-memory lane quadrant each) into the accumulator and, at the end
//                              of a unit, dV and dK into their tensors. Warp 9 publishes the units to
//                              the drain warps; the compute warps and the issuers learn about a step
//                              from its control word alone.
//                              Code size is a first-order concern here: five roles' loops run at
//                              the same time and have to share the SM's instruction cache (at
//                              67 KB of code its hit rate was 68 % and instruction fetch was the
//                              top stall; at 48 KB it is above 93 %). Hence the compact wait loop,
//                              divisions by multiply-high, and the compute role as a function that is
//                              not inlined. (The MMA-issue loops are unrolled: rolled, a thread issues
//                              an N = 64 MMA every 45-58 clocks instead of every 32.)
//                              Measured (dense 32 x 8 x 4096, repeated for 0.3 s, at the power limit;
//                              whole backward): A operands from shared memory, one row per thread
//                              3.82 ms; this form 3.37 ms.
//   attn_bwd_epilogue_kernel : dQ = bf16(scale * accumulator). HBM-bound.
//
// Packed calls with many (sequence, head) pairs of not too many tiles have a second kind of unit, a run: one CTA works
// off all key tiles of a pair and keeps its dQ in tiles of its own (see BwdRun). Clearing the accumulator in the
// prologue and reading it again in the epilogue is 16 % of the backward of such a call; for a run both fall away and
// delta is all that the prologue computes. Whole backward, us, without and with runs: 256 sequences of 720..920 tokens
// x 12 heads 2204 and 1932, 128 of them 1088 and 983, 64 537 and 507, 32 270 and 262; 500 of 1..300 490 and 383; 300 of
// 200 372 and 292. The form of the main kernel that knows runs is an instantiation of its own: its code is 2 KB larger,
// and with its waits inlined like the others' 7 KB, which made it 5 to 20 % slower on calls without any run.
//
// Packed mode: block 0 of the prologue also builds the scheduler's work list of key tiles
// (sched_kernel.cuh); the main kernel's work units are list entries x heads (the heads of one entry
// adjacent), taken by the CTAs in the list's order of decreasing cost.
// A ragged tile is computed at full width and masked: rows of the NEXT packed sequence that it
// brings into shared memory are
// multiplied by exact zeros of P^T / dS^T. For finite data that is exact; if the next sequence's
// first rows hold Inf or NaN, 0 x Inf makes this sequence's gradients NaN as well (the forward
// kernel clears such rows and keeps sequences isolated; measured here, clearing them in this
// kernel cost 7 % of its time, and cutting the MMAs of ragged tiles to their live rows gained
// nothing, so neither is done).
#pragma once

#include "fwd_kernel.cuh"
#include "ptx.cuh"

namespace nb {

#ifndef NB_BWD_L2_HINTS
#define NB_BWD_L2_HINTS 1
#endif

constexpr int kBwdPartFloats = 2 * kTile * kHeadDim;  // a cut unit's dV and dK

struct BwdParams {
  const __nv_bfloat16 *o, *d_o;
  int64_t o_sb, o_st, o_sh, do_sb, do_st, do_sh;
  __nv_bfloat16 *dq, *dk, *dv;
  int64_t dq_sb, dq_st, dq_sh, dk_sb, dk_st, dk_sh, dv_sb, dv_st, dv_sh;
  const float* lse;
  float* delta;     // same indexing as lse
  float* dq_accum;  // fp32 [total_q][heads][64]
  const int32_t* cu_q;
  const int32_t* cu_k;
  const SchedItem* items;  // packed mode: work list of key tiles; a unit is an entry and a head
  SchedParams sched;       // packed mode: what block 0 of the prologue builds (items == NULL: nothing)
  int32_t batch, heads;
  int32_t lq, lk;
  int32_t n_work;  // work units of the main kernel: key tiles x heads x sequences, or list entries x heads
  int32_t n_kt;    // dense mode: key tiles per (sequence, head)
  FastDiv div_heads, div_n_kt;  // the main kernel splits a work index without a division routine
  // Dense mode with few units: a CTA takes an equal run of (unit, query tile) steps, units are cut between
  // CTAs (see bwd_work) and the epilogue adds their parts up. NULL: whole units.
  float* parts;  // [2 * CTAs][kBwdPartFloats]
  uint32_t split_base, split_extra;  // CTA c starts at step c * base + min(c, extra)
  int32_t n_qt;                      // dense mode: query tiles per sequence
  FastDiv div_n_qt;
  FastDiv div_lq;
  int32_t rows32;      // (token, head) rows can be counted in 31 bits
  int32_t row_blocks;  // blocks of the epilogue that convert dQ; the ones after them add up parts
  // Runs: units that stand for all key tiles of a (sequence, head). Their dQ is summed up in the CTA's own
  // tiles and leaves as bf16 with the last key tile, so the accumulator and the epilogue are for the others.
  float* own;         // [CTAs][own_tiles][128 x 64]
  int32_t own_tiles;  // query tiles per CTA
  int32_t* rest;      // packed mode with runs: see sched_write_rest; NULL: every sequence is single tiles
  int64_t total_q, total_k;
  float scale, scale_log2;
  int32_t* status;
  int32_t pad[2];  // see below
};
// The host needs 1.9 us to launch a kernel whose parameters leave a remainder of 24 or 32 bytes by 64, and 2.2 to 2.3
// us with any other remainder (an empty kernel, sizes of 200..1144 bytes). It is these bytes for the prologue and
// epilogue, these and five tensor maps of 128 bytes for the main kernel: a backward's host time is 12.6 us with 24 and
// 13.4 us with 16.
static_assert(sizeof(BwdParams) % 64 == 24 || sizeof(BwdParams) % 64 == 32, "choose the size of `pad`");

// ----------------------------------------------------------------------------------------
// Prologue: one quarter-warp (8 lanes x 16 bytes) per (token, head) row.
// ----------------------------------------------------------------------------------------
constexpr int kAuxThreads = 256;

// Token, head and (dense mode) sequence and position of a (token, head) row. 64-bit divisions are routines of some
// hundred instructions, so rows that fit 31 bits are divided by multiply-high. In packed mode b = 0 and tok = t.
struct AuxRow {
  int64_t t, b, tok;
  int h;
  __device__ __forceinline__ AuxRow(const BwdParams& p, int64_t row) {
    b = 0;
    if (p.rows32) {
      const uint32_t t32 = p.div_heads.quot(uint32_t(row));
      t = tok = t32, h = int(uint32_t(row) - t32 * uint32_t(p.heads));
      if (p.cu_q == nullptr) {
        const uint32_t b32 = p.div_lq.quot(t32);
        b = b32, tok = t32 - b32 * uint32_t(p.lq);
      }
    } else {
      t = tok = row / p.heads, h = int(row - t * p.heads);
      if (p.cu_q == nullptr) b = t / p.lq, tok = t - b * p.lq;
    }
  }
};
// A block's part of `n_rows` rows where it takes consecutive ones: an equal share each.
__device__ __forceinline__ int64_t aux_begin(int64_t n_rows, uint32_t blocks, uint32_t block) {
  return min(int64_t(block) * ((n_rows + blocks - 1) / blocks), n_rows);
}

struct BwdPrologueShared {
  SchedRunShared runs;
  int end[kSchedRunSeqs + 1];  // last query row of each sequence + 1, and of the rows past the last one; bit 31: a run
  int first;                   // the sequence in which the block's rows start
  int lead;                    // rows before the first sequence
};

template <bool kRuns>
__global__ void __launch_bounds__(kAuxThreads) attn_bwd_prologue_kernel(const BwdParams p) {
  __shared__ SchedShared sched_sm;
  __shared__ std::conditional_t<kRuns, BwdPrologueShared, int> sm;
  pdl_wait();  // O comes from the forward kernel, dO from whatever ran before this call
  pdl_launch_dependents();
  const int64_t n_rows = p.total_q * p.heads;
  const int lane8 = threadIdx.x & 7;
  int64_t first = int64_t(blockIdx.x) * (kAuxThreads / 8), step = int64_t(gridDim.x) * (kAuxThreads / 8), end = n_rows;
  SchedRuns rule = {-1, 0};
  // With runs every block finds out by itself which sequences are: their accumulator needs no clearing.
  if constexpr (kRuns) rule = sched_runs<kAuxThreads>(p.sched, sm.runs);
  if (blockIdx.x == 0 && p.sched.items != nullptr) {
    sched_build<kAuxThreads>(p.sched, sched_sm, rule);
    if constexpr (kRuns) sched_write_rest<kAuxThreads>(p.sched, rule, sm.runs);
  }
  int seq = 0, lead = 0;
  if constexpr (kRuns) {
    // (The first block has the list to build, which the main kernel waits for: the others share its rows.)
    const uint32_t others = gridDim.x - 1;
    if (others > 0 && blockIdx.x == 0) return;
    const uint32_t part = others > 0 ? blockIdx.x - 1 : 0, parts = others > 0 ? others : 1;
    first = aux_begin(n_rows, parts, part), end = aux_begin(n_rows, parts, part + 1), step = kAuxThreads / 8;
    const int tok = int(min(first, n_rows - 1) / p.heads);
    if (threadIdx.x == 0) sm.first = 0;
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i <= p.batch; i += kAuxThreads) {
      int begin = 0, stop = int(p.total_q);
      bool run = false;
      if (!sm.runs.bad) {
        begin = p.cu_q[i];
        if (i < p.batch) {
          stop = p.cu_q[i + 1];
          const int keys = p.cu_k[i + 1] - p.cu_k[i], cost = sm.runs.cost[i];
          run = keys > kTile ? i < rule.below && cost > 0 && cost <= rule.max_cost : keys > 0 && stop > begin;
        }
      }
      sm.end[i] = stop | (run ? int(0x80000000u) : 0);
      if (begin <= tok && tok < stop) sm.first = i;
      if (i == 0) sm.lead = begin;
    }
    __syncthreads();
    seq = sm.first, lead = sm.lead;
  }
#if NB_BWD_L2_HINTS
  const uint64_t keep = l2_policy_evict_last();
#endif
  struct Loaded {
    uint4 o, g;
    int64_t row, didx;
    bool clear;
  };
  auto load = [&](int64_t row, Loaded& l) {
    const AuxRow w(p, row);
    l.row = row, l.clear = true;
    if (p.cu_q == nullptr) {
      l.didx = (w.b * p.heads + w.h) * p.lq + w.tok;
    } else {
      l.didx = int64_t(w.h) * p.total_q + w.tok;
      if constexpr (kRuns) {
        int stop = sm.end[seq];
        while (w.tok >= (stop & 0x7fffffff) && seq < p.batch) stop = sm.end[++seq];
        l.clear = stop >= 0 || w.tok < lead;
      }
    }
    l.o = *reinterpret_cast<const uint4*>(p.o + w.b * p.o_sb + w.tok * p.o_st + w.h * p.o_sh + lane8 * 8);
    l.g = *reinterpret_cast<const uint4*>(p.d_o + w.b * p.do_sb + w.tok * p.do_st + w.h * p.do_sh + lane8 * 8);
  };
  auto finish = [&](const Loaded& l) {
    const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&l.o);
    const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&l.g);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = __bfloat1622float2(o2[i]);
      const float2 g = __bfloat1622float2(g2[i]);
      acc = fmaf(a.x, g.x, acc);
      acc = fmaf(a.y, g.y, acc);
    }
    const uint32_t group = 0xffu << (threadIdx.x & 24);
    acc += __shfl_xor_sync(group, acc, 4);
    acc += __shfl_xor_sync(group, acc, 2);
    acc += __shfl_xor_sync(group, acc, 1);
    if (lane8 == 0) p.delta[l.didx] = acc;
    if (!l.clear) return;
    float4* acc_row = reinterpret_cast<float4*>(p.dq_accum + l.row * kHeadDim);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#if NB_BWD_L2_HINTS
    st_global_v4_hint(acc_row + lane8 * 2, z, keep);
    st_global_v4_hint(acc_row + lane8 * 2 + 1, z, keep);
#else
    acc_row[lane8 * 2] = z;
    acc_row[lane8 * 2 + 1] = z;
#endif
  };
  if constexpr (kRuns) {
    // Two rows at a time, so that twice the bytes are in flight: the stores keep the compiler from requesting the second
    // row before the first is done. (Where every row is cleared too, the writes are more than half of the traffic and
    // one row at a time is as fast.)
#pragma unroll 1
    for (int64_t row = first + (threadIdx.x >> 3); row < end; row += 2 * step) {
      Loaded l0, l1;
      load(row, l0);
      const bool two = row + step < end;
      if (two) load(row + step, l1);
      finish(l0);
      if (two) finish(l1);
    }
  } else {
    for (int64_t row = first + (threadIdx.x >> 3); row < end; row += step) {
      Loaded l;
      load(row, l);
      finish(l);
    }
  }
}

__device__ __forceinline__ uint32_t bwd_split_start(const BwdParams& p, uint32_t c) {
  return c * p.split_base + min(c, p.split_extra);
}

// dV and dK of a cut unit from its parts, in each of them 16 groups of four columns x 128 rows of fp32.
// Four blocks look after the unit in which CTA b's run starts, if that is the first cut in it: dV / dK
// times two halves of the rows; thread = (row, four groups).
__device__ __forceinline__ void bwd_combine(const BwdParams& p, uint32_t block) {
  const uint32_t b = (block >> 2) + 1, s0 = bwd_split_start(p, b);
  const uint32_t u = p.div_n_qt.quot(s0), first = u * uint32_t(p.n_qt), end = first + uint32_t(p.n_qt);
  if (s0 == first || bwd_split_start(p, b - 1) > first) return;
  const bool is_dk = (block & 1u) != 0;
  const int row = int(block >> 1 & 1u) * 64 + int(threadIdx.x & 63), g0 = int(threadIdx.x >> 6) * 4;
  const uint32_t t = p.div_n_kt.quot(u), seq = p.div_heads.quot(t), h = t - seq * uint32_t(p.heads);
  const int tok = int(u - t * uint32_t(p.n_kt)) * kTile + row;
  if (tok >= p.lk) return;
  float4 o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) o[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t c = b - 1; bwd_split_start(p, c) < end; ++c) {
    const float* part = p.parts + int64_t(2 * c + (c == b - 1)) * kBwdPartFloats + (is_dk ? kTile * kHeadDim : 0);
    const float4* src = reinterpret_cast<const float4*>(part) + g0 * kTile + row;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 a = src[j * kTile];
      o[j].x += a.x, o[j].y += a.y, o[j].z += a.z, o[j].w += a.w;
    }
  }
  __nv_bfloat16* out = is_dk ? p.dk + int64_t(seq) * p.dk_sb + int64_t(h) * p.dk_sh + int64_t(tok) * p.dk_st
                             : p.dv + int64_t(seq) * p.dv_sb + int64_t(h) * p.dv_sh + int64_t(tok) * p.dv_st;
#pragma unroll
  for (int j = 0; j < 2; ++j)
    reinterpret_cast<uint4*>(out)[g0 / 2 + j] =
        make_uint4(pack_bf16(o[2 * j].x, o[2 * j].y), pack_bf16(o[2 * j].z, o[2 * j].w),
                   pack_bf16(o[2 * j + 1].x, o[2 * j + 1].y), pack_bf16(o[2 * j + 1].z, o[2 * j + 1].w));
}

// ----------------------------------------------------------------------------------------
// Epilogue: dQ = bf16(scale * accumulator), 8 lanes per (token, head) row; dK and dV of cut units.
// ----------------------------------------------------------------------------------------
template <bool kRuns>
__global__ void __launch_bounds__(kAuxThreads) attn_bwd_epilogue_kernel(const BwdParams p) {
  __shared__ SchedRest rest_sm[kRuns ? kSchedRunSeqs + 1 : 1];
  __shared__ int first_sm;
  pdl_wait();  // the accumulator is complete when the main kernel is
  pdl_launch_dependents();
  if (int(blockIdx.x) >= p.row_blocks) return bwd_combine(p, blockIdx.x - uint32_t(p.row_blocks));
#if NB_BWD_L2_HINTS
  const uint64_t drop = l2_policy_evict_first();
#endif
  const int lane8 = threadIdx.x & 7;
  int64_t first = int64_t(blockIdx.x) * (kAuxThreads / 8), step = int64_t(p.row_blocks) * (kAuxThreads / 8),
          end = p.total_q * p.heads;
  int seq = 0;
  if constexpr (kRuns) {
    const int64_t n_rows = int64_t(p.rest[0]) * p.heads;
    first = aux_begin(n_rows, uint32_t(p.row_blocks), blockIdx.x);
    end = aux_begin(n_rows, uint32_t(p.row_blocks), blockIdx.x + 1), step = kAuxThreads / 8;
    if (first >= end) return;  // the whole block
    const int tok = int(first / p.heads);
    const SchedRest* rest = reinterpret_cast<const SchedRest*>(p.rest + 4);
#pragma unroll 1
    for (int i = threadIdx.x; i <= p.batch; i += kAuxThreads) {
      const SchedRest r = rest[i];
      rest_sm[i] = r;
      if (tok < r.end && (i == 0 || tok >= rest[i - 1].end)) first_sm = i;
    }
    __syncthreads();
    seq = first_sm;
  }
  for (int64_t row = first + (threadIdx.x >> 3); row < end; row += step) {
    const AuxRow w(p, row);
    const int64_t b = w.b;
    const int h = w.h;
    int64_t tok = w.tok, at = row;
    if constexpr (kRuns) {
      while (tok >= rest_sm[seq].end) ++seq;
      tok += rest_sm[seq].shift;
      at = tok * p.heads + h;
    }
    const float4* acc_row = reinterpret_cast<const float4*>(p.dq_accum + at * kHeadDim);
#if NB_BWD_L2_HINTS
    const float4 x = ld_global_v4_hint(acc_row + lane8 * 2, drop), y = ld_global_v4_hint(acc_row + lane8 * 2 + 1, drop);
#else
    const float4 x = acc_row[lane8 * 2], y = acc_row[lane8 * 2 + 1];
#endif
    uint4 v;
    v.x = pack_bf16(x.x * p.scale, x.y * p.scale);
    v.y = pack_bf16(x.z * p.scale, x.w * p.scale);
    v.z = pack_bf16(y.x * p.scale, y.y * p.scale);
    v.w = pack_bf16(y.z * p.scale, y.w * p.scale);
    *reinterpret_cast<uint4*>(p.dq + b * p.dq_sb + tok * p.dq_st + h * p.dq_sh + lane8 * 8) = v;
  }
}

// ----------------------------------------------------------------------------------------
// Main backward kernel
// ----------------------------------------------------------------------------------------
constexpr int kBwdThreads = 512;
constexpr int kBwdStages = 3;  // Q/dO ring
constexpr int kBwdOutStageBytes = 8192;  // dK/dV read-out: 2 KB per drain warp
// K (two buffers), V, 3x(Q, dO), dS (two 64-column halves), fp32 dQ staging (two 32-column halves),
// the dK/dV read-out staging, LSE/delta stages, the steps' control words and alignment slack
constexpr int kBwdSmemBytes =
    (3 + 2 * kBwdStages + 4) * kTileBytes + kBwdOutStageBytes + kBwdStages * 2 * kTile * 4 + 64 + 1024;
// Tensor memory: S^T 0 (P^T over it), dP^T 128 (dS^T over it), dV 256, dK 320, dQ 384, K 448, V 480
constexpr int kBwdTmemCols = 512;
// Register re-partitioning. The CTA launches with 512 threads x 128 registers (the whole register file); setmaxnreg
// only moves registers inside that allocation, so the budget must balance exactly or the growing warps would wait for
// ever. Every warp of an aligned warpgroup executes the same setmaxnreg instruction. The compute role needs 144. With
// 640 threads x 96 registers (TMA and LSE/delta rows in a warpgroup of their own; drain 64, loaders 48) ptxas spilled
// 40 to 72 bytes in the other roles' step loops (8 bytes are left in the form of whole units, none in the others): the
// change was worth 6 % of the whole backward of 2 x 12 x 820, 3 % of 1 x 12 x 3476 and 32 x 12 x 820, 2 % of 256
// sequences of 720..920 tokens. (Many sequences of two tiles, 300 of 200 tokens, gain nothing: the one warp's reads of
// list and rows follow each other.)
constexpr int kBwdLaunchRegs = 128;
constexpr int kBwdComputeRegs = 152;
constexpr int kBwdIssuerRegs = 104;  // issuers and loader
constexpr int kBwdDrainRegs = 104;
static_assert(256 * kBwdComputeRegs + 128 * (kBwdIssuerRegs + kBwdDrainRegs) == kBwdThreads * kBwdLaunchRegs,
              "register budget");

constexpr int kBwdWorkSlots = 4;

enum BwdBar : int {
  kBarKFull = 0,                            // [2] K is double-buffered across a CTA's work items
  kBarKFree = 2,                            // [2] the item's last dQ MMA has read K
  kBarVFull = 4,
  kBarVFree,                                // the item's V has been copied into tensor memory
  kBarQdoFull,                              // [kBwdStages] TMA issue + LSE/delta staged
  kBarQdoEmpty = kBarQdoFull + kBwdStages,  // [kBwdStages], 2 arrivals: both issuers
  // [2]: one per half of the step's query columns (= per compute warpgroup)
  kBarSFull = kBarQdoEmpty + kBwdStages,
  kBarDpFull = kBarSFull + 2,
  kBarPFull = kBarDpFull + 2,    // 4 arrivals (one per compute warp): P^T is in tensor memory
  kBarDstFull = kBarPFull + 2,   // 4: dS^T is in tensor memory
  kBarDsFull = kBarDstFull + 2,  // 4: dS is in shared memory
  kBarDsFree = kBarDsFull + 2,   // the step's dQ MMAs have read dS from shared memory
  kBarDqFull,
  kBarDqFree,   // 4 (dQ drain warps)
  kBarDvDone,   // the item's last dV MMA is complete
  kBarDkDone,
  kBarDvOut,    // 4: the drain warps have read the item's dV accumulator
  kBarDkOut,    // 4
  kBarWorkFull,                                  // [kBwdWorkSlots] the ring of published units
  kBarWorkEmpty = kBarWorkFull + kBwdWorkSlots,  // [kBwdWorkSlots], 4: drain warps
  kBarOwnFull = kBarWorkEmpty + kBwdWorkSlots,   // [4], only with runs: a drain warp's part of the CTA's own dQ tile
                                                 // has been read back
  kBwdNumBars = kBarOwnFull + 4
};

// One unit of a CTA's work: a 128-row K/V tile of one (sequence, head).
struct BwdWork {
  int n_q;  // query tiles to walk; 0: keys without queries (dK = dV = 0, not published); -1: no more work
  int kt, h, b, bcoord;
  int k_begin, lk, q_begin, lq;
};

// Key tiles of a run go one after the other through the same CTA, each in the order of query tiles that it has as a
// unit of its own (so dK and dV are the same either way). dQ of the first key tile is stored into the CTA's own tiles,
// that of the others added to them, and the last one's leaves as bf16 together with what is there. So the accumulator
// of a run is neither cleared nor read by a pass of its own, and 148 x own_tiles x 32 KB stay in the L2 from run to
// run.
enum BwdRun : int { kRunTile = 1, kRunFirst = 2, kRunLast = 4 };
// Most query tiles of a run: 148 CTAs' own tiles, Q and dO then take 148 x 10 x 64 KB = 97 of the L2's 126 MB. 64
// sequences of 1030..1150 tokens (nine tiles) x 12 heads take 814 us instead of 863, of 1160..1280 1017 instead of
// 1041; but with twelve tiles 64 of 1400..1536 take 1646 instead of 1409. (The tenth tile is allowed from five rounds of
// pairs on, see bwd_runs in nb_attn.cu.)
constexpr int kBwdRunTiles = 10;

// Query tile an item starts at. Concurrent CTAs work on the key tiles of one (sequence, head) and
// all add into the same dQ tiles, so they start at different ones: key tile kt at query tile kt,
// and where there are more key tiles than query tiles at a tile picked by a multiplicative hash
// (a multiply-high maps it into [0, n_q) without a division routine).
__device__ __forceinline__ int bwd_first_tile(int kt, int n_q) {
  return kt < n_q ? kt : int(__umulhi(uint32_t(kt) * 0x9E3779B9u, uint32_t(n_q)));
}

// The same where units may be cut between CTAs. The two forms are separate instantiations of the kernel:
// with the extra fields and the drain warps' second way out in one kernel, calls without cut units took
// 1.5 % (long sequences) to 7 % (short ones) longer.
struct BwdCutWork : BwdWork {
  int jt0, n_qt;  // first query tile of the walk, query tiles of the sequence
  int part;       // >= 0: the unit is cut; where this CTA's dV and dK go
};
// And where there may be runs.
struct BwdRunWork : BwdWork {
  int run;  // a key tile of a run: BwdRun bits; 0: a unit of its own
};
// The kernel's forms.
enum BwdMode : int { kBwdWhole, kBwdCut, kBwdRuns };
__device__ __forceinline__ int bwd_run(const BwdWork&) { return 0; }
__device__ __forceinline__ int bwd_run(const BwdRunWork& w) { return w.run; }
__device__ __forceinline__ int bwd_start(const BwdWork& w) { return bwd_first_tile(w.kt, w.n_q); }
__device__ __forceinline__ int bwd_start(const BwdCutWork& w) { return w.jt0; }
__device__ __forceinline__ int bwd_tiles(const BwdWork& w) { return w.n_q; }
__device__ __forceinline__ int bwd_tiles(const BwdCutWork& w) { return w.n_qt; }
__device__ __forceinline__ int bwd_part(const BwdWork&) { return -1; }
__device__ __forceinline__ int bwd_part(const BwdCutWork& w) { return w.part; }
template <int kMode>
using BwdWorkOf = std::conditional_t<kMode == kBwdCut, BwdCutWork,
                                     std::conditional_t<kMode == kBwdRuns, BwdRunWork, BwdWork>>;

// Unit g of the call; n_q = -1 past the last one. The loader fetches a CTA's units and publishes them to
// the other roles through a small ring. Dense units all cost the same: CTA c of G takes c, G + c, ...
// Packed units are taken from the list's counter, most expensive first. Where whole dense units would
// leave CTAs idle, CTA c takes an equal run of (unit, query tile) steps; g then counts the units that run
// touches, and at most two of them are cut: the one that run starts in and the one it ends in.
// kt = -1: all key tiles of the (sequence, head), a run.
template <int kMode>
__device__ __forceinline__ BwdWorkOf<kMode> bwd_work(const BwdParams& p, uint32_t g) {
  constexpr bool kCut = kMode == kBwdCut, kRuns = kMode == kBwdRuns;
  BwdWorkOf<kMode> w;
  w.n_q = -1, w.kt = 0, w.h = 0, w.b = 0, w.bcoord = 0, w.k_begin = 0, w.lk = 0, w.q_begin = 0, w.lq = 0;
  if constexpr (kRuns) w.run = 0;
  if constexpr (kCut) {
    w.jt0 = w.n_qt = 0, w.part = -1;
    const int s0 = int(bwd_split_start(p, blockIdx.x)), s1 = int(bwd_split_start(p, blockIdx.x + 1));
    const uint32_t u = p.div_n_qt.quot(uint32_t(s0)) + g;
    const int first = int(u) * p.n_qt;
    const int tile0 = g == 0 ? s0 - first : 0;
    if (first + tile0 >= s1) return w;
    const int tile1 = min(s1 - first, p.n_qt);
    if (tile0 > 0 || tile1 < p.n_qt) w.part = 2 * int(blockIdx.x) + (tile0 == 0);
    w.jt0 = tile0, w.n_q = tile1 - tile0, w.n_qt = p.n_qt;
    g = u;
  } else if (g >= uint32_t(p.n_work)) {
    return w;
  }
  if (kRuns || (!kCut && p.cu_q != nullptr)) {
    // One 32-byte read tells all about the item (the sequence index `batch` stands for the rows past
    // the last sequence: keys without queries). Unused entries sit at the end of the list.
    const uint32_t idx = p.div_heads.quot(g);
    const SchedItem item = sched_load(p.items, idx);
    if (item.seq < 0) return w;
    w.h = int(g - idx * uint32_t(p.heads));
    w.b = item.seq, w.kt = item.tile;
    w.k_begin = item.own_begin, w.lk = item.own_len;
    w.q_begin = item.other_begin, w.lq = item.other_len;
  } else {
    const uint32_t t = p.div_n_kt.quot(g);
    w.kt = int(g - t * uint32_t(p.n_kt));
    w.b = w.bcoord = int(p.div_heads.quot(t));
    w.h = int(t - uint32_t(w.b) * uint32_t(p.heads));
    w.lk = p.lk, w.lq = p.lq;
  }
  if constexpr (kCut) {
    if (w.part < 0) w.jt0 = bwd_first_tile(w.kt, w.n_qt);
  } else {
    w.n_q = (w.lq + kTile - 1) / kTile;
  }
  return w;
}

// Running position of a role in the CTA's stream of steps: step count, Q/dO stage and the phase of
// that stage's barriers. Steps run on through the boundaries between work items.
struct BwdStepPos {
  uint32_t s = 0, qs = 0, qph = 0;
  __device__ __forceinline__ void advance() {
    ++s;
    if (++qs == uint32_t(kBwdStages)) qs = 0, qph ^= 1u;
  }
};

// Control word of a step, staged with the step's LSE/delta rows (one per Q/dO stage). The compute
// warps and the MMA issuers learn everything about a step from it, so they never read the work
// list or leave their step loops: between two items of a persistent CTA they would otherwise run
// cold code behind a global-memory read (measured: 1500-3000 cycles per item boundary).
enum BwdCtrl : uint32_t {
  kCtrlFirst = 1u,  // first step of a work item
  kCtrlLast = 2u,   // last step of a work item
  kCtrlKb = 4u,     // which K buffer the item uses
  kCtrlStop = 8u,   // no step: the CTA's work has ended
  // bits 8 and up: live key rows of the item's tile (1..128)
};

// The compute warps' role: for every step of the CTA, P^T from S^T, then dS^T from dP^T.
// Not inlined on purpose: compiled by itself the step body keeps its instruction schedule (it needs
// 144 of the compute warps' 152 registers, and inlined into the kernel it came out 10-60 % slower
// whenever the code around it changed).
__device__ __noinline__ void bwd_compute_role(const uint32_t bar0, int* abort_flag, const uint32_t tmem_base,
                                              const float* sLse, const float* sDelta, const volatile uint32_t* sCtrl,
                                              const uint32_t ds_smem, const float scale_log2) {
  const int warp = threadIdx.x >> 5;
  const int w = warp >> 2;                       // warpgroup: query columns [64w, 64w+64)
  const int t = threadIdx.x & 31, quad = warp & 3;
  const uint32_t tm_lane = tmem_base + (uint32_t(quad * 32) << 16);
  // This warpgroup's score columns; its P^T (dS^T) takes the first half of the S^T (dP^T) columns it
  // has just read.
  const uint32_t tm_s = tm_lane + 64 * w, tm_dp = tm_lane + 128 + 64 * w;
  // A thread owns key rows row0 + {0, 8, 16, 24} of the tile and query columns 8i + col0 + {0, 1} of its
  // warpgroup's 64 (the register layout of the 16-lane tensor-memory loads below): it needs 16 values
  // of -lse and of -delta per step where a thread owning a whole row would need 64.
  const int row0 = quad * 32 + (t >> 2), col0 = 2 * (t & 3);
  const uint32_t lane0 = t == 0;
  const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2);
  auto bar = [&](int i) { return bar0 + 8u * uint32_t(i); };
  // stmatrix: this lane's row of the 8x8 block it addresses (blocks: column block 0 / 1 x row half).
  const uint32_t st_row = uint32_t(quad * 32 + ((t >> 3) & 1) * 8 + (t & 7)), st_chunk = uint32_t(t >> 4);
  const uint32_t st_base = ds_smem + w * kTileBytes + st_row * 128u, st_xor = st_row & 7u;
  BwdStepPos pos;
  for (;; pos.advance()) {
    const uint32_t s = pos.s, qs = pos.qs;
    const float2* lse2 = reinterpret_cast<const float2*>(sLse + qs * kTile + 64 * w + col0);   // -lse (log2)
    const float2* dl2 = reinterpret_cast<const float2*>(sDelta + qs * kTile + 64 * w + col0);  // -delta
    uint64_t pf[32];  // P^T values of this thread as packed fp32 pairs: [16 * lane half + 2 * block + row half]

    // ---- phase A: P^T = exp2(S^T * scale_log2 - lse) ----
    if (!mbar_wait2(bar(kBarQdoFull + qs), pos.qph, bar(kBarSFull + w), s & 1, abort_flag)) break;
    const uint32_t ctrl = sCtrl[qs];
    __syncwarp();
    tc_fence_after();
    bool dp_ok;
    {
      uint32_t ra[2][32];
      tmem_ld_16x256b_x8(tm_s, ra[0]);
      tmem_ld_16x256b_x8(tm_s + (16u << 16), ra[1]);
      uint64_t l[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 v = lse2[4 * i];
        l[i] = pack_f32x2(v.x, v.y);
      }
      tmem_wait_ld();
      // Look at the barrier needed after the exponentials now; the latency overlaps them.
      dp_ok = mbar_test_wait(bar(kBarDpFull + w), s & 1);
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int i = 0; i < 16; ++i) {  // pair i: column block i >> 1, row half i & 1
          const uint64_t x = fma_f32x2(
              pack_f32x2(__uint_as_float(ra[half][2 * i]), __uint_as_float(ra[half][2 * i + 1])), scale2, l[i >> 1]);
          // All on the MUFU unit: with a quarter of them evaluated as a polynomial on the FMA pipe the
          // kernel takes 5 % longer (issue slots and power, not the MUFU unit, are what is short).
          // Query columns past the end of the sequence have -lse = -inf and come out as exactly 0.
          float x0, x1;
          unpack_f32x2(x, x0, x1);
          pf[16 * half + i] = pack_f32x2(fast_exp2(x0), fast_exp2(x1));
        }
    }
    if (ctrl & kCtrlStop) {
      // The dQ issuer learns of the end here -- once it has seen the step before (a barrier must never
      // run two phases ahead of a waiter that tests by parity).
      if (s > 0) mbar_wait_inline(bar(kBarDsFree), (s - 1) & 1, abort_flag);
      __syncwarp();
      mbar_arrive_if(bar(kBarDsFull + w), lane0);
      break;
    }
    const int rows_live = int(ctrl >> 8);
    if (rows_live < kTile) {
      // Key rows past the end of the sequence must not contribute to dQ.
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (row0 + 16 * half + 8 * (i & 1) >= rows_live) pf[16 * half + i] = 0ull;
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t pk[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float a0, a1;
        unpack_f32x2(pf[16 * half + i], a0, a1);
        pk[i] = pack_bf16(a0, a1);
      }
      tmem_st_16x128b_x8(tm_s + (uint32_t(16 * half) << 16), pk);
    }
    tmem_wait_st();
    tc_fence_before();
    __syncwarp();
    mbar_arrive_if(bar(kBarPFull + w), lane0);

    // ---- phase B: dS^T = P^T o (dP^T - delta) -> tensor memory (for dK) and shared memory (for dQ) ----
    uint32_t ra[2][32];
    uint64_t nd[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 v = dl2[4 * i];
      nd[i] = pack_f32x2(v.x, v.y);
    }
    if (!dp_ok) mbar_wait_inline(bar(kBarDpFull + w), s & 1, abort_flag);
    __syncwarp();
    tc_fence_after();
    tmem_ld_16x256b_x8(tm_dp, ra[0]);
    tmem_ld_16x256b_x8(tm_dp + (16u << 16), ra[1]);
    tmem_wait_ld();
    const bool ds_ok = s == 0 || mbar_test_wait(bar(kBarDsFree), (s - 1) & 1);
    uint32_t ds[2][16];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint64_t dp2 = pack_f32x2(__uint_as_float(ra[half][2 * i]), __uint_as_float(ra[half][2 * i + 1]));
        float a0, a1;
        unpack_f32x2(mul_f32x2(pf[16 * half + i], add_f32x2(dp2, nd[i >> 1])), a0, a1);
        ds[half][i] = pack_bf16(a0, a1);
      }
      tmem_st_16x128b_x8(tm_dp + (uint32_t(16 * half) << 16), ds[half]);
    }
    tmem_wait_st();
    tc_fence_before();
    __syncwarp();
    mbar_arrive_if(bar(kBarDstFull + w), lane0);
    if (!ds_ok) mbar_wait_inline(bar(kBarDsFree), (s - 1) & 1, abort_flag);
    __syncwarp();  // lanes leave a wait one by one; the aligned instructions below need the whole warp
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
      for (int c = 0; c < 8; c += 2)  // two 16-byte chunks (column blocks c, c + 1) of 16 key rows
        stmatrix_x4(st_base + half * (16 * 128) + (((c + st_chunk) ^ st_xor) << 4), ds[half][2 * c], ds[half][2 * c + 1],
                    ds[half][2 * c + 2], ds[half][2 * c + 3]);
    fence_proxy_async_smem();
    __syncwarp();
    mbar_arrive_if(bar(kBarDsFull + w), lane0);
  }
}

template <int kMode>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                const __grid_constant__ CUtensorMap tmap_dq, const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[kBwdNumBars];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  constexpr bool kCut = kMode == kBwdCut, kRuns = kMode == kBwdRuns;
  __shared__ BwdWorkOf<kMode> work_ring[kBwdWorkSlots];

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  // delta, the cleared dQ accumulator and the work list come from the prologue kernel.
  pdl_wait();
  pdl_launch_dependents();

  uint8_t* smem_al = smem_raw + (((smem_u32(smem_raw) + 1023u) & ~1023u) - smem_u32(smem_raw));
  const uint32_t smem_base = smem_u32(smem_al);
  auto sK = [&](uint32_t kb) { return smem_base + kb * kTileBytes; };
  const uint32_t sV = smem_base + 2 * kTileBytes;
  auto sQ = [&](uint32_t s) { return smem_base + (3 + 2 * s) * kTileBytes; };
  auto sDO = [&](uint32_t s) { return smem_base + (4 + 2 * s) * kTileBytes; };
  constexpr int kDsTile0 = 3 + 2 * kBwdStages;
  const uint32_t sDS = smem_base + kDsTile0 * kTileBytes;  // 32 KB bf16: q columns 0..63 | 64..127
  uint8_t* sDQ_ptr = smem_al + (kDsTile0 + 2) * kTileBytes;  // 32 KB fp32: d columns 0..31 | 32..63
  uint8_t* sOut_ptr = smem_al + (kDsTile0 + 4) * kTileBytes;  // dK/dV read-out staging
  float* sLse = reinterpret_cast<float*>(sOut_ptr + kBwdOutStageBytes);  // [stages][128], log2 domain
  float* sDelta = sLse + kBwdStages * kTile;                             // [stages][128]
  uint32_t* sCtrl = reinterpret_cast<uint32_t*>(sDelta + kBwdStages * kTile);  // [stages], see BwdCtrl
  uint32_t* sCtrlQ = sCtrl + 4;  // [8], indexed by step & 7: the dQ issuer's copy (it does not hold the stage)

  const uint32_t bar0 = smem_u32(&bars[0]);
  auto bar = [&](int i) { return bar0 + 8u * uint32_t(i); };
  // In the form with runs a wait's loop is called instead of inlined, 5 KB less code: 3 % of 256 sequences of 720..920
  // tokens. The others, small enough, do not gain (2 x 12 x 820: 31.7 -> 32.6).
  auto wait = [&](uint32_t b, uint32_t parity) {
    return kRuns ? mbar_wait(b, parity, &abort_flag) : mbar_wait_inline(b, parity, &abort_flag);
  };

  if (tid == 9 * 32) {
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_do);
    abort_flag = 0;
    // Unrolled by request: by itself the compiler keeps a loop of 41 barriers, which one thread walks while all the others
    // wait for it. Whole backward, us, loop and unrolled: 1 x 2 x 33 10.9 and 9.9, 2 x 12 x 820 31.9 and 30.8.
#pragma unroll
    for (int i = 0; i < (kRuns ? int(kBwdNumBars) : int(kBarOwnFull)); ++i) {
      uint32_t count = 1;
      if (i >= kBarQdoFull && i < kBarQdoFull + kBwdStages) count = 2;  // TMA issue + LSE/delta staged
      if (i >= kBarQdoEmpty && i < kBarQdoEmpty + kBwdStages) count = 2;
      if (i >= kBarPFull && i < kBarDsFull + 2) count = 4;
      if (i == kBarDqFree || i == kBarDvOut || i == kBarDkOut) count = 4;
      if (i >= kBarWorkEmpty && i < kBarOwnFull) count = 4;
      mbar_init(bar(i), count);
    }
    fence_mbar_init();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(&tmem_base_slot), kBwdTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128;
  const uint32_t tm_dv = tmem_base + 256, tm_dk = tmem_base + 320, tm_dq = tmem_base + 384;
  const uint32_t tm_k = tmem_base + 448, tm_v = tmem_base + 480;

  constexpr uint32_t kIdescSH = make_idesc(128, 64, 0, 0);   // K-major x K-major, N = 64
  constexpr uint32_t kIdescKN = make_idesc(128, 64, 0, 1);   // A K-major / tensor memory, B MN-major
  constexpr uint32_t kIdescNN = make_idesc(128, 64, 1, 1);   // A MN-major, B MN-major
  const bool packed = kRuns || (!kCut && p.cu_q != nullptr);

  // The CTA's unit number `round`, read by a whole warp from the loader's ring.
  auto next_work = [&](uint32_t round) {
    const uint32_t slot = round % kBwdWorkSlots;
    BwdWorkOf<kMode> w;
    w.n_q = -1;
    if (wait(bar(kBarWorkFull + slot), (round / kBwdWorkSlots) & 1)) w = work_ring[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(kBarWorkEmpty + slot));
    return w;
  };

  if (warp >= 8 && warp < 12) setmaxnreg_dec<kBwdIssuerRegs>();
  if (warp == 9) {
    // ---------------- loader: units, TMA (lane 0), LSE/delta rows and the steps' control words ----------------
    // K of the next item goes into the other K buffer; V is reloaded as soon as it has been
    // copied into tensor memory; Q/dO tiles run through the ring without regard to item boundaries.
    // A step's LSE/delta rows are requested before the wait for a free stage, so that this latency does not
    // sit between a stage becoming free and becoming full again. They are staged negated: -lse in
    // the log2 domain and -delta. Rows past the end of the sequence get -lse = -inf, which makes
    // their P^T column 0.
    BwdStepPos pos;
    uint32_t ni = 0;  // items with queries so far
    auto next_unit = [&](uint32_t g) {
      if (!packed) return kCut ? g + 1 : g + gridDim.x;
      uint32_t token = 0;
      if (lane == 0) token = sched_next(p.items);
      return __shfl_sync(0xffffffffu, token, 0);
    };
    uint32_t g = packed ? next_unit(0) : kCut ? 0u : blockIdx.x;
    BwdWorkOf<kMode> wk;
    int kt_end = 0;  // of a run
    uint32_t round = 0;  // units published
#pragma unroll 1
    for (;;) {
      if (kt_end == 0) wk = bwd_work<kMode>(p, g);
      if constexpr (kRuns) {
        if (wk.kt < 0) kt_end = (wk.lk + kTile - 1) / kTile, wk.kt = 0;
        if (kt_end > 0) wk.run = kRunTile | (wk.kt == 0 ? kRunFirst : 0) | (wk.kt == kt_end - 1 ? kRunLast : 0);
      }
      const uint32_t slot = round % kBwdWorkSlots, kb = ni & 1u;
      const int krow = wk.k_begin + wk.kt * kTile;
      const int rows_live = min(wk.lk - wk.kt * kTile, kTile);
      if (!kCut && wk.n_q == 0) {
        // Keys without queries: dK = dV = 0, written here. Such units have no step, and the drain warps hold a unit until
        // the issuers have seen the next step: published, a few of them in a row would fill the ring and nothing would move.
        // (One warp writes what four did: one 512-byte store at a time, 63 sequences of 300 keys without queries x 12
        // heads take 48.8 us, four at a time 37.2; 56 of 64 sequences of 800 keys 158 and 136.)
        auto clear = [&](__nv_bfloat16* rows, int64_t st) {
#pragma unroll 4
          for (int c = lane; c < rows_live * 8; c += 32)
            *reinterpret_cast<uint4*>(rows + int64_t(c >> 3) * st + (c & 7) * 8) = make_uint4(0, 0, 0, 0);
        };
        clear(p.dv + (int64_t(wk.bcoord) * p.dv_sb + int64_t(wk.h) * p.dv_sh + krow * p.dv_st), p.dv_st);
        clear(p.dk + (int64_t(wk.bcoord) * p.dk_sb + int64_t(wk.h) * p.dk_sh + krow * p.dk_st), p.dk_st);
        g = next_unit(g);
        continue;
      }
      const int64_t stat_base =
          packed ? int64_t(wk.h) * p.total_q + wk.q_begin : (int64_t(wk.b) * p.heads + wk.h) * p.lq;
      int jt = bwd_start(wk);
      float l2[4], dl[4];  // (as they are: arithmetic on them here would wait for them before the TMA loads are issued)
      auto rows = [&] {
#pragma unroll
        for (int r4 = 0; r4 < 4; ++r4) {
          const int r = jt * kTile + r4 * 32 + lane;
          l2[r4] = INFINITY, dl[r4] = 0.f;
          if (r < wk.lq) l2[r4] = p.lse[stat_base + r], dl[r4] = p.delta[stat_base + r];
        }
      };
      // The first step's rows are requested before the waits for a slot, the K buffer and a stage, or on short sequences
      // their latency would come on top of the list's: 2100 sequences of 200 tokens x 2 heads 468 us without, 437 with;
      // 300 x 12 heads 412 and 382. (As runs, whose units are longer, these take 291 us without and 295 with.)
      if (!kRuns && wk.n_q > 0) rows();
      if (lane == 0) {
        if (round >= uint32_t(kBwdWorkSlots))
          wait(bar(kBarWorkEmpty + slot), ((round / kBwdWorkSlots) - 1) & 1);
        work_ring[slot] = wk;
        mbar_arrive(bar(kBarWorkFull + slot));
        if (wk.n_q > 0) {
          if (ni >= 2) wait(bar(kBarKFree + kb), ((ni >> 1) - 1) & 1);
          mbar_arrive_expect_tx(bar(kBarKFull + kb), kTileBytes);
          tma_load_4d(sK(kb), &tmap_k, bar(kBarKFull + kb), 0, krow, wk.h, wk.bcoord);
        }
      }
      ++round;
      if (wk.n_q < 0) break;
#pragma unroll 1
      for (int j = 0; j < wk.n_q; ++j) {
        if (kRuns || j > 0) rows();
        if (lane == 0) {
          if (pos.s >= uint32_t(kBwdStages)) wait(bar(kBarQdoEmpty + pos.qs), pos.qph ^ 1u);
          mbar_arrive_expect_tx(bar(kBarQdoFull + pos.qs), 2 * kTileBytes);
          tma_load_4d(sQ(pos.qs), &tmap_q, bar(kBarQdoFull + pos.qs), 0, wk.q_begin + jt * kTile, wk.h, wk.bcoord);
          tma_load_4d(sDO(pos.qs), &tmap_do, bar(kBarQdoFull + pos.qs), 0, wk.q_begin + jt * kTile, wk.h, wk.bcoord);
          const uint32_t ctrl = (j == 0 ? kCtrlFirst : 0u) | (j == wk.n_q - 1 ? kCtrlLast : 0u) | (kb ? kCtrlKb : 0u) |
                                (uint32_t(rows_live) << 8);
          sCtrl[pos.qs] = ctrl;
          sCtrlQ[pos.s & 7u] = ctrl;
        }
        __syncwarp();
#pragma unroll
        for (int r4 = 0; r4 < 4; ++r4) {
          sLse[pos.qs * kTile + r4 * 32 + lane] = l2[r4] * -1.4426950408889634f;
          sDelta[pos.qs * kTile + r4 * 32 + lane] = -dl[r4];
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar(kBarQdoFull + pos.qs));
          if (j == 0) {
            if (ni >= 1) wait(bar(kBarVFree), (ni - 1) & 1);
            mbar_arrive_expect_tx(bar(kBarVFull), kTileBytes);
            tma_load_4d(sV, &tmap_v, bar(kBarVFull), 0, krow, wk.h, wk.bcoord);
          }
        }
        pos.advance();
        jt = jt + 1 == bwd_tiles(wk) ? 0 : jt + 1;
      }
      ++ni;
      if constexpr (kRuns) {
        if (++wk.kt < kt_end) continue;
        kt_end = 0;
      }
      // The next unit is taken as late as can be: this warp is about three steps ahead of the MMAs, which covers the
      // counter's and the list's latency, and a unit taken earlier would wait behind a long one while other CTAs run
      // dry. (Taken before the wait for the last step's stage: 300 sequences of 200 tokens lose 2 %.)
      g = next_unit(g);
    }
    // One more stage carries the stop mark (no data).
    if (lane == 0) {
      if (pos.s >= uint32_t(kBwdStages)) wait(bar(kBarQdoEmpty + pos.qs), pos.qph ^ 1u);
      sCtrl[pos.qs] = kCtrlStop;
      sCtrlQ[pos.s & 7u] = kCtrlStop;
      mbar_arrive(bar(kBarQdoFull + pos.qs));
      mbar_arrive(bar(kBarQdoFull + pos.qs));
    }
  } else if (warp >= 12) {
    // ---------------- drain warps: dQ tiles every step, dV and dK once per item ----------------
    // Warp 12+q owns tensor-memory lane quadrant q. dQ: it stages its 32 rows (two 32-column
    // halves, 128-byte swizzled rows) in shared memory and one lane issues the TMA add-reductions,
    // so only warp-level synchronisation is needed and L2 receives whole 128-byte lines. Rows past
    // the end of the sequence are staged as exact zeros, so adding them is harmless. dV / dK: when
    // the item's last MMA into the accumulator is complete every lane pulls its row into registers
    // as bf16 and the warp stores the rows through a 2 KB scratch area; the issuers start the next
    // item's first dV / dK MMA as soon as the accumulator has been read. dV is complete half a step
    // before the item's last dQ tile, so it is taken out before that tile is drained; dK follows the
    // tile. (With both after it, every item's second step waited ~2900 cycles for the next dV / dK
    // MMA.)
    setmaxnreg_dec<kBwdDrainRegs>();
    const int quad = warp & 3;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    uint8_t* stage = sDQ_ptr + quad * 4096;
    uint8_t* ostage = sOut_ptr + quad * (kBwdOutStageBytes / 4);
    uint32_t s = 0, ni = 0, own_phase = 0;
#if NB_BWD_L2_HINTS
    const uint64_t keep = l2_policy_evict_last();
#endif
#pragma unroll 1
    for (uint32_t round = 0;; ++round) {
      const BwdWorkOf<kMode> wk = next_work(round);
      const int n_q = wk.n_q;
      if (n_q < 0) break;
      const int h = wk.h;
      const int rows_live = wk.lk - wk.kt * kTile - quad * 32;  // this warp's rows below that exist
      const int out_row = wk.k_begin + wk.kt * kTile + quad * 32, bcoord = wk.bcoord;
      auto dv_rows = [&] { return p.dv + (int64_t(bcoord) * p.dv_sb + int64_t(h) * p.dv_sh + out_row * p.dv_st); };
      auto dk_rows = [&] { return p.dk + (int64_t(bcoord) * p.dk_sb + int64_t(h) * p.dk_sh + out_row * p.dk_st); };
      const int n_qt = bwd_tiles(wk), part = bwd_part(wk);
      int row = (packed ? 0 : wk.b * p.lq) + wk.q_begin + quad * 32 + bwd_start(wk) * kTile;
      const int row_end = (packed ? 0 : wk.b * p.lq) + wk.q_begin + quad * 32 + n_qt * kTile;
      // A run: this warp's part of the CTA's own dQ tiles, and reading one of them back into the staging rows.
      const int run = bwd_run(wk);
      float* const own0 = p.own + (int64_t(blockIdx.x) * p.own_tiles * 4 + quad) * 2048;
      int jt = kRuns && run ? bwd_start(wk) : 0;
      // Key tile kt starts one query tile behind the key tile before it, so a query tile's turns are n_q - 1
      // steps apart, or further; where there are more key than query tiles they may be neighbours.
      const bool far_apart = n_q > 2 && wk.kt < n_q;
      const bool read_back = kRuns && (run & (kRunFirst | kRunLast)) == kRunLast;
      // Waits until what was done to the own tile that is next, n_q - 1 steps ago or earlier, is complete.
      auto own_order = [&] {
        if (!far_apart) bulk_wait_group<0>();
        else if (n_q < 5) bulk_wait_group<1>();
        else if (n_q < 7) bulk_wait_group<3>();
        else bulk_wait_group<5>();
      };
      auto own_load = [&] {
        const float* own = own0 + jt * 8192;
        mbar_arrive_expect_tx(bar(kBarOwnFull + quad), 8192);
        bulk_load(smem_u32(stage), own, 4096, bar(kBarOwnFull + quad));
        bulk_load(smem_u32(stage + kTileBytes), own + 1024, 4096, bar(kBarOwnFull + quad));
      };
      if (read_back && lane == 0) {
        // (The last addition may still read the staging rows.)
        bulk_wait_group_read0();
        own_order();
        own_load();
      }
      // Events of an item, in order: the dQ tiles of steps 0 .. n_q-2, dV, the last dQ tile, dK.
#pragma unroll 1
      for (int e = 0; e < n_q + 2; ++e) {
        const bool is_out = e == n_q - 1 || e == n_q + 1, is_dk = e > n_q;
        const bool is_dq = kRuns && !is_out;
        if (is_out || (is_dq && (run & kRunLast))) {
          wait(bar(is_dq ? kBarDqFull : is_dk ? kBarDkDone : kBarDvDone), (is_dq ? s : ni) & 1);
          tc_fence_after();
          const uint32_t tm_acc = (is_dq ? tm_dq : is_dk ? tm_dk : tm_dv) + lane_off;
          const float out_scale = is_dk || is_dq ? p.scale : 1.f;
          const bool add = is_dq && read_back;
          if (add) {
            wait(bar(kBarOwnFull + quad), own_phase);
            own_phase ^= 1u;
          }
          // The whole 64-column row of this lane becomes 32 packed registers (four 16-column loads)
          // and the accumulator is handed back at once. The rows then go out 32 columns at a time
          // through a 2 KB scratch area, four lanes per 64-byte half row (a row per lane straight
          // from the registers was measured slower: 32 separate lines per store instruction).
          if (kCut && part >= 0) {
            // A cut unit: the fp32 rows go to the workspace (the layout bwd_combine reads).
            float4* dst = reinterpret_cast<float4*>(p.parts + int64_t(part) * kBwdPartFloats) +
                          (is_dk ? 16 * kTile : 0) + quad * 32 + lane;
#pragma unroll 1
            for (int q4 = 0; q4 < 4; ++q4) {
              uint32_t r[16];
              tmem_ld16(tm_acc + 16 * q4, r);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 4; ++i)
                dst[(4 * q4 + i) * kTile] =
                    make_float4(__uint_as_float(r[4 * i]) * out_scale, __uint_as_float(r[4 * i + 1]) * out_scale,
                                __uint_as_float(r[4 * i + 2]) * out_scale, __uint_as_float(r[4 * i + 3]) * out_scale);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(is_dk ? kBarDkOut : kBarDvOut));
            continue;
          }
          uint32_t pk[32];
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint32_t r[16];
            tmem_ld16(tm_acc + 16 * q4, r);
            tmem_wait_ld();
            if (kRuns && add) {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const float4 a = *reinterpret_cast<const float4*>(stage + (q4 >> 1) * kTileBytes +
                                                                  swz128(lane, (q4 & 1) * 4 + c));
                r[4 * c] = __float_as_uint(__uint_as_float(r[4 * c]) + a.x);
                r[4 * c + 1] = __float_as_uint(__uint_as_float(r[4 * c + 1]) + a.y);
                r[4 * c + 2] = __float_as_uint(__uint_as_float(r[4 * c + 2]) + a.z);
                r[4 * c + 3] = __float_as_uint(__uint_as_float(r[4 * c + 3]) + a.w);
              }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
              pk[8 * q4 + i] =
                  pack_bf16(__uint_as_float(r[2 * i]) * out_scale, __uint_as_float(r[2 * i + 1]) * out_scale);
          }
          tc_fence_before();
          if (kRuns && add) fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(is_dq ? kBarDqFree : is_dk ? kBarDkOut : kBarDvOut));  // the accumulator is free
          __nv_bfloat16* out = is_dk ? dk_rows() : dv_rows();
          int64_t out_st = is_dk ? p.dk_st : p.dv_st;
          int out_live = rows_live;
          if (kRuns && is_dq) {
            out = p.dq + (int64_t(bcoord) * p.dq_sb + int64_t(h) * p.dq_sh +
                          (wk.q_begin + jt * kTile + quad * 32) * p.dq_st);
            out_st = p.dq_st;
            out_live = wk.lq - jt * kTile - quad * 32;
            ++s;
            jt = jt + 1 == n_q ? 0 : jt + 1;
            if (add && e < n_q && lane == 0) {  // the next one (the last is event n_q)
              bulk_wait_group<0>();
              own_load();
            }
          }
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            // Row `lane` of the scratch holds 32 bf16 = four 16-byte chunks, XOR-ed with the row
            // pair's index so that neither the writes (a row per lane) nor the reads (four lanes per
            // row) collide on banks.
#pragma unroll
            for (int c = 0; c < 4; ++c)
              *reinterpret_cast<uint4*>(ostage + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = make_uint4(
                  pk[16 * half + 4 * c], pk[16 * half + 4 * c + 1], pk[16 * half + 4 * c + 2], pk[16 * half + 4 * c + 3]);
            __syncwarp();
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              const int rloc = it * 8 + (lane >> 2), c = lane & 3;
              const uint4 v = *reinterpret_cast<const uint4*>(ostage + rloc * 64 + ((c ^ ((rloc >> 1) & 3)) << 4));
              if (rloc < out_live) *reinterpret_cast<uint4*>(out + int64_t(rloc) * out_st + half * 32 + c * 8) = v;
            }
            __syncwarp();
          }
          continue;
        }
        wait(bar(kBarDqFull), s & 1);
        tc_fence_after();
        if (lane == 0) {
          bulk_wait_group_read0();  // the previous reductions have read the staging rows
          // Additions to an own tile have to find the ones before them done.
          if (kRuns && run) own_order();
        }
        __syncwarp();
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t r[32];
          tmem_ld32(tm_dq + lane_off + 32 * half, r);
          tmem_wait_ld();
          if (half == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kBarDqFree));  // the dQ tile is out of tensor memory
          }
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(stage + half * kTileBytes + swz128(lane, c)) =
                make_uint4(r[4 * c], r[4 * c + 1], r[4 * c + 2], r[4 * c + 3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (kRuns && run) {
          if (lane == 0) {
            float* own = own0 + jt * 8192;
            if (run & kRunFirst) {
              bulk_store(own, smem_u32(stage), 4096);
              bulk_store(own + 1024, smem_u32(stage + kTileBytes), 4096);
            } else {
              bulk_reduce_add(own, smem_u32(stage), 4096);
              bulk_reduce_add(own + 1024, smem_u32(stage + kTileBytes), 4096);
            }
            bulk_commit_group();
          }
          jt = jt + 1 == n_q ? 0 : jt + 1;
        } else if (lane == 0) {
#if NB_BWD_L2_HINTS
          tma_reduce_add_3d_hint(&tmap_dq, smem_u32(stage), 0, row, h, keep);
          tma_reduce_add_3d_hint(&tmap_dq, smem_u32(stage + kTileBytes), 32, row, h, keep);
#else
          tma_reduce_add_3d(&tmap_dq, smem_u32(stage), 0, row, h);
          tma_reduce_add_3d(&tmap_dq, smem_u32(stage + kTileBytes), 32, row, h);
#endif
          bulk_commit_group();
        }
        ++s;
        row += kTile;
        if (row == row_end) row -= n_qt * kTile;
      }
      ++ni;
    }
    if (lane == 0) bulk_wait_group_read0();  // the staging rows must outlive the TMA engine's reads
  } else if (warp >= 8) {
    // Three issuers, one elected thread each, that walk the CTA's steps by their control words. The two
    // halves of a step's query columns (one per compute warpgroup) run half a step apart, so one
    // warpgroup's exponentials overlap the other's dS arithmetic and the MMAs of both. P^T takes the
    // columns of the S^T it came from and dS^T those of its dP^T, so the next S^T (dP^T) may only be
    // written after the dV (dK) MMAs have read them: each pair is issued by one thread in that order, and
    // MMAs of one thread execute in order.
    if (elect_one()) {
      BwdStepPos pos;
      uint32_t ni = 0;  // items started
      volatile uint32_t* ctrl_ring = sCtrl;
      uint32_t ctrl = 0;
      if (warp == 8) {
        // ---------------- S^T = K Q^T of step s+1 after dV += P^T dO of step s, half by half ----------------
        // K goes into tensor memory once per item, so S^T takes its A operand from there and the
        // shared-memory port carries only Q.
        auto copy_k = [&](uint32_t c) {
          const uint32_t kb = (c & kCtrlKb) ? 1u : 0u;
          const uint64_t kd = make_sdesc(sK(kb), 16, 1024);
          wait(bar(kBarKFull + kb), (ni >> 1) & 1);
          ++ni;
#pragma unroll 1
          for (int k = 0; k < 4; ++k) tmem_copy_128x256b(tm_k + 8 * k, kd + 2 * k);
        };
        auto issue_s = [&](uint32_t stage, int h) {
          const uint64_t qd = make_sdesc(sQ(stage) + h * (kTileBytes / 2), 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_ts(tm_s + 64 * h, tm_k + 8 * k, qd + 2 * k, kIdescSH, k > 0);
          tc_commit(bar(kBarSFull + h));
        };
        wait(bar(kBarQdoFull), 0);
        ctrl = ctrl_ring[0];
        if (!(ctrl & kCtrlStop)) {
          copy_k(ctrl);
          issue_s(0, 0);
        } else {
          mbar_arrive(bar(kBarSFull));
          mbar_arrive(bar(kBarSFull + 1));
        }
#pragma unroll 1
        while (!(ctrl & kCtrlStop)) {
          const bool first = (ctrl & kCtrlFirst) != 0;
          BwdStepPos next = pos;
          next.advance();
          // The previous item's dV has to be out of tensor memory before this one's first MMA.
          if (first && ni > 1) wait(bar(kBarDvOut), (ni - 2) & 1);
          const uint64_t gd_mn = make_sdesc(sDO(pos.qs), 1024, 1024);
          uint32_t next_ctrl = 0;
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            if (!wait(bar(kBarPFull + h), pos.s & 1)) next_ctrl = kCtrlStop;
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < 4; ++k)  // A: P^T of query columns [64h + 16k, +16)
              mma_ts(tm_dv, tm_s + 64 * h + 8 * k, gd_mn + 512 * h + 128 * k, kIdescKN, !first || (h + k > 0));
            if (h == 0) {
              if (pos.s == 0) issue_s(0, 1);  // the second half starts later: see above
              wait(bar(kBarQdoFull + next.qs), next.qph);
              next_ctrl |= ctrl_ring[next.qs];
              if ((next_ctrl & (kCtrlFirst | kCtrlStop)) == kCtrlFirst) {
                // The MMAs that read the previous item's K must be complete.
                wait(bar(kBarSFull + 1), pos.s & 1);
                tc_fence_after();
                copy_k(next_ctrl);
              }
            } else {
              tc_commit(bar(kBarQdoEmpty + pos.qs));
              if (ctrl & kCtrlLast) tc_commit(bar(kBarDvDone));
            }
            // The compute warps wait for the stage and for S^T together, so the stop mark needs an
            // arrival on the S^T barrier (they have consumed the phase before: P^T was full).
            if (next_ctrl & kCtrlStop) mbar_arrive(bar(kBarSFull + h));
            else issue_s(next.qs, h);
          }
          ctrl = next_ctrl;
          pos = next;
        }
      } else if (warp == 10) {
        // ---------------- dP^T = V dO^T of step s+1 after dK += dS^T Q of step s, half by half ----------------
        const uint64_t vd = make_sdesc(sV, 16, 1024);
        auto copy_v = [&] {
          wait(bar(kBarVFull), ni & 1);
          ++ni;
#pragma unroll 1
          for (int k = 0; k < 4; ++k) tmem_copy_128x256b(tm_v + 8 * k, vd + 2 * k);
          tc_commit(bar(kBarVFree));
        };
        auto issue_dp = [&](uint32_t stage, int h) {
          const uint64_t gd = make_sdesc(sDO(stage) + h * (kTileBytes / 2), 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_ts(tm_dp + 64 * h, tm_v + 8 * k, gd + 2 * k, kIdescSH, k > 0);
          tc_commit(bar(kBarDpFull + h));
        };
        wait(bar(kBarQdoFull), 0);
        ctrl = ctrl_ring[0];
        if (!(ctrl & kCtrlStop)) {
          copy_v();
          issue_dp(0, 0);
          issue_dp(0, 1);
        }
#pragma unroll 1
        while (!(ctrl & kCtrlStop)) {
          const bool first = (ctrl & kCtrlFirst) != 0;
          BwdStepPos next = pos;
          next.advance();
          if (first && ni > 1) wait(bar(kBarDkOut), (ni - 2) & 1);
          const uint64_t qd_mn = make_sdesc(sQ(pos.qs), 1024, 1024);
          uint32_t next_ctrl = 0;
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            if (!wait(bar(kBarDstFull + h), pos.s & 1)) next_ctrl = kCtrlStop;
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < 4; ++k)  // A: dS^T of query columns [64h + 16k, +16)
              mma_ts(tm_dk, tm_dp + 64 * h + 8 * k, qd_mn + 512 * h + 128 * k, kIdescKN, !first || (h + k > 0));
            if (h == 0) {
              wait(bar(kBarQdoFull + next.qs), next.qph);
              next_ctrl |= ctrl_ring[next.qs];
              if ((next_ctrl & (kCtrlFirst | kCtrlStop)) == kCtrlFirst) {
                // The MMAs that read the previous item's V must be complete.
                wait(bar(kBarDpFull + 1), pos.s & 1);
                tc_fence_after();
                copy_v();
              }
            } else {
              tc_commit(bar(kBarQdoEmpty + pos.qs));
              if (ctrl & kCtrlLast) tc_commit(bar(kBarDkDone));
            }
            if (!(next_ctrl & kCtrlStop)) issue_dp(next.qs, h);
          }
          ctrl = next_ctrl;
          pos = next;
        }
      } else {
        // ---------------- dQ = dS K ----------------
        // A: MN-major view of the dS bytes in shared memory; one K step = 16 key rows.
        const uint64_t ds_mn = make_sdesc(sDS, kTileBytes, 1024);
        uint64_t kd_mn = 0;
        uint32_t kb = 0;
#pragma unroll 1
        for (;; pos.advance()) {
          // This issuer does not hold the stage (the path from a stage becoming free to becoming full
          // again is the tightest in the pipeline), so it reads a copy of the control word from a ring of
          // eight: the word of step s+8 is written after step s+5 has freed its stage, hence after the
          // dQ MMAs of step s+3. The compute warps have seen the word before they arrive here.
          if (!wait(bar(kBarDsFull), pos.s & 1)) break;
          ctrl = (reinterpret_cast<volatile uint32_t*>(sCtrlQ))[pos.s & 7u];
          if (ctrl & kCtrlStop) break;
          if (ctrl & kCtrlFirst) {
            kb = (ctrl & kCtrlKb) ? 1u : 0u;
            kd_mn = make_sdesc(sK(kb), 1024, 1024);
            wait(bar(kBarKFull + kb), (ni >> 1) & 1);
          }
          if (pos.s > 0) wait(bar(kBarDqFree), (pos.s - 1) & 1);
          wait(bar(kBarDsFull + 1), pos.s & 1);
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 8; ++k) mma_ss(tm_dq, ds_mn + 128 * k, kd_mn + 128 * k, kIdescNN, k > 0);
          tc_commit(bar(kBarDqFull));
          tc_commit(bar(kBarDsFree));
          if (ctrl & kCtrlLast) {
            tc_commit(bar(kBarKFree + kb));
            ++ni;
          }
        }
      }
    }
  } else {
    // ---------------- compute warpgroups: w = 0 / 1 owns query columns [64w, 64w+64) ----------------
    setmaxnreg_inc<kBwdComputeRegs>();
    bwd_compute_role(bar0, &abort_flag, tmem_base, sLse, sDelta, sCtrl, sDS, p.scale_log2);
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0) report_abort(&abort_flag, p.status);
  if (warp == 8) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kBwdTmemCols);
  }
}

}  // namespace nb
