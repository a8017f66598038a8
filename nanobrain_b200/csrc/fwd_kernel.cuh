// Forward attention kernel: O = softmax(Q K^T * scale) V, bf16 in / bf16 out, fp32 softmax
// statistics and accumulation, head_dim 64, non-causal.
//
// A work unit is one 128-row query tile of one (sequence, head), walked over the sequence's keys in
// 128-row tiles, each in two halves of 64 key columns. CTAs are persistent, two per SM (256
// tensor-memory columns and 99 KB of shared memory each, so one CTA's softmax overlaps the other's MMAs);
// the producer warp fetches the units and runs on into the next one -- its descriptor, Q, first K / V
// tiles and first scores are there before the softmax warps have stored the unit before it. Packed units
// come from the scheduler's list (sched_kernel.cuh), dense ones by position, and where whole dense units
// would leave SMs idle each CTA takes an equal share of all key tiles (fwd_unit). A ragged last key tile
// is trimmed: its MMAs cover the live columns rounded up to 16, and a second half without live columns
// is left out. Warp roles (192 threads):
//
//   warps 0-3 : softmax warpgroup. Thread r owns row r of the tile (tensor-memory lane r). Per half it
//               pulls its 64 fp32 scores into registers and writes P = exp2(S*scale_log2 - m) as bf16
//               over the first half of the columns they came from. The offset m is the row max of the
//               first tile; later halves compute no max at all: fp32 and bf16 carry exponents up
//               to 2^127, so scores may rise 60 (in log2 units) above the first ones before anything
//               has to be rescaled. Only if a row's sum ends above 2^60 (or Inf / NaN), or above 2^14
//               with a P V that is not finite, or the polynomial met an argument beyond its range,
//               does the CTA list the unit and walk it a second time, with the running max of every
//               half. At the end of a unit the warps normalise and store O and the log-sum-exp. O is
//               divided (where there is more than one tile) by the sum of
//               P as the product sees it, rounded to bf16, which the tensor core forms from 16 columns
//               of ones behind V: where few keys dominate a row, the rounding of their P then cancels.
//               Scores of standard deviation 9 and 16 nats, relative error of O against 64 bits: 2.2e-3
//               and 2.0e-3 divided by the sum before rounding, 1.7e-3 and 1.5e-3 this way (with the running
//               max as the offset 1.9e-3 and 1.7e-3). The columns cost 1 % (dense 32 x 8 x 4096, sustained:
//               1428 -> 1442 us), the max of the whole first tile instead of its first half 0.3 %.
//   warp 4    : one elected thread issues every tcgen05.mma. Q is copied into tensor memory once
//               per unit (tcgen05.cp), so S = Q K^T takes its A operand from there, as O += P V does. After P of
//               half h of tile i is complete it issues P V of that half and then S of half h of tile
//               i+1 over the same columns (MMAs of one thread execute in order), which run while the
//               softmax warps work on the other half: the warps never wait for a score tile in steady
//               state although P has no tensor memory of its own.
//   warp 5    : one elected thread fetches units and drives TMA: Q once per unit, K and V tiles through
//               two-stage rings (SWIZZLE_128B; every CTA loads its own tiles).
//
// What bounds it: the instructions of the softmax warps and the board's power limit (at 1 kW the SMs
// run at 1.65-1.8 GHz of 1.965). Measured on dense 32 x 8 x 4096, repeated for 0.3 s: with a score tile
// and P of 128 columns each, Q from shared memory and P handed over once per tile 1550 us (1540 clocks
// per 128 x 128 tile and SM); this form 1402 us before `top`, the columns of ones and the first tile's max,
// 1448 with them (exact scores and NaN cost 1.5 %, precision 1.4 %). Against the form before it, in GPU time between
// unrelated kernels: packed 32 x U[720,920] x 12 heads 138 -> 113 us, 500 sequences of 1..300 tokens 258 -> 165,
// 1 x 12 x 3476 77 -> 58, 2 x 12 x 820 15.7 -> 15.4. Calls of at most 300 tokens lose 1 to 2 us (1 x 12 x 128: 4.5 -> 6.4,
// 1 x 12 x 300: 7.2 -> 8.1): a block that has one unit runs through twice the code once, cold. Loads issued before the
// tensor memory is there (6.3) and a rolled epilogue (6.3, 500 short sequences 165 -> 169) were not worth their code.
//
// Tensor memory (256 columns): S / P [0,128) O [128,192) row sums of P [192,208) Q [208,240).
#pragma once

#include <type_traits>

#include "ptx.cuh"
#include "sched_kernel.cuh"

namespace nb {

// Division of a number below 2^31 by a fixed divisor as a multiply-high and a shift (the divisor's
// magic numbers come from the host). The work-index split is inlined in several warp roles, and
// an integer division routine in each of them is code the instruction cache has no room for.
struct FastDiv {
  uint32_t mul, shr, div;
  __device__ __forceinline__ uint32_t quot(uint32_t n) const { return div == 1u ? n : __umulhi(n, mul) >> shr; }
};
inline FastDiv make_fast_div(uint32_t d) {
  FastDiv f;
  f.div = d, f.mul = 0, f.shr = 0;
  if (d > 1) {
    uint32_t lg = 0;
    while ((1ull << lg) < d) ++lg;  // ceil(log2 d)
    const uint64_t p = 31 + lg;
    f.mul = uint32_t(((1ull << p) + d - 1) / d);
    f.shr = uint32_t(p - 32);
  }
  return f;
}

struct FwdParams {
  __nv_bfloat16* o;
  int64_t o_sb, o_st, o_sh;  // element strides of O: batch, token, head
  float* lse;
  const int32_t* cu_q;  // NULL => dense
  const int32_t* cu_k;
  const SchedItem* items;  // packed mode: the scheduler's work list; a unit is an entry and a head
  int32_t batch, heads;
  int32_t lq, lk;  // dense lengths (max_seqlen in varlen mode)
  int64_t total_q, total_k;
  float scale_log2;  // scale * log2(e)
  int32_t* status;
  // Work units: query tiles x heads x sequences (dense), or list entries x heads (packed).
  int32_t n_units;
  int32_t n_qt, n_kt;  // dense: query and key tiles per (sequence, head)
  FastDiv div_heads, div_n_qt;
  // Dense mode with few units: a CTA takes an equal run of (unit, key tile) steps, units are cut between
  // CTAs (see fwd_unit) and put together by attn_fwd_combine_kernel. NULL: whole units.
  float* parts;  // [2 * CTAs][kFwdPartFloats]
  uint32_t split_base, split_extra;  // CTA c starts at step c * base + min(c, extra)
  FastDiv div_n_kt;
};

__device__ __forceinline__ uint32_t fwd_split_start(const FwdParams& p, uint32_t c) {
  return c * p.split_base + min(c, p.split_extra);
}

constexpr int kTile = 128;  // rows per Q tile and per K/V tile
constexpr int kHeadDim = 64;
constexpr int kTileBytes = kTile * kHeadDim * 2;  // 16 KB

constexpr int kFwdThreads = 192;
constexpr int kFwdQRows = kTile;  // query rows per CTA
constexpr int kFwdStages = 2;
constexpr int kFwdOnesBytes = 2048;
// Q, K and V rings, O staging, the block of ones, alignment slack
constexpr int kFwdSmemBytes = (2 + 2 * kFwdStages) * kTileBytes + kFwdOnesBytes + 1024;
constexpr int kFwdRedoSlots = 16;
constexpr int kFwdPartFloats = kTile * (kHeadDim + 3);  // a cut unit's O (not normalised), offsets and both sums
constexpr int kFwdTmemCols = 256;
constexpr float kRescaleThreshold = 8.f;                       // log2 units
constexpr float kFirstPassSumLimit = 1152921504606846976.f;  // 2^60
constexpr float kNoOffset = -1.2676506002282294e30f;  // -2^100
constexpr float kPlainSumLimit = 16384.f;
constexpr float kPolyLimit = 126.f;                          // log2 units

enum FwdBar : int {
  kFwdQFull = 0,                          // [2]: Q and the unit's descriptor (by descriptor slot)
  kFwdQEmpty = 2,                         // Q has been copied into tensor memory
  kFwdKFull,                              // [stages]
  kFwdKEmpty = kFwdKFull + kFwdStages,    // [stages]
  kFwdVFull = kFwdKEmpty + kFwdStages,    // [stages]
  kFwdVEmpty = kFwdVFull + kFwdStages,    // [stages]
  kFwdSFull = kFwdVEmpty + kFwdStages,    // [2]: per half of a key tile
  kFwdPFull = kFwdSFull + 2,              // [2], 4 arrivals (one per softmax warp)
  // [2]: P V of the half is complete. One barrier per half: the softmax warps hand over two halves
  // before they look, and a barrier must never be two phases behind a waiter that tests by parity.
  kFwdPvDone = kFwdPFull + 2,
  kFwdOFree = kFwdPvDone + 2,             // 4: the unit's O is out of tensor memory
  kFwdUnitDone,                           // [2], 4: the unit in this descriptor slot is finished
  kFwdNumBars = kFwdUnitDone + 2
};

// A CTA's next unit as the producer publishes it to the other roles (two slots in shared memory).
struct FwdUnit {
  int lk;        // key rows to walk; 0: queries without keys; -1: no more work
  int safe;      // walk with the running max of every half (second time)
  uint32_t token;  // see fwd_unit
  int q_row0, q_begin, lq, h, b;
  int part;      // >= 0: the unit is cut between CTAs; where this CTA's part goes
  int k_begin, bcoord;
};

// The unit a token stands for (lk = -1: none). Packed mode: token = unit, taken from the list's counter,
// most expensive first. Dense mode, whole units: token = unit, CTA c of G takes c, G + c, ... Where whole
// units would leave CTAs idle, CTA c takes an equal run of (unit, key tile) steps, units counted with the
// query tile fastest; its token counts the units that run touches. A CTA has at most two cut units: the
// one its run starts in and the one it ends in.
__device__ __forceinline__ FwdUnit fwd_unit(const FwdParams& p, uint32_t token) {
  FwdUnit w;
  w.lk = -1, w.safe = 0, w.token = token, w.part = -1;
  w.q_row0 = w.q_begin = w.lq = w.h = w.b = w.k_begin = w.bcoord = 0;
  uint32_t u = token;
  int tile0 = 0, tile1 = p.n_kt;
  if (p.parts != nullptr) {
    const int s0 = int(fwd_split_start(p, blockIdx.x)), s1 = int(fwd_split_start(p, blockIdx.x + 1));
    u = p.div_n_kt.quot(uint32_t(s0)) + token;
    const int first = int(u) * p.n_kt;
    if (token == 0) tile0 = s0 - first;
    if (first + tile0 >= s1) return w;
    tile1 = min(s1 - first, p.n_kt);
    if (tile0 > 0 || tile1 < p.n_kt) w.part = 2 * int(blockIdx.x) + (tile0 == 0);
  } else if (u >= uint32_t(p.n_units)) {
    return w;
  }
  if (p.cu_q != nullptr) {
    // One read tells everything about an item (the sequence index `batch` stands for the rows past the
    // last sequence: queries without keys, which get O = 0 and LSE = -inf). Unused entries sit at the
    // end of the list.
    const uint32_t at = p.div_heads.quot(u);
    const SchedItem item = sched_load(p.items, at);
    if (item.seq < 0) return w;
    w.h = int(u - at * uint32_t(p.heads));
    w.b = item.seq;
    w.q_row0 = item.tile * kTile, w.q_begin = item.own_begin, w.lq = item.own_len;
    w.k_begin = item.other_begin, w.lk = item.other_len;
  } else {
    const uint32_t t = p.div_n_qt.quot(u);
    w.q_row0 = int(u - t * uint32_t(p.n_qt)) * kTile, w.lq = p.lq;
    w.b = w.bcoord = int(p.div_heads.quot(t));
    w.h = int(t - uint32_t(w.b) * uint32_t(p.heads));
    w.k_begin = tile0 * kTile;
    w.lk = min(p.lk, tile1 * kTile) - w.k_begin;
  }
  return w;
}

// Row maximum of 32 raw scores with two independent chains of 3-input max.
__device__ __forceinline__ void chunk_max(const uint32_t (&r)[32], float& mx0, float& mx1) {
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    mx0 = max3(mx0, __uint_as_float(r[j]), __uint_as_float(r[j + 1]));
    mx1 = max3(mx1, __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
  }
}

// Columns >= valid (only on a ragged last key tile) count as -inf.
__device__ __forceinline__ void chunk_mask(uint32_t (&r)[32], int col0, int valid) {
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (col0 + j >= valid) r[j] = 0xff800000u;
}

// P = exp2(s*scale_log2 - m_scaled) for 32 scores, packed to bf16; four partial row sums kept as
// two packed fp32 pairs. Packed f32x2 arithmetic halves the issue slots of the FMA and the add. `top` collects
// the largest argument that took the polynomial, NaN if one was: its results mean nothing from 2^128 on and
// do not show a NaN, so the caller has to look.
__device__ __forceinline__ void chunk_exp(const uint32_t (&r)[32], uint64_t scale2, uint64_t neg_m2, float& top,
                                          uint64_t& l01, uint64_t& l23, uint32_t* pk) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float x0, x1;
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), scale2, neg_m2),
                 x0, x1);
    float p0, p1;
    // One pair in eight takes the polynomial on the FMA pipe: the MUFU unit gives 16 results per clock
    // and SM, 1024 clocks for a 128 x 128 tile. Dense 32 x 8 x 4096, sustained: none 1453 us, one in eight
    // 1424, one in four 1430; 1 x 12 x 3476, not power-limited: 60.4, 57.5, 56.3. One in four would
    // double what the polynomial adds to the error of the log-sum-exp (a bias of 5e-7 over many
    // keys). Without `top`: 1412 and 57.7.
    if ((j & 7) == 7) {
      unpack_f32x2(exp2_poly_f32x2(pack_f32x2(x0, x1)), p0, p1);
      top = max3_nan(top, x0, x1);
    } else {
      p0 = fast_exp2(x0), p1 = fast_exp2(x1);
    }
    if (j & 1) l23 = add_f32x2(l23, pack_f32x2(p0, p1)); else l01 = add_f32x2(l01, pack_f32x2(p0, p1));
    pk[j] = pack_bf16(p0, p1);
  }
}

// Puts the cut units together: block (b, half) looks after the unit in which CTA b's run starts, if it
// is the first cut in that unit, and 64 of its rows; thread = (row, four groups of four columns).
__global__ void __launch_bounds__(256) attn_fwd_combine_kernel(const __grid_constant__ FwdParams p) {
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t b = blockIdx.x + 1, s0 = fwd_split_start(p, b);
  const uint32_t u = p.div_n_kt.quot(s0), first = u * uint32_t(p.n_kt), end = first + uint32_t(p.n_kt);
  if (s0 == first || fwd_split_start(p, b - 1) > first) return;
  const int row = int(blockIdx.y) * 64 + int(threadIdx.x & 63), g0 = int(threadIdx.x >> 6) * 4;
  const uint32_t t = p.div_n_qt.quot(u);
  const int tok = int(u - t * uint32_t(p.n_qt)) * kTile + row;
  if (tok >= p.lq) return;
  auto part = [&](uint32_t c) { return p.parts + int64_t(2 * c + (c == b - 1)) * kFwdPartFloats; };
  auto stat = [&](uint32_t c) { return reinterpret_cast<const float2*>(part(c) + kTile * kHeadDim)[row]; };
  float m = -INFINITY, l = 0.f, w = 0.f;
  for (uint32_t c = b - 1; fwd_split_start(p, c) < end; ++c) m = fmaxf(m, stat(c).x);
  float4 o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) o[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t c = b - 1; fwd_split_start(p, c) < end; ++c) {
    const float2 st = stat(c);
    const float4* src = reinterpret_cast<const float4*>(part(c)) + g0 * kTile + row;
    const float f = fast_exp2((st.x - m) * p.scale_log2);
    l += st.y * f;
    w += part(c)[kTile * (kHeadDim + 2) + row] * f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 a = src[j * kTile];
      o[j].x = fmaf(a.x, f, o[j].x), o[j].y = fmaf(a.y, f, o[j].y);
      o[j].z = fmaf(a.z, f, o[j].z), o[j].w = fmaf(a.w, f, o[j].w);
    }
  }
  const float inv_l = 1.f / fmaf(l, 0.f, w);
  const uint32_t seq = p.div_heads.quot(t), h = t - seq * uint32_t(p.heads);
  uint4* dst = reinterpret_cast<uint4*>(p.o + int64_t(seq) * p.o_sb + int64_t(h) * p.o_sh + int64_t(tok) * p.o_st) + g0 / 2;
#pragma unroll
  for (int j = 0; j < 2; ++j)
    dst[j] = make_uint4(pack_bf16(o[2 * j].x * inv_l, o[2 * j].y * inv_l), pack_bf16(o[2 * j].z * inv_l, o[2 * j].w * inv_l),
                        pack_bf16(o[2 * j + 1].x * inv_l, o[2 * j + 1].y * inv_l),
                        pack_bf16(o[2 * j + 1].z * inv_l, o[2 * j + 1].w * inv_l));
  if (g0 == 0)
    p.lse[(int64_t(seq) * p.heads + h) * p.lq + tok] = (m * p.scale_log2 + log2f(l)) * 0.6931471805599453f;
}

__global__ void __launch_bounds__(kFwdThreads, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[kFwdNumBars];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ FwdUnit units[2];
  // Units to be walked again: a ring of tokens, and whether the unit in a slot has been listed.
  __shared__ uint32_t redo_tokens[kFwdRedoSlots];
  __shared__ int redo_count, redo_listed[2];

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = smem_base;
  auto sK = [&](uint32_t s) { return smem_base + (1 + 2 * s) * kTileBytes; };
  auto sV = [&](uint32_t s) { return smem_base + (2 + 2 * s) * kTileBytes; };
  const uint32_t sO = smem_base + (1 + 2 * kFwdStages) * kTileBytes;
  const uint32_t sOnes = sO + kTileBytes;
  const uint32_t bar0 = smem_u32(&bars[0]);
  auto bar = [&](uint32_t i) { return bar0 + 8u * i; };

  if (tid == 5 * 32) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    abort_flag = 0, redo_count = 0;
    for (int i = 0; i < kFwdNumBars; ++i) {
      const bool warps =
          (i >= kFwdPFull && i < kFwdPFull + 2) || i >= kFwdOFree;
      mbar_init(bar(i), warps ? 4 : 1);
    }
    fence_mbar_init();
  }
  if (tid < kFwdOnesBytes / 16) {
    constexpr uint32_t kOnes = 0x3f803f80u;
    reinterpret_cast<uint4*>(smem_raw + (sOnes - smem_u32(smem_raw)))[tid] = make_uint4(kOnes, kOnes, kOnes, kOnes);
    fence_proxy_async_smem();
  }
  // Everything this kernel reads may come from the kernel right before it in the stream. Tensor memory is taken
  // behind the wait: the kernel before may be a foreign one (a library GEMM) with blocks that have yet
  // to take theirs, and neither side's wait would end. For the same reason dependents may start only when this block has
  // its own.
  pdl_wait();
  if (warp == 4) {
    tmem_alloc(smem_u32(&tmem_base_slot), kFwdTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  const uint32_t tmem_base = tmem_base_slot;
  const uint32_t tm_s = tmem_base, tm_o = tmem_base + 128, tm_q = tmem_base + 208;

  if (warp == 5) {
    // ---------------- producer: unit descriptors, Q, K and V ----------------
    if (elect_one()) {
      uint32_t u = 0;     // units published so far
      uint32_t t = 0;     // key tiles requested so far
      uint32_t redo = 0;  // units walked again so far
      const bool packed = p.cu_q != nullptr;
      auto wait_done = [&](uint32_t v) {  // unit v is finished
        mbar_wait(bar(kFwdUnitDone + (v & 1u)), (v >> 1) & 1u, &abort_flag);
      };
      uint32_t token = packed ? sched_next(p.items) : p.parts != nullptr ? 0u : blockIdx.x;
#pragma unroll 1
      for (;;) {
        FwdUnit w = fwd_unit(p, token);
        // Again: when there is no new unit, or the list is about to overflow (two units may be in flight).
        const bool again = w.lk < 0 || *reinterpret_cast<volatile int*>(&redo_count) - int(redo) >= kFwdRedoSlots - 3;
        if (again) {
          if (w.lk < 0) {  // whether there is anything to walk again is known once all units are finished
            if (u >= 2) wait_done(u - 2);
            if (u >= 1) wait_done(u - 1);
          }
          if (redo == uint32_t(*reinterpret_cast<volatile int*>(&redo_count))) break;
          w = fwd_unit(p, reinterpret_cast<volatile uint32_t*>(redo_tokens)[redo++ % kFwdRedoSlots]);
          w.safe = 1;
        }
        if (u >= 2) wait_done(u - 2);  // the descriptor slot's last user
        if (u >= 1) mbar_wait(bar(kFwdQEmpty), (u - 1) & 1u, &abort_flag);
        units[u & 1u] = w;
        redo_listed[u & 1u] = 0;
        if (w.lk == 0) {
          mbar_arrive(bar(kFwdQFull + (u & 1u)));
        } else {
          mbar_arrive_expect_tx(bar(kFwdQFull + (u & 1u)), kTileBytes);
          tma_load_4d(sQ, &tmap_q, bar(kFwdQFull + (u & 1u)), 0, w.q_begin + w.q_row0, w.h, w.bcoord);
        }
        ++u;
        if (abort_flag) break;
#pragma unroll 1
        for (int row = 0; row < w.lk; row += kTile, ++t) {
          const uint32_t s = t % kFwdStages, ph = ((t / kFwdStages) - 1) & 1;
          if (t >= uint32_t(kFwdStages)) mbar_wait(bar(kFwdKEmpty + s), ph, &abort_flag);
          mbar_arrive_expect_tx(bar(kFwdKFull + s), kTileBytes);
          tma_load_4d(sK(s), &tmap_k, bar(kFwdKFull + s), 0, w.k_begin + row, w.h, w.bcoord);
          if (t >= uint32_t(kFwdStages)) mbar_wait(bar(kFwdVEmpty + s), ph, &abort_flag);
          mbar_arrive_expect_tx(bar(kFwdVFull + s), kTileBytes);
          tma_load_4d(sV(s), &tmap_v, bar(kFwdVFull + s), 0, w.k_begin + row, w.h, w.bcoord);
        }
        // The next unit is taken as late as can be: this thread is two key tiles ahead of the softmax warps, which
        // covers the counter's and the list's latency, and a unit taken earlier waits behind this one while
        // other CTAs run dry (one sequence of 3476 tokens and 12 heads: 88 us with the next unit taken before this
        // one's loads, 74 this way).
        if (!again) token = packed ? sched_next(p.items) : p.parts != nullptr ? token + 1 : token + gridDim.x;
      }
      units[u & 1u].lk = -1;
      mbar_arrive(bar(kFwdQFull + (u & 1u)));
      if (packed) sched_leave(p.items, gridDim.x);
    }
  } else if (warp == 4) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t kIdescS = make_idesc(128, 64, 0, 0);
      // P V with 16 more columns of B, all ones: the first of them sums up the rows of P as the product
      // sees it, rounded to bf16. They lie behind V at the descriptor's leading offset, which therefore shrinks by what
      // the start address grows from K step to K step.
      constexpr uint32_t kIdescPV = make_idesc(128, 80, 0, 1);
      constexpr uint64_t kVStep = 128 - (128ull << 16);
      const uint64_t qd = make_sdesc(sQ, 16, 1024);
      uint32_t t = 0;   // key tiles so far
      uint32_t t1 = 0;  // of them with a second half
      uint32_t uo = 0;  // units with keys so far
#pragma unroll 1
      for (uint32_t u = 0;; ++u) {
        if (!mbar_wait(bar(kFwdQFull + (u & 1u)), (u >> 1) & 1u, &abort_flag)) break;
        const int lk = reinterpret_cast<volatile FwdUnit*>(units)[u & 1u].lk;
        if (lk < 0) break;
        if (lk == 0) {
          mbar_arrive(bar(kFwdQEmpty));
          continue;
        }
        const int n_kv = (lk + kTile - 1) / kTile;
        // Live key columns of the last tile, rounded up to the MMA's granularity of 16.
        const int last_n16 = (lk - (n_kv - 1) * kTile + 15) & ~15;
        // S of half hf of tile i (the t-th of the CTA); its columns hold no live P any more.
        auto issue_s = [&](int i, uint32_t tt, int hf) {
          const uint64_t kd = make_sdesc(sK(tt % kFwdStages) + hf * (kTileBytes / 2), 16, 1024);
          const int n = i == n_kv - 1 ? min(last_n16 - 64 * hf, 64) : 64;
          const uint32_t idesc = idesc_with_n(kIdescS, n);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_ts(tm_s + 64 * hf, tm_q + 8 * k, kd + 2 * k, idesc, k > 0);
          tc_commit(bar(kFwdSFull + hf));
        };
        auto halves = [&](int i) { return i == n_kv - 1 && last_n16 <= 64 ? 1 : 2; };
        // (The MMAs that read the previous unit's Q are complete: their scores have been consumed.)
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k) tmem_copy_128x256b(tm_q + 8 * k, qd + 2 * k);
        tc_commit(bar(kFwdQEmpty));
        mbar_wait(bar(kFwdKFull + t % kFwdStages), (t / kFwdStages) & 1, &abort_flag);
        tc_fence_after();
        const int nh0 = halves(0);
        issue_s(0, t, 0);
        if (nh0 > 1) issue_s(0, t, 1);
        tc_commit(bar(kFwdKEmpty + t % kFwdStages));
        // O of the previous unit has to be out of tensor memory before the first P V product.
        if (uo > 0) mbar_wait(bar(kFwdOFree), (uo - 1) & 1u, &abort_flag);
        ++uo;
#pragma unroll 1
        for (int i = 0; i < n_kv; ++i, ++t) {
          const uint32_t s = t % kFwdStages, s1 = (t + 1) % kFwdStages;
          mbar_wait(bar(kFwdVFull + s), (t / kFwdStages) & 1, &abort_flag);
          const uint64_t vd = make_sdesc(sV(s), sOnes - sV(s), 1024);
          const int nh = halves(i), nh1 = i + 1 < n_kv ? halves(i + 1) : 0;
#pragma unroll 1
          for (int hf = 0; hf < nh; ++hf) {
            mbar_wait(bar(kFwdPFull + hf), (hf ? t1 : t) & 1, &abort_flag);
            tc_fence_after();
            // P of this half times V (the softmax warps have cleared the V rows between the last live
            // key and the next multiple of 16).
            const int ksteps = i == n_kv - 1 ? min((last_n16 >> 4) - 4 * hf, 4) : 4;
            if (ksteps == 4) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                mma_ts(tm_o, tm_s + 64 * hf + 8 * k, vd + kVStep * (4 * hf + k), kIdescPV, (i | hf | k) > 0);
            } else {
#pragma unroll 1
              for (int k = 0; k < ksteps; ++k)
                mma_ts(tm_o, tm_s + 64 * hf + 8 * k, vd + kVStep * (4 * hf + k), kIdescPV, (i | hf | k) > 0);
            }
            tc_commit(bar(kFwdPvDone + hf));
            if (hf == nh - 1) tc_commit(bar(kFwdVEmpty + s));
            if (hf < nh1) {
              if (hf == 0) {
                mbar_wait(bar(kFwdKFull + s1), ((t + 1) / kFwdStages) & 1, &abort_flag);
                tc_fence_after();
              }
              issue_s(i + 1, t + 1, hf);
              if (hf == nh1 - 1) tc_commit(bar(kFwdKEmpty + s1));
            }
          }
          t1 += nh - 1;
        }
      }
    }
  } else {
    // ---------------- softmax warpgroup ----------------
    const uint32_t lane_off = uint32_t(warp * 32) << 16;
    const uint32_t s_addr = tm_s + lane_off, o_addr = tm_o + lane_off;
    const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
    const uint32_t lane0 = lane == 0;
    uint32_t t[2] = {0, 0};  // first and second halves so far
#pragma unroll 1
    for (uint32_t u = 0;; ++u) {
      if (!mbar_wait(bar(kFwdQFull + (u & 1u)), (u >> 1) & 1u, &abort_flag)) break;
      const volatile FwdUnit& meta = reinterpret_cast<volatile FwdUnit*>(units)[u & 1u];
      const int lk = meta.lk;
      if (lk < 0) break;
      const bool safe = meta.safe != 0;
      float m_run = -INFINITY;  // raw (unscaled) offset of the exponent
      float l_run = 0.f;
      float top = -INFINITY;  // see chunk_exp
      bool s_ok = false;
#pragma unroll 1
      for (int c0 = 0; c0 < lk; c0 += 64) {  // one half tile: key columns [c0, c0 + 64)
        const int hf = (c0 >> 6) & 1;
        const int valid = lk - c0;  // live columns, if below 64
        const uint32_t th = hf ? t[1] : t[0];
        if (!s_ok) mbar_wait(bar(kFwdSFull + hf), th & 1, &abort_flag);
        __syncwarp();
        tc_fence_after();
        uint32_t ra[32], rb[32], pk[32];
        tmem_ld32(s_addr + 64 * hf, ra);
        tmem_ld32(s_addr + 64 * hf + 32, rb);
        tmem_wait_ld();
        if (valid < 64) {
          chunk_mask(ra, 0, valid);
          chunk_mask(rb, 32, valid);
          if (warp == 0 && p.cu_q != nullptr) {
            // Packed mode: V rows [lk, lk rounded up to 16) of this tile belong to the next sequence.
            // Their P columns are 0, but 0 x Inf would still poison this sequence, so the rows are
            // cleared before P is handed to the MMA warp. (The swizzle only permutes 16-byte chunks
            // inside a 128-byte row: whole rows are contiguous.)
            const uint32_t tile = hf ? t[0] - 1 : t[0], st = tile % kFwdStages;
            mbar_wait(bar(kFwdVFull + st), (tile / kFwdStages) & 1, &abort_flag);
            uint8_t* v_rows = smem_raw + (sV(st) - smem_u32(smem_raw)) + hf * (kTileBytes / 2);
            for (int c = valid * 8 + lane; c < ((valid + 15) & ~15) * 8; c += 32)
              reinterpret_cast<uint4*>(v_rows)[c] = make_uint4(0, 0, 0, 0);
            fence_proxy_async_smem();
            __syncwarp();
          }
        }
        if (c0 == 0 || safe) {
          float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
          chunk_max(ra, mx0, mx1);
          chunk_max(rb, mx2, mx3);
          if (c0 == 0 && lk > 64) {  // the first offset is the max of the whole tile
            mbar_wait(bar(kFwdSFull + 1), t[1] & 1, &abort_flag);
            __syncwarp();
            tc_fence_after();
#pragma unroll 1
            for (int c = 64; c < 128; c += 32) {
              uint32_t r[32];
              tmem_ld32(s_addr + c, r);
              tmem_wait_ld();
              if (lk < 128) chunk_mask(r, c, lk);
              chunk_max(r, mx0, mx1);
            }
          }
          const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)));
          const bool need = (m_new - m_run) * p.scale_log2 > kRescaleThreshold;
          if (c0 == 0) {
            // Where all scores of the tile are -inf, the first walk goes on with that offset: P becomes Inf or NaN, which
            // leads to the second. There any finite offset makes their P 0.
            m_run = safe && m_new == -INFINITY ? kNoOffset : m_new;
          } else if (__any_sync(0xffffffffu, need)) {
            // Second time: refresh the offset of the rows that need it, rescale their running sum and
            // their row of the O accumulator (complete up to the previous half).
            mbar_wait(bar(kFwdPvDone + (hf ^ 1)), ((hf ? t[0] : t[1]) - 1) & 1, &abort_flag);
            __syncwarp();
            tc_fence_after();
            const float alpha = need ? fast_exp2((m_run - m_new) * p.scale_log2) : 1.f;
            if (need) m_run = m_new;
            l_run *= alpha;
#pragma unroll 1
            for (int c = 0; c < 5; ++c) {
              uint32_t o[16];
              tmem_ld16(o_addr + c * 16, o);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
              tmem_st16(o_addr + c * 16, o);
            }
          }
        }
        const float nm = -m_run * p.scale_log2;
        const uint64_t neg_m2 = pack_f32x2(nm, nm);
        uint64_t l01 = 0ull, l23 = 0ull;
        chunk_exp(ra, scale2, neg_m2, top, l01, l23, pk);
        chunk_exp(rb, scale2, neg_m2, top, l01, l23, pk + 16);
        tmem_st32(s_addr + 64 * hf, pk);
        // The next half's scores are usually there already; look while the stores complete.
        if (hf) ++t[1]; else ++t[0];
        s_ok = mbar_test_wait(bar(kFwdSFull + (hf ^ 1)), (hf ? t[0] : t[1]) & 1);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(bar(kFwdPFull + hf), lane0);
        float a0, a1, a2, a3;
        unpack_f32x2(l01, a0, a1);
        unpack_f32x2(l23, a2, a3);
        l_run += (a0 + a1) + (a2 + a3);
      }

      // End of the unit: O / l -> bf16, natural-log LSE; or this CTA's part of a cut unit.
      const int e_q_begin = meta.q_begin, e_lq = meta.lq, e_h = meta.h, e_b = meta.b, e_row0 = meta.q_row0;
      const int row = e_row0 + tid;
      bool store = true;
      if (lk > 0) {
        const int hf = ((lk - 1) >> 6) & 1;  // the last half; MMAs complete in order
        mbar_wait(bar(kFwdPvDone + hf), ((hf ? t[1] : t[0]) - 1) & 1, &abort_flag);
        __syncwarp();
        tc_fence_after();
        if (!(top < kPolyLimit)) l_run = NAN;
        if (!safe) {
          bool again = !(l_run <= kFirstPassSumLimit);
          if (__any_sync(0xffffffffu, l_run > kPlainSumLimit)) {
            // P has been far above 1, so P V may have left fp32's range where the result would not.
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t o[16];
              tmem_ld16(o_addr + c * 16, o);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 16; ++j) again |= (o[j] & 0x7f800000u) == 0x7f800000u;
            }
          }
          if (__any_sync(0xffffffffu, again)) {
            // Some exponent ran far above the first tile's offset: the unit is walked again.
            if (lane == 0 && atomicExch(&redo_listed[u & 1u], 1) == 0)
              redo_tokens[uint32_t(atomicAdd(&redo_count, 1)) % kFwdRedoSlots] = meta.token;
            store = false;
          }
        }
      }
      // Each warp turns its 32 rows into bf16 in a 4 KB staging area and writes them out with eight lanes
      // per 128-byte row, so the stores are whole lines; a warp only reads what it wrote.
      uint8_t* scratch = smem_raw + (sO - smem_u32(smem_raw)) + warp * 4096;
      // What O is divided by is the sum of the rounded P: the rounding of a key's P then weighs nothing in a row which that
      // key dominates. The sum before rounding is the one for the log-sum-exp (and carries NaN, see `top`).
      float w_run = 1.f;
      if (lk > 0) {
        uint32_t w[16];
        tmem_ld16(o_addr + 64, w);
        tmem_wait_ld();
        // (A sequence of one tile has its max as the offset, whose P is exactly 1: nothing to gain there.)
        w_run = lk <= kTile && meta.part < 0 ? l_run : fmaf(l_run, 0.f, __uint_as_float(w[0]));
      }
      if (meta.part >= 0) {
        // This CTA's part of a cut unit: O as it is, then offset and sum of every row. O is laid out as 16
        // groups of four columns x 128 rows, so that a warp's stores are whole lines.
        float* part = p.parts + int64_t(meta.part) * kFwdPartFloats;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t o[32];
          tmem_ld32(o_addr + c * 32, o);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            reinterpret_cast<uint4*>(part)[(c * 8 + j) * kTile + tid] =
                make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        }
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(bar(kFwdOFree), lane0);
        reinterpret_cast<float2*>(part + kTile * kHeadDim)[tid] = make_float2(m_run, l_run);
        part[kTile * (kHeadDim + 2) + tid] = w_run;
        store = false;
      } else {
        const float inv_l = lk > 0 ? 1.f / w_run : 0.f;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t o[32];
          if (lk > 0) {
            tmem_ld32(o_addr + c * 32, o);
            tmem_wait_ld();
            if (c == 1) {
              tc_fence_before();
              __syncwarp();
              mbar_arrive_if(bar(kFwdOFree), lane0);
            }
          } else {
            // No keys at all: the output is defined as zero and the LSE as -inf.
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = 0u;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(o[8 * j + 0]) * inv_l, __uint_as_float(o[8 * j + 1]) * inv_l);
            v.y = pack_bf16(__uint_as_float(o[8 * j + 2]) * inv_l, __uint_as_float(o[8 * j + 3]) * inv_l);
            v.z = pack_bf16(__uint_as_float(o[8 * j + 4]) * inv_l, __uint_as_float(o[8 * j + 5]) * inv_l);
            v.w = pack_bf16(__uint_as_float(o[8 * j + 6]) * inv_l, __uint_as_float(o[8 * j + 7]) * inv_l);
            *reinterpret_cast<uint4*>(scratch + swz128(lane, c * 4 + j)) = v;
          }
        }
      }
      __syncwarp();
      if (store) {
        __nv_bfloat16* out_base =
            p.o + (p.cu_q != nullptr ? int64_t(0) : int64_t(e_b) * p.o_sb) + int64_t(e_h) * p.o_sh;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int rloc = it * 4 + (lane >> 3);
          const int orow = e_row0 + warp * 32 + rloc;
          const uint4 v = *reinterpret_cast<const uint4*>(scratch + swz128(rloc, lane & 7));
          if (orow < e_lq)
            *reinterpret_cast<uint4*>(out_base + int64_t(e_q_begin + orow) * p.o_st + (lane & 7) * 8) = v;
        }
        if (row < e_lq) {
          const float lse = lk > 0 ? (m_run * p.scale_log2 + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
          const int64_t lse_idx = p.cu_q != nullptr ? int64_t(e_h) * p.total_q + e_q_begin + row
                                                    : (int64_t(e_b) * p.heads + e_h) * p.lq + row;
          p.lse[lse_idx] = lse;
        }
      }
      __syncwarp();
      mbar_arrive_if(bar(kFwdUnitDone + (u & 1u)), lane0);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0) report_abort(&abort_flag, p.status);
  if (warp == 4) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kFwdTmemCols);
  }
}

}  // namespace nb
