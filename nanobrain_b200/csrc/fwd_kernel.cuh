// Forward attention kernel: O = softmax(Q K^T * scale) V, bf16 in / bf16 out, fp32 softmax
// statistics and accumulation, head_dim 64, non-causal.
//
// One CTA owns one 128-row query tile of one (sequence, head) and walks the sequence's keys in
// 128-row tiles, each in two halves of 64 key columns. In packed mode the CTA takes its (sequence,
// tile) from the scheduler's work list (sched_kernel.cuh: grid = items x heads with the heads of one
// item adjacent, so that launch order is most expensive first over the whole grid; running the list
// once per head instead was measured slower on mixes of short and long sequences); in dense mode the
// grid is (tiles, heads, batch). Two CTAs are resident per SM (256 tensor-memory columns and 81 KB of
// shared memory each), so one CTA's softmax, prologue and epilogue overlap the other's MMAs. A ragged
// last key tile is trimmed: its MMAs cover the live columns rounded up to 16, and a second half
// without live columns is left out. Warp roles (192 threads):
//
//   warps 0-3 : softmax warpgroup. Thread r owns row r of the tile (tensor-memory lane r). Per half it
//               pulls its 64 fp32 scores into registers and writes P = exp2(S*scale_log2 - m) as bf16
//               over the first half of the columns they came from. The offset m is the row max of the
//               first half tile; later halves compute no max at all: fp32 and bf16 carry exponents up
//               to 2^127, so scores may rise 60 (in log2 units) above the first ones before anything
//               has to be rescaled. Only if a row's sum ends above 2^60 (or Inf / NaN) does the CTA walk
//               the keys a second time, now with the running max of every half. At the end the warps
//               normalise and store O and the log-sum-exp.
//   warp 4    : one elected thread issues every tcgen05.mma. Q is copied into tensor memory once
//               (tcgen05.cp), so S = Q K^T takes its A operand from there, as O += P V does. After P of
//               half h of tile i is complete it issues P V of that half and then S of half h of tile
//               i+1 over the same columns (MMAs of one thread execute in order), which run while the
//               softmax warps work on the other half: the warps never wait for a score tile in steady
//               state although P has no tensor memory of its own.
//   warp 5    : one elected thread drives TMA: the Q tile once, then K and V tiles through two-stage
//               rings (SWIZZLE_128B; every CTA loads its own tiles).
//
// What bounds it: the instructions of the softmax warps and the board's power limit (at 1 kW the SMs
// run at 1.65-1.8 GHz of 1.965). Measured on dense 32 x 8 x 4096, repeated for 0.3 s: with a score tile
// and P of 128 columns each, Q from shared memory and P handed over once per tile 1550 us (1540 clocks
// per 128 x 128 tile and SM); this form 1455 us (1363 clocks); 24 sequences of 820 tokens 15.0 -> 12.7 us.
//
// Tensor memory (256 columns): S / P [0,128) O [128,192) Q [192,224).
#pragma once

#include <type_traits>

#include "ptx.cuh"
#include "sched_kernel.cuh"

namespace nb {

struct FwdParams {
  __nv_bfloat16* o;
  int64_t o_sb, o_st, o_sh;  // element strides of O: batch, token, head
  float* lse;
  const int32_t* cu_q;  // NULL => dense
  const int32_t* cu_k;
  const SchedItem* items;  // packed mode: the scheduler's work list; CTA x runs entry x / heads for head x % heads
  int32_t batch, heads;
  int32_t lq, lk;  // dense lengths (max_seqlen in varlen mode)
  int64_t total_q, total_k;
  float scale_log2;  // scale * log2(e)
  int32_t* status;
};

constexpr int kTile = 128;  // rows per Q tile and per K/V tile
constexpr int kHeadDim = 64;
constexpr int kTileBytes = kTile * kHeadDim * 2;  // 16 KB

constexpr int kFwdThreads = 192;
constexpr int kFwdQRows = kTile;  // query rows per CTA
constexpr int kFwdStages = 2;
constexpr int kFwdSmemBytes = (1 + 2 * kFwdStages) * kTileBytes + 1024;
constexpr int kFwdTmemCols = 256;
constexpr float kRescaleThreshold = 8.f;                       // log2 units
constexpr float kFirstPassSumLimit = 1152921504606846976.f;  // 2^60

enum FwdBar : int {
  kFwdQFull = 0,
  kFwdKFull,                              // [stages]
  kFwdKEmpty = kFwdKFull + kFwdStages,    // [stages]
  kFwdVFull = kFwdKEmpty + kFwdStages,    // [stages]
  kFwdVEmpty = kFwdVFull + kFwdStages,    // [stages]
  kFwdSFull = kFwdVEmpty + kFwdStages,    // [2]: per half of a key tile
  kFwdPFull = kFwdSFull + 2,              // [2], 4 arrivals (one per softmax warp)
  // [2]: P V of the half is complete. One barrier per half: the softmax warps hand over two halves
  // before they look, and a barrier must never be two phases behind a waiter that tests by parity.
  kFwdPvDone = kFwdPFull + 2,
  kFwdVerdict = kFwdPvDone + 2,           // 4 arrivals: the first pass is judged
  kFwdNumBars
};

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
// two packed fp32 pairs. Packed f32x2 arithmetic halves the issue slots of the FMA and the add.
__device__ __forceinline__ void chunk_exp(const uint32_t (&r)[32], uint64_t scale2, uint64_t neg_m2,
                                          uint64_t& l01, uint64_t& l23, uint32_t* pk) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float x0, x1;
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), scale2, neg_m2),
                 x0, x1);
    float p0, p1;
    // One pair in four takes the polynomial on the FMA pipe: the MUFU unit gives 16 results per clock
    // and SM, 1024 clocks for a 128 x 128 tile, and the rest of the loop leaves room for about that
    // much (dense 32 x 8 x 4096: none 1468 us, one in eight 1462, one in four 1455; 24 sequences of
    // 820 tokens, not power-limited: 13.8, 13.2, 12.7).
    if ((j & 3) == 3) unpack_f32x2(exp2_poly_f32x2(pack_f32x2(x0, x1)), p0, p1);
    else p0 = fast_exp2(x0), p1 = fast_exp2(x1);
    if (j & 1) l23 = add_f32x2(l23, pack_f32x2(p0, p1)); else l01 = add_f32x2(l01, pack_f32x2(p0, p1));
    pk[j] = pack_bf16(p0, p1);
  }
}

__global__ void __launch_bounds__(kFwdThreads, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[kFwdNumBars];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag, redo_flag;
  // What only the epilogue needs of the work item (re-read there, so that the softmax warps do not
  // hold it in registers through their loop): q_begin, lq, head, sequence, first row of the tile.
  __shared__ int epi_meta[5];

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  int qt = blockIdx.x, h = blockIdx.y, b = blockIdx.z;

  // Everything this kernel reads may come from the kernel right before it in the stream.
  pdl_wait();
  pdl_launch_dependents();

  int q_begin = 0, k_begin = 0, lq = p.lq, lk = p.lk, bcoord = b;
  if (p.cu_q != nullptr) {
    // One read tells the CTA everything about its item (the sequence index `batch` stands for the
    // rows past the last sequence: queries without keys, which get O = 0 and LSE = -inf).
    const SchedItem item = sched_load(p.items, blockIdx.x / uint32_t(p.heads));
    if (item.seq < 0) return;
    h = blockIdx.x % uint32_t(p.heads);
    b = item.seq;
    qt = item.tile;
    q_begin = item.own_begin;
    lq = item.own_len;
    k_begin = item.other_begin;
    lk = item.other_len;
    bcoord = 0;
  }
  const int q_row0 = qt * kTile;
  if (q_row0 >= lq) return;  // this tile lies past the end of the sequence
  const int n_kv = (lk + kTile - 1) / kTile;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = smem_base;
  auto sK = [&](int s) { return smem_base + (1 + 2 * s) * kTileBytes; };
  auto sV = [&](int s) { return smem_base + (2 + 2 * s) * kTileBytes; };
  const uint32_t bar0 = smem_u32(&bars[0]);
  auto bar = [&](uint32_t i) { return bar0 + 8u * i; };

  // The producer's own thread initialises the barriers, so it can start the first loads (Q and both
  // K/V stages) at once; the other threads meet the barriers only after the __syncthreads below.
  if (tid == 5 * 32) {
    epi_meta[0] = q_begin, epi_meta[1] = lq, epi_meta[2] = h, epi_meta[3] = b, epi_meta[4] = q_row0;
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    abort_flag = 0, redo_flag = 0;
    for (int i = 0; i < kFwdNumBars; ++i)
      mbar_init(bar(i), (i == kFwdPFull || i == kFwdPFull + 1 || i == kFwdVerdict) ? 4 : 1);
    fence_mbar_init();
    if (n_kv > 0) {
      mbar_arrive_expect_tx(bar(kFwdQFull), kTileBytes);
      tma_load_4d(sQ, &tmap_q, bar(kFwdQFull), 0, q_begin + q_row0, h, bcoord);
      for (int i = 0; i < kFwdStages && i < n_kv; ++i) {
        mbar_arrive_expect_tx(bar(kFwdKFull + i), kTileBytes);
        tma_load_4d(sK(i), &tmap_k, bar(kFwdKFull + i), 0, k_begin + i * kTile, h, bcoord);
        mbar_arrive_expect_tx(bar(kFwdVFull + i), kTileBytes);
        tma_load_4d(sV(i), &tmap_v, bar(kFwdVFull + i), 0, k_begin + i * kTile, h, bcoord);
      }
    }
  }
  if (warp == 4) {
    tmem_alloc(smem_u32(&tmem_base_slot), kFwdTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  const uint32_t tm_s = tmem_base, tm_o = tmem_base + 128, tm_q = tmem_base + 192;

  // The roles below ask this once, after the first pass: do the keys have to be walked again?
  auto second_pass_wanted = [&] {
    mbar_wait(bar(kFwdVerdict), 0, &abort_flag, p.status);
    return *const_cast<volatile int*>(&redo_flag) != 0;
  };

  if (n_kv > 0) {
    if (warp == 5) {
      // ---------------- TMA producer ----------------
      if (elect_one()) {
        uint32_t t = uint32_t(min(kFwdStages, n_kv));  // tiles requested so far, over both passes
        int i = int(t);                                // (the first ones at start-up)
#pragma unroll 1
        for (int pass = 0;; ++pass) {
#pragma unroll 1
          for (; i < n_kv; ++i, ++t) {
            const uint32_t s = t % kFwdStages, ph = ((t / kFwdStages) - 1) & 1;
            if (t >= uint32_t(kFwdStages)) mbar_wait(bar(kFwdKEmpty + s), ph, &abort_flag, p.status);
            mbar_arrive_expect_tx(bar(kFwdKFull + s), kTileBytes);
            tma_load_4d(sK(s), &tmap_k, bar(kFwdKFull + s), 0, k_begin + i * kTile, h, bcoord);
            if (t >= uint32_t(kFwdStages)) mbar_wait(bar(kFwdVEmpty + s), ph, &abort_flag, p.status);
            mbar_arrive_expect_tx(bar(kFwdVFull + s), kTileBytes);
            tma_load_4d(sV(s), &tmap_v, bar(kFwdVFull + s), 0, k_begin + i * kTile, h, bcoord);
          }
          if (pass == 1 || !second_pass_wanted()) break;
          i = 0;
        }
      }
    } else if (warp == 4) {
      // ---------------- MMA issuer ----------------
      if (elect_one()) {
        constexpr uint32_t kIdescS = make_idesc(128, 64, 0, 0);
        constexpr uint32_t kIdescPV = make_idesc(128, 64, 0, 1);
        // Live key columns of the last tile, rounded up to the MMA's granularity of 16.
        const int last_n16 = (lk - (n_kv - 1) * kTile + 15) & ~15;
        // S of half hf of tile i (the t-th of both passes); its columns hold no live P any more.
        auto issue_s = [&](int i, uint32_t t, int hf) {
          const uint64_t kd = make_sdesc(sK(t % kFwdStages) + hf * (kTileBytes / 2), 16, 1024);
          const int n = i == n_kv - 1 ? min(last_n16 - 64 * hf, 64) : 64;
          const uint32_t idesc = idesc_with_n(kIdescS, n);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_ts(tm_s + 64 * hf, tm_q + 8 * k, kd + 2 * k, idesc, k > 0);
          tc_commit(bar(kFwdSFull + hf));
        };
        auto halves = [&](int i) { return i == n_kv - 1 && last_n16 <= 64 ? 1 : 2; };
        mbar_wait(bar(kFwdQFull), 0, &abort_flag, p.status);
        tc_fence_after();
        const uint64_t qd = make_sdesc(sQ, 16, 1024);
#pragma unroll
        for (int k = 0; k < 4; ++k) tmem_copy_128x256b(tm_q + 8 * k, qd + 2 * k);
        uint32_t t = 0;   // key tiles so far, over both passes
        uint32_t t1 = 0;  // tiles with a second half so far
#pragma unroll 1
        for (int pass = 0;; ++pass) {
          mbar_wait(bar(kFwdKFull + t % kFwdStages), (t / kFwdStages) & 1, &abort_flag, p.status);
          tc_fence_after();
          for (int hf = 0; hf < halves(0); ++hf) issue_s(0, t, hf);
          tc_commit(bar(kFwdKEmpty + t % kFwdStages));
#pragma unroll 1
          for (int i = 0; i < n_kv; ++i, ++t) {
            const uint32_t s = t % kFwdStages, s1 = (t + 1) % kFwdStages;
            mbar_wait(bar(kFwdVFull + s), (t / kFwdStages) & 1, &abort_flag, p.status);
            const uint64_t vd = make_sdesc(sV(s), 1024, 1024);
            const int nh = halves(i), nh1 = i + 1 < n_kv ? halves(i + 1) : 0;
#pragma unroll 1
            for (int hf = 0; hf < nh; ++hf) {
              mbar_wait(bar(kFwdPFull + hf), (hf ? t1 : t) & 1, &abort_flag, p.status);
              tc_fence_after();
              // P of this half times V (the softmax warps have cleared the V rows between the last live
              // key and the next multiple of 16).
              const int ksteps = i == n_kv - 1 ? min((last_n16 >> 4) - 4 * hf, 4) : 4;
              if (ksteps == 4) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  mma_ts(tm_o, tm_s + 64 * hf + 8 * k, vd + 512 * hf + 128 * k, kIdescPV, (i | hf | k) > 0);
              } else {
#pragma unroll 1
                for (int k = 0; k < ksteps; ++k)
                  mma_ts(tm_o, tm_s + 64 * hf + 8 * k, vd + 512 * hf + 128 * k, kIdescPV, (i | hf | k) > 0);
              }
              tc_commit(bar(kFwdPvDone + hf));
              if (hf == nh - 1) tc_commit(bar(kFwdVEmpty + s));
              if (hf < nh1) {
                if (hf == 0) {
                  mbar_wait(bar(kFwdKFull + s1), ((t + 1) / kFwdStages) & 1, &abort_flag, p.status);
                  tc_fence_after();
                }
                issue_s(i + 1, t + 1, hf);
                if (hf == nh1 - 1) tc_commit(bar(kFwdKEmpty + s1));
              }
            }
            t1 += nh - 1;
          }
          if (pass == 1 || !second_pass_wanted()) break;
        }
      }
    } else {
      // ---------------- softmax warpgroup ----------------
      const uint32_t lane_off = uint32_t(warp * 32) << 16;
      const uint32_t s_addr = tm_s + lane_off, o_addr = tm_o + lane_off;
      const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
      const uint32_t lane0 = lane == 0;
      float m_run = -INFINITY;  // raw (unscaled) offset of the exponent
      float l_run = 0.f;
      uint32_t t[2] = {0, 0};  // first and second halves so far, over both passes
#pragma unroll 1
      for (int pass = 0;; ++pass) {
        bool s_ok = false;
#pragma unroll 1
        for (int c0 = 0; c0 < lk; c0 += 64) {  // one half tile: key columns [c0, c0 + 64)
          const int hf = (c0 >> 6) & 1;
          const int valid = lk - c0;  // live columns, if below 64
          const uint32_t th = hf ? t[1] : t[0];
          if (!s_ok) mbar_wait(bar(kFwdSFull + hf), th & 1, &abort_flag, p.status);
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
              mbar_wait(bar(kFwdVFull + st), (tile / kFwdStages) & 1, &abort_flag, p.status);
              uint8_t* v_rows = smem_raw + (sV(st) - smem_u32(smem_raw)) + hf * (kTileBytes / 2);
              for (int c = valid * 8 + lane; c < ((valid + 15) & ~15) * 8; c += 32)
                reinterpret_cast<uint4*>(v_rows)[c] = make_uint4(0, 0, 0, 0);
              fence_proxy_async_smem();
              __syncwarp();
            }
          }
          if (c0 == 0 || pass == 1) {
            float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
            chunk_max(ra, mx0, mx1);
            chunk_max(rb, mx2, mx3);
            const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)));
            const bool need = (m_new - m_run) * p.scale_log2 > kRescaleThreshold;
            if (c0 == 0) {
              m_run = m_new;
            } else if (__any_sync(0xffffffffu, need)) {
              // Second pass: refresh the offset of the rows that need it, rescale their running sum and
              // their row of the O accumulator (complete up to the previous half).
              mbar_wait(bar(kFwdPvDone + (hf ^ 1)), ((hf ? t[0] : t[1]) - 1) & 1, &abort_flag, p.status);
              __syncwarp();
              tc_fence_after();
              const float alpha = need ? fast_exp2((m_run - m_new) * p.scale_log2) : 1.f;
              if (need) m_run = m_new;
              l_run *= alpha;
#pragma unroll 1
              for (int c = 0; c < 4; ++c) {
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
          chunk_exp(ra, scale2, neg_m2, l01, l23, pk);
          chunk_exp(rb, scale2, neg_m2, l01, l23, pk + 16);
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
        if (pass == 1) break;
        if (__any_sync(0xffffffffu, !(l_run <= kFirstPassSumLimit)) && lane == 0) redo_flag = 1;
        __syncwarp();
        mbar_arrive_if(bar(kFwdVerdict), lane0);
        if (!second_pass_wanted()) break;
        __syncwarp();
        m_run = -INFINITY, l_run = 0.f;
      }

      // Epilogue: O / l -> bf16, natural-log LSE.
      const int last_half = ((lk - 1) >> 6) & 1;  // MMAs complete in order
      mbar_wait(bar(kFwdPvDone + last_half), ((last_half ? t[1] : t[0]) - 1) & 1, &abort_flag, p.status);
      __syncwarp();
      tc_fence_after();
      const volatile int* meta = epi_meta;
      const int e_q_begin = meta[0], e_lq = meta[1], e_h = meta[2], e_b = meta[3], e_row0 = meta[4];
      const int e_bcoord = p.cu_q != nullptr ? 0 : e_b;
      const int row = e_row0 + tid;
      const float inv_l = l_run > 0.f ? 1.f / l_run : 0.f;
      // Each warp turns its 32 rows into bf16 in a 4 KB scratch area (the Q tile, dead since
      // it was copied into tensor memory, which the completed MMAs imply) and writes them out with eight
      // lanes per 128-byte row, so the stores are whole lines; a warp only reads what it wrote.
      uint8_t* scratch = smem_raw + (smem_base - smem_u32(smem_raw)) + warp * 4096;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t o[32];
        tmem_ld32(o_addr + c * 32, o);
        tmem_wait_ld();
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
      __syncwarp();
      __nv_bfloat16* out_base = p.o + int64_t(e_bcoord) * p.o_sb + int64_t(e_h) * p.o_sh;
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int rloc = it * 4 + (lane >> 3);
        const int orow = e_row0 + warp * 32 + rloc;
        const uint4 v = *reinterpret_cast<const uint4*>(scratch + swz128(rloc, lane & 7));
        if (orow < e_lq) *reinterpret_cast<uint4*>(out_base + int64_t(e_q_begin + orow) * p.o_st + (lane & 7) * 8) = v;
      }
      if (row < e_lq) {
        const float lse = (m_run * p.scale_log2 + log2f(l_run)) * 0.6931471805599453f;
        const int64_t lse_idx = p.cu_q != nullptr ? int64_t(e_h) * p.total_q + e_q_begin + row
                                                  : (int64_t(e_b) * p.heads + e_h) * p.lq + row;
        p.lse[lse_idx] = lse;
      }
    }
  } else if (warp < 4) {
    // No keys at all: the output is defined as zero and the LSE as -inf.
    const int row = q_row0 + tid;
    if (row < lq) {
      __nv_bfloat16* optr = p.o + int64_t(bcoord) * p.o_sb + int64_t(q_begin + row) * p.o_st + int64_t(h) * p.o_sh;
      for (int c = 0; c < 8; ++c) reinterpret_cast<uint4*>(optr)[c] = make_uint4(0, 0, 0, 0);
      const int64_t lse_idx = p.cu_q != nullptr ? int64_t(h) * p.total_q + q_begin + row
                                                : (int64_t(b) * p.heads + h) * p.lq + row;
      p.lse[lse_idx] = -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kFwdTmemCols);
  }
}

}  // namespace nb
