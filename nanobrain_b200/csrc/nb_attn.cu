// Host side of the C ABI declared in include/nb_attn.h: argument validation, TMA tensor-map
// construction and kernel launches. No device memory is allocated here and nothing is kept
// between calls except per-process one-time state (the driver entry point used to encode
// tensor maps and the per-device "large dynamic shared memory" opt-in).
#include "../../include/nb_attn.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>
#include <utility>
#include <vector>

#include "bwd_kernel.cuh"
#include "fwd_kernel.cuh"
#include "sched_kernel.cuh"
#include "selftest_kernel.cuh"

// Build-time switch: 0 launches every kernel with plain stream order instead of programmatic
// dependent launch (the kernels' griddepcontrol instructions are then no-ops).
#ifndef NB_ATTN_PDL
#define NB_ATTN_PDL 1
#endif

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

using CtxGetCurrentFn = CUresult (*)(CUcontext*);

EncodeTiledFn g_encode = nullptr;
CtxGetCurrentFn g_ctx_get_current = nullptr;
std::once_flag g_encode_once;

EncodeTiledFn get_encode() {
  std::call_once(g_encode_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    }
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(fn);
    }
  });
  return g_encode;
}

// Encoding a tensor map is a driver call and needs a current context. A thread whose first CUDA call
// this is (autograd's device thread, when the allocator serves the scratch from its cache) has none
// yet: the runtime would bind it at its first launch.
int bind_context(int dev) {
  if (get_encode() == nullptr || g_ctx_get_current == nullptr) return NB_ATTN_ERR_TENSOR_MAP;
  CUcontext ctx = nullptr;
  if (g_ctx_get_current(&ctx) == CUDA_SUCCESS && ctx != nullptr) return NB_ATTN_OK;
  return cudaSetDevice(dev) == cudaSuccess ? NB_ATTN_OK : NB_ATTN_ERR_LAUNCH;
}

constexpr int kMaxDevices = 64;
std::mutex g_dev_mutex;
int g_dev_state[kMaxDevices];  // 0 = not set up, 1 = ready, <0 = error code (negated)
int g_dev_sms[kMaxDevices];    // SM count, valid once the device is ready

// Bind the thread's context, and once per device: check the architecture and opt the kernels into
// their dynamic shared memory.
int ensure_device_ready() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return NB_ATTN_ERR_LAUNCH;
  if (dev < 0 || dev >= kMaxDevices) return NB_ATTN_ERR_DEVICE;
  if (const int rc = bind_context(dev)) return rc;
  std::lock_guard<std::mutex> lock(g_dev_mutex);
  if (g_dev_state[dev] == 1) return NB_ATTN_OK;
  if (g_dev_state[dev] < 0) return -g_dev_state[dev];
  int major = 0;
  int rc = NB_ATTN_OK;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&g_dev_sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      g_dev_sms[dev] <= 0) {
    rc = NB_ATTN_ERR_LAUNCH;
  } else if (major != 10) {
    rc = NB_ATTN_ERR_DEVICE;
  } else if (cudaFuncSetAttribute(nb::attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  nb::kFwdSmemBytes) != cudaSuccess ||
             cudaFuncSetAttribute(nb::attn_bwd_kernel<nb::kBwdWhole>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  nb::kBwdSmemBytes) != cudaSuccess ||
             cudaFuncSetAttribute(nb::attn_bwd_kernel<nb::kBwdCut>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  nb::kBwdSmemBytes) != cudaSuccess ||
             cudaFuncSetAttribute(nb::attn_bwd_kernel<nb::kBwdRuns>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  nb::kBwdSmemBytes) != cudaSuccess ||
             cudaFuncSetAttribute(nb::mma_selftest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  nb::kSelftestSmemBytes) != cudaSuccess) {
    rc = NB_ATTN_ERR_LAUNCH;
  }
  g_dev_state[dev] = rc == NB_ATTN_OK ? 1 : -rc;
  return rc;
}

// SM count of the current device (after ensure_device_ready succeeded on it). An entry point asks once and hands the
// number on to the rules: asked for by each of them a dense backward took the lock eight times (0.1 us of 14).
int device_sm_count() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 1;
  std::lock_guard<std::mutex> lock(g_dev_mutex);
  return g_dev_sms[dev] > 0 ? g_dev_sms[dev] : 1;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_tensor(const nb_attn_tensor& t, bool dense) {
  if (t.ptr == nullptr) return NB_ATTN_ERR_NULL;
  if (!aligned16(t.ptr)) return NB_ATTN_ERR_ALIGN;
  if (t.stride_token <= 0 || t.stride_head <= 0 || (t.stride_token % 8) != 0 || (t.stride_head % 8) != 0)
    return NB_ATTN_ERR_ALIGN;
  if (dense && (t.stride_batch <= 0 || (t.stride_batch % 8) != 0)) return NB_ATTN_ERR_ALIGN;
  return NB_ATTN_OK;
}

int check_shape(const nb_attn_shape& s) {
  if (s.head_dim != nb::kHeadDim) return NB_ATTN_ERR_HEAD_DIM;
  if (s.batch <= 0 || s.heads <= 0 || s.max_seqlen_q <= 0 || s.max_seqlen_k <= 0) return NB_ATTN_ERR_SHAPE;
  if (s.batch > 65534 || s.heads > 65535) return NB_ATTN_ERR_SHAPE;
  if ((s.cu_seqlens_q == nullptr) != (s.cu_seqlens_k == nullptr)) return NB_ATTN_ERR_SHAPE;
  if (s.total_q <= 0 || s.total_k <= 0) return NB_ATTN_ERR_SHAPE;
  if (s.cu_seqlens_q == nullptr) {
    if (s.total_q != int64_t(s.batch) * s.max_seqlen_q || s.total_k != int64_t(s.batch) * s.max_seqlen_k)
      return NB_ATTN_ERR_SHAPE;
    // The kernels count their work units (query or key tiles x heads x sequences) in 32 bits.
    if ((int64_t(s.max_seqlen_k) + nb::kTile - 1) / nb::kTile * s.heads * s.batch > INT32_MAX ||
        (int64_t(s.max_seqlen_q) + nb::kTile - 1) / nb::kTile * s.heads * s.batch > INT32_MAX)
      return NB_ATTN_ERR_SHAPE;
  } else {
    if (s.total_q > INT32_MAX || s.total_k > INT32_MAX) return NB_ATTN_ERR_SHAPE;
    // Units (items x heads) are counted in 32 bits.
    if (nb::sched_capacity(s.total_q, s.batch) * s.heads > INT32_MAX ||
        nb::sched_capacity(s.total_k, s.batch) * s.heads > INT32_MAX)
      return NB_ATTN_ERR_SHAPE;
  }
  if (!(s.scale > 0.f)) return NB_ATTN_ERR_SHAPE;
  return NB_ATTN_OK;
}

// 4-D map over (head_dim, token, head, batch) with a 64 x 128 x 1 x 1 box and 128-byte swizzle.
// Rows outside the token extent read as zeros.
int make_tmap(CUtensorMap* map, const nb_attn_tensor& t, const nb_attn_shape& s, bool is_q) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return NB_ATTN_ERR_TENSOR_MAP;
  const bool dense = s.cu_seqlens_q == nullptr;
  const uint64_t tokens = dense ? uint64_t(is_q ? s.max_seqlen_q : s.max_seqlen_k) : uint64_t(is_q ? s.total_q : s.total_k);
  const uint64_t nbatch = dense ? uint64_t(s.batch) : 1u;
  cuuint64_t dims[4] = {uint64_t(nb::kHeadDim), tokens, uint64_t(s.heads), nbatch};
  const uint64_t batch_stride = dense ? uint64_t(t.stride_batch) : tokens * uint64_t(t.stride_token);
  cuuint64_t strides[3] = {uint64_t(t.stride_token) * 2u, uint64_t(t.stride_head) * 2u, batch_stride * 2u};
  cuuint32_t box[4] = {uint32_t(nb::kHeadDim), uint32_t(nb::kTile), 1u, 1u};
  cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, t.ptr, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? NB_ATTN_OK : NB_ATTN_ERR_TENSOR_MAP;
}

// 3-D fp32 map over the dQ accumulator [token][head][64]: (64, tokens, heads), box 32 x 32 x 1 with
// 128-byte swizzle, used by the backward kernel's TMA add-reductions.
int make_dq_accum_tmap(CUtensorMap* map, float* accum, int64_t total_q, int heads) {
  EncodeTiledFn enc = get_encode();
  if (enc == nullptr) return NB_ATTN_ERR_TENSOR_MAP;
  cuuint64_t dims[3] = {uint64_t(nb::kHeadDim), uint64_t(total_q), uint64_t(heads)};
  cuuint64_t strides[2] = {uint64_t(heads) * nb::kHeadDim * sizeof(float), uint64_t(nb::kHeadDim) * sizeof(float)};
  cuuint32_t box[3] = {32u, 32u, 1u};
  cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, accum, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? NB_ATTN_OK : NB_ATTN_ERR_TENSOR_MAP;
}

constexpr float kLog2e = 1.4426950408889634f;

// Launch with programmatic stream serialization: the kernel may become resident while its
// predecessor in the stream drains; it orders itself with griddepcontrol.wait (ptx.cuh).
template <typename... KArgs, typename... Args>
cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = NB_ATTN_PDL ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// side 0: query tiles are the items; side 1: key tiles are.
nb::SchedParams make_sched(const nb_attn_shape& s, int side, nb::SchedItem* items, int64_t n_items, int32_t* status) {
  nb::SchedParams sp;
  const bool fwd = side == 0;
  sp.cu_own = fwd ? s.cu_seqlens_q : s.cu_seqlens_k;
  sp.cu_other = fwd ? s.cu_seqlens_k : s.cu_seqlens_q;
  sp.batch = s.batch;
  sp.max_own = fwd ? s.max_seqlen_q : s.max_seqlen_k;
  sp.max_other = fwd ? s.max_seqlen_k : s.max_seqlen_q;
  sp.total_own = fwd ? s.total_q : s.total_k;
  sp.total_other = fwd ? s.total_k : s.total_q;
  sp.items = items;
  sp.n_items = int32_t(n_items);
  sp.status = status;
  sp.merged = 0;
  sp.run_tiles = 0, sp.heads = s.heads, sp.sms = 1, sp.rest = nullptr;
  return sp;
}

// Layout of the backward workspace: fp32 dQ accumulator | fp32 delta | work list (varlen only).
size_t bwd_accum_bytes(const nb_attn_shape& s) { return size_t(s.total_q) * size_t(s.heads) * nb::kHeadDim * sizeof(float); }
size_t bwd_delta_bytes(const nb_attn_shape& s) { return size_t(s.total_q) * size_t(s.heads) * sizeof(float); }
size_t bwd_items_offset(const nb_attn_shape& s) { return align_up(bwd_accum_bytes(s) + bwd_delta_bytes(s), 256); }

int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Scratch for nb_attn_bwd_builtin_scratch: one fixed array in the library image per GPU. The name
// below is only a host-side handle; kernels get the device address looked up per device.
constexpr size_t kBuiltinScratchBytes =
    size_t(NB_ATTN_BUILTIN_SCRATCH_ROWS) * (nb::kHeadDim * sizeof(float) + sizeof(float)) + 256 +
    size_t(NB_ATTN_BUILTIN_SCRATCH_ITEMS) * sizeof(nb::SchedItem);
static __device__ __align__(256) unsigned char g_builtin_scratch[kBuiltinScratchBytes];
void* g_builtin_scratch_addr[kMaxDevices];  // device address of the array, per device, once looked up

// Once per device, with that device current: resolve the array's device address.
int builtin_scratch_address(void** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return NB_ATTN_ERR_LAUNCH;
  if (dev < 0 || dev >= kMaxDevices) return NB_ATTN_ERR_DEVICE;
  std::lock_guard<std::mutex> lock(g_dev_mutex);
  if (g_builtin_scratch_addr[dev] == nullptr) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_builtin_scratch) != cudaSuccess || ptr == nullptr) return NB_ATTN_ERR_LAUNCH;
    g_builtin_scratch_addr[dev] = ptr;
  }
  *out = g_builtin_scratch_addr[dev];
  return NB_ATTN_OK;
}

// Should a dense forward cut its units (query tiles) between CTAs, and into how many CTAs? Whole units
// leave SMs idle where the last round over the SMs is short or there is not even one round: one image of
// 3476 tokens and 12 heads has 336 units for 148 SMs of two CTAs each. In key tiles per CTA, with k
// units on the busiest SM whole units take about (k/2 rounded down, plus 0.9 where k is odd: a CTA that
// has the SM for itself is only a little faster) x tiles; cut ones take an equal share plus about four
// tiles' time for the parts and the kernel that puts them together. An eighth has to be gained, because
// at the power limit SMs that wait let the others run faster (1024 units of 32 tiles: 186 us whole, 189
// cut; the image: 73.5 whole, 58.5 cut). A CTA gets at least four tiles. Where every unit has an SM for itself
// but its parts would share SMs, whole units take 5.2 us + 1.05 per tile and cut ones 12 us + 1.55 per tile of
// their share: 1 x 8 x 2048 22.3 whole, 24.1 cut; x 1800 20.9 and 21.7; x 1500 18.1 and 17.2; 1 x 4 x 2000 22.0
// and 17.8.
struct FwdSplit {
  unsigned ctas = 0;  // 0: whole units
  size_t bytes = 0;
};
FwdSplit fwd_split(const nb_attn_shape& s, int sms) {
  FwdSplit r;
  if (s.cu_seqlens_q != nullptr) return r;
  const int64_t n_kt = ceil_div(s.max_seqlen_k, nb::kTile);
  const int64_t units = int64_t(ceil_div(s.max_seqlen_q, nb::kFwdQRows)) * s.heads * s.batch;
  const int64_t slots = 2 * int64_t(sms), steps = units * n_kt;
  const int64_t ctas = steps / 4 < slots ? steps / 4 : slots;
  if (ctas < 2 || steps > INT32_MAX) return r;
  const int64_t k = (units + slots / 2 - 1) / (slots / 2);
  const int64_t share = (steps + ctas - 1) / ctas;
  if ((k / 2 * 10 + (k & 1) * 9) * n_kt * 8 <= 90 * (share + 4)) return r;
  if (k == 1 && ctas > slots / 2 && 10 * n_kt < 60 + 15 * share) return r;
  r.ctas = unsigned(ctas);
  r.bytes = 2 * size_t(ctas) * nb::kFwdPartFloats * sizeof(float);
  return r;
}

// The same question for a dense backward (units are key tiles, steps are query tiles, one CTA per SM).
// Whole units take ceil(units / SMs) x tiles steps; cut ones an equal share plus about three steps' time
// for the parts. At least a twelfth has to be gained, and a CTA gets at least two steps.
struct BwdSplit {
  unsigned ctas = 0;
  size_t parts_offset = 0, bytes = 0;  // of the whole workspace
};
BwdSplit bwd_split(const nb_attn_shape& s, int64_t sms) {
  BwdSplit r;
  if (s.cu_seqlens_q != nullptr) return r;
  const int64_t n_qt = ceil_div(s.max_seqlen_q, nb::kTile);
  const int64_t units = int64_t(ceil_div(s.max_seqlen_k, nb::kTile)) * s.heads * s.batch;
  const int64_t steps = units * n_qt;
  const int64_t ctas = steps / 2 < sms ? steps / 2 : sms;
  if (ctas < 2 || steps > INT32_MAX) return r;
  if ((units + sms - 1) / sms * n_qt * 12 <= 13 * ((steps + ctas - 1) / ctas + 3)) return r;
  r.ctas = unsigned(ctas);
  r.parts_offset = align_up(bwd_accum_bytes(s) + bwd_delta_bytes(s), 256);
  r.bytes = r.parts_offset + 2 * size_t(ctas) * nb::kBwdPartFloats * sizeof(float);
  return r;
}

// May sequences of a packed backward be runs (see BwdRun)? Which of them are the device decides (sched_runs), and every
// block of the prologue has to look at all sequences for it, 3 to 5 us. So there have to be
//   * two rounds of (sequence, head) pairs over the SMs, or most of the work stays single tiles anyway. 12 heads, us
//     without and with runs: 20 x 820 tokens (1.6 rounds) 178.6 and 180.0, 24 (1.95) 212.0 and 210.0, 26 (2.1) 227.9 and
//     220.3, 32 of 720..920 (2.6) 270.4 and 261.6; 25 of 500..1100 (2.03) still 209.7 and 213.2;
//   * 21 steps per SM, about 30 us, to save from, by the mean length (skewed lengths have more, but spread over fewer
//     units: 30 of 200 and one of 2000, 10.2 by the mean and 30.5 in fact, 79.2 and 88.4). 35 x 300 (15.6 steps) 79.8 and
//     85.1, 80 x 200 (15.8) 101.5 and 96.3, 40 x 300 (17.8) 90.7 and 91.8, 26 x 400 (20.6) 93.9 and 96.4, 110 x 200 (21.8)
//     139.7 and 125.3, 50 x 300 (22.3) 112.1 and 109.6, 40 x 400 (31.7) 142.0 and 135.5;
//   * no more tiles per sequence on average than a run has at most, or few could be one. Ten are allowed from five rounds
//     on: sequences of 1160..1280 tokens, without and with ten, 32 (2.6 rounds) 518.8 and 537.9, 44 (3.6) 713 and 737, 50
//     (4.05) 811 and 787, 56 (4.5) 908 and 929, 60 (4.9) 976 and 1000, 64 (5.2) 1041 and 1017, 72 (5.8) 1170 and 1185, 80
//     (6.5) 1305 and 1295: it is the part of a round left over that decides, and it weighs less the more rounds there are.
// Sequences of one key tile are runs without more ado, which pays from four rounds on: x 128 tokens x 8 heads, 40 (2.2)
// 23.4 and 24.3, 60 (3.2) 29.7 and 29.1, 80 (4.3) 36.2 and 34.0, 100 (5.4) 42.1 and 39.3.
struct BwdRuns {
  int tiles = 0;  // SchedParams::run_tiles
  int own_tiles = 0;
  size_t rest_offset = 0, own_offset = 0, bytes = 0;  // of the whole workspace; bytes = 0: no
};
BwdRuns bwd_runs(const nb_attn_shape& s, int64_t sms) {
  BwdRuns r;
  if (s.cu_seqlens_q == nullptr) return r;
  const int64_t pairs = int64_t(s.batch) * s.heads;
  const int n_qt = ceil_div(s.max_seqlen_q, nb::kTile), n_kt = ceil_div(s.max_seqlen_k, nb::kTile);
  const int most = pairs < 5 * sms ? nb::kBwdRunTiles - 1 : nb::kBwdRunTiles;
  // (Rows past the last sequence, of a buffer with room to spare, are no work.)
  const int64_t most_q = int64_t(s.batch) * s.max_seqlen_q, most_k = int64_t(s.batch) * s.max_seqlen_k;
  const int64_t rows_q = s.total_q < most_q ? s.total_q : most_q, rows_k = s.total_k < most_k ? s.total_k : most_k;
  if (s.batch > nb::kSchedRunSeqs || pairs < (n_kt == 1 ? 4 : 2) * sms || rows_q > int64_t(s.batch) * most * nb::kTile)
    return r;
  const double steps = double(rows_q) / nb::kTile * (double(rows_k) / nb::kTile) * s.heads / s.batch;  // or more
  if (n_kt > 1 && steps < 21. * double(sms)) return r;
  r.tiles = n_kt == 1 ? -1 : n_qt < most ? n_qt : most;
  r.own_tiles = n_kt == 1 ? 0 : r.tiles;
  r.rest_offset =
      align_up(bwd_items_offset(s) + size_t(nb::sched_capacity(s.total_k, s.batch)) * sizeof(nb::SchedItem), 256);
  r.own_offset = align_up(r.rest_offset + nb::sched_rest_bytes(s.batch), 256);
  r.bytes = r.own_offset + size_t(sms) * r.own_tiles * nb::kTile * nb::kHeadDim * sizeof(float);
  return r;
}

// Everything about a backward call that can be checked without touching CUDA.
int validate_bwd(const nb_attn_bwd_args* a) {
  if (a == nullptr) return NB_ATTN_ERR_NULL;
  int rc = check_shape(a->shape);
  if (rc) return rc;
  const bool dense = a->shape.cu_seqlens_q == nullptr;
  const nb_attn_tensor* ts[] = {&a->q, &a->k, &a->v, &a->o, &a->d_o, &a->dq, &a->dk, &a->dv};
  for (const nb_attn_tensor* t : ts)
    if ((rc = check_tensor(*t, dense))) return rc;
  if (a->lse == nullptr) return NB_ATTN_ERR_NULL;
  return NB_ATTN_OK;
}

// `a` has passed validate_bwd and the device is ready.
int launch_bwd(const nb_attn_bwd_args* a, void* workspace, size_t workspace_bytes, void* stream) {
  int rc = NB_ATTN_OK;
  const nb_attn_shape& s = a->shape;
  const bool dense = s.cu_seqlens_q == nullptr;
  if (workspace_bytes < nb_attn_bwd_workspace_bytes(&s)) return NB_ATTN_ERR_WORKSPACE;

  CUtensorMap tq, tk, tv, tg, tdq;
  if ((rc = make_tmap(&tq, a->q, s, true)) || (rc = make_tmap(&tk, a->k, s, false)) ||
      (rc = make_tmap(&tv, a->v, s, false)) || (rc = make_tmap(&tg, a->d_o, s, true)) ||
      (rc = make_dq_accum_tmap(&tdq, static_cast<float*>(workspace), s.total_q, s.heads)))
    return rc;

  nb::BwdParams p;
  p.o = static_cast<const __nv_bfloat16*>(a->o.ptr);
  p.d_o = static_cast<const __nv_bfloat16*>(a->d_o.ptr);
  p.o_sb = dense ? a->o.stride_batch : 0;
  p.o_st = a->o.stride_token;
  p.o_sh = a->o.stride_head;
  p.do_sb = dense ? a->d_o.stride_batch : 0;
  p.do_st = a->d_o.stride_token;
  p.do_sh = a->d_o.stride_head;
  p.dq = static_cast<__nv_bfloat16*>(a->dq.ptr);
  p.dk = static_cast<__nv_bfloat16*>(a->dk.ptr);
  p.dv = static_cast<__nv_bfloat16*>(a->dv.ptr);
  p.dq_sb = dense ? a->dq.stride_batch : 0;
  p.dq_st = a->dq.stride_token;
  p.dq_sh = a->dq.stride_head;
  p.dk_sb = dense ? a->dk.stride_batch : 0;
  p.dk_st = a->dk.stride_token;
  p.dk_sh = a->dk.stride_head;
  p.dv_sb = dense ? a->dv.stride_batch : 0;
  p.dv_st = a->dv.stride_token;
  p.dv_sh = a->dv.stride_head;
  p.lse = a->lse;
  p.dq_accum = static_cast<float*>(workspace);
  p.delta = p.dq_accum + size_t(s.total_q) * s.heads * nb::kHeadDim;
  p.cu_q = s.cu_seqlens_q;
  p.cu_k = s.cu_seqlens_k;
  p.batch = s.batch;
  p.heads = s.heads;
  p.lq = s.max_seqlen_q;
  p.lk = s.max_seqlen_k;
  p.total_q = s.total_q;
  p.total_k = s.total_k;
  p.scale = s.scale;
  p.scale_log2 = s.scale * kLog2e;
  p.status = a->status;
  // The main kernel's CTAs are persistent: one per SM, each walking its share of the work units
  // (key tiles x heads x sequences, or work-list entries x heads).
  int64_t n_work = 0;
  p.n_kt = ceil_div(s.max_seqlen_k, nb::kTile);
  p.n_qt = ceil_div(s.max_seqlen_q, nb::kTile);
  p.parts = nullptr;
  const int sms = device_sm_count();
  unsigned ctas = unsigned(sms);
  const BwdRuns runs = bwd_runs(s, sms);
  const bool use_runs = runs.bytes > 0 && workspace_bytes >= runs.bytes;
  p.own = use_runs ? reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + runs.own_offset) : nullptr;
  p.own_tiles = runs.own_tiles;
  p.rest = nullptr;
  if (dense) {
    p.items = nullptr;
    p.sched = nb::SchedParams{};
    n_work = int64_t(p.n_kt) * s.heads * s.batch;
    const BwdSplit split = bwd_split(s, sms);
    if (split.ctas > 0 && workspace_bytes >= split.bytes) {
      const uint32_t steps = uint32_t(n_work * p.n_qt);
      p.parts = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + split.parts_offset);
      ctas = split.ctas;
      p.split_base = steps / ctas, p.split_extra = steps % ctas;
    }
  } else {
    // Block 0 of the prologue builds the list of key tiles; units are items x heads.
    const int64_t n_items = nb::sched_capacity(s.total_k, s.batch);
    nb::SchedItem* items =
        reinterpret_cast<nb::SchedItem*>(static_cast<unsigned char*>(workspace) + bwd_items_offset(s));
    p.items = items;
    p.sched = make_sched(s, 1, items, n_items, a->status);
    p.sched.merged = 1;
    if (use_runs) {
      p.rest = reinterpret_cast<int32_t*>(static_cast<unsigned char*>(workspace) + runs.rest_offset);
      p.sched.run_tiles = runs.tiles, p.sched.sms = int32_t(ctas), p.sched.rest = p.rest;
    }
    n_work = n_items * s.heads;
  }
  p.n_work = int32_t(n_work);
  p.rows32 = s.total_q * s.heads <= INT32_MAX;
  p.div_lq = nb::make_fast_div(uint32_t(s.max_seqlen_q));
  p.div_heads = nb::make_fast_div(uint32_t(s.heads));
  p.div_n_kt = nb::make_fast_div(uint32_t(p.n_kt));
  p.div_n_qt = nb::make_fast_div(uint32_t(p.n_qt));
  const dim3 grid(p.parts == nullptr && n_work < int64_t(ctas) ? unsigned(n_work) : ctas, 1, 1);

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t rows = s.total_q * s.heads;
  const int64_t want_blocks = (rows * 8 + 255) / 256;
  // (With runs a block first looks at all sequences and takes consecutive rows: no more blocks than are resident. 300
  // sequences of 200 tokens gain 4 us by four per SM instead of eight.)
  const int64_t most_blocks = (p.rest != nullptr ? 4 : 16) * int64_t(sms);
  const int aux_blocks = int(want_blocks < most_blocks ? want_blocks : most_blocks);
  p.row_blocks = aux_blocks;
  const int combine_blocks = p.parts != nullptr ? 4 * (int(ctas) - 1) : 0;
  const auto main = p.parts != nullptr ? nb::attn_bwd_kernel<nb::kBwdCut>
                    : use_runs           ? nb::attn_bwd_kernel<nb::kBwdRuns>
                                         : nb::attn_bwd_kernel<nb::kBwdWhole>;
  const auto prologue = use_runs ? nb::attn_bwd_prologue_kernel<true> : nb::attn_bwd_prologue_kernel<false>;
  const auto epilogue = use_runs ? nb::attn_bwd_epilogue_kernel<true> : nb::attn_bwd_epilogue_kernel<false>;
  bool ok = launch(prologue, dim3(aux_blocks), dim3(nb::kAuxThreads), 0, st, p) == cudaSuccess;
  if (a->event_main_begin) cudaEventRecord(static_cast<cudaEvent_t>(a->event_main_begin), st);
  ok = ok && launch(main, grid, dim3(nb::kBwdThreads), nb::kBwdSmemBytes, st, tq, tk, tv, tg, tdq, p) ==
                 cudaSuccess;
  if (a->event_main_end) cudaEventRecord(static_cast<cudaEvent_t>(a->event_main_end), st);
  ok = ok && launch(epilogue, dim3(aux_blocks + combine_blocks), dim3(nb::kAuxThreads), 0, st, p) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();  // leave no sticky "last error" behind for the caller's own checks
    return NB_ATTN_ERR_LAUNCH;
  }
  return cudaGetLastError() == cudaSuccess ? NB_ATTN_OK : NB_ATTN_ERR_LAUNCH;
}

// `listed`: the workspace holds the list of an earlier call.
int run_fwd(const nb_attn_fwd_args* a, bool listed, void* stream) {
  if (a == nullptr) return NB_ATTN_ERR_NULL;
  int rc = check_shape(a->shape);
  if (rc) return rc;
  const nb_attn_shape& s = a->shape;
  const bool dense = s.cu_seqlens_q == nullptr;
  if ((rc = check_tensor(a->q, dense)) || (rc = check_tensor(a->k, dense)) || (rc = check_tensor(a->v, dense)) ||
      (rc = check_tensor(a->o, dense)))
    return rc;
  if (a->lse == nullptr) return NB_ATTN_ERR_NULL;
  const size_t ws_need = nb_attn_fwd_workspace_bytes(&s);
  if (ws_need > 0 && (a->workspace == nullptr || a->workspace_bytes < ws_need ||
                      (reinterpret_cast<uintptr_t>(a->workspace) & 255u) != 0))
    return NB_ATTN_ERR_WORKSPACE;
  if ((rc = ensure_device_ready())) return rc;

  CUtensorMap tq, tk, tv;
  if ((rc = make_tmap(&tq, a->q, s, true)) || (rc = make_tmap(&tk, a->k, s, false)) ||
      (rc = make_tmap(&tv, a->v, s, false)))
    return rc;

  nb::FwdParams p;
  p.o = static_cast<__nv_bfloat16*>(a->o.ptr);
  p.o_sb = dense ? a->o.stride_batch : 0;
  p.o_st = a->o.stride_token;
  p.o_sh = a->o.stride_head;
  p.lse = a->lse;
  p.cu_q = s.cu_seqlens_q;
  p.cu_k = s.cu_seqlens_k;
  p.batch = s.batch;
  p.heads = s.heads;
  p.lq = s.max_seqlen_q;
  p.lk = s.max_seqlen_k;
  p.total_q = s.total_q;
  p.total_k = s.total_k;
  p.scale_log2 = s.scale * kLog2e;
  p.status = a->status;

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  bool ok = true;
  p.items = nullptr;
  p.parts = nullptr;
  p.n_qt = ceil_div(s.max_seqlen_q, nb::kFwdQRows);
  p.n_kt = ceil_div(s.max_seqlen_k, nb::kTile);
  int64_t n_units = int64_t(p.n_qt) * s.heads * s.batch;
  const int sms = device_sm_count();
  unsigned slots = 2 * unsigned(sms);  // CTAs are persistent, two per SM
  if (dense) {
    const FwdSplit split = fwd_split(s, sms);
    if (split.ctas > 0 && a->workspace != nullptr && a->workspace_bytes >= split.bytes &&
        (reinterpret_cast<uintptr_t>(a->workspace) & 255u) == 0) {
      const uint32_t steps = uint32_t(n_units * p.n_kt);
      p.parts = static_cast<float*>(a->workspace);
      slots = split.ctas;
      p.split_base = steps / split.ctas, p.split_extra = steps % split.ctas;
    }
  } else {
    // The scheduler's list of query tiles; a unit is an entry and a head.
    const int64_t n_items = nb::sched_capacity(s.total_q, s.batch);
    nb::SchedItem* items = static_cast<nb::SchedItem*>(a->workspace);
    if (!listed) {
      nb::SchedParams sp = make_sched(s, 0, items, n_items, a->status);
      sp.merged = 1;
      ok = launch(nb::attn_sched_kernel, dim3(1), dim3(nb::kSchedThreads), 0, st, sp) == cudaSuccess;
    }
    p.items = items;
    n_units = n_items * s.heads;
  }
  p.n_units = int32_t(n_units);
  p.div_heads = nb::make_fast_div(uint32_t(s.heads));
  p.div_n_qt = nb::make_fast_div(uint32_t(p.n_qt));
  p.div_n_kt = nb::make_fast_div(uint32_t(p.n_kt));
  const dim3 grid(p.parts != nullptr || n_units > int64_t(slots) ? slots : unsigned(n_units), 1, 1);
  ok = ok && launch(nb::attn_fwd_kernel, grid, dim3(nb::kFwdThreads), nb::kFwdSmemBytes, st, tq, tk, tv, p) == cudaSuccess;
  if (p.parts != nullptr)
    ok = ok && launch(nb::attn_fwd_combine_kernel, dim3(slots - 1, 2), dim3(256), 0, st, p) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    return NB_ATTN_ERR_LAUNCH;
  }
  return cudaGetLastError() == cudaSuccess ? NB_ATTN_OK : NB_ATTN_ERR_LAUNCH;
}

}  // namespace

extern "C" {

int nb_attn_abi_version(void) { return NB_ATTN_ABI_VERSION; }

const char* nb_attn_strerror(int code) {
  switch (code) {
    case NB_ATTN_OK: return "ok";
    case NB_ATTN_ERR_NULL: return "a required pointer is NULL";
    case NB_ATTN_ERR_HEAD_DIM: return "head_dim must be 64";
    case NB_ATTN_ERR_SHAPE: return "invalid or inconsistent sizes";
    case NB_ATTN_ERR_ALIGN: return "pointers must be 16-byte aligned and strides positive multiples of 8 elements";
    case NB_ATTN_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
    case NB_ATTN_ERR_TENSOR_MAP: return "could not encode a TMA tensor map";
    case NB_ATTN_ERR_LAUNCH: return "a CUDA runtime call failed";
    case NB_ATTN_ERR_DEVICE: return "the current device is not an sm_100 GPU";
    case NB_ATTN_ERR_TOO_LARGE:
      return "total_q * heads exceeds NB_ATTN_BUILTIN_SCRATCH_ROWS; use nb_attn_bwd with a caller workspace";
    default: return "unknown error code";
  }
}

size_t nb_attn_bwd_workspace_bytes(const nb_attn_shape* shape) {
  if (shape == nullptr || check_shape(*shape) != NB_ATTN_OK) return 0;
  const nb_attn_shape& s = *shape;
  if (s.cu_seqlens_q == nullptr) return bwd_accum_bytes(s) + bwd_delta_bytes(s);
  return bwd_items_offset(s) + size_t(nb::sched_capacity(s.total_k, s.batch)) * sizeof(nb::SchedItem);
}

size_t nb_attn_bwd_split_workspace_bytes(const nb_attn_shape* shape) {
  if (shape == nullptr || check_shape(*shape) != NB_ATTN_OK || ensure_device_ready() != NB_ATTN_OK) return 0;
  const int sms = device_sm_count();
  return shape->cu_seqlens_q == nullptr ? bwd_split(*shape, sms).bytes : bwd_runs(*shape, sms).bytes;
}

size_t nb_attn_fwd_workspace_bytes(const nb_attn_shape* shape) {
  if (shape == nullptr || check_shape(*shape) != NB_ATTN_OK || shape->cu_seqlens_q == nullptr) return 0;
  return size_t(nb::sched_capacity(shape->total_q, shape->batch)) * sizeof(nb::SchedItem);
}

size_t nb_attn_fwd_split_workspace_bytes(const nb_attn_shape* shape) {
  if (shape == nullptr || check_shape(*shape) != NB_ATTN_OK || ensure_device_ready() != NB_ATTN_OK) return 0;
  return fwd_split(*shape, device_sm_count()).bytes;
}

int nb_attn_fwd(const nb_attn_fwd_args* a, void* stream) { return run_fwd(a, false, stream); }

int nb_attn_fwd_again(const nb_attn_fwd_args* a, void* stream) { return run_fwd(a, true, stream); }

int nb_attn_bwd(const nb_attn_bwd_args* a, void* stream) {
  int rc = validate_bwd(a);
  if (rc) return rc;
  if (a->workspace == nullptr || a->workspace_bytes < nb_attn_bwd_workspace_bytes(&a->shape) ||
      (reinterpret_cast<uintptr_t>(a->workspace) & 255u) != 0)
    return NB_ATTN_ERR_WORKSPACE;
  if ((rc = ensure_device_ready())) return rc;
  return launch_bwd(a, a->workspace, a->workspace_bytes, stream);
}

int nb_attn_bwd_builtin_scratch(const nb_attn_bwd_args* a, void* stream) {
  // Same argument checks, in the same order, as nb_attn_bwd; CUDA is touched only after them.
  int rc = validate_bwd(a);
  if (rc) return rc;
  const nb_attn_shape& s = a->shape;
  if (s.total_q * int64_t(s.heads) > int64_t(NB_ATTN_BUILTIN_SCRATCH_ROWS)) return NB_ATTN_ERR_TOO_LARGE;
  if (s.cu_seqlens_q != nullptr && nb::sched_capacity(s.total_k, s.batch) > int64_t(NB_ATTN_BUILTIN_SCRATCH_ITEMS))
    return NB_ATTN_ERR_TOO_LARGE;
  if ((rc = ensure_device_ready())) return rc;
  void* scratch = nullptr;
  if ((rc = builtin_scratch_address(&scratch))) {
    cudaGetLastError();
    return rc;
  }
  return launch_bwd(a, scratch, kBuiltinScratchBytes, stream);
}

int nb_attn_selftest_mma(int mode, const void* a, const void* b, float* d, int32_t* status, void* stream) {
  if (a == nullptr || b == nullptr || d == nullptr) return NB_ATTN_ERR_NULL;
  if (mode < 0 || mode > 3) return NB_ATTN_ERR_SHAPE;
  if (!aligned16(a) || !aligned16(b)) return NB_ATTN_ERR_ALIGN;
  int rc = ensure_device_ready();
  if (rc) return rc;
  nb::mma_selftest_kernel<<<1, 128, nb::kSelftestSmemBytes, static_cast<cudaStream_t>(stream)>>>(
      mode, static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(b), d, status);
  return cudaGetLastError() == cudaSuccess ? NB_ATTN_OK : NB_ATTN_ERR_LAUNCH;
}

int nb_attn_selftest_wait(uint64_t limit_ns, int32_t* status, int32_t* out, void* stream) {
  if (status == nullptr) return NB_ATTN_ERR_NULL;
  if (limit_ns == 0 || limit_ns > 1000000000ull) return NB_ATTN_ERR_SHAPE;  // at most one second
  int rc = ensure_device_ready();
  if (rc) return rc;
  nb::wait_selftest_kernel<<<1, 128, 0, static_cast<cudaStream_t>(stream)>>>(limit_ns, status, out);
  return cudaGetLastError() == cudaSuccess ? NB_ATTN_OK : NB_ATTN_ERR_LAUNCH;
}

int64_t nb_attn_schedule_capacity(int64_t total_tokens, int32_t batch) {
  if (total_tokens < 0 || batch <= 0) return 0;
  return nb::sched_capacity(total_tokens, batch);
}

int nb_attn_schedule_build(const nb_attn_shape* shape, int side, nb_attn_sched_item* items, int64_t n_items,
                           int32_t* status, void* stream) {
  if (shape == nullptr || items == nullptr) return NB_ATTN_ERR_NULL;
  int rc = check_shape(*shape);
  if (rc) return rc;
  if (shape->cu_seqlens_q == nullptr || (side != 0 && side != 1)) return NB_ATTN_ERR_SHAPE;
  if (n_items < nb::sched_capacity(side == 0 ? shape->total_q : shape->total_k, shape->batch) || n_items > INT32_MAX)
    return NB_ATTN_ERR_WORKSPACE;
  if ((rc = ensure_device_ready())) return rc;
  const nb::SchedParams sp = make_sched(*shape, side, reinterpret_cast<nb::SchedItem*>(items), n_items, status);
  if (launch(nb::attn_sched_kernel, dim3(1), dim3(nb::kSchedThreads), 0, static_cast<cudaStream_t>(stream), sp) !=
      cudaSuccess) {
    cudaGetLastError();
    return NB_ATTN_ERR_LAUNCH;
  }
  return NB_ATTN_OK;
}

int nb_attn_schedule_host(const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k, int32_t batch,
                          int32_t max_seqlen_q, int32_t max_seqlen_k, int64_t total_q, int64_t total_k, int side,
                          nb_attn_sched_item* items_out, int64_t n_items) {
  if (cu_seqlens_q == nullptr || cu_seqlens_k == nullptr || items_out == nullptr) return NB_ATTN_ERR_NULL;
  nb::SchedItem* items = reinterpret_cast<nb::SchedItem*>(items_out);
  if (batch <= 0 || batch > 65534 || (side != 0 && side != 1) || n_items > INT32_MAX) return NB_ATTN_ERR_SHAPE;
  nb_attn_shape s = {};
  s.batch = batch;
  s.max_seqlen_q = max_seqlen_q;
  s.max_seqlen_k = max_seqlen_k;
  s.total_q = total_q;
  s.total_k = total_k;
  s.cu_seqlens_q = cu_seqlens_q;
  s.cu_seqlens_k = cu_seqlens_k;
  const nb::SchedParams sp = make_sched(s, side, items, n_items, nullptr);
  if (n_items < nb::sched_capacity(sp.total_own, batch)) return NB_ATTN_ERR_WORKSPACE;
  // Same classification as the device kernel; buckets in order, sequences ascending inside one.
  std::vector<std::vector<int>> by_bucket(nb::kSchedBuckets);
  for (int i = 0; i <= batch; ++i) {  // i == batch: the rows past the last sequence
    const nb::SchedSeq q = nb::sched_classify(sp, i);
    if (!q.ok) return NB_ATTN_ERR_SHAPE;
    by_bucket[q.bucket].push_back(i);
  }
  int64_t at = 0;
  for (const auto& seqs : by_bucket)
    for (int i : seqs) {
      const nb::SchedSeq q = nb::sched_classify(sp, i);
      for (int t = 0; t < q.full; ++t) items[at++] = nb::sched_item(q, i, t);
    }
  for (const auto& seqs : by_bucket)
    for (int i : seqs) {
      const nb::SchedSeq q = nb::sched_classify(sp, i);
      if (q.ragged) items[at++] = nb::sched_item(q, i, q.full);
    }
  for (; at < n_items; ++at) items[at] = nb::sched_no_item();
  return NB_ATTN_OK;
}

}  // extern "C"
