// The token-wise kernels of include/nb_encoder.h. All of them are bound by memory traffic: a row (or a
// 16-byte piece) is read once, everything that follows is computed in registers and what the next
// matrix product needs is written in its own type. In separate elementwise kernels the same work moved
// the fp32 residual stream and its bf16 copies through memory eleven times per block; here it is six.
#include "../../include/nb_encoder.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/nb_attn.h"
#include "ptx.cuh"

namespace {

constexpr int kWarps = 8;  // rows in flight per block: one warp per row
constexpr int kThreads = kWarps * 32;

int launched() { return cudaGetLastError() == cudaSuccess ? NB_ATTN_OK : NB_ATTN_ERR_LAUNCH; }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack2(uint32_t v) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// A row of `dim` fp32 values in one warp: lane l holds the float4s l, l + 32, ... (kChunks of them).
template <int kChunks>
struct Row {
  float4 v[kChunks];
  __device__ __forceinline__ static bool has(int c, int dim) { return c * 128 + int(threadIdx.x & 31) * 4 < dim; }
  __device__ __forceinline__ static int at(int c) { return c * 128 + int(threadIdx.x & 31) * 4; }
  __device__ __forceinline__ void load(const float* p, int dim) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      v[c] = has(c, dim) ? *reinterpret_cast<const float4*>(p + at(c)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ void add(const float* p, int dim) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (has(c, dim)) {
        const float4 a = *reinterpret_cast<const float4*>(p + at(c));
        v[c].x += a.x, v[c].y += a.y, v[c].z += a.z, v[c].w += a.w;
      }
  }
  __device__ __forceinline__ void add(const __nv_bfloat16* p, int dim) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (has(c, dim)) {
        const uint2 a = *reinterpret_cast<const uint2*>(p + at(c));
        const float2 lo = unpack2(a.x), hi = unpack2(a.y);
        v[c].x += lo.x, v[c].y += lo.y, v[c].z += hi.x, v[c].w += hi.y;
      }
  }
  __device__ __forceinline__ void store(float* p, int dim) const {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (has(c, dim)) *reinterpret_cast<float4*>(p + at(c)) = v[c];
  }
  __device__ __forceinline__ void store(__nv_bfloat16* p, int dim) const {
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (has(c, dim))
        *reinterpret_cast<uint2*>(p + at(c)) = make_uint2(pack2(v[c].x, v[c].y), pack2(v[c].z, v[c].w));
  }
  // LayerNorm in place; the variance from the centred values.
  __device__ __forceinline__ void norm(const nb_enc_norm& n, int dim) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) s += (v[c].x + v[c].y) + (v[c].z + v[c].w);
    const float mean = warp_sum(s) / float(dim);
    float q = 0.f;
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (has(c, dim)) {
        const float a = v[c].x - mean, b = v[c].y - mean, d = v[c].z - mean, e = v[c].w - mean;
        q += (a * a + b * b) + (d * d + e * e);
      }
    const float rstd = rsqrtf(warp_sum(q) / float(dim) + n.eps);
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (has(c, dim)) {
        const float4 g = *reinterpret_cast<const float4*>(n.gamma + at(c));
        const float4 b = *reinterpret_cast<const float4*>(n.beta + at(c));
        v[c].x = (v[c].x - mean) * rstd * g.x + b.x;
        v[c].y = (v[c].y - mean) * rstd * g.y + b.y;
        v[c].z = (v[c].z - mean) * rstd * g.z + b.z;
        v[c].w = (v[c].w - mean) * rstd * g.w + b.w;
      }
  }
};

// Launch with programmatic stream serialization: the kernel's blocks may be resident while its
// predecessor drains; every kernel launched this way begins with griddepcontrol.wait.
template <typename... KArgs, typename... Args>
void launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, void* stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// f(integral_constant<kChunks>) for the smallest kChunks that holds a row of `dim` values.
template <typename F>
int with_chunks(int dim, F f) {
  switch ((dim + 127) / 128) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    default: return NB_ATTN_ERR_SHAPE;
  }
  return launched();
}
bool dim_ok(int dim) { return dim > 0 && dim % 64 == 0 && dim <= NB_ENC_MAX_DIM; }
unsigned row_blocks(int64_t rows) { return unsigned((rows + kWarps - 1) / kWarps); }

// ---- casts -------------------------------------------------------------------------------
constexpr int kCastItems = 96;      // per launch (kernel parameters are limited to 4 KB)
constexpr int kCastChunk = 8192;    // elements per block
struct CastTable {
  nb_enc_cast_item item[kCastItems];
  int32_t first_block[kCastItems + 1];
  int32_t n;
};
__global__ void __launch_bounds__(256) cast_kernel(const __grid_constant__ CastTable t) {
  int lo = 0, hi = t.n - 1;  // the last item that starts at or before this block
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (int(blockIdx.x) >= t.first_block[mid]) lo = mid;
    else hi = mid - 1;
  }
  const nb_enc_cast_item it = t.item[lo];
  const int64_t begin = int64_t(int(blockIdx.x) - t.first_block[lo]) * kCastChunk;
  const int64_t end = begin + kCastChunk < it.n ? begin + kCastChunk : it.n;
  __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(it.dst);
  if ((it.n & 3) == 0) {
#pragma unroll 4
    for (int64_t i = begin + threadIdx.x * 4; i < end; i += 256 * 4) {
      const float4 v = *reinterpret_cast<const float4*>(it.src + i);
      *reinterpret_cast<uint2*>(dst + i) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
    }
  } else {
    for (int64_t i = begin + threadIdx.x; i < end; i += 256) dst[i] = __float2bfloat16(it.src[i]);
  }
}

// ---- selection of in-mask patches ----------------------------------------------------------
struct MaskTable {
  const uint8_t* mask[NB_ENC_MAX_IMAGES];
};
// One block of 1024 threads per image: every thread a run of consecutive patches, one block-wide scan.
__global__ void __launch_bounds__(1024) select_kernel(const __grid_constant__ MaskTable t, int first, int patches,
                                                      int32_t* ids, int32_t* rank, int32_t* counts) {
  __shared__ int warp_total[32];
  const uint8_t* mask = t.mask[blockIdx.x];
  const int64_t image = first + blockIdx.x;
  ids += image * patches, rank += image * patches;
  const int per = (patches + 1023) / 1024;
  const int begin = min(int(threadIdx.x) * per, patches), end = min(begin + per, patches);
  int mine = 0;
  for (int p = begin; p < end; ++p) mine += mask[p] != 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += up;
  }
  if (lane == 31) warp_total[warp] = incl;
  __syncthreads();
  int before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < 32; ++w) {
    if (w < warp) before += warp_total[w];
    total += warp_total[w];
  }
  int at = before + incl - mine;
  for (int p = begin; p < end; ++p) {
    const bool in = mask[p] != 0;
    rank[p] = in ? at : -1;
    if (in) ids[at++] = p;
  }
  if (threadIdx.x == 0) counts[image] = total;
}

__global__ void offsets_kernel(const int32_t* counts, int images, int class_tokens, int32_t* cu, int32_t* cu_r,
                               int32_t* host_counts) {
  int sum = 0;
  for (int i = 0; i < images; ++i) {
    cu[i] = sum, cu_r[i] = sum + class_tokens * i;
    const int n = counts[i];
    host_counts[i] = n;
    sum += n;
  }
  cu[images] = sum, cu_r[images] = sum + class_tokens * images;
}

// ---- gather of the selected patches ---------------------------------------------------------
struct ValueTable {
  const float* values[NB_ENC_MAX_IMAGES];
};
__global__ void __launch_bounds__(kThreads) gather_kernel(const __grid_constant__ ValueTable t, int first, int patches,
                                                          int dim, const int32_t* ids, const int32_t* counts,
                                                          const int32_t* cu, __nv_bfloat16* tokens) {
  const int64_t image = first + blockIdx.y;
  const int j = blockIdx.x * kWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (j >= counts[image]) return;
  const float* src = t.values[blockIdx.y] + int64_t(ids[image * patches + j]) * dim;
  __nv_bfloat16* dst = tokens + (int64_t(cu[image]) + j) * dim;
  for (int i = lane * 4; i < dim; i += 128) {
    const float4 v = *reinterpret_cast<const float4*>(src + i);
    *reinterpret_cast<uint2*>(dst + i) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
  }
}

// ---- embeddings, residual + norm, GELU -------------------------------------------------------
template <int kChunks>
__global__ void __launch_bounds__(kThreads)
    embed_kernel(const __nv_bfloat16* h, const int32_t* ids, const int32_t* cu, const int32_t* cu_r, int images,
                 int patches, int class_tokens, int64_t rows, int dim, const int64_t* coord, const float* table_x,
                 const float* table_y, const float* table_z, const float* cls, float* x, nb_enc_norm norm,
                 __nv_bfloat16* y) {
  const int64_t row = int64_t(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  int lo = 0, hi = images - 1;  // the last image that starts at or before this row
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (row >= cu_r[mid]) lo = mid;
    else hi = mid - 1;
  }
  const int local = int(row - cu_r[lo]) - class_tokens;
  Row<kChunks> r;
  if (local < 0) {
    r.load(cls + int64_t(local + class_tokens) * dim, dim);
  } else {
    const int64_t* c = coord + int64_t(ids[int64_t(lo) * patches + local]) * 3;
    r.load(table_x + c[0] * dim, 0);  // zeros
    r.add(h + (int64_t(cu[lo]) + local) * dim, dim);
    r.add(table_x + c[0] * dim, dim);
    r.add(table_y + c[1] * dim, dim);
    r.add(table_z + c[2] * dim, dim);
  }
  r.store(x + row * dim, dim);
  r.norm(norm, dim);
  r.store(y + row * dim, dim);
}

template <int kChunks>
__global__ void __launch_bounds__(kThreads)
    add_norm_kernel(float* x, const __nv_bfloat16* add, int64_t rows, int dim, nb_enc_norm norm, __nv_bfloat16* y) {
  nb::pdl_wait();
  nb::pdl_launch_dependents();
  const int64_t row = int64_t(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  Row<kChunks> r;
  r.load(x + row * dim, dim);
  r.add(add + row * dim, dim);
  r.store(x + row * dim, dim);
  r.norm(norm, dim);
  r.store(y + row * dim, dim);
}

// GELU of bf16 values through a table in shared memory. Bound by instructions otherwise: 14 000 x 3072
// values took 47 us with erff for each, 31 us with a rational approximation (and other roundings than the
// modules' GELU); from the table 34.6 us, 26 of them memory traffic. Only 17 binary exponents need
// entries, 2^-14 <= |v| < 8: above them the result is v or -0, below them v / 2 (both exactly what the
// formula gives). Every block makes its own table, so a thread should have a few hundred values to look
// up: below kGeluTableMin elements the formula is evaluated directly, with the same results.
__device__ __forceinline__ float gelu(float v) { return v * 0.5f * (1.f + erff(v * 0.70710678118654752f)); }
constexpr uint32_t kGeluFirst = 113u << 7, kGeluCodes = 17u << 7;  // bf16 bits of 2^-14; codes per sign
constexpr int64_t kGeluTableMin = int64_t(1) << 22;
__device__ __forceinline__ uint32_t gelu_bits(uint32_t code) {
  const __nv_bfloat16 r = __float2bfloat16(gelu(__uint_as_float(code << 16)));
  return *reinterpret_cast<const uint16_t*>(&r);
}
template <bool kTable>
__global__ void __launch_bounds__(512) gelu_kernel(__nv_bfloat16* v, int64_t n) {
  __shared__ uint16_t table[kTable ? 2 * kGeluCodes : 1];
  if (kTable) {
    for (uint32_t i = threadIdx.x; i < 2 * kGeluCodes; i += 512)
      table[i] = uint16_t(gelu_bits(i < kGeluCodes ? kGeluFirst + i : 0x8000u + kGeluFirst + (i - kGeluCodes)));
    __syncthreads();
  }
  nb::pdl_wait();
  nb::pdl_launch_dependents();
  auto one = [&](uint32_t code) -> uint32_t {
    const uint32_t at = (code & 0x7fffu) - kGeluFirst;
    if (kTable && at < kGeluCodes) return table[at + (code >> 15) * kGeluCodes];
    return gelu_bits(code);
  };
  auto eight = [&](uint4 u) {
    uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = one(w[k] & 0xffffu) | one(w[k] >> 16) << 16;
    return u;
  };
  // Two pieces at a time: the second one's load is under way while the first is looked up.
  const int64_t step = int64_t(gridDim.x) * 512 * 8;
#pragma unroll 1
  for (int64_t i = (int64_t(blockIdx.x) * 512 + threadIdx.x) * 8; i < n; i += 2 * step) {
    const bool two = i + step < n;
    const uint4 a = *reinterpret_cast<const uint4*>(v + i);
    uint4 b = make_uint4(0, 0, 0, 0);
    if (two) b = *reinterpret_cast<const uint4*>(v + i + step);
    *reinterpret_cast<uint4*>(v + i) = eight(a);
    if (two) *reinterpret_cast<uint4*>(v + i + step) = eight(b);
  }
}

// ---- final norm: dense grid and mean ----------------------------------------------------------
constexpr int kFinishPatches = 64;  // patches per block, eight per warp
struct DenseTable {
  float* dense[NB_ENC_MAX_IMAGES];
};
template <int kChunks>
__global__ void __launch_bounds__(kThreads)
    finish_kernel(const float* x, const __nv_bfloat16* add, const int32_t* rank, const int32_t* cu_r, int first,
                  int patches, int class_tokens, int dim, nb_enc_norm norm, const __grid_constant__ DenseTable t,
                  float* partial) {
  __shared__ float4 sums[kWarps][32];
  const int64_t image = first + blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* dense = t.dense[blockIdx.y];
  Row<kChunks> total;
  total.load(x, 0);  // zeros
  for (int k = 0; k < kFinishPatches / kWarps; ++k) {
    const int p = blockIdx.x * kFinishPatches + k * kWarps + warp;
    if (p >= patches) break;
    const int at = rank[image * patches + p];
    Row<kChunks> r;
    if (at >= 0) {
      const int64_t row = int64_t(cu_r[image]) + class_tokens + at;
      r.load(x + row * dim, dim);
      r.add(add + row * dim, dim);
      r.norm(norm, dim);
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
        total.v[c].x += r.v[c].x, total.v[c].y += r.v[c].y, total.v[c].z += r.v[c].z, total.v[c].w += r.v[c].w;
    } else {
      r.load(x, 0);
    }
    if (dense != nullptr) r.store(dense + int64_t(p) * dim, dim);
  }
  float* out = partial + (int64_t(blockIdx.y) * gridDim.x + blockIdx.x) * dim;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    sums[warp][lane] = total.v[c];
    __syncthreads();
    if (warp == 0 && Row<kChunks>::has(c, dim)) {
      float4 s = sums[0][lane];
#pragma unroll
      for (int w = 1; w < kWarps; ++w) {
        const float4 a = sums[w][lane];
        s.x += a.x, s.y += a.y, s.z += a.z, s.w += a.w;
      }
      *reinterpret_cast<float4*>(out + Row<kChunks>::at(c)) = s;
    }
    __syncthreads();
  }
}
// One block per image and 64 columns: four threads per column share the partial sums.
__global__ void __launch_bounds__(256) mean_kernel(const float* partial, int blocks, int dim, const int32_t* counts,
                                                   int first, float* means) {
  __shared__ float sums[4][64];
  const int64_t image = first + blockIdx.x;
  const int d = blockIdx.y * 64 + (threadIdx.x & 63), part = threadIdx.x >> 6;
  float s = 0.f;
#pragma unroll 8
  for (int b = part; b < blocks; b += 4) s += partial[(int64_t(blockIdx.x) * blocks + b) * dim + d];
  sums[part][threadIdx.x & 63] = s;
  __syncthreads();
  if (part == 0) {
    s = (sums[0][threadIdx.x] + sums[1][threadIdx.x]) + (sums[2][threadIdx.x] + sums[3][threadIdx.x]);
    means[image * dim + d] = s / float(counts[image] > 1 ? counts[image] : 1);
  }
}

}  // namespace

extern "C" {

int nb_enc_cast(const nb_enc_cast_item* items, int n_items, void* stream) {
  if (items == nullptr || n_items < 0) return NB_ATTN_ERR_NULL;
  for (int i = 0; i < n_items; ++i) {
    if (items[i].src == nullptr || items[i].dst == nullptr) return NB_ATTN_ERR_NULL;
    if (!aligned16(items[i].src) || (reinterpret_cast<uintptr_t>(items[i].dst) & 7u) != 0) return NB_ATTN_ERR_ALIGN;
    if (items[i].n <= 0 || items[i].n > (int64_t(1) << 40)) return NB_ATTN_ERR_SHAPE;
  }
  for (int at = 0; at < n_items; at += kCastItems) {
    CastTable t;
    t.n = n_items - at < kCastItems ? n_items - at : kCastItems;
    int64_t blocks = 0;
    for (int i = 0; i < t.n; ++i) {
      t.item[i] = items[at + i];
      t.first_block[i] = int32_t(blocks);
      blocks += (items[at + i].n + kCastChunk - 1) / kCastChunk;
      if (blocks > INT32_MAX) return NB_ATTN_ERR_SHAPE;
    }
    cast_kernel<<<unsigned(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(t);
    if (const int rc = launched()) return rc;
  }
  return NB_ATTN_OK;
}

int nb_enc_select(const uint8_t* const* masks, int first, int n, int patches, int32_t* ids, int32_t* rank,
                  int32_t* counts, void* stream) {
  if (masks == nullptr || ids == nullptr || rank == nullptr || counts == nullptr) return NB_ATTN_ERR_NULL;
  if (n <= 0 || n > NB_ENC_MAX_IMAGES || patches <= 0 || first < 0) return NB_ATTN_ERR_SHAPE;
  MaskTable t;
  for (int i = 0; i < n; ++i)
    if ((t.mask[i] = masks[i]) == nullptr) return NB_ATTN_ERR_NULL;
  select_kernel<<<n, 1024, 0, static_cast<cudaStream_t>(stream)>>>(t, first, patches, ids, rank, counts);
  return launched();
}

int nb_enc_offsets(const int32_t* counts, int images, int class_tokens, int32_t* cu, int32_t* cu_r,
                   int32_t* host_counts, void* stream) {
  if (counts == nullptr || cu == nullptr || cu_r == nullptr || host_counts == nullptr) return NB_ATTN_ERR_NULL;
  if (images <= 0 || class_tokens < 0) return NB_ATTN_ERR_SHAPE;
  offsets_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(counts, images, class_tokens, cu, cu_r, host_counts);
  return launched();
}

int nb_enc_gather(const float* const* values, int first, int n, int patches, int dim, const int32_t* ids,
                  const int32_t* counts, const int32_t* cu, void* tokens, void* stream) {
  if (values == nullptr || ids == nullptr || counts == nullptr || cu == nullptr || tokens == nullptr)
    return NB_ATTN_ERR_NULL;
  if (n <= 0 || n > NB_ENC_MAX_IMAGES || patches <= 0 || first < 0 || dim <= 0 || dim % 4 != 0) return NB_ATTN_ERR_SHAPE;
  ValueTable t;
  for (int i = 0; i < n; ++i) {
    if ((t.values[i] = values[i]) == nullptr) return NB_ATTN_ERR_NULL;
    if (!aligned16(values[i])) return NB_ATTN_ERR_ALIGN;
  }
  gather_kernel<<<dim3(row_blocks(patches), n), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      t, first, patches, dim, ids, counts, cu, static_cast<__nv_bfloat16*>(tokens));
  return launched();
}

int nb_enc_embed(const void* h, const int32_t* ids, const int32_t* cu, const int32_t* cu_r, int images, int patches,
                 int class_tokens, int64_t rows, int dim, const int64_t* coord, const float* table_x,
                 const float* table_y, const float* table_z, const float* cls, float* x, const nb_enc_norm* norm,
                 void* y, void* stream) {
  if (h == nullptr || ids == nullptr || cu == nullptr || cu_r == nullptr || coord == nullptr || table_x == nullptr ||
      table_y == nullptr || table_z == nullptr || (cls == nullptr && class_tokens > 0) || x == nullptr ||
      norm == nullptr || y == nullptr)
    return NB_ATTN_ERR_NULL;
  if (!dim_ok(dim) || rows <= 0 || images <= 0 || patches <= 0 || class_tokens < 0) return NB_ATTN_ERR_SHAPE;
  return with_chunks(dim, [&](auto c) {
    embed_kernel<decltype(c)::value><<<row_blocks(rows), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(h), ids, cu, cu_r, images, patches, class_tokens, rows, dim, coord, table_x,
        table_y, table_z, cls, x, *norm, static_cast<__nv_bfloat16*>(y));
  });
}

int nb_enc_add_norm(float* x, const void* add, int64_t rows, int dim, const nb_enc_norm* norm, void* y, void* stream) {
  if (x == nullptr || add == nullptr || norm == nullptr || y == nullptr) return NB_ATTN_ERR_NULL;
  if (!dim_ok(dim) || rows <= 0) return NB_ATTN_ERR_SHAPE;
  return with_chunks(dim, [&](auto c) {
    launch(add_norm_kernel<decltype(c)::value>, dim3(row_blocks(rows)), dim3(kThreads), stream, x,
           static_cast<const __nv_bfloat16*>(add), rows, dim, *norm, static_cast<__nv_bfloat16*>(y));
  });
}

int nb_enc_gelu(void* v, int64_t n, void* stream) {
  if (v == nullptr) return NB_ATTN_ERR_NULL;
  if (!aligned16(v)) return NB_ATTN_ERR_ALIGN;
  if (n <= 0 || n % 8 != 0) return NB_ATTN_ERR_SHAPE;
  const int64_t blocks = (n / 8 + 511) / 512;
  const bool table = n >= kGeluTableMin;  // four resident blocks on each of 148 SMs then walk the array
  launch(table ? gelu_kernel<true> : gelu_kernel<false>, dim3(unsigned(table ? (blocks < 592 ? blocks : 592) : blocks)),
         dim3(512), stream, static_cast<__nv_bfloat16*>(v), n);
  return launched();
}

size_t nb_enc_finish_scratch_bytes(int n, int patches, int dim) {
  if (n <= 0 || patches <= 0 || !dim_ok(dim)) return 0;
  return size_t(n) * size_t((patches + kFinishPatches - 1) / kFinishPatches) * size_t(dim) * sizeof(float);
}

int nb_enc_finish(const float* x, const void* add, const int32_t* rank, const int32_t* counts, const int32_t* cu_r,
                  int first, int n, int patches, int class_tokens, int dim, const nb_enc_norm* norm,
                  float* const* dense, float* means, void* scratch, void* stream) {
  if (x == nullptr || add == nullptr || rank == nullptr || counts == nullptr || cu_r == nullptr || norm == nullptr ||
      means == nullptr || scratch == nullptr)
    return NB_ATTN_ERR_NULL;
  if (!dim_ok(dim) || n <= 0 || n > NB_ENC_MAX_IMAGES || patches <= 0 || first < 0 || class_tokens < 0)
    return NB_ATTN_ERR_SHAPE;
  DenseTable t;
  for (int i = 0; i < n; ++i) t.dense[i] = dense == nullptr ? nullptr : dense[i];
  const int blocks = (patches + kFinishPatches - 1) / kFinishPatches;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* partial = static_cast<float*>(scratch);
  const int rc = with_chunks(dim, [&](auto c) {
    finish_kernel<decltype(c)::value><<<dim3(blocks, n), kThreads, 0, st>>>(
        x, static_cast<const __nv_bfloat16*>(add), rank, cu_r, first, patches, class_tokens, dim, *norm, t, partial);
  });
  if (rc) return rc;
  mean_kernel<<<dim3(n, dim / 64), 256, 0, st>>>(partial, blocks, dim, counts, first, means);
  return launched();
}

}  // extern "C"
