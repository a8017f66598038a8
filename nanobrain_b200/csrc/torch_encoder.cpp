// The packed inference encoder (ViTMAE3D.embed_packed) in native code: selection and gather of the
// in-mask patches, embeddings, the block loop and the final norm, over the kernels of nb_encoder.h, the
// attention of nb_attn.h and library GEMMs for the Linears.
//
// Why: module by module a pass over twelve blocks cost the host 5.2 ms (about forty Python-level calls
// and 195 casts of weights, biases and activations per pass, and a synchronisation per image), whatever
// the number of images, and the casts and elementwise kernels were half of the GPU's 8 ms on eight images. Here the weights are cast
// by one kernel per 96 tensors, Q, K and V are one product, residual additions, LayerNorms and the
// casts around them are one kernel each, and the only synchronisation is for the patch counts.
//
// Precision is that of the modules under bf16 autocast: fp32 residual stream and LayerNorm, bf16
// operands and results of the Linears, exact GELU evaluated in fp32 on the bf16 values.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>

#include <exception>
#include <optional>
#include <vector>

#include "../../include/nb_encoder.h"
#include "torch_common.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

constexpr int kBlockParams = 16;  // norm1 w b, q w b, k w b, v w b, proj w b, norm2 w b, fc1 w b, fc2 w b
constexpr int64_t kHeadDim = 64;

// Can the kernels read this tensor in place: plain contiguous fp32 on one device, 16-byte aligned?
bool readable(const Tensor& t, const Tensor& like) {
  return t.scalar_type() == at::kFloat && t.device() == like.device() && t.layout() == at::kStrided &&
         !t.unsafeGetTensorImpl()->is_python_dispatch() && t.has_storage() && !t.is_neg() && t.is_contiguous() &&
         (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) == 0;
}

// Are these parameters, in the order of encode_images, what it takes? (Anything else is for the modules.)
bool takes_params(const std::vector<OptTensor>& stem, const std::vector<OptTensor>& blocks) {
  if (stem.size() != 8 || blocks.empty() || blocks.size() % kBlockParams != 0 || !stem[2].has_value()) return false;
  const Tensor& like = *stem[2];
  if (like.dim() != 2) return false;
  const int64_t dim = like.size(1);
  for (const auto* list : {&stem, &blocks})
    for (const OptTensor& t : *list)
      if (t.has_value() && !readable(*t, like)) return false;
  auto is = [](const OptTensor& t, at::IntArrayRef sizes) { return t.has_value() && t->sizes() == sizes; };
  auto absent_or = [&](const OptTensor& t, at::IntArrayRef sizes) { return !t.has_value() || t->sizes() == sizes; };
  auto matrix = [](const OptTensor& t) { return t.has_value() && t->dim() == 2; };
  auto norm = [&](const OptTensor& w, const OptTensor& b) { return is(w, {dim}) && is(b, {dim}); };
  if (!matrix(stem[0]) || stem[0]->size(0) != dim || !absent_or(stem[1], {dim}) || !norm(stem[6], stem[7])) return false;
  for (int i : {3, 4})
    if (!matrix(stem[i]) || stem[i]->size(1) != dim) return false;
  if (stem[5].has_value() && (stem[5]->dim() != 3 || stem[5]->size(0) != 1 || stem[5]->size(2) != dim)) return false;
  for (size_t at = 0; at < blocks.size(); at += kBlockParams) {
    const OptTensor* b = blocks.data() + at;
    for (int i : {2, 4, 6, 8})
      if (!is(b[i], {dim, dim}) || !absent_or(b[i + 1], {dim})) return false;
    if (b[3].has_value() != b[5].has_value() || b[3].has_value() != b[7].has_value()) return false;
    if (!norm(b[0], b[1]) || !norm(b[10], b[11]) || !matrix(b[12])) return false;
    const int64_t hidden = b[12]->size(0);
    if (hidden % 8 != 0 || !is(b[12], {hidden, dim}) || !absent_or(b[13], {hidden})) return false;
    if (!is(b[14], {dim, hidden}) || !absent_or(b[15], {dim})) return false;
  }
  return true;
}

void check_param(const Tensor& t, const Tensor& like) {
  TORCH_CHECK(readable(t, like), "nanobrain_b200 encoder: parameters must be contiguous float32 on one device");
}

// bf16 copies of fp32 parameters in one buffer, cast together.
struct Casts {
  struct Slot {
    int64_t offset = -1;
    std::vector<int64_t> shape;
  };
  std::vector<nb_enc_cast_item> items;
  std::vector<int64_t> offsets;
  int64_t total = 0;
  Tensor buffer;

  // The rows of `parts` one after the other; parts are all there or all absent (a missing bias).
  Slot add(std::initializer_list<const OptTensor*> parts, const Tensor& like) {
    Slot s;
    if (!(*parts.begin())->has_value()) return s;
    total = (total + 7) / 8 * 8;
    s.offset = total;
    for (const OptTensor* part : parts) {
      TORCH_CHECK(part->has_value(), "nanobrain_b200 encoder: biases of q, k and v must be all there or all absent");
      const Tensor& t = **part;
      check_param(t, like);
      if (s.shape.empty()) s.shape = t.sizes().vec();
      else s.shape[0] += t.size(0);
      items.push_back({t.data_ptr<float>(), nullptr, t.numel()});
      offsets.push_back(total);
      total += t.numel();
    }
    return s;
  }
  void allocate(const Tensor& like) {
    buffer = at::empty({total}, like.options().dtype(at::kBFloat16));
    auto* base = static_cast<at::BFloat16*>(buffer.data_ptr());
    for (size_t i = 0; i < items.size(); ++i) items[i].dst = base + offsets[i];
  }
  void run(cudaStream_t stream) const {
    nbt::check_rc(nb_enc_cast(items.data(), int(items.size()), stream), "nb_enc_cast");
  }
  Tensor view(int64_t offset, at::IntArrayRef sizes, at::IntArrayRef strides) const {
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(buffer.storage()),
                                                        buffer.key_set(), buffer.dtype());
    t.unsafeGetTensorImpl()->set_sizes_and_strides(sizes, strides, offset);
    return t;
  }
};

// Waits for a stream at the end of a scope that is left by an exception.
struct Finished {
  cudaStream_t stream;
  const int exceptions = std::uncaught_exceptions();
  ~Finished() {
    if (std::uncaught_exceptions() > exceptions) cudaStreamSynchronize(stream);
  }
};

// x W^T + b, with the views of W^T and b made once per pass without the dispatcher: narrow, view, t and
// linear were five dispatched calls per product, a fifth of the host's time for a pass.
struct Product {
  Tensor wt, b;
  Product(const Casts& casts, const Casts::Slot& w, const Casts::Slot& bias) {
    const int64_t out = w.shape[0], in = w.shape[1];
    wt = casts.view(w.offset, {in, out}, {1, in});
    if (bias.offset >= 0) b = casts.view(bias.offset, {out}, {1});
  }
  Tensor operator()(const Tensor& x) const { return b.defined() ? at::addmm(b, x, wt) : at::mm(x, wt); }
};

struct BlockWeights {
  Casts::Slot wqkv, bqkv, wproj, bproj, w1, b1, w2, b2;
};

nb_enc_norm make_norm(const OptTensor& w, const OptTensor& b, double eps, const Tensor& like) {
  TORCH_CHECK(w.has_value() && b.has_value(), "nanobrain_b200 encoder: LayerNorm needs weight and bias");
  check_param(*w, like), check_param(*b, like);
  return {w->data_ptr<float>(), b->data_ptr<float>(), float(eps)};
}

// Returns (means [N, D], one dense [P, D] tensor per image or an empty list).
std::tuple<Tensor, std::vector<Tensor>> encode_images(const std::vector<Tensor>& patches,
                                                      const std::vector<Tensor>& masks, const Tensor& coord,
                                                      const std::vector<OptTensor>& stem,
                                                      const std::vector<OptTensor>& blocks,
                                                      const std::vector<double>& eps, int64_t heads,
                                                      bool return_dense) {
  const int64_t n_images = int64_t(patches.size()), n_patches = coord.size(0);
  TORCH_CHECK(n_images > 0 && masks.size() == patches.size() && stem.size() == 8 && !blocks.empty() &&
                  blocks.size() % kBlockParams == 0,
              "nanobrain_b200 encoder: inconsistent arguments");
  const int64_t depth = int64_t(blocks.size()) / kBlockParams;
  TORCH_CHECK(int64_t(eps.size()) == 2 * depth + 1, "nanobrain_b200 encoder: inconsistent arguments");
  const Tensor& table_x = *stem[2];
  const c10::cuda::CUDAGuard guard(table_x.device());
  const c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
  cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
  const int64_t dim = table_x.size(1), patch_dim = patches[0].size(1);
  const auto f32 = table_x.options(), bf16 = f32.dtype(at::kBFloat16), i32 = f32.dtype(at::kInt);
  TORCH_CHECK(coord.device() == table_x.device() && coord.scalar_type() == at::kLong && coord.is_contiguous(),
              "nanobrain_b200 encoder: coordinates must be contiguous int64 on the parameters' device");

  // In-mask patches of every image.
  std::vector<const uint8_t*> mask_ptrs;
  std::vector<const float*> patch_ptrs;
  for (int64_t i = 0; i < n_images; ++i) {
    const Tensor &m = masks[i], &p = patches[i];
    TORCH_CHECK(m.device() == table_x.device() && m.scalar_type() == at::kBool && m.is_contiguous() &&
                    m.numel() == n_patches && p.device() == table_x.device() && p.scalar_type() == at::kFloat &&
                    p.is_contiguous() && p.dim() == 2 && p.size(0) == n_patches && p.size(1) == patch_dim,
                "nanobrain_b200 encoder: every image needs contiguous float32 patches and a bool mask");
    mask_ptrs.push_back(static_cast<const uint8_t*>(m.data_ptr()));
    patch_ptrs.push_back(p.data_ptr<float>());
  }
  const bool has_cls = stem[5].has_value();
  const int class_tokens = has_cls ? int(stem[5]->size(-2)) : 0;
  // What can be wrong with the parameters is found before anything is launched.
  Casts casts;
  const auto w_patch = casts.add({&stem[0]}, table_x), b_patch = casts.add({&stem[1]}, table_x);
  std::vector<BlockWeights> weights(depth);
  std::vector<nb_enc_norm> norms;  // norm1 and norm2 of every block, then the final one
  for (int64_t i = 0; i < depth; ++i) {
    const OptTensor* b = blocks.data() + i * kBlockParams;
    BlockWeights& w = weights[i];
    w.wqkv = casts.add({&b[2], &b[4], &b[6]}, table_x), w.bqkv = casts.add({&b[3], &b[5], &b[7]}, table_x);
    w.wproj = casts.add({&b[8]}, table_x), w.bproj = casts.add({&b[9]}, table_x);
    w.w1 = casts.add({&b[12]}, table_x), w.b1 = casts.add({&b[13]}, table_x);
    w.w2 = casts.add({&b[14]}, table_x), w.b2 = casts.add({&b[15]}, table_x);
    norms.push_back(make_norm(b[0], b[1], eps[2 * i], table_x));
    norms.push_back(make_norm(b[10], b[11], eps[2 * i + 1], table_x));
  }
  norms.push_back(make_norm(stem[6], stem[7], eps[2 * depth], table_x));
  for (int i : {2, 3, 4}) check_param(*stem[i], table_x);
  if (has_cls) check_param(*stem[5], table_x);
  casts.allocate(table_x);
  const Product patch_product(casts, w_patch, b_patch);
  std::vector<Product> products;
  products.reserve(4 * depth);
  for (const BlockWeights& w : weights) {
    products.emplace_back(casts, w.wqkv, w.bqkv);
    products.emplace_back(casts, w.wproj, w.bproj);
    products.emplace_back(casts, w.w1, w.b1);
    products.emplace_back(casts, w.w2, w.b2);
  }

  Tensor ids = at::empty({n_images, n_patches}, i32), rank = at::empty({n_images, n_patches}, i32);
  Tensor counts = at::empty({n_images}, i32), cu = at::empty({n_images + 1}, i32), cu_r = at::empty({n_images + 1}, i32);
  // A kernel writes the counts into pinned host memory, which the caching host allocator may hand out again as soon as
  // the tensor is gone: whichever way this function is left, the write has happened before that.
  Tensor host_counts = at::empty({n_images}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
  const Finished counts_written{stream};
  auto chunks = [&](auto f) {
    for (int64_t at = 0; at < n_images; at += NB_ENC_MAX_IMAGES)
      f(int(at), int(std::min<int64_t>(NB_ENC_MAX_IMAGES, n_images - at)));
  };
  chunks([&](int first, int n) {
    nbt::check_rc(nb_enc_select(mask_ptrs.data() + first, first, n, int(n_patches), ids.data_ptr<int32_t>(),
                                rank.data_ptr<int32_t>(), counts.data_ptr<int32_t>(), stream),
                  "nb_enc_select");
  });
  nbt::check_rc(nb_enc_offsets(counts.data_ptr<int32_t>(), int(n_images), class_tokens, cu.data_ptr<int32_t>(),
                               cu_r.data_ptr<int32_t>(), host_counts.data_ptr<int32_t>(), stream),
                "nb_enc_offsets");
  at::cuda::CUDAEvent counted;
  counted.record(at::cuda::getCurrentCUDAStream());
  casts.run(stream);  // while the host waits for the counts

  counted.synchronize();
  const int32_t* n_tokens = host_counts.data_ptr<int32_t>();
  int64_t tokens = 0, longest = 0;
  for (int64_t i = 0; i < n_images; ++i) {
    TORCH_CHECK_VALUE(n_tokens[i] > 0, "every image needs at least one in-mask patch");
    tokens += n_tokens[i];
    longest = std::max<int64_t>(longest, n_tokens[i]);
  }
  const int64_t rows = tokens + class_tokens * n_images;

  Tensor x = at::empty({rows, dim}, f32), y = at::empty({rows, dim}, bf16);
  {
    Tensor packed = at::empty({tokens, patch_dim}, bf16);
    chunks([&](int first, int n) {
      nbt::check_rc(nb_enc_gather(patch_ptrs.data() + first, first, n, int(n_patches), int(patch_dim),
                                  ids.data_ptr<int32_t>(), counts.data_ptr<int32_t>(), cu.data_ptr<int32_t>(),
                                  packed.data_ptr(), stream),
                    "nb_enc_gather");
    });
    const Tensor h = patch_product(packed);
    nbt::check_rc(nb_enc_embed(h.data_ptr(), ids.data_ptr<int32_t>(), cu.data_ptr<int32_t>(), cu_r.data_ptr<int32_t>(),
                               int(n_images), int(n_patches), class_tokens, rows, int(dim), coord.data_ptr<int64_t>(),
                               table_x.data_ptr<float>(), stem[3]->data_ptr<float>(), stem[4]->data_ptr<float>(),
                               has_cls ? stem[5]->data_ptr<float>() : nullptr, x.data_ptr<float>(), &norms[0],
                               y.data_ptr(), stream),
                  "nb_enc_embed");
  }

  nb_attn_fwd_args a{};
  a.shape.batch = int32_t(n_images), a.shape.heads = int32_t(heads), a.shape.head_dim = int32_t(kHeadDim);
  a.shape.max_seqlen_q = a.shape.max_seqlen_k = int32_t(longest + class_tokens);
  a.shape.total_q = a.shape.total_k = rows;
  a.shape.cu_seqlens_q = a.shape.cu_seqlens_k = cu_r.data_ptr<int32_t>();
  a.shape.scale = 0.125f;
  volatile int32_t* word = nbt::status_ptr(table_x.get_device());
  nbt::raise_for_status(word);
  a.status = const_cast<int32_t*>(word);
  a.workspace_bytes = nb_attn_fwd_workspace_bytes(&a.shape);
  Tensor workspace = at::empty({int64_t(a.workspace_bytes)}, f32.dtype(at::kByte));
  Tensor attn = at::empty({rows, dim}, bf16), lse = at::empty({heads, rows}, f32);
  a.workspace = workspace.data_ptr();
  a.lse = lse.data_ptr<float>();
  a.o = {attn.data_ptr(), 0, dim, kHeadDim};
  Tensor branch;
  for (int64_t i = 0; i < depth; ++i) {
    const Product* w = products.data() + 4 * i;
    const Tensor qkv = w[0](y);
    auto* base = static_cast<at::BFloat16*>(qkv.data_ptr());
    a.q = {base, 0, 3 * dim, kHeadDim};
    a.k = {base + dim, 0, 3 * dim, kHeadDim};
    a.v = {base + 2 * dim, 0, 3 * dim, kHeadDim};
    // The blocks share one work list: building it took 4.5 us of each, on one SM.
    nbt::check_rc(i == 0 ? nb_attn_fwd(&a, stream) : nb_attn_fwd_again(&a, stream), "nb_attn_fwd");
    branch = w[1](attn);
    nbt::check_rc(nb_enc_add_norm(x.data_ptr<float>(), branch.data_ptr(), rows, int(dim), &norms[2 * i + 1],
                                  y.data_ptr(), stream),
                  "nb_enc_add_norm");
    const Tensor hidden = w[2](y);
    nbt::check_rc(nb_enc_gelu(hidden.data_ptr(), hidden.numel(), stream), "nb_enc_gelu");
    branch = w[3](hidden);
    if (i + 1 < depth)
      nbt::check_rc(nb_enc_add_norm(x.data_ptr<float>(), branch.data_ptr(), rows, int(dim), &norms[2 * i + 2],
                                    y.data_ptr(), stream),
                    "nb_enc_add_norm");
  }
  nbt::after_launch(word);

  Tensor means = at::empty({n_images, dim}, f32);
  std::vector<Tensor> dense;
  std::vector<float*> dense_ptrs(n_images, nullptr);
  if (return_dense)
    for (int64_t i = 0; i < n_images; ++i) {
      dense.push_back(at::empty({n_patches, dim}, f32));
      dense_ptrs[i] = dense.back().data_ptr<float>();
    }
  chunks([&](int first, int n) {
    Tensor scratch = at::empty({int64_t(nb_enc_finish_scratch_bytes(n, int(n_patches), int(dim)))}, f32.dtype(at::kByte));
    nbt::check_rc(nb_enc_finish(x.data_ptr<float>(), branch.data_ptr(), rank.data_ptr<int32_t>(),
                                counts.data_ptr<int32_t>(), cu_r.data_ptr<int32_t>(), first, n, int(n_patches),
                                class_tokens, int(dim), &norms[2 * depth], dense_ptrs.data() + first,
                                means.data_ptr<float>(), scratch.data_ptr(), stream),
                  "nb_enc_finish");
  });
  return {std::move(means), std::move(dense)};
}

}  // namespace

namespace nbt {

void bind_encoder(pybind11::module_& m) {
  m.def("takes_params", &takes_params);
  m.def("encode_images", &encode_images, pybind11::call_guard<pybind11::gil_scoped_release>());
}

}  // namespace nbt
