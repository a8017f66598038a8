// PyTorch side of the operator in native code: the CUDA and autograd kernels of the four
// nanobrain_b200::* ops (their schemas and fake kernels are declared in ops.py) and the two entry
// points that Python calls.
//
// Why native: a small attention call is bound by host work. With the ops' bodies in Python (argument
// checks, ctypes structures, the Python autograd function and the custom-op wrapper around each) one
// forward + backward cost the host 297 us for 12 us of GPU work; here it is argument checks on
// tensor metadata, one call of the C ABI per direction and the C++ autograd function.
//
// Everything numeric stays behind the C ABI of include/nb_attn.h. Arguments outside the supported
// subset raise; there is no fallback and no CPU kernel.
#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>
#include <torch/library.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <tuple>

#include "../../include/nb_attn.h"
#include "torch_common.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using Two = std::tuple<Tensor, Tensor>;
using Three = std::tuple<Tensor, Tensor, Tensor>;

constexpr int64_t kHeadDim = 64;

#define NB_REQUIRE(cond, ...) TORCH_CHECK(cond, "nanobrain_b200.sdpa: ", __VA_ARGS__)

// ------------------------------------------------------------------------------------------
// Status words: one pinned int32 per device that kernels write to when something went wrong. The GPU
// addresses it directly, the host looks at it without synchronising.
// ------------------------------------------------------------------------------------------
constexpr int kMaxDevices = 64;
std::mutex g_status_mutex;
Tensor* g_status_tensors[kMaxDevices];             // never freed: a kernel may still hold the address
std::atomic<volatile int32_t*> g_status_ptrs[kMaxDevices];

Tensor status_word(int64_t device) {
  TORCH_CHECK(device >= 0 && device < kMaxDevices, "nanobrain_b200: no such device");
  std::lock_guard<std::mutex> lock(g_status_mutex);
  if (g_status_tensors[device] == nullptr) {
    auto* t = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt)).pin_memory());
    g_status_tensors[device] = t;
    g_status_ptrs[device].store(t->data_ptr<int32_t>(), std::memory_order_release);
  }
  return *g_status_tensors[device];
}

}  // namespace

namespace nbt {

volatile int32_t* status_ptr(int64_t device) {
  volatile int32_t* p = g_status_ptrs[device].load(std::memory_order_acquire);
  if (p == nullptr) {
    status_word(device);
    p = g_status_ptrs[device].load(std::memory_order_acquire);
  }
  return p;
}

void raise_for_status(volatile int32_t* word) {
  const int32_t code = *word;
  if (C10_LIKELY(code == 0)) return;
  *word = 0;
  TORCH_CHECK(false, "nanobrain_b200 attention kernel reported device status ", code, ": ",
              code == NB_ATTN_STATUS_WAIT_TIMEOUT
                  ? "a bounded wait inside a kernel gave up; results are garbage"
                  : code == NB_ATTN_STATUS_BAD_SEQLENS
                        ? "cu_seqlens is not a valid packing (offsets decreasing, a sequence longer than max_seqlen, "
                          "or the last offset beyond the token count); outputs were not written"
                        : "unknown code");
}

void after_launch(volatile int32_t* word) {
  static const bool debug = [] {
    const char* v = std::getenv("NB_ATTN_DEBUG");
    return v != nullptr && std::strcmp(v, "1") == 0;
  }();
  if (debug) {
    c10::cuda::device_synchronize();
    raise_for_status(word);
  }
}

void check_rc(int rc, const char* what) {
  TORCH_CHECK(rc == NB_ATTN_OK, what, " failed: ", nb_attn_strerror(rc), " (code ", rc, ")");
}

}  // namespace nbt

namespace {

using nbt::after_launch;
using nbt::check_rc;
using nbt::raise_for_status;
using nbt::status_ptr;

// ------------------------------------------------------------------------------------------
// Argument checks and layouts
// ------------------------------------------------------------------------------------------
void check_one(const Tensor& t, const char* name, int64_t ndim) {
  NB_REQUIRE(t.is_cuda(), name, " must be a CUDA tensor (there is no CPU path)");
  NB_REQUIRE(t.scalar_type() == at::kBFloat16, name, " must be bfloat16, got ", t.scalar_type());
  NB_REQUIRE(t.dim() == ndim, name, " must have ", ndim, " dimensions, got ", t.dim());
  NB_REQUIRE(t.size(-1) == kHeadDim, "head_dim must be ", kHeadDim, ", got ", t.size(-1));
}

void check_qkv(const Tensor& q, const Tensor& k, const Tensor& v, int64_t ndim) {
  check_one(q, "query", ndim);
  check_one(k, "key", ndim);
  check_one(v, "value", ndim);
  NB_REQUIRE(q.device() == k.device() && k.device() == v.device(), "query, key and value must be on the same device");
  NB_REQUIRE(k.sizes() == v.sizes(), "key and value must have the same shape");
}

void check_cu(const Tensor& cu, const char* name, const Tensor& like) {
  NB_REQUIRE(cu.scalar_type() == at::kInt && cu.dim() == 1 && cu.numel() >= 2, name, " must be int32 [B+1]");
  NB_REQUIRE(cu.device() == like.device(), name, " must live on the same device as the tokens");
  NB_REQUIRE(cu.is_contiguous(), name, " must be contiguous");
}

// Can the kernels address this tensor in place (head_dim contiguous, 16-byte rows)?
bool strides_ok(const Tensor& t) {
  const int64_t n = t.dim();
  if (t.stride(n - 1) != 1 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) != 0) return false;
  for (int64_t i = 0; i + 1 < n; ++i)
    if (t.size(i) > 1 && (t.stride(i) <= 0 || t.stride(i) % 8 != 0)) return false;
  return true;
}

// Logical [B, H, L, 64]: as it is, or a copy in [B, L, H, 64] memory.
Tensor dense_layout(const Tensor& t) {
  return strides_ok(t) ? t : t.transpose(1, 2).contiguous().transpose(1, 2);
}
Tensor packed_layout(const Tensor& t) { return strides_ok(t) ? t : t.contiguous(); }

nb_attn_tensor dense_desc(const Tensor& t) {
  const int64_t b = t.size(0), h = t.size(1), l = t.size(2);
  return {t.data_ptr(), b > 1 ? t.stride(0) : h * l * kHeadDim, l > 1 ? t.stride(2) : h * kHeadDim,
          h > 1 ? t.stride(1) : kHeadDim};
}
nb_attn_tensor packed_desc(const Tensor& t) {
  const int64_t n = t.size(0), h = t.size(1);
  return {t.data_ptr(), 0, n > 1 ? t.stride(0) : h * kHeadDim, h > 1 ? t.stride(1) : kHeadDim};
}

// Uninitialised tensors on the device of `like`, which is current here: from the caching allocator as
// at::empty's, without its two dispatched calls (seven tensors per forward + backward).
Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}
// Logical [B, H, L, 64] in [B, L, H, 64] memory.
Tensor new_dense(const Tensor& like) {
  const int64_t b = like.size(0), h = like.size(1), l = like.size(2);
  return at::detail::empty_strided_cuda({b, h, l, kHeadDim}, {l * h * kHeadDim, kHeadDim, h * kHeadDim, 1},
                                        at::kBFloat16, like.device());
}

nb_attn_shape dense_shape(const Tensor& q, const Tensor& k, double scale) {
  const int64_t b = q.size(0), lq = q.size(2), lk = k.size(2);
  nb_attn_shape s{};
  s.batch = int32_t(b), s.heads = int32_t(q.size(1)), s.head_dim = int32_t(kHeadDim);
  s.max_seqlen_q = int32_t(lq), s.max_seqlen_k = int32_t(lk);
  s.total_q = b * lq, s.total_k = b * lk;
  s.scale = float(scale);
  return s;
}
nb_attn_shape packed_shape(const Tensor& q, const Tensor& k, const Tensor& cu_q, const Tensor& cu_k, int64_t max_q,
                           int64_t max_k, double scale) {
  nb_attn_shape s{};
  s.batch = int32_t(cu_q.numel() - 1), s.heads = int32_t(q.size(1)), s.head_dim = int32_t(kHeadDim);
  s.max_seqlen_q = int32_t(max_q), s.max_seqlen_k = int32_t(max_k);
  s.total_q = q.size(0), s.total_k = k.size(0);
  s.cu_seqlens_q = cu_q.data_ptr<int32_t>(), s.cu_seqlens_k = cu_k.data_ptr<int32_t>();
  s.scale = float(scale);
  return s;
}

// ------------------------------------------------------------------------------------------
// CUDA kernels of the ops
// ------------------------------------------------------------------------------------------
void launch_fwd(nb_attn_fwd_args& a, const Tensor& q, Tensor& workspace) {
  volatile int32_t* word = status_ptr(q.get_device());
  raise_for_status(word);
  a.status = const_cast<int32_t*>(word);
  a.workspace_bytes = a.shape.cu_seqlens_q != nullptr ? nb_attn_fwd_workspace_bytes(&a.shape)  // the work list
                                                      : nb_attn_fwd_split_workspace_bytes(&a.shape);
  if (a.workspace_bytes > 0) {
    workspace = new_tensor({int64_t(a.workspace_bytes)}, at::kByte, q);
    a.workspace = workspace.data_ptr();
  }
  check_rc(nb_attn_fwd(&a, at::cuda::getCurrentCUDAStream().stream()), "nb_attn_fwd");
  after_launch(word);
}

void launch_bwd(nb_attn_bwd_args& a, const Tensor& q, const Tensor& lse) {
  volatile int32_t* word = status_ptr(q.get_device());
  raise_for_status(word);
  a.lse = lse.data_ptr<float>();
  a.status = const_cast<int32_t*>(word);
  // With room to cut units between CTAs or for their own dQ tiles.
  a.workspace_bytes = std::max(nb_attn_bwd_workspace_bytes(&a.shape), nb_attn_bwd_split_workspace_bytes(&a.shape));
  Tensor workspace = new_tensor({int64_t(a.workspace_bytes)}, at::kByte, q);
  a.workspace = workspace.data_ptr();
  check_rc(nb_attn_bwd(&a, at::cuda::getCurrentCUDAStream().stream()), "nb_attn_bwd");
  after_launch(word);
}

Two sdpa_fwd_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale) {
  check_qkv(q_, k_, v_, 4);
  const int64_t b = q_.size(0), h = q_.size(1), lq = q_.size(2);
  NB_REQUIRE(k_.size(0) == b && k_.size(1) == h, "query and key must agree on batch and heads (no GQA)");
  NB_REQUIRE(b > 0 && h > 0 && lq > 0 && k_.size(2) > 0, "empty tensors are not supported");
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = dense_layout(q_), k = dense_layout(k_), v = dense_layout(v_);
  Tensor out = new_dense(q), workspace;
  Tensor lse = new_tensor({b, h, lq}, at::kFloat, q);
  nb_attn_fwd_args a{};
  a.shape = dense_shape(q, k, scale);
  a.q = dense_desc(q), a.k = dense_desc(k), a.v = dense_desc(v), a.o = dense_desc(out);
  a.lse = lse.data_ptr<float>();
  launch_fwd(a, q, workspace);
  return {std::move(out), std::move(lse)};
}

Three sdpa_bwd_cuda(const Tensor& d_out_, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& out_,
                    const Tensor& lse_, double scale) {
  check_qkv(q_, k_, v_, 4);
  NB_REQUIRE(d_out_.scalar_type() == at::kBFloat16 && out_.scalar_type() == at::kBFloat16,
             "out and d_out must be bfloat16");
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = dense_layout(q_), k = dense_layout(k_), v = dense_layout(v_);
  const Tensor out = dense_layout(out_), d_out = dense_layout(d_out_), lse = lse_.contiguous();
  Tensor dq = new_dense(q), dk = new_dense(k), dv = new_dense(v);
  nb_attn_bwd_args a{};
  a.shape = dense_shape(q, k, scale);
  a.q = dense_desc(q), a.k = dense_desc(k), a.v = dense_desc(v), a.o = dense_desc(out), a.d_o = dense_desc(d_out);
  a.dq = dense_desc(dq), a.dk = dense_desc(dk), a.dv = dense_desc(dv);
  launch_bwd(a, q, lse);
  return {std::move(dq), std::move(dk), std::move(dv)};
}

Two sdpa_varlen_fwd_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& cu_q, const Tensor& cu_k,
                         int64_t max_q, int64_t max_k, double scale) {
  check_qkv(q_, k_, v_, 3);
  check_cu(cu_q, "cu_seqlens_q", q_);
  check_cu(cu_k, "cu_seqlens_k", q_);
  NB_REQUIRE(cu_q.numel() == cu_k.numel(), "cu_seqlens_q and cu_seqlens_k must have the same length");
  const int64_t tq = q_.size(0), h = q_.size(1);
  NB_REQUIRE(k_.size(1) == h, "query and key must agree on heads (no GQA)");
  NB_REQUIRE(tq > 0 && k_.size(0) > 0 && max_q > 0 && max_k > 0, "empty tensors are not supported");
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = packed_layout(q_), k = packed_layout(k_), v = packed_layout(v_);
  Tensor out = new_tensor({tq, h, kHeadDim}, at::kBFloat16, q), workspace;
  Tensor lse = new_tensor({h, tq}, at::kFloat, q);
  nb_attn_fwd_args a{};
  a.shape = packed_shape(q, k, cu_q, cu_k, max_q, max_k, scale);
  a.q = packed_desc(q), a.k = packed_desc(k), a.v = packed_desc(v), a.o = packed_desc(out);
  a.lse = lse.data_ptr<float>();
  launch_fwd(a, q, workspace);
  return {std::move(out), std::move(lse)};
}

Three sdpa_varlen_bwd_cuda(const Tensor& d_out_, const Tensor& q_, const Tensor& k_, const Tensor& v_,
                           const Tensor& out_, const Tensor& lse_, const Tensor& cu_q, const Tensor& cu_k,
                           int64_t max_q, int64_t max_k, double scale) {
  check_qkv(q_, k_, v_, 3);
  NB_REQUIRE(d_out_.scalar_type() == at::kBFloat16 && out_.scalar_type() == at::kBFloat16,
             "out and d_out must be bfloat16");
  const c10::cuda::CUDAGuard guard(q_.device());
  const Tensor q = packed_layout(q_), k = packed_layout(k_), v = packed_layout(v_);
  const Tensor out = packed_layout(out_), d_out = packed_layout(d_out_), lse = lse_.contiguous();
  Tensor dq = new_tensor(q.sizes(), at::kBFloat16, q), dk = new_tensor(k.sizes(), at::kBFloat16, q),
         dv = new_tensor(k.sizes(), at::kBFloat16, q);
  nb_attn_bwd_args a{};
  a.shape = packed_shape(q, k, cu_q, cu_k, max_q, max_k, scale);
  a.q = packed_desc(q), a.k = packed_desc(k), a.v = packed_desc(v), a.o = packed_desc(out), a.d_o = packed_desc(d_out);
  a.dq = packed_desc(dq), a.dk = packed_desc(dk), a.dv = packed_desc(dv);
  launch_bwd(a, q, lse);
  return {std::move(dq), std::move(dk), std::move(dv)};
}

// ------------------------------------------------------------------------------------------
// Autograd. The functions call the ops again below autograd, so dispatch modes (fake tensors, tracing,
// the FLOP counter) see every forward and backward op.
// ------------------------------------------------------------------------------------------
using FwdSig = Two(const Tensor&, const Tensor&, const Tensor&, double);
using BwdSig = Three(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, double);
using VarFwdSig = Two(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, c10::SymInt,
                      c10::SymInt, double);
using VarBwdSig = Three(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                        const Tensor&, const Tensor&, c10::SymInt, c10::SymInt, double);

template <typename Sig>
c10::TypedOperatorHandle<Sig> find_op(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}
const auto& fwd_op() {
  static const auto op = find_op<FwdSig>("nanobrain_b200::sdpa_fwd");
  return op;
}
const auto& bwd_op() {
  static const auto op = find_op<BwdSig>("nanobrain_b200::sdpa_bwd");
  return op;
}
const auto& varlen_fwd_op() {
  static const auto op = find_op<VarFwdSig>("nanobrain_b200::sdpa_varlen_fwd");
  return op;
}
const auto& varlen_bwd_op() {
  static const auto op = find_op<VarBwdSig>("nanobrain_b200::sdpa_varlen_bwd");
  return op;
}

bool wants_grad(const Tensor& q, const Tensor& k, const Tensor& v) {
  return at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
}

// The gradient of `out`; the log-sum-exp's own gradient is not used (it exists for the backward op).
Tensor grad_of_out(const variable_list& grads, const Tensor& out) {
  return grads[0].defined() ? grads[0] : at::zeros_like(out);
}

struct SdpaFunction : public torch::autograd::Function<SdpaFunction> {
  static constexpr bool is_traceable = true;  // compiled autograd may trace through backward
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, double scale) {
    at::AutoDispatchBelowADInplaceOrView guard;
    auto [out, lse] = fwd_op().call(q, k, v, scale);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({q, k, v, out, lse});
    ctx->saved_data["scale"] = scale;
    return {out, lse};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    auto [dq, dk, dv] = bwd_op().call(grad_of_out(grads, s[3]), s[0], s[1], s[2], s[3], s[4],
                                      ctx->saved_data["scale"].toDouble());
    return {dq, dk, dv, Tensor()};
  }
};

struct SdpaVarlenFunction : public torch::autograd::Function<SdpaVarlenFunction> {
  static constexpr bool is_traceable = true;  // compiled autograd may trace through backward
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                               const Tensor& cu_q, const Tensor& cu_k, c10::SymInt max_q, c10::SymInt max_k,
                               double scale) {
    at::AutoDispatchBelowADInplaceOrView guard;
    auto [out, lse] = varlen_fwd_op().call(q, k, v, cu_q, cu_k, max_q, max_k, scale);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({q, k, v, out, lse, cu_q, cu_k});
    ctx->saved_data["max_q"] = std::move(max_q);
    ctx->saved_data["max_k"] = std::move(max_k);
    ctx->saved_data["scale"] = scale;
    return {out, lse};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    auto [dq, dk, dv] = varlen_bwd_op().call(grad_of_out(grads, s[3]), s[0], s[1], s[2], s[3], s[4], s[5], s[6],
                                             ctx->saved_data["max_q"].toSymInt(), ctx->saved_data["max_k"].toSymInt(),
                                             ctx->saved_data["scale"].toDouble());
    return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Two sdpa_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, double scale) {
  if (!wants_grad(q, k, v)) {
    at::AutoDispatchBelowADInplaceOrView guard;
    return fwd_op().call(q, k, v, scale);
  }
  auto r = SdpaFunction::apply(q, k, v, scale);
  return {r[0], r[1]};
}

Two sdpa_varlen_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu_q, const Tensor& cu_k,
                             c10::SymInt max_q, c10::SymInt max_k, double scale) {
  if (!wants_grad(q, k, v)) {
    at::AutoDispatchBelowADInplaceOrView guard;
    return varlen_fwd_op().call(q, k, v, cu_q, cu_k, max_q, max_k, scale);
  }
  auto r = SdpaVarlenFunction::apply(q, k, v, cu_q, cu_k, max_q, max_k, scale);
  return {r[0], r[1]};
}

// What Python's sdpa() and sdpa_varlen() call outside of tracing: straight to the dispatcher, without
// the boxed call of torch.ops.
Tensor sdpa(const Tensor& q, const Tensor& k, const Tensor& v, double scale) {
  return std::get<0>(fwd_op().call(q, k, v, scale));
}
Tensor sdpa_varlen(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu_q, const Tensor& cu_k,
                   int64_t max_q, int64_t max_k, double scale) {
  return std::get<0>(varlen_fwd_op().call(q, k, v, cu_q, cu_k, max_q, max_k, scale));
}

}  // namespace

TORCH_LIBRARY_IMPL(nanobrain_b200, CUDA, m) {
  m.impl("sdpa_fwd", sdpa_fwd_cuda);
  m.impl("sdpa_bwd", sdpa_bwd_cuda);
  m.impl("sdpa_varlen_fwd", sdpa_varlen_fwd_cuda);
  m.impl("sdpa_varlen_bwd", sdpa_varlen_bwd_cuda);
}

TORCH_LIBRARY_IMPL(nanobrain_b200, Autograd, m) {
  m.impl("sdpa_fwd", sdpa_fwd_autograd);
  m.impl("sdpa_varlen_fwd", sdpa_varlen_fwd_autograd);
  // There is no second derivative.
  m.impl("sdpa_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("sdpa_varlen_bwd", torch::autograd::autogradNotImplementedFallback());
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("sdpa", &sdpa, py::call_guard<py::gil_scoped_release>());
  m.def("sdpa_varlen", &sdpa_varlen, py::call_guard<py::gil_scoped_release>());
  m.def("status_word", &status_word);
  nbt::bind_encoder(m);
}
