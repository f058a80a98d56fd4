// Python module `attention_cuda`: the three functions the reference's pybind shim
// exports (reference csrc/attention_ext.cpp:19-35) with the same names, keyword
// names, argument order and list-of-tensors results, backed by libattn_b200.so.
//
// Differences, all additive: a trailing `mask_mode` keyword (0 = the reference's
// causal + sliding-window + validity mask, 1 = no mask) and an `impl` keyword
// (0 auto, 1 fp32 SIMT kernels, 2 tensor-core kernels); float32 inputs and head
// dimensions up to 128 are accepted.  Kernels run on the current PyTorch stream
// of the tensors' device.
//
// `flash_attention` is the twice-differentiable call of attention.py with its two chained autograd
// functions written in C++: the autograd engine then runs both backward passes on its own thread
// without taking the interpreter lock.  A Python autograd function costs 25-30 us per use on the
// host (four of them in a second-order step) against about 5 us here.  Calls that a Python
// autograd function handles better (tracers, forward-mode tangents) are left to it.
#include <torch/extension.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <ATen/FuncTorchTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>

#include <atomic>
#include <cstdio>
#include <initializer_list>
#include <mutex>
#include <vector>

#include "attn_b200.h"

namespace {

int dtype_code(const torch::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kHalf: return ATTN_F16;
    case at::kBFloat16: return ATTN_BF16;
    case at::kFloat: return ATTN_F32;
    default: TORCH_CHECK(false, "V7 requires fp16, bf16 or fp32, got ", t.scalar_type());
  }
  return -1;
}

// Contiguous, and re-materialised if a view starts at an address TMA cannot use.
torch::Tensor dense(const torch::Tensor& t) {
  torch::Tensor c = t.contiguous();
  if (reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 != 0) c = c.clone();
  return c;
}

// New tensors of a contiguous shape on t's device, straight from the caching allocator: the
// dispatcher's factory functions take twice as long, and a call makes three to five tensors.  A tracer
// has to see where its tensors come from.
torch::Tensor fresh(at::IntArrayRef sizes, at::ScalarType type, const torch::Tensor& t) {
  if (torch::jit::tracer::isTracing()) return torch::empty(sizes, t.options().dtype(type));
  return at::detail::empty_cuda(sizes, type, t.device(), c10::nullopt);
}
torch::Tensor fresh_like(const torch::Tensor& t) { return fresh(t.sizes(), t.scalar_type(), t); }

void check_qkv(const torch::Tensor& Q, const torch::Tensor& K, const torch::Tensor& V) {
  TORCH_CHECK(Q.is_cuda(), "Q must be a CUDA tensor");
  TORCH_CHECK(K.is_cuda() && V.is_cuda(), "K and V must be CUDA tensors");
  TORCH_CHECK(Q.dim() == 4 && K.dim() == 4 && V.dim() == 4, "Q, K, V must be [B, H, N, D]");
  TORCH_CHECK(K.sizes() == V.sizes(), "K and V must have the same shape");
  TORCH_CHECK(Q.size(0) == K.size(0) && Q.size(1) == K.size(1) && Q.size(3) == K.size(3),
              "Q and K must agree in B, H and D");
  TORCH_CHECK(Q.scalar_type() == K.scalar_type() && Q.scalar_type() == V.scalar_type(),
              "Q, K, V must have the same dtype");
  TORCH_CHECK(Q.device() == K.device() && Q.device() == V.device(), "Q, K, V must be on one device");
}

void check_like(const torch::Tensor& x, const torch::Tensor& ref, const char* name) {
  TORCH_CHECK(x.is_cuda() && x.device() == ref.device(), name, " must be on the same device as Q");
  TORCH_CHECK(x.sizes() == ref.sizes(), name, " has the wrong shape");
  TORCH_CHECK(x.scalar_type() == ref.scalar_type(), name, " has the wrong dtype");
}

attn_shape_t make_shape(const torch::Tensor& Q, const torch::Tensor& K, int window_size, int chunk_id,
                        int mask_mode, int impl) {
  attn_shape_t s;
  s.B = (int32_t)Q.size(0);
  s.H = (int32_t)Q.size(1);
  s.N_q = (int32_t)Q.size(2);
  s.N_kv = (int32_t)K.size(2);
  s.D = (int32_t)Q.size(3);
  s.window_size = window_size;
  s.chunk_id = chunk_id;
  s.mask_mode = mask_mode;
  s.dtype = dtype_code(Q);
  s.impl = impl;
  return s;
}

void check_rc(int rc, const char* what) {
  TORCH_CHECK(rc == ATTN_OK, what, " failed (", rc, "): ", attn_b200_last_error());
}

// A kernel that gives up on a bounded wait stores a code in the device's status word and returns;
// its outputs are then meaningless.  This module registers one page-locked host word per device
// as a mirror of that status word (the failing kernel writes its code there too) and looks at it
// at the start of every call: a time-out of an earlier call is reported as an exception of the
// first call that starts after it, and the good path costs one read of host memory.
uint32_t* status_mirror(int device) {
  static torch::Tensor words[64];
  static std::atomic<uint32_t*> known[64];
  static std::mutex mu;
  TORCH_CHECK(device >= 0 && device < 64, "device index out of range");
  if (uint32_t* w = known[device].load(std::memory_order_acquire)) return w;
  std::lock_guard<std::mutex> lock(mu);
  if (!words[device].defined()) {
    words[device] = torch::zeros({1}, torch::dtype(torch::kInt32).pinned_memory(true));
    check_rc(attn_b200_set_status_mirror(reinterpret_cast<uint32_t*>(words[device].data_ptr<int32_t>())),
             "attn_b200_set_status_mirror");
  }
  uint32_t* w = reinterpret_cast<uint32_t*>(words[device].data_ptr<int32_t>());
  known[device].store(w, std::memory_order_release);
  return w;
}

void raise_if_earlier_call_timed_out(int device) {
  volatile uint32_t* w = status_mirror(device);
  if (*w == 0u) return;
  *w = 0u;
  uint32_t code = 0;
  int rc = attn_b200_device_status(&code);     // synchronises, reads and clears the device word
  char hex[16];
  snprintf(hex, sizeof(hex), "0x%x", code);
  TORCH_CHECK(rc == ATTN_OK && code == 0u, "an earlier attention kernel on this device gave up on a bounded wait (status ",
              hex, "); its outputs are invalid");
}

}  // namespace

std::vector<torch::Tensor> v7_forward_cuda(torch::Tensor Q, torch::Tensor K, torch::Tensor V, int window_size,
                                           int chunk_id, int mask_mode, int impl) {
  check_qkv(Q, K, V);
  c10::cuda::CUDAGuard guard(Q.device());
  raise_if_earlier_call_timed_out(Q.device().index());
  Q = dense(Q); K = dense(K); V = dense(V);
  attn_shape_t s = make_shape(Q, K, window_size, chunk_id, mask_mode, impl);
  auto O = fresh_like(Q);
  auto L = fresh({Q.size(0), Q.size(1), Q.size(2)}, at::kFloat, Q);
  check_rc(attn_b200_forward(&s, Q.data_ptr(), K.data_ptr(), V.data_ptr(), O.data_ptr(), L.data_ptr<float>(),
                             at::cuda::getCurrentCUDAStream().stream()),
           "v7_forward");
  return {O, L};
}

std::vector<torch::Tensor> v7_backward_cuda(torch::Tensor dO, torch::Tensor Q, torch::Tensor K, torch::Tensor V,
                                            torch::Tensor O, torch::Tensor L, int window_size, int chunk_id,
                                            int mask_mode, int impl) {
  check_qkv(Q, K, V);
  check_like(dO, Q, "dO");
  check_like(O, Q, "O");
  TORCH_CHECK(L.is_cuda() && L.scalar_type() == at::kFloat && L.numel() == Q.size(0) * Q.size(1) * Q.size(2),
              "L must be a float32 CUDA tensor of shape [B, H, N_q]");
  c10::cuda::CUDAGuard guard(Q.device());
  raise_if_earlier_call_timed_out(Q.device().index());
  dO = dense(dO); Q = dense(Q); K = dense(K); V = dense(V); O = dense(O); L = L.contiguous();
  attn_shape_t s = make_shape(Q, K, window_size, chunk_id, mask_mode, impl);
  auto dQ = fresh_like(Q);
  auto dK = fresh_like(K);
  auto dV = fresh_like(V);
  auto scratch = fresh({(int64_t)(attn_b200_backward_scratch_bytes(&s) / sizeof(float)) + 4}, at::kFloat, Q);
  check_rc(attn_b200_backward(&s, dO.data_ptr(), Q.data_ptr(), K.data_ptr(), V.data_ptr(), O.data_ptr(),
                              L.data_ptr<float>(), dQ.data_ptr(), dK.data_ptr(), dV.data_ptr(),
                              scratch.data_ptr<float>(), at::cuda::getCurrentCUDAStream().stream()),
           "v7_backward");
  return {dQ, dK, dV};
}

std::vector<torch::Tensor> v7_double_backward_cuda(torch::Tensor g_dQ, torch::Tensor g_dK, torch::Tensor g_dV,
                                                   torch::Tensor dO, torch::Tensor Q, torch::Tensor K,
                                                   torch::Tensor V, torch::Tensor O, torch::Tensor L,
                                                   int window_size, int chunk_id, int mask_mode, int impl) {
  check_qkv(Q, K, V);
  check_like(dO, Q, "dO");
  check_like(g_dQ, Q, "g_dQ");
  check_like(g_dK, K, "g_dK");
  check_like(g_dV, V, "g_dV");
  TORCH_CHECK(L.is_cuda() && L.scalar_type() == at::kFloat && L.numel() == Q.size(0) * Q.size(1) * Q.size(2),
              "L must be a float32 CUDA tensor of shape [B, H, N_q]");
  c10::cuda::CUDAGuard guard(Q.device());
  raise_if_earlier_call_timed_out(Q.device().index());
  g_dQ = dense(g_dQ); g_dK = dense(g_dK); g_dV = dense(g_dV);
  dO = dense(dO); Q = dense(Q); K = dense(K); V = dense(V); L = L.contiguous();
  attn_shape_t s = make_shape(Q, K, window_size, chunk_id, mask_mode, impl);
  auto g_dO = fresh_like(Q);
  auto g_Q = fresh_like(Q);
  auto g_K = fresh_like(K);
  auto g_V = fresh_like(V);
  auto scratch = fresh({(int64_t)(attn_b200_double_backward_scratch_bytes(&s) / sizeof(float)) + 4}, at::kFloat, Q);
  check_like(O, Q, "O");
  O = dense(O);
  check_rc(attn_b200_double_backward(&s, g_dQ.data_ptr(), g_dK.data_ptr(), g_dV.data_ptr(), dO.data_ptr(),
                                     Q.data_ptr(), K.data_ptr(), V.data_ptr(), O.data_ptr(), L.data_ptr<float>(),
                                     g_dO.data_ptr(), g_Q.data_ptr(), g_K.data_ptr(), g_V.data_ptr(),
                                     scratch.data_ptr<float>(), at::cuda::getCurrentCUDAStream().stream()),
           "v7_double_backward");
  return {g_dO, g_Q, g_K, g_V};
}

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

bool has_tangent(std::initializer_list<const torch::Tensor*> inputs) {
  for (const torch::Tensor* t : inputs)
    if (t->defined() && t->_fw_grad(/*level=*/0).defined()) return true;
  return false;
}

// A call for the Python autograd functions: torch.jit.trace records them, and they refuse a tangent,
// which kernels called directly would drop.  Under a functorch transform neither kind of function has
// a rule: refused here, whether or not gradients are asked for.
bool leave_to_python(std::initializer_list<const torch::Tensor*> inputs) {
  if (const auto& functorch = at::functorch::functorchTLSAccessor()) functorch->checkSupportsCppAutogradFunction();
  return torch::jit::tracer::isTracing() || has_tangent(inputs);
}

struct MaskArgs { int window_size, chunk_id, mask_mode; };

void save_mask(AutogradContext* ctx, int64_t window_size, int64_t chunk_id, int64_t mask_mode) {
  ctx->saved_data["window_size"] = window_size;
  ctx->saved_data["chunk_id"] = chunk_id;
  ctx->saved_data["mask_mode"] = mask_mode;
}

MaskArgs saved_mask(AutogradContext* ctx) {
  return {(int)ctx->saved_data["window_size"].toInt(), (int)ctx->saved_data["chunk_id"].toInt(),
          (int)ctx->saved_data["mask_mode"].toInt()};
}

// First backward as a differentiable function of dO, Q, K, V; its own backward is the double
// backward.  O and L come in detached: gradients are total derivatives with O and L treated as
// functions of Q, K, V, so nothing flows back through them.
struct AttentionBackward : public torch::autograd::Function<AttentionBackward> {
  static variable_list forward(AutogradContext* ctx, const torch::Tensor& dO, const torch::Tensor& Q, const torch::Tensor& K,
                               const torch::Tensor& V, const torch::Tensor& O, const torch::Tensor& L, int64_t window_size,
                               int64_t chunk_id, int64_t mask_mode) {
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({dO, Q, K, V, O, L});
    save_mask(ctx, window_size, chunk_id, mask_mode);
    return v7_backward_cuda(dO, Q, K, V, O, L, (int)window_size, (int)chunk_id, (int)mask_mode, 0);
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list out(9);      // dO, Q, K, V, O, L, window_size, chunk_id, mask_mode
    if (!g[0].defined() && !g[1].defined() && !g[2].defined()) return out;
    const variable_list s = ctx->get_saved_variables();
    const MaskArgs m = saved_mask(ctx);
    auto tangent = [](const torch::Tensor& t, const torch::Tensor& like) { return t.defined() ? t : torch::zeros_like(like); };
    variable_list r = v7_double_backward_cuda(tangent(g[0], s[1]), tangent(g[1], s[2]), tangent(g[2], s[3]), s[0], s[1], s[2],
                                              s[3], s[4], s[5], m.window_size, m.chunk_id, m.mask_mode, 0);
    for (int i = 0; i < 4; ++i) out[i] = std::move(r[i]);
    return out;
  }
};

struct Attention : public torch::autograd::Function<Attention> {
  static torch::Tensor forward(AutogradContext* ctx, const torch::Tensor& Q, const torch::Tensor& K, const torch::Tensor& V,
                               int64_t window_size, int64_t chunk_id, int64_t mask_mode) {
    variable_list r = v7_forward_cuda(Q, K, V, (int)window_size, (int)chunk_id, (int)mask_mode, 0);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({Q, K, V, r[0], r[1]});
    save_mask(ctx, window_size, chunk_id, mask_mode);
    return r[0];
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list out(6);      // Q, K, V, window_size, chunk_id, mask_mode
    if (!g[0].defined()) return out;
    const variable_list s = ctx->get_saved_variables();
    const MaskArgs m = saved_mask(ctx);
    // without create_graph nothing will ask for the derivative of this backward (but a tangent has to be refused)
    variable_list r = at::GradMode::is_enabled() || has_tangent({&g[0], &s[0], &s[1], &s[2]})
                          ? AttentionBackward::apply(g[0], s[0], s[1], s[2], s[3].detach(), s[4], (int64_t)m.window_size,
                                                     (int64_t)m.chunk_id, (int64_t)m.mask_mode)
                          : v7_backward_cuda(g[0], s[0], s[1], s[2], s[3], s[4], m.window_size, m.chunk_id, m.mask_mode, 0);
    for (int i = 0; i < 3; ++i) out[i] = std::move(r[i]);
    return out;
  }
};

}  // namespace

// Nothing: a call for the Python function (attention.py).
c10::optional<torch::Tensor> flash_attention(const torch::Tensor& Q, const torch::Tensor& K, const torch::Tensor& V, int window_size,
                                             int chunk_id, int mask_mode) {
  if (leave_to_python({&Q, &K, &V})) return c10::nullopt;
  const bool graph = at::GradMode::is_enabled() && (Q.requires_grad() || K.requires_grad() || V.requires_grad());
  if (!graph) return v7_forward_cuda(Q, K, V, window_size, chunk_id, mask_mode, 0)[0];
  return Attention::apply(Q, K, V, (int64_t)window_size, (int64_t)chunk_id, (int64_t)mask_mode);
}

// x [n_tok, H, d] -> [1, H, n_tok, d]: RMS normalisation (rows >= norm_from, when a weight is given),
// rotary embedding with freqs [positions, d/2, 2] (float32 cos, sin), layout change; one kernel.
torch::Tensor qk_norm_rope_cuda(torch::Tensor x, c10::optional<torch::Tensor> weight, torch::Tensor freqs, int pos0,
                                double eps, int norm_from) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 3, "x must be a CUDA tensor [n_tok, H, d]");
  TORCH_CHECK(freqs.is_cuda() && freqs.scalar_type() == at::kFloat && freqs.dim() == 3 && freqs.size(2) == 2 &&
              freqs.size(1) * 2 == x.size(2), "freqs must be float32 [positions, d/2, 2]");
  TORCH_CHECK(pos0 >= 0 && pos0 + x.size(0) <= freqs.size(0), "positions out of the range of freqs");
  c10::cuda::CUDAGuard guard(x.device());
  x = x.contiguous();
  freqs = freqs.contiguous();
  torch::Tensor w;
  if (weight.has_value() && weight->defined()) {
    TORCH_CHECK(weight->is_cuda() && weight->numel() == x.size(2), "weight must be a CUDA tensor [d]");
    w = weight->to(x.scalar_type()).contiguous();
  }
  auto out = fresh({1, x.size(1), x.size(0), x.size(2)}, x.scalar_type(), x);
  check_rc(attn_b200_qk_norm_rope(x.data_ptr(), w.defined() ? w.data_ptr() : nullptr, freqs.data_ptr<float>(), out.data_ptr(),
                                  (int32_t)x.size(0), (int32_t)x.size(1), (int32_t)x.size(2), pos0, norm_from, (float)eps,
                                  dtype_code(x), at::cuda::getCurrentCUDAStream().stream()),
           "qk_norm_rope");
  return out;
}

namespace {

// The differentiable form: the forward and the first backward run the fused kernels; the second
// backward differentiates the formulas below with the autograd engine.
struct PrepArgs { int pos0; double eps; int norm_from; };

// "No weight" is an empty tensor between the autograd functions, which take defined tensors only.
torch::Tensor weight_or_none(const torch::Tensor& w) { return w.numel() > 0 ? w : torch::Tensor(); }

// The same computation out of ordinary operations, with the kernel's rounding points.
torch::Tensor qk_norm_rope_formula(const torch::Tensor& x, const torch::Tensor& weight, const torch::Tensor& freqs, const PrepArgs& a) {
  const int64_t n_tok = x.size(0), H = x.size(1), d = x.size(2);
  torch::Tensor y = x;
  if (weight.defined()) {
    const torch::Tensor xf = x.to(torch::kFloat);
    torch::Tensor normed = (xf * torch::rsqrt(xf.pow(2).mean({-1}, true) + a.eps)).to(x.scalar_type()) * weight.to(x.scalar_type());
    if (a.norm_from > 0) {
      const torch::Tensor keep = (torch::arange(n_tok, x.options().dtype(torch::kLong)) < a.norm_from).view({n_tok, 1, 1});
      normed = torch::where(keep, x, normed);
    }
    y = normed;
  }
  const torch::Tensor f = freqs.slice(0, a.pos0, a.pos0 + n_tok).unsqueeze(1);
  const torch::Tensor pair = y.to(torch::kFloat).reshape({n_tok, H, d / 2, 2});
  const torch::Tensor u = pair.select(-1, 0), v = pair.select(-1, 1), c = f.select(-1, 0), s = f.select(-1, 1);
  return torch::stack({u * c - v * s, u * s + v * c}, -1).reshape({n_tok, H, d}).to(x.scalar_type()).permute({1, 0, 2}).unsqueeze(0);
}

// {gx, gw}; gw is undefined without a weight or when it is not wanted
variable_list qk_norm_rope_backward(const torch::Tensor& g_in, const torch::Tensor& x_in, const torch::Tensor& weight,
                                    const torch::Tensor& freqs_in, const PrepArgs& a, bool want_gw) {
  const int64_t n_tok = x_in.size(0), H = x_in.size(1), d = x_in.size(2);
  if (d % 8 != 0 || x_in.numel() == 0) {      // no 16-byte accesses at these widths: the kernels do not take them
    at::AutoGradMode on(true);
    variable_list wrt{x_in.detach().requires_grad_(true)};
    if (weight.defined()) wrt.push_back(weight.detach().requires_grad_(true));
    const torch::Tensor y = qk_norm_rope_formula(wrt[0], weight.defined() ? wrt[1] : weight, freqs_in, a);
    variable_list r = torch::autograd::grad({y}, wrt, {g_in});
    r.resize(2);
    return r;
  }
  c10::cuda::CUDAGuard guard(x_in.device());
  const torch::Tensor x = dense(x_in), g = dense(g_in), freqs = dense(freqs_in);
  torch::Tensor w, gw, scratch;
  if (weight.defined()) w = dense(weight.to(x.scalar_type()));
  torch::Tensor gx = fresh_like(x);
  want_gw = want_gw && w.defined();
  if (want_gw) {
    gw = fresh(weight.sizes(), x.scalar_type(), x);
    scratch = fresh({(int64_t)(attn_b200_qk_norm_rope_backward_scratch_bytes((int32_t)n_tok, (int32_t)H, (int32_t)d) / sizeof(float))},
                    at::kFloat, x);
  }
  check_rc(attn_b200_qk_norm_rope_backward(x.data_ptr(), w.defined() ? w.data_ptr() : nullptr, freqs.data_ptr<float>(), g.data_ptr(),
                                           gx.data_ptr(), want_gw ? gw.data_ptr() : nullptr, want_gw ? scratch.data_ptr<float>() : nullptr,
                                           (int32_t)n_tok, (int32_t)H, (int32_t)d, a.pos0, a.norm_from, (float)a.eps, dtype_code(x),
                                           at::cuda::getCurrentCUDAStream().stream()),
           "qk_norm_rope_backward");
  if (want_gw && weight.scalar_type() != gw.scalar_type()) gw = gw.to(weight.scalar_type());
  return {gx, gw};
}

void save_prep(AutogradContext* ctx, int64_t pos0, double eps, int64_t norm_from) {
  ctx->set_materialize_grads(false);
  ctx->saved_data["pos0"] = pos0;
  ctx->saved_data["eps"] = eps;
  ctx->saved_data["norm_from"] = norm_from;
}
PrepArgs saved_prep(AutogradContext* ctx) {
  return {(int)ctx->saved_data["pos0"].toInt(), ctx->saved_data["eps"].toDouble(), (int)ctx->saved_data["norm_from"].toInt()};
}

struct QKNormRopeBackward : public torch::autograd::Function<QKNormRopeBackward> {
  static variable_list forward(AutogradContext* ctx, const torch::Tensor& g, const torch::Tensor& x, const torch::Tensor& weight,
                               const torch::Tensor& freqs, int64_t pos0, double eps, int64_t norm_from) {
    save_prep(ctx, pos0, eps, norm_from);
    ctx->save_for_backward({g, x, weight, freqs});
    variable_list r = qk_norm_rope_backward(g, x, weight_or_none(weight), freqs, {(int)pos0, eps, (int)norm_from}, true);
    if (weight.numel() == 0) r.resize(1);
    return r;
  }

  static variable_list backward(AutogradContext* ctx, variable_list tangents) {
    variable_list out(7);      // g, x, weight, freqs, pos0, eps, norm_from
    const variable_list s = ctx->get_saved_variables();
    const PrepArgs a = saved_prep(ctx);
    const bool keep_graph = at::GradMode::is_enabled();
    at::AutoGradMode on(true);
    // aliases of the inputs, so that the derivatives are partial ones even where the inputs depend on
    // one another (g often depends on x); connected to them when a third derivative may be asked for
    auto alias = [&](const torch::Tensor& t) {
      return keep_graph && t.requires_grad() ? t.view_as(t) : t.detach().requires_grad_(true);
    };
    const torch::Tensor g = alias(s[0]), x = alias(s[1]);
    variable_list first_wrt{x}, wrt{g, x};
    torch::Tensor w;
    if (s[2].numel() > 0) {
      w = alias(s[2]);
      first_wrt.push_back(w);
      wrt.push_back(w);
    }
    const variable_list first = torch::autograd::grad({qk_norm_rope_formula(x, w, s[3], a)}, first_wrt, {g}, true, true);
    variable_list of, with;
    for (size_t i = 0; i < first.size(); ++i)
      if (tangents[i].defined()) { of.push_back(first[i]); with.push_back(tangents[i]); }
    if (of.empty()) return out;
    const variable_list r = torch::autograd::grad(of, wrt, with, true, keep_graph, true);
    for (size_t i = 0; i < r.size(); ++i) out[i] = r[i];
    return out;
  }
};

struct QKNormRope : public torch::autograd::Function<QKNormRope> {
  static torch::Tensor forward(AutogradContext* ctx, const torch::Tensor& x, const torch::Tensor& weight, const torch::Tensor& freqs,
                               int64_t pos0, double eps, int64_t norm_from) {
    save_prep(ctx, pos0, eps, norm_from);
    ctx->save_for_backward({x, weight, freqs});
    return qk_norm_rope_cuda(x, weight_or_none(weight), freqs, (int)pos0, eps, (int)norm_from);
  }

  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list out(6);      // x, weight, freqs, pos0, eps, norm_from
    if (!g[0].defined()) return out;
    const variable_list s = ctx->get_saved_variables();
    const PrepArgs a = saved_prep(ctx);
    if (has_tangent({&g[0], &s[0], &s[1]})) {      // forward mode over this backward: the formulas have the rules
      const bool keep_graph = at::GradMode::is_enabled();
      at::AutoGradMode on(true);
      auto leaf = [](const torch::Tensor& t) { return t.requires_grad() ? t : t.detach().requires_grad_(true); };
      variable_list wrt{leaf(s[0])};
      if (s[1].numel() > 0) wrt.push_back(leaf(s[1]));
      const torch::Tensor y = qk_norm_rope_formula(wrt[0], wrt.size() > 1 ? wrt[1] : torch::Tensor(), s[2], a);
      const variable_list r = torch::autograd::grad({y}, wrt, {g[0]}, c10::nullopt, keep_graph, true);
      for (size_t i = 0; i < r.size(); ++i) out[i] = r[i];
      return out;
    }
    variable_list r = at::GradMode::is_enabled()
                          ? QKNormRopeBackward::apply(g[0], s[0], s[1], s[2], (int64_t)a.pos0, a.eps, (int64_t)a.norm_from)
                          : qk_norm_rope_backward(g[0], s[0], weight_or_none(s[1]), s[2], a, ctx->needs_input_grad(1));
    for (size_t i = 0; i < r.size(); ++i) out[i] = r[i];
    return out;
  }
};

}  // namespace

// Nothing: a call for the Python function (qk_prep.py).
c10::optional<torch::Tensor> qk_norm_rope_diff(const torch::Tensor& x, c10::optional<torch::Tensor> weight, const torch::Tensor& freqs,
                                               int pos0, double eps, int norm_from) {
  const bool has_weight = weight.has_value() && weight->defined();
  if (leave_to_python({&x, has_weight ? &*weight : &x, &freqs})) return c10::nullopt;
  // the table has no gradient, but a table that asks for one makes the output part of the graph
  if (!at::GradMode::is_enabled() || !(x.requires_grad() || freqs.requires_grad() || (has_weight && weight->requires_grad())))
    return qk_norm_rope_cuda(x, weight, freqs, pos0, eps, norm_from);
  return QKNormRope::apply(x, has_weight ? *weight : fresh({0}, x.scalar_type(), x), freqs, (int64_t)pos0, eps, (int64_t)norm_from);
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("qk_norm_rope", &qk_norm_rope_cuda, "fused RMS norm + rotary embedding + [n_tok,H,d] -> [1,H,n_tok,d]",
        py::arg("x"), py::arg("weight"), py::arg("freqs"), py::arg("pos0") = 0, py::arg("eps") = 1e-6, py::arg("norm_from") = 0);
  m.def("qk_norm_rope_diff", &qk_norm_rope_diff, "qk_norm_rope, twice differentiable (None: a call for the Python function)",
        py::arg("x"), py::arg("weight"), py::arg("freqs"), py::arg("pos0") = 0, py::arg("eps") = 1e-6, py::arg("norm_from") = 0,
        py::call_guard<py::gil_scoped_release>());
  m.def("flash_attention", &flash_attention, "Rectangular sliding-window flash attention, twice differentiable -> O (None: a call for the Python function)",
        py::arg("Q"), py::arg("K"), py::arg("V"), py::arg("window_size"), py::arg("chunk_id"), py::arg("mask_mode") = 0,
        py::call_guard<py::gil_scoped_release>());
  m.def("v7_forward", &v7_forward_cuda, "Rectangular sliding-window flash attention forward -> [O, L]",
        py::arg("Q"), py::arg("K"), py::arg("V"), py::arg("window_size"), py::arg("chunk_id"),
        py::arg("mask_mode") = 0, py::arg("impl") = 0);
  m.def("v7_backward", &v7_backward_cuda, "Rectangular sliding-window flash attention backward -> [dQ, dK, dV]",
        py::arg("dO"), py::arg("Q"), py::arg("K"), py::arg("V"), py::arg("O"), py::arg("L"),
        py::arg("window_size"), py::arg("chunk_id"), py::arg("mask_mode") = 0, py::arg("impl") = 0);
  m.def("v7_double_backward", &v7_double_backward_cuda,
        "Rectangular sliding-window flash attention double backward -> [g_dO, g_Q, g_K, g_V]",
        py::arg("g_dQ"), py::arg("g_dK"), py::arg("g_dV"), py::arg("dO"), py::arg("Q"), py::arg("K"),
        py::arg("V"), py::arg("O"), py::arg("L"), py::arg("window_size"), py::arg("chunk_id"),
        py::arg("mask_mode") = 0, py::arg("impl") = 0);
  m.def("last_launch_count", &attn_b200_last_launch_count, "kernels launched by the last call of this thread");
  m.def("device_status", []() {
    uint32_t code = 0;
    int rc = attn_b200_device_status(&code);
    return py::make_tuple(rc, code);
  }, "(return code, status word) of the current device; synchronises");
}
