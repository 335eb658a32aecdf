// Differentiable operators of the `algebraic` namespace with their autograd formulas in C++, and the entry points through
// which the Python functions reach them.
//
// A call of a fused operator on a few thousand elements takes 2-4 us on the GPU; what it costs is the host.  With Python
// autograd Functions over torch.ops, a pass of forward and backward took 77 us for softmax [4096, 4096], where the GPU needs 41,
// and 123 us for residual add + norm [64, 768] (17 on the GPU); this way 48 and 83.  The forward is one typed dispatcher call from a
// METH_FASTCALL function, the graph
// node is a plain C++ Node with SavedVariables, and its backward calls the backward operator without going through the
// interpreter.  The operators below the autograd key are the ones of torch_ops.cpp and are reached through the dispatcher,
// so modes that watch operators (fake tensors, profilers, functionalisation) see what they saw before.
#include <ATen/PythonTorchFunctionTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/core/dispatch/Dispatcher.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/library.h>

#include <string>
#include <tuple>
#include <type_traits>

namespace {

using at::Tensor;
using c10::optional;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

template <typename Sig>
c10::TypedOperatorHandle<Sig> handle(const char* name) {
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}

// ------------------------------------------------------------------------------------- the operators underneath
Tensor op_softmax_fwd(const Tensor& x, double eps) {
  static const auto op = handle<Tensor(const Tensor&, double)>("algebraic::softmax_fwd");
  return op.call(x, eps);
}
Tensor op_softmax_bwd(const Tensor& d, const Tensor& x, double eps) {
  static const auto op = handle<Tensor(const Tensor&, const Tensor&, double)>("algebraic::softmax_bwd");
  return op.call(d, x, eps);
}
Tensor op_swiglu_fwd(const Tensor& g, const Tensor& v) {
  static const auto op = handle<Tensor(const Tensor&, const Tensor&)>("algebraic::swiglu_fwd");
  return op.call(g, v);
}
Tensor op_swiglu_bwd_packed(const Tensor& d, const Tensor& g, const Tensor& v) {
  static const auto op = handle<Tensor(const Tensor&, const Tensor&, const Tensor&)>("algebraic::swiglu_bwd_packed");
  return op.call(d, g, v);
}
std::tuple<Tensor, Tensor> op_swiglu_bwd_dense(const Tensor& d, const Tensor& g, const Tensor& v) {
  static const auto op = handle<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&)>("algebraic::swiglu_bwd_dense");
  return op.call(d, g, v);
}
std::tuple<Tensor, Tensor> op_norm_fwd(const Tensor& x, const Tensor& w, double eps) {
  static const auto op = handle<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, double)>("algebraic::norm_fwd");
  return op.call(x, w, eps);
}
std::tuple<Tensor, Tensor> op_norm_bwd(const Tensor& d, const Tensor& x, const Tensor& w, const Tensor& mean, double eps) {
  static const auto op = handle<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, double)>("algebraic::norm_bwd");
  return op.call(d, x, w, mean, eps);
}
std::tuple<Tensor, Tensor, Tensor> op_add_norm_fwd(const Tensor& x, const Tensor& r, const Tensor& w, double eps) {
  static const auto op = handle<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, double)>("algebraic::add_norm_fwd");
  return op.call(x, r, w, eps);
}
std::tuple<Tensor, Tensor> op_add_norm_bwd(const Tensor& dy, const optional<Tensor>& dh, const Tensor& h, const Tensor& w, const Tensor& mean, double eps) {
  static const auto op = handle<std::tuple<Tensor, Tensor>(const Tensor&, const optional<Tensor>&, const Tensor&, const Tensor&, const Tensor&, double)>("algebraic::add_norm_bwd");
  return op.call(dy, dh, h, w, mean, eps);
}
Tensor op_pack_key_mask(const Tensor& m) {
  static const auto op = handle<Tensor(const Tensor&)>("algebraic::pack_key_mask");
  return op.call(m);
}
std::tuple<Tensor, Tensor, Tensor> op_attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& slopes, double scale, bool causal,
                                               double eps, const optional<Tensor>& bits, bool residual) {
  static const auto op = handle<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, double, bool, double,
                                                                  int64_t, bool, const optional<Tensor>&, bool)>("algebraic::attn_fwd");
  return op.call(q, k, v, slopes, scale, causal, eps, 0, false, bits, residual);
}
std::tuple<Tensor, Tensor, Tensor> op_attn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lo, const Tensor& L,
                                               const Tensor& d, const Tensor& slopes, double scale, bool causal, double eps, const optional<Tensor>& bits) {
  static const auto op = handle<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                                  const Tensor&, const Tensor&, const Tensor&, double, bool, double, int64_t,
                                                                  const optional<Tensor>&)>("algebraic::attn_bwd");
  return op.call(q, k, v, out, lo, L, d, slopes, scale, causal, eps, 0, bits);
}
std::tuple<Tensor, Tensor, Tensor> op_attn_fwd_packed(const Tensor& qkv, const Tensor& slopes, double scale, double eps, const optional<Tensor>& bits, bool residual) {
  static const auto op = handle<std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, double, double, const optional<Tensor>&, bool)>("algebraic::attn_fwd_packed");
  return op.call(qkv, slopes, scale, eps, bits, residual);
}
Tensor op_attn_bwd_packed(const Tensor& qkv, const Tensor& out, const Tensor& lo, const Tensor& L, const Tensor& d, const Tensor& slopes, double scale,
                          double eps, const optional<Tensor>& bits) {
  static const auto op = handle<Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&, double, double,
                                       const optional<Tensor>&)>("algebraic::attn_bwd_packed");
  return op.call(qkv, out, lo, L, d, slopes, scale, eps, bits);
}

// ------------------------------------------------------------------------------------- nodes
using BelowAutograd = at::AutoDispatchBelowADInplaceOrView;

// In a backward without create_graph nothing below is differentiated: the operators are called below the autograd keys.
struct BackwardScope {
  optional<BelowAutograd> guard;
  BackwardScope() { if (!at::GradMode::is_enabled()) guard.emplace(); }
};

template <typename N, typename... Ts>
std::shared_ptr<N> new_node(const Ts&... inputs) {
  std::shared_ptr<N> node(new N(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  return node;
}

// Custom operators have no forward-mode formula: say so instead of dropping the tangent.
template <typename... Ts>
void no_forward_mode(const char* what, const Ts&... ts) {
  const bool any = (... || (ts.defined() && ts._fw_grad(/*level=*/0).defined()));
  TORCH_CHECK_NOT_IMPLEMENTED(!any, "algebraic::", what, " does not support forward-mode automatic differentiation");
}

// What the nodes have in common.  N::attributes(f) shows f everything the backward depends on: f(SavedVariable&, is_output) and
// f(constant).  Compiled autograd collects it and runs apply() on tensors of its own in the saved ones' place; the gradients it
// passes have no shape yet, so an apply() hands them to its operator as they are.
template <typename N>
struct OperatorNode : Node {
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    self().attributes([](auto& a, bool = false) {
      if constexpr (std::is_same_v<std::decay_t<decltype(a)>, SavedVariable>) a.reset_data();
    });
  }
  void compiled_args(torch::dynamo::autograd::CompiledNodeArgs& args) const override {
    const_cast<OperatorNode*>(this)->self().attributes([&](auto& a, bool is_output = false) {
      if constexpr (std::is_same_v<std::decay_t<decltype(a)>, SavedVariable>) args.collect(a, is_output);
      else args.collect(a);
    });
  }
  variable_list apply_with_saved(const variable_list& inputs, torch::dynamo::autograd::SwapSavedVariables& saved) override {
    self().attributes([&](auto& a, bool = false) { saved.before(a); });
    traced = true;
    variable_list out = this->apply(variable_list(inputs));
    traced = false;
    self().attributes([&](auto& a, bool = false) { saved.after(a); });
    return out;
  }

 protected:
  bool traced = false;

 private:
  N& self() { return static_cast<N&>(*this); }
};

struct RationalSoftmaxBackward : OperatorNode<RationalSoftmaxBackward> {
  SavedVariable x;
  double eps = 0;
  template <typename F> void attributes(F&& f) { f(x, false); f(eps); }
  std::string name() const override { return "RationalSoftmaxBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return {Tensor()};
    const Tensor xt = x.unpack();
    BackwardScope scope;
    return {op_softmax_bwd(grads[0], xt, eps)};
  }
};

// The two inputs are often the halves of one packed projection, `gate, value = gv.chunk(2, -1)`.  Autograd would then
// concatenate the two gradients into the projection's (113 us of 291 at [8192, 2 x 2730] bfloat16).  When the halves are
// found to be such a pair, the node has a third edge straight to the projection, and its backward sends ONE packed gradient
// along it and nothing to the halves - unless somebody wants to see the halves' gradients themselves (hooks, retain_grad,
// torch.autograd.grad with respect to them), in which case they get them as before.
struct RationalSwiGLUBackward : OperatorNode<RationalSwiGLUBackward> {
  SavedVariable gate, value;
  bool halves = false;                                  // edge 2 leads to the packed tensor
  template <typename F> void attributes(F&& f) { f(gate, false); f(value, false); f(halves); }
  std::string name() const override { return "RationalSwiGLUBackward"; }

  static bool watched(Node* n) {
    if (!n->tensor_pre_hooks().empty() || !n->pre_hooks().empty() || !n->post_hooks().empty() || !n->retains_grad_hooks().empty()) return true;
    const auto* info = torch::autograd::get_current_graph_task_exec_info();
    if (info && !info->empty()) {
      const auto it = info->find(n);
      if (it == info->end() || it->second.captures_) return true;      // wanted for itself (or not on the way at all)
    }
    return false;
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(num_outputs());
    if (!grads[0].defined()) return out;
    const Tensor g = gate.unpack(), v = value.unpack();
    const bool to_packed = halves && !traced && task_should_compute_output(2) &&
                           !watched(next_edge(0).function.get()) && !watched(next_edge(1).function.get());
    BackwardScope scope;
    if (to_packed) {
      out[2] = op_swiglu_bwd_packed(grads[0], g, v);
    } else {
      std::tie(out[0], out[1]) = op_swiglu_bwd_dense(grads[0], g, v);
    }
    return out;
  }
};

// Whether gate and value are the two halves along the last dimension of one dense tensor that they were taken from by
// differentiable views, and if so the gradient edge of that tensor.
optional<torch::autograd::Edge> packed_edge(const Tensor& gate, const Tensor& value) {
  if (!gate.is_view() || !value.is_view() || gate.dim() == 0 || gate.sizes() != value.sizes() || gate.strides() != value.strides()) return {};
  const auto &fg = gate.grad_fn(), &fv = value.grad_fn();
  if (!fg || !fv || fg->num_outputs() != 1 || fv->num_outputs() != 1 || gate.requires_grad() != value.requires_grad()) return {};
  const at::TensorBase& base = gate._base();
  const int64_t n = gate.size(-1);
  if (!value._base().is_same(base) || !base.is_contiguous() || base.dim() != gate.dim() || base.size(-1) != 2 * n) return {};
  for (int64_t d = 0; d + 1 < gate.dim(); ++d)
    if (gate.size(d) != base.size(d) || (gate.size(d) != 1 && gate.stride(d) != base.stride(d))) return {};
  if (gate.storage_offset() != base.storage_offset() || value.storage_offset() != base.storage_offset() + n || (n != 1 && gate.stride(-1) != 1)) return {};
  const torch::autograd::Edge to = torch::autograd::impl::gradient_edge(Tensor(base));
  if (!to.is_valid() || fg->next_edge(0) != to || fv->next_edge(0) != to) return {};
  return to;
}

struct MeanErrorNormBackward : OperatorNode<MeanErrorNormBackward> {
  SavedVariable x, weight, mean;
  double eps = 0;
  template <typename F> void attributes(F&& f) { f(x, false); f(weight, false); f(mean, false); f(eps); }
  std::string name() const override { return "MeanErrorNormBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    const Tensor xt = x.unpack(), wt = weight.unpack(), mt = mean.unpack();
    BackwardScope scope;
    auto [dx, dw] = op_norm_bwd(grads[0], xt, wt, mt, eps);
    return {dx, dw};
  }
};

struct AddMeanErrorNormBackward : OperatorNode<AddMeanErrorNormBackward> {
  SavedVariable h, weight, mean;                        // h (an output), not x and residual: the backward only needs their sum
  double eps = 0;
  template <typename F> void attributes(F&& f) { f(h, true); f(weight, false); f(mean, false); f(eps); }
  std::string name() const override { return "AddMeanErrorNormBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor dh = grads[0], dy = grads[1];
    grads.clear();
    if (!dy.defined()) return {dh, dh, Tensor()};       // only the sum was used downstream
    const Tensor ht = h.unpack(shared_from_this()), wt = weight.unpack(), mt = mean.unpack();
    BackwardScope scope;
    auto [ds, dw] = op_add_norm_bwd(dy, dh.defined() ? optional<Tensor>(dh) : optional<Tensor>(), ht, wt, mt, eps);
    return {ds, ds, dw};
  }
};

struct RationalAttentionBackward : OperatorNode<RationalAttentionBackward> {
  SavedVariable q, k, v, out, L, lo, slopes, bits;
  double scale = 0, eps = 0;
  bool causal = true;
  template <typename F> void attributes(F&& f) {
    f(q, false); f(k, false); f(v, false); f(out, true); f(L, false); f(lo, false); f(slopes, false); f(bits, false);
    f(scale); f(eps); f(causal);
  }
  std::string name() const override { return "RationalAttentionBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined() || !(should_compute_output(0) || should_compute_output(1) || should_compute_output(2))) return {Tensor(), Tensor(), Tensor(), Tensor()};
    const Tensor qt = q.unpack(), kt = k.unpack(), vt = v.unpack(), ot = out.unpack(shared_from_this()), Lt = L.unpack(), lt = lo.unpack(),
                 st = slopes.unpack(), bt = bits.unpack();
    BackwardScope scope;
    auto [dq, dk, dv] = op_attn_bwd(qt, kt, vt, ot, lt, Lt, grads[0], st, scale, causal, eps, bt.defined() ? optional<Tensor>(bt) : optional<Tensor>());
    return {dq, dk, dv, Tensor()};                      // (the slopes have an edge and no gradient)
  }
};

struct RationalAttentionPackedBackward : OperatorNode<RationalAttentionPackedBackward> {
  SavedVariable qkv, out, L, lo, slopes, bits;          // out: the result [B,T,H*D] itself, so that a change in place is noticed
  double scale = 0, eps = 0;
  template <typename F> void attributes(F&& f) { f(qkv, false); f(out, true); f(L, false); f(lo, false); f(slopes, false); f(bits, false); f(scale); f(eps); }
  std::string name() const override { return "RationalAttentionPackedBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined() || !should_compute_output(0)) return {Tensor(), Tensor()};
    const Tensor pt = qkv.unpack(), ot = out.unpack(shared_from_this()), Lt = L.unpack(), lt = lo.unpack(), st = slopes.unpack(), bt = bits.unpack();
    BackwardScope scope;
    return {op_attn_bwd_packed(pt, ot, lt, Lt, grads[0], st, scale, eps, bt.defined() ? optional<Tensor>(bt) : optional<Tensor>()), Tensor()};
  }
};

// ------------------------------------------------------------------------------------- forwards (autograd key)
using torch::autograd::compute_requires_grad;
using torch::autograd::set_history;

Tensor softmax_autograd(const Tensor& x, double eps) {
  no_forward_mode("rational_softmax", x);
  std::shared_ptr<RationalSoftmaxBackward> node;
  if (compute_requires_grad(x)) {
    node = new_node<RationalSoftmaxBackward>(x);
    node->x = SavedVariable(x, false);
    node->eps = eps;
  }
  Tensor p;
  { BelowAutograd guard; p = op_softmax_fwd(x, eps); }
  if (node) set_history(p, node);
  return p;
}

Tensor swiglu_autograd(const Tensor& gate, const Tensor& value) {
  no_forward_mode("rational_swiglu", gate, value);
  std::shared_ptr<RationalSwiGLUBackward> node;
  if (compute_requires_grad(gate, value)) {
    node = new_node<RationalSwiGLUBackward>(gate, value);
    if (auto edge = packed_edge(gate, value)) {
      node->add_next_edge(*edge);
      node->halves = true;
    }
    node->gate = SavedVariable(gate, false);
    node->value = SavedVariable(value, false);
  }
  Tensor out;
  { BelowAutograd guard; out = op_swiglu_fwd(gate, value); }
  if (node) set_history(out, node);
  return out;
}

Tensor norm_autograd(const Tensor& x, const Tensor& weight, double eps) {
  no_forward_mode("mean_error_norm", x, weight);
  std::shared_ptr<MeanErrorNormBackward> node;
  if (compute_requires_grad(x, weight)) {
    node = new_node<MeanErrorNormBackward>(x, weight);
    node->x = SavedVariable(x, false);
    node->weight = SavedVariable(weight, false);
    node->eps = eps;
  }
  Tensor y, mean;
  { BelowAutograd guard; std::tie(y, mean) = op_norm_fwd(x, weight, eps); }
  if (node) {
    set_history(y, node);
    node->mean = SavedVariable(mean, false);
  }
  return y;
}

std::tuple<Tensor, Tensor> add_norm_autograd(const Tensor& x, const Tensor& residual, const Tensor& weight, double eps) {
  no_forward_mode("add_mean_error_norm", x, residual, weight);
  std::shared_ptr<AddMeanErrorNormBackward> node;
  if (compute_requires_grad(x, residual, weight)) {
    node = new_node<AddMeanErrorNormBackward>(x, residual, weight);
    node->weight = SavedVariable(weight, false);
    node->eps = eps;
  }
  Tensor h, y, mean;
  { BelowAutograd guard; std::tie(h, y, mean) = op_add_norm_fwd(x, residual, weight, eps); }
  if (node) {
    set_history(h, node);
    set_history(y, node);
    node->h = SavedVariable(h, true);
    node->mean = SavedVariable(mean, false);
  }
  return {h, y};
}

// The bits of a padding mask that is given as a [B, T] mask (mask_tokens < 0) or already packed for mask_tokens tokens.
optional<Tensor> bits_of(const optional<Tensor>& key_mask, int64_t mask_tokens, int64_t n_tokens) {
  if (!key_mask.has_value() || !key_mask->defined()) return {};
  if (mask_tokens < 0) TORCH_CHECK_VALUE(key_mask->dim() == 2, "a padding mask must be [B, T]");
  const int64_t covers = mask_tokens < 0 ? key_mask->size(1) : mask_tokens;
  TORCH_CHECK_VALUE(covers == n_tokens, "the padding mask covers ", covers, " tokens, the sequence has ", n_tokens);
  return mask_tokens < 0 ? op_pack_key_mask(*key_mask) : *key_mask;
}

Tensor attention_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& slopes, double scale, bool causal, double eps,
                          const optional<Tensor>& key_mask, int64_t mask_tokens) {
  no_forward_mode("rational_attention", q, k, v, slopes);
  std::shared_ptr<RationalAttentionBackward> node;
  if (compute_requires_grad(q, k, v, slopes)) {
    node = new_node<RationalAttentionBackward>(q, k, v, slopes);
    node->q = SavedVariable(q, false);
    node->k = SavedVariable(k, false);
    node->v = SavedVariable(v, false);
    node->slopes = SavedVariable(slopes, false);
    node->scale = scale;
    node->eps = eps;
    node->causal = causal;
  }
  Tensor out, L, lo;
  optional<Tensor> bits;
  {
    BelowAutograd guard;
    bits = bits_of(key_mask, mask_tokens, q.size(2));
    std::tie(out, L, lo) = op_attn_fwd(q, k, v, slopes, scale, causal, eps, bits, node && compute_requires_grad(q, k, v));
  }
  if (node) {
    set_history(out, node);
    node->out = SavedVariable(out, true);
    node->L = SavedVariable(L, false);
    node->lo = SavedVariable(lo, false);
    if (bits) node->bits = SavedVariable(*bits, false);
  }
  return out;
}

Tensor attention_packed_autograd(const Tensor& qkv, const Tensor& slopes, double scale, double eps, const optional<Tensor>& key_mask,
                                 int64_t mask_tokens) {
  no_forward_mode("rational_attention_packed", qkv, slopes);
  std::shared_ptr<RationalAttentionPackedBackward> node;
  if (compute_requires_grad(qkv, slopes)) {
    node = new_node<RationalAttentionPackedBackward>(qkv, slopes);
    node->qkv = SavedVariable(qkv, false);
    node->slopes = SavedVariable(slopes, false);
    node->scale = scale;
    node->eps = eps;
  }
  Tensor out, L, lo, tokens;
  optional<Tensor> bits;
  {
    BelowAutograd guard;
    bits = bits_of(key_mask, mask_tokens, qkv.size(1));
    std::tie(out, L, lo) = op_attn_fwd_packed(qkv, slopes, scale, eps, bits, node && compute_requires_grad(qkv));
    tokens = out.permute({0, 2, 1, 3}).reshape({qkv.size(0), qkv.size(1), qkv.size(3) * qkv.size(4)});     // a view: the memory order is [B,T,H,D]
  }
  if (node) {
    set_history(tokens, node);
    node->out = SavedVariable(tokens, true);
    node->L = SavedVariable(L, false);
    node->lo = SavedVariable(lo, false);
    if (bits) node->bits = SavedVariable(*bits, false);
  }
  return tokens;
}

// ------------------------------------------------------------------------------------- forwards (no autograd: inference mode)
Tensor attention_plain(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& slopes, double scale, bool causal, double eps,
                       const optional<Tensor>& key_mask, int64_t mask_tokens) {
  return std::get<0>(op_attn_fwd(q, k, v, slopes, scale, causal, eps, bits_of(key_mask, mask_tokens, q.size(2)), false));
}
Tensor attention_packed_plain(const Tensor& qkv, const Tensor& slopes, double scale, double eps, const optional<Tensor>& key_mask, int64_t mask_tokens) {
  return std::get<0>(op_attn_fwd_packed(qkv, slopes, scale, eps, bits_of(key_mask, mask_tokens, qkv.size(1)), false))
      .permute({0, 2, 1, 3}).reshape({qkv.size(0), qkv.size(1), qkv.size(3) * qkv.size(4)});
}
Tensor norm_plain(const Tensor& x, const Tensor& weight, double eps) { return std::get<0>(op_norm_fwd(x, weight, eps)); }
std::tuple<Tensor, Tensor> add_norm_plain(const Tensor& x, const Tensor& residual, const Tensor& weight, double eps) {
  auto [h, y, mean] = op_add_norm_fwd(x, residual, weight, eps);
  return {h, y};
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(algebraic, m) {
  m.def("rational_softmax(Tensor x, float eps) -> Tensor");
  m.def("rational_swiglu(Tensor gate, Tensor value) -> Tensor");
  m.def("mean_error_norm(Tensor x, Tensor weight, float eps) -> Tensor");
  m.def("add_mean_error_norm(Tensor x, Tensor residual, Tensor weight, float eps) -> (Tensor, Tensor)");
  m.def("rational_attention(Tensor q, Tensor k, Tensor v, Tensor slopes, float scale, bool causal, float eps, Tensor? key_mask, int mask_tokens) -> Tensor");
  m.def("rational_attention_packed(Tensor qkv, Tensor slopes, float scale, float eps, Tensor? key_mask, int mask_tokens) -> Tensor");
}
TORCH_LIBRARY_IMPL(algebraic, AutogradCUDA, m) {
  m.impl("rational_softmax", &softmax_autograd);
  m.impl("rational_swiglu", &swiglu_autograd);
  m.impl("mean_error_norm", &norm_autograd);
  m.impl("add_mean_error_norm", &add_norm_autograd);
  m.impl("rational_attention", &attention_autograd);
  m.impl("rational_attention_packed", &attention_packed_autograd);
}
TORCH_LIBRARY_IMPL(algebraic, CUDA, m) {
  m.impl("rational_softmax", &op_softmax_fwd);
  m.impl("rational_swiglu", &op_swiglu_fwd);
  m.impl("mean_error_norm", &norm_plain);
  m.impl("add_mean_error_norm", &add_norm_plain);
  m.impl("rational_attention", &attention_plain);
  m.impl("rational_attention_packed", &attention_packed_plain);
}

// ------------------------------------------------------------------------------------- the way in from Python
namespace {

bool tensor_arg(PyObject* o, const char* what, const Tensor*& out) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor, not %s", what, Py_TYPE(o)->tp_name);
    return false;
  }
  out = &THPVariable_Unpack(o);
  return true;
}
bool cuda_arg(const Tensor& t, const char* fn) {
  if (t.is_cuda()) return true;
  PyErr_SetString(PyExc_RuntimeError, (std::string(fn) + ": CUDA tensor required — this build has no CPU fallback").c_str());
  return false;
}
// Whether a call has to be seen by __torch_function__ (a mode, or a tensor of a class that defines it) or by a functorch transform:
// the autograd Functions' business, and the caller is told so with NotImplemented.  (A plain tensor costs a type and a bit test.)
bool not_ours(PyObject* o) {
  const Tensor& t = THPVariable_Unpack(o);
  if (t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper}))) return true;
  if (THPVariable_CheckExact(o)) return false;
  static PyObject* const disabled = [] {
    PyObject* m = PyImport_ImportModule("torch._C");
    PyObject* f = m ? PyObject_GetAttrString(m, "_disabled_torch_function_impl") : nullptr;
    Py_XDECREF(m);
    if (!f) PyErr_Clear();
    return f;
  }();
  PyObject* f = PyObject_GetAttrString(reinterpret_cast<PyObject*>(Py_TYPE(o)), "__torch_function__");
  if (!f) PyErr_Clear();
  Py_XDECREF(f);
  return f != nullptr && f != disabled;
}
template <typename... Os>
bool not_ours(PyObject* o, Os... os) { return not_ours(o) || not_ours(os...); }
#define FAT_LEAVE_TO_PYTHON(...) \
  if (at::impl::torch_function_mode_enabled() || not_ours(__VA_ARGS__)) Py_RETURN_NOTIMPLEMENTED

bool number_arg(PyObject* o, double& out) {
  out = PyFloat_AsDouble(o);
  return !(out == -1.0 && PyErr_Occurred());
}
bool count_args(Py_ssize_t n, Py_ssize_t want, const char* fn) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "%s: %zd arguments expected, got %zd", fn, want, n);
  return false;
}
// key_mask: None, a [B, T] mask, or (packed bits, tokens they cover)
bool mask_arg(PyObject* o, PyObject* tokens, optional<Tensor>& mask, int64_t& n) {
  n = PyLong_AsLongLong(tokens);
  if (n == -1 && PyErr_Occurred()) return false;
  if (o == Py_None) return true;
  const Tensor* t = nullptr;
  if (!tensor_arg(o, "key_mask", t)) return false;
  mask = *t;
  return true;
}

PyObject* py_softmax(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor* x; double eps;
  if (!count_args(n, 2, "rational_softmax") || !tensor_arg(a[0], "x", x) || !number_arg(a[1], eps) || !cuda_arg(*x, "rational_softmax")) return nullptr;
  FAT_LEAVE_TO_PYTHON(a[0]);
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    static const auto op = handle<Tensor(const Tensor&, double)>("algebraic::rational_softmax");
    r = op.call(*x, eps);
  }
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

PyObject* py_swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *g, *v;
  if (!count_args(n, 2, "rational_swiglu") || !tensor_arg(a[0], "gate", g) || !tensor_arg(a[1], "value", v) || !cuda_arg(*g, "rational_swiglu")) return nullptr;
  if (!v->is_cuda()) { PyErr_SetString(PyExc_AssertionError, "Inputs must be on CUDA"); return nullptr; }
  FAT_LEAVE_TO_PYTHON(a[0], a[1]);
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    static const auto op = handle<Tensor(const Tensor&, const Tensor&)>("algebraic::rational_swiglu");
    r = op.call(*g, *v);
  }
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

PyObject* py_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *x, *w; double eps;
  if (!count_args(n, 3, "mean_error_norm") || !tensor_arg(a[0], "x", x) || !tensor_arg(a[1], "weight", w) || !number_arg(a[2], eps) ||
      !cuda_arg(*x, "mean_error_norm")) return nullptr;
  FAT_LEAVE_TO_PYTHON(a[0], a[1]);
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    static const auto op = handle<Tensor(const Tensor&, const Tensor&, double)>("algebraic::mean_error_norm");
    r = op.call(*x, *w, eps);
  }
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

PyObject* py_add_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *x, *res, *w; double eps;
  if (!count_args(n, 4, "add_mean_error_norm") || !tensor_arg(a[0], "x", x) || !tensor_arg(a[1], "residual", res) || !tensor_arg(a[2], "weight", w) ||
      !number_arg(a[3], eps) || !cuda_arg(*x, "add_mean_error_norm")) return nullptr;
  if (!res->is_cuda()) { PyErr_SetString(PyExc_AssertionError, "Input must be on CUDA"); return nullptr; }
  FAT_LEAVE_TO_PYTHON(a[0], a[1], a[2]);
  std::tuple<Tensor, Tensor> r;
  {
    pybind11::gil_scoped_release nogil;
    static const auto op = handle<std::tuple<Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, double)>("algebraic::add_mean_error_norm");
    r = op.call(*x, *res, *w, eps);
  }
  PyObject* pair = PyTuple_New(2);
  if (!pair) return nullptr;
  PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(std::get<0>(r)));
  PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(std::get<1>(r)));
  return pair;
  END_HANDLE_TH_ERRORS
}

PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *q, *k, *v, *slopes; double scale, eps; optional<Tensor> mask; int64_t tokens;
  if (!count_args(n, 9, "rational_attention") || !tensor_arg(a[0], "q", q) || !tensor_arg(a[1], "k", k) || !tensor_arg(a[2], "v", v) ||
      !tensor_arg(a[3], "alibi_slopes", slopes) || !number_arg(a[4], scale) || !number_arg(a[6], eps) || !mask_arg(a[7], a[8], mask, tokens)) return nullptr;
  const int causal = PyObject_IsTrue(a[5]);
  if (causal < 0) return nullptr;
  if (!q->is_cuda()) { PyErr_SetString(PyExc_RuntimeError, "rational_attention: CUDA tensors required — this build has no CPU fallback"); return nullptr; }
  if (!k->is_cuda() || !v->is_cuda() || q->sizes() != k->sizes() || q->sizes() != v->sizes()) {
    PyErr_SetString(PyExc_AssertionError, "q, k and v must be CUDA tensors of one shape");
    return nullptr;
  }
  FAT_LEAVE_TO_PYTHON(a[0], a[1], a[2], a[3]);
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    static const auto op = handle<Tensor(const Tensor&, const Tensor&, const Tensor&, const Tensor&, double, bool, double, const optional<Tensor>&,
                                         int64_t)>("algebraic::rational_attention");
    r = op.call(*q, *k, *v, *slopes, scale, causal != 0, eps, mask, tokens);
  }
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

PyObject* py_attention_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *qkv, *slopes; double scale, eps; optional<Tensor> mask; int64_t tokens;
  if (!count_args(n, 6, "rational_attention_packed") || !tensor_arg(a[0], "qkv", qkv) || !tensor_arg(a[1], "alibi_slopes", slopes) ||
      !number_arg(a[2], scale) || !number_arg(a[3], eps) || !mask_arg(a[4], a[5], mask, tokens)) return nullptr;
  if (!qkv->is_cuda() || qkv->dim() != 5 || qkv->size(2) != 3) {
    PyErr_SetString(PyExc_AssertionError, "a packed projection must be a CUDA tensor [B,T,3,H,D]");
    return nullptr;
  }
  FAT_LEAVE_TO_PYTHON(a[0], a[1]);
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    static const auto op = handle<Tensor(const Tensor&, const Tensor&, double, double, const optional<Tensor>&, int64_t)>("algebraic::rational_attention_packed");
    r = op.call(*qkv, *slopes, scale, eps, mask, tokens);
  }
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyMethodDef fast(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)), METH_FASTCALL, nullptr};
}

PyMethodDef kMethods[] = {
    fast<py_softmax>("rational_softmax"), fast<py_swiglu>("rational_swiglu"), fast<py_norm>("mean_error_norm"),
    fast<py_add_norm>("add_mean_error_norm"), fast<py_attention>("rational_attention"),
    fast<py_attention_packed>("rational_attention_packed"), {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "libfat_torch_ops", "Entry points of the algebraic operators.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_libfat_torch_ops(void) { return PyModule_Create(&kModule); }
