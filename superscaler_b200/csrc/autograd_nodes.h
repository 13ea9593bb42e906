// The differentiable ops of a transformer as native autograd nodes: LayerNorm, linear (+ activation, dropout, residual), MLP, flash
// attention, the embedding lookup and the head with its loss.  Included by bindings.cpp behind the wrappers it calls; the same kernels in the same order as the
// autograd functions of ops/functional.py, which stay the path of CPU tensors and of traced or transformed calls.
//
// Why: a layer of a small model spends more time on the host than on the GPU.  A Python autograd function costs 20 to 40 us a
// call in either direction (argument checks, context, a kernel call each through the interpreter, which the backward thread
// has to share with the main thread); a node costs the kernels' launches and allocations.  Back to back on the host: scoring one
// prompt of 512 tokens with four layers 779 -> 456 us, a step of a two-layer model with two micro-batches 3387 -> 2797, forward
// and backward of one attention call 112 -> 85; with the lookup and the head as nodes too the step 2501 -> 2195 and the scoring
// 433 -> 400.
//
// (Included inside the anonymous namespace of bindings.cpp, so it includes nothing itself.)
#pragma once

std::atomic<long long> g_node_kernels{0}, g_node_calls{0};  // launches issued by nodes (the counterpart of the Python counter)

void count_kernels(int n) {
  g_node_kernels.fetch_add(n, std::memory_order_relaxed);
  g_node_calls.fetch_add(1, std::memory_order_relaxed);
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int64_t kEwBiasGeluBwd = 1, kEwDropoutBwd = 4, kEwReluBwd = 6;

// A parameter whose gradient a node takes.  Its fp32 buffer `main_grad` is an attribute of the Python object and is asked for
// when the backward runs, as the other autograd functions do: it may be attached, replaced or taken away after the forward.
// The reference does not own the parameter (whoever may look at its gradient does).
struct ParamRef {
  c10::optional<c10::weak_intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl>> ref;
  c10::ScalarType type = torch::kFloat32;
};
ParamRef param_ref(const OptTensor& param) {
  ParamRef r;
  if (param.has_value()) {
    r.ref.emplace(param->getIntrusivePtr());
    r.type = param->scalar_type();
  }
  return r;
}

// Gradient of a parameter: added to its fp32 buffer when it has one (nothing to return then), else returned in its type.
struct ParamGrad {
  OptTensor main;
  c10::ScalarType type;
};
template <size_t N>
std::array<ParamGrad, N> param_grads(const ParamRef* const (&params)[N]) {
  std::array<ParamGrad, N> out;
  pybind11::gil_scoped_acquire gil;
  for (size_t i = 0; i < N; ++i) {
    out[i].type = params[i]->type;
    if (!params[i]->ref.has_value()) continue;
    auto impl = params[i]->ref->lock();
    if (!impl.defined()) continue;
    const pybind11::object main = pybind11::getattr(pybind11::cast(Tensor(std::move(impl))), "main_grad", pybind11::none());
    if (!main.is_none()) out[i].main = main.cast<Tensor>();
  }
  return out;
}
OptTensor some(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }
const OptTensor kNone;

Tensor node_gemm(const Tensor& a, const Tensor& b, Tensor out, bool a_mn, bool b_mn, const OptTensor& bias, int64_t act,
                 const OptTensor& aux, const OptTensor& preact, const OptTensor& residual, bool accumulate, double dropout_p,
                 int64_t seed) {
  if (!out.defined()) out = torch::empty({a.size(a_mn ? 1 : 0), b.size(b_mn ? 1 : 0)}, a.options());
  gemm(a, b, out, a_mn, b_mn, bias, act, aux, preact, residual, accumulate, 1.0, dropout_p, seed);
  count_kernels(1);
  return out;
}
Tensor node_wgrad(const ParamGrad& w, const Tensor& g, const Tensor& x) {
  if (w.main.has_value()) {
    node_gemm(g, x, w.main->view({g.size(1), x.size(1)}), true, true, kNone, 0, kNone, kNone, kNone, true, 0.0, 0);
    return Tensor();
  }
  Tensor out = torch::empty({g.size(1), x.size(1)}, g.options().dtype(torch::kFloat32));
  return node_gemm(g, x, out, true, true, kNone, 0, kNone, kNone, kNone, false, 0.0, 0).to(w.type);
}
Tensor node_bgrad(const ParamGrad& b, const Tensor& g) {
  Tensor out = b.main.has_value() ? *b.main : torch::empty({g.size(1)}, g.options().dtype(torch::kFloat32));
  colsum(g, out, b.main.has_value());
  count_kernels(1);
  return b.main.has_value() ? Tensor() : out.to(b.type);
}
Tensor node_elementwise(int64_t op, const Tensor& x, const OptTensor& a, double p, int64_t seed) {
  count_kernels(1);
  return elementwise(op, x, a, kNone, p, seed);
}
Tensor node_dropout_bwd(const Tensor& g, double p, int64_t seed) {
  return p == 0.0 ? g : node_elementwise(kEwDropoutBwd, g, kNone, p, seed);
}

bool any_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}
bool wants(const OptTensor& t) { return t.has_value() && t->requires_grad(); }

// What a node keeps beside its saved tensors.
struct NodeArgs : torch::CustomClassHolder {
  bool has_bias = false, has_res = false, has_lens = false, has_table = false, same_qkv = false, same_kv = false;
  bool want_x = false, want_w = false, want_b = false;
  int64_t act = 0, seed = 0;
  double dropout_p = 0.0;
  ParamRef w, b, w2, b2;
  // attention
  int64_t B = 0, NH = 0, SQ = 0, SK = 0, HD = 0, qc = 0, kc = 0, vc = 0;
  double scale = 1.0;
  bool causal = false;
  // embedding: the tables, whose gradients need their sizes and gradient buffers; not saved tensors, which may not change in place
  Tensor table, places;
  int64_t v0 = 0;
};
using NodeArgsPtr = c10::intrusive_ptr<NodeArgs>;
void keep_args(AutogradContext* ctx, const NodeArgsPtr& a) { ctx->saved_data["args"] = c10::IValue::make_capsule(a); }
NodeArgsPtr args_of(AutogradContext* ctx) {
  return c10::static_intrusive_pointer_cast<NodeArgs>(ctx->saved_data["args"].toCapsule());
}

struct LinearNode : torch::autograd::Function<LinearNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias, const OptTensor& res,
                        const NodeArgsPtr& a, bool training) {
    Tensor pre;
    if (a->act != 0 && training) pre = torch::empty({x.size(0), w.size(0)}, x.options());
    Tensor y = node_gemm(x, w, Tensor(), false, false, bias, a->act, kNone, some(pre), res, false, a->dropout_p, a->seed);
    ctx->save_for_backward({x, w, pre});
    keep_args(ctx, a);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &pre = saved[2];
    const NodeArgsPtr a = args_of(ctx);
    const Tensor dy = grads[0].contiguous();
    Tensor g = node_dropout_bwd(dy, a->dropout_p, a->seed);
    if (a->act != 0) g = node_elementwise(a->act == ssb::kActGelu ? kEwBiasGeluBwd : kEwReluBwd, pre, g, 0.0, 0);
    Tensor dx, dw, db;
    if (a->want_x) dx = node_gemm(g, w, Tensor(), false, true, kNone, 0, kNone, kNone, kNone, false, 0.0, 0);
    if (a->want_w || a->want_b) {
      const auto pg = param_grads({&a->w, &a->b});
      if (a->want_w) dw = node_wgrad(pg[0], g, x);
      if (a->want_b) db = node_bgrad(pg[1], g);
    }
    return {dx, dw, db, a->has_res ? dy : Tensor(), Tensor(), Tensor()};
  }
};

Tensor linear_node(const Tensor& x, const Tensor& w, const OptTensor& bias, const OptTensor& res, int64_t act, double dropout_p,
                   int64_t seed) {
  auto a = c10::make_intrusive<NodeArgs>();
  a->has_res = res.has_value();
  a->want_x = x.requires_grad();
  a->want_w = w.requires_grad();
  a->want_b = wants(bias);
  a->act = act;
  a->dropout_p = dropout_p;
  a->seed = seed;
  a->w = param_ref(w);
  a->b = param_ref(bias);
  const bool training = at::GradMode::is_enabled() && (a->want_x || a->want_w || a->want_b || wants(res));
  return LinearNode::apply(x, w, bias, res, a, training);
}

struct MlpNode : torch::autograd::Function<MlpNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const OptTensor& b1, const Tensor& w2,
                        const OptTensor& b2, const OptTensor& res, const NodeArgsPtr& a, bool training) {
    Tensor pre;
    if (training) pre = torch::empty({x.size(0), w1.size(0)}, x.options());
    Tensor h = node_gemm(x, w1, Tensor(), false, false, b1, a->act, kNone, some(pre), kNone, false, 0.0, 0);
    Tensor y = node_gemm(h, w2, Tensor(), false, false, b2, 0, kNone, kNone, res, false, a->dropout_p, a->seed);
    ctx->save_for_backward({x, w1, w2, pre, h});
    keep_args(ctx, a);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w1 = saved[1], &w2 = saved[2], &pre = saved[3], &h = saved[4];
    const NodeArgsPtr a = args_of(ctx);
    const Tensor dy = grads[0].contiguous();
    const Tensor g2 = node_dropout_bwd(dy, a->dropout_p, a->seed);
    Tensor dx, db1, db2;
    const auto pg = param_grads({&a->w, &a->b, &a->w2, &a->b2});
    Tensor dw2 = node_wgrad(pg[2], g2, h);
    if (a->has_bias) db2 = node_bgrad(pg[3], g2);
    const Tensor g1 = node_gemm(g2, w2, Tensor(), false, true, kNone, a->act == ssb::kActGelu ? ssb::kActDGelu : ssb::kActDRelu,
                                pre, kNone, kNone, false, 0.0, 0);
    Tensor dw1 = node_wgrad(pg[0], g1, x);
    if (a->want_b) db1 = node_bgrad(pg[1], g1);
    if (a->want_x) dx = node_gemm(g1, w1, Tensor(), false, true, kNone, 0, kNone, kNone, kNone, false, 0.0, 0);
    return {dx, dw1, db1, dw2, db2, a->has_res ? dy : Tensor(), Tensor(), Tensor()};
  }
};

Tensor mlp_node(const Tensor& x, const Tensor& w1, const OptTensor& b1, const Tensor& w2, const OptTensor& b2,
                const OptTensor& res, int64_t act, double dropout_p, int64_t seed) {
  auto a = c10::make_intrusive<NodeArgs>();
  a->has_res = res.has_value();
  a->has_bias = b2.has_value();   // the biases' gradients are taken whenever the layer has them
  a->want_b = b1.has_value();
  a->want_x = x.requires_grad();
  a->act = act;
  a->dropout_p = dropout_p;
  a->seed = seed;
  a->w = param_ref(w1);
  a->b = param_ref(b1);
  a->w2 = param_ref(w2);
  a->b2 = param_ref(b2);
  const bool training = any_grad({&x, &w1, &w2}) || (at::GradMode::is_enabled() && (wants(b1) || wants(b2) || wants(res)));
  return MlpNode::apply(x, w1, b1, w2, b2, res, a, training);
}

struct LayerNormNode : torch::autograd::Function<LayerNormNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps,
                               bool pass_through, const NodeArgsPtr& a) {
    auto out = layernorm_fwd(x, kNone, gamma, beta, eps);
    count_kernels(1);
    ctx->save_for_backward({x, gamma, out[1], out[2]});
    ctx->set_materialize_grads(false);
    keep_args(ctx, a);
    if (pass_through) return {out[0], x.view_as(x)};
    return {out[0]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &gamma = saved[1], &mean = saved[2], &rstd = saved[3];
    const NodeArgsPtr a = args_of(ctx);
    Tensor dres = grads.size() > 1 ? grads[1] : Tensor();
    if (!grads[0].defined()) return {dres, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};  // only the residual branch was used
    const Tensor dy = grads[0].contiguous();
    if (dres.defined()) dres = dres.contiguous();
    const auto pg = param_grads({&a->w, &a->b});
    const bool accumulate = pg[0].main.has_value() && pg[1].main.has_value();
    Tensor dg = accumulate ? *pg[0].main : torch::empty_like(gamma, torch::kFloat32);
    Tensor db = accumulate ? *pg[1].main : torch::empty_like(gamma, torch::kFloat32);
    Tensor dx = layernorm_bwd(dy, x, gamma, mean, rstd, some(dres), dg, db, accumulate);
    count_kernels(2);
    if (accumulate) return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    return {dx, dg.to(pg[0].type), db.to(pg[1].type), Tensor(), Tensor(), Tensor()};
  }
};

variable_list layernorm_node(const Tensor& x, const Tensor& gamma, const Tensor& beta, double eps, bool pass_through) {
  auto a = c10::make_intrusive<NodeArgs>();
  a->w = param_ref(gamma);
  a->b = param_ref(beta);
  return LayerNormNode::apply(x, gamma, beta, eps, pass_through, a);
}

struct AttentionNode : torch::autograd::Function<AttentionNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& kv_lens,
                        const OptTensor& table, const NodeArgsPtr& a) {
    Tensor bt;
    if (table.has_value()) bt = table->to(torch::kFloat32).contiguous();
    auto out = attn_fwd(q, k, v, a->B, a->NH, a->SQ, a->SK, a->HD, a->qc, a->kc, a->vc, a->scale, a->causal, kv_lens,
                        a->dropout_p, a->seed, some(bt));
    count_kernels(1);
    ctx->save_for_backward({q, k, v, out[0], out[1], kv_lens.has_value() ? *kv_lens : Tensor(), bt});
    keep_args(ctx, a);
    return out[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
    const NodeArgsPtr a = args_of(ctx);
    const OptTensor lens = a->has_lens ? OptTensor(saved[5]) : kNone, bt = a->has_table ? OptTensor(saved[6]) : kNone;
    Tensor dbias;
    if (bt.has_value()) dbias = torch::zeros_like(*bt);
    const Tensor dout = grads[0].contiguous();
    // gradients land in matrices laid out like their inputs, so a fused QKV input gets ONE gradient; columns no head
    // writes (a wider carrier matrix) must read as zero
    const int64_t w = a->NH * a->HD;
    auto like = [](const Tensor& t, int64_t cols) { return t.size(1) == cols ? torch::empty_like(t) : torch::zeros_like(t); };
    Tensor dq = like(q, a->same_qkv ? 3 * w : w);
    Tensor dk = a->same_qkv ? dq : like(k, a->same_kv ? 2 * w : w);
    Tensor dv = a->same_qkv || a->same_kv ? dk : like(v, w);
    attn_bwd(q, k, v, saved[3], saved[4], dout, dq, dk, dv, a->B, a->NH, a->SQ, a->SK, a->HD, a->qc, a->kc, a->vc, a->qc, a->kc,
             a->vc, a->scale, a->causal, lens, a->dropout_p, a->seed, bt, some(dbias));
    count_kernels(3);
    return {dq, a->same_qkv ? Tensor() : dk, a->same_qkv || a->same_kv ? Tensor() : dv, Tensor(), dbias, Tensor()};
  }
};

Tensor attention_node(const Tensor& q, const Tensor& k, const Tensor& v, int64_t B, int64_t NH, int64_t SQ, int64_t SK, int64_t HD,
                      int64_t qc, int64_t kc, int64_t vc, double scale, bool causal, const OptTensor& kv_lens, double dropout_p,
                      int64_t seed, const OptTensor& table) {
  auto a = c10::make_intrusive<NodeArgs>();
  a->B = B; a->NH = NH; a->SQ = SQ; a->SK = SK; a->HD = HD;
  a->qc = qc; a->kc = kc; a->vc = vc;
  a->scale = scale;
  a->causal = causal;
  a->dropout_p = dropout_p;
  a->seed = seed;
  a->has_lens = kv_lens.has_value();
  a->has_table = table.has_value();
  a->same_kv = k.data_ptr() == v.data_ptr() && k.sizes() == v.sizes();
  a->same_qkv = a->same_kv && q.data_ptr() == k.data_ptr() && q.sizes() == k.sizes();
  return AttentionNode::apply(q, k, v, kv_lens, table, a);
}

// Which kernel sums the embedding gradient (set_deterministic_embedding_grad of ops/functional.py): rows in token order, or float
// atomics.  Read by the threads that run a backward.
std::atomic<bool> g_embedding_in_order{true};

struct EmbeddingNode : torch::autograd::Function<EmbeddingNode> {
  // The tables are passed for the graph alone; the values come with the arguments.
  static Tensor forward(AutogradContext* ctx, const Tensor& ids, const OptTensor& pos, const Tensor& W, const OptTensor& P,
                        const NodeArgsPtr& a) {
    Tensor flat_pos;
    if (pos.has_value()) flat_pos = pos->contiguous().view(-1);
    Tensor y = embedding_fwd(ids.contiguous().view(-1), some(flat_pos), W, P, a->v0, a->dropout_p, a->seed);
    count_kernels(1);
    ctx->save_for_backward({ids, pos.has_value() ? *pos : Tensor()});
    keep_args(ctx, a);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const NodeArgsPtr a = args_of(ctx);
    const Tensor g = grads[0].contiguous(), ids = saved[0].contiguous().view(-1);
    Tensor pos;
    if (saved[1].defined()) pos = saved[1].contiguous().view(-1);
    const auto pg = param_grads({&a->w, &a->b});
    auto buffer = [&](const ParamGrad& p, const Tensor& t) {
      return p.main.has_value() ? *p.main : torch::zeros(t.sizes(), g.options().dtype(torch::kFloat32));
    };
    Tensor dW = buffer(pg[0], a->table), dP;
    if (a->places.defined()) dP = buffer(pg[1], a->places);
    if (!g_embedding_in_order) {
      embedding_bwd(ids, some(pos), g, dW, some(dP), a->v0, a->dropout_p, a->seed);
      count_kernels(1);
    } else if (ids.numel() <= ssb::embedding_group_max_tokens()) {
      embedding_bwd_grouped(ids, some(pos), g, dW, some(dP), a->v0, a->dropout_p, a->seed);
      count_kernels(2);
    } else {
      auto sorted = [&](const Tensor& keys_of, const Tensor& dst, int64_t k0) {
        const auto order = torch::sort(embedding_keys(keys_of, k0, dst.size(0)), /*stable=*/true, 0, false);
        count_kernels(1);
        embedding_bwd_sorted(std::get<0>(order), std::get<1>(order), g, dst, 0, a->dropout_p, a->seed);
      };
      sorted(ids, dW, a->v0);
      if (pos.defined() && dP.defined()) sorted(pos, dP, 0);
    }
    return {Tensor(), Tensor(), pg[0].main.has_value() ? Tensor() : dW.to(a->table.scalar_type()),
            !dP.defined() || pg[1].main.has_value() ? Tensor() : dP.to(a->places.scalar_type()), Tensor()};
  }
};

Tensor embedding_node(const Tensor& ids, const OptTensor& pos, const Tensor& W, const OptTensor& P, int64_t v0, double dropout_p,
                      int64_t seed) {
  auto a = c10::make_intrusive<NodeArgs>();
  a->v0 = v0;
  a->dropout_p = dropout_p;
  a->seed = seed;
  a->table = W;
  a->w = param_ref(W);
  if (P.has_value()) {
    a->places = *P;
    a->b = param_ref(P);
  }
  return EmbeddingNode::apply(ids, pos, W, P, a);
}

struct HeadLossNode : torch::autograd::Function<HeadLossNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& W, const Tensor& targets, const OptTensor& mask,
                        const NodeArgsPtr& a) {
    Tensor logits = node_gemm(x, W, Tensor(), false, false, kNone, 0, kNone, kNone, kNone, false, 0.0, 0);
    const Tensor losses = ce_loss_grad(logits, targets.contiguous().view(-1), mask, a->v0, a->scale);
    count_kernels(1);
    ctx->save_for_backward({x, W, logits});
    keep_args(ctx, a);
    return losses.sum() * a->scale;
  }
  static variable_list backward(AutogradContext* ctx, variable_list) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &W = saved[1], &g = saved[2];
    const NodeArgsPtr a = args_of(ctx);
    Tensor dx, dw;
    if (a->want_x) dx = node_gemm(g, W, Tensor(), false, true, kNone, 0, kNone, kNone, kNone, false, 0.0, 0);
    if (a->want_w) dw = node_wgrad(param_grads({&a->w})[0], g, x);
    return {dx, dw, Tensor(), Tensor(), Tensor()};
  }
};

Tensor head_loss_node(const Tensor& x, const Tensor& W, const Tensor& targets, const OptTensor& mask, int64_t v0, double loss_scale) {
  auto a = c10::make_intrusive<NodeArgs>();
  a->v0 = v0;
  a->scale = loss_scale;
  a->want_x = x.requires_grad();
  a->want_w = W.requires_grad();
  a->w = param_ref(W);
  return HeadLossNode::apply(x, W, targets, mask, a);
}
