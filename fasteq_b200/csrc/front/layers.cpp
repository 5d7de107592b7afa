// SO3Linear, the dense layer, SiLU and the radial chain.  The first two are bilinear, so each term of the second backward is one of their
// three launches again with a cotangent in an operand's place.
#include "front.h"

namespace front {
namespace {

// ------------------------------------------------------------------------------------------------ SO3Linear
constexpr int64_t kTf32 = 0;

struct Geometry : torch::CustomClassHolder {
  std::vector<int32_t> in_row, out_row, rows;
  std::vector<int64_t> block;          // weight block of each path
  std::vector<double> coeff;
  int u = 0, v = 0, in_rows = 0, out_rows = 0;
  bool in_order = true;
  std::string key;
  PyKeep wgrad;                        // (x, grad_out, precision, batch, shape of w) -> grad_w

  Geometry(std::vector<std::array<int64_t, 4>> mapping, std::vector<double> c, int u_, int v_, int I, int J, py::object wg)
      : coeff(std::move(c)), u(u_), v(v_), in_rows(I), out_rows(J), wgrad(std::move(wg)) {
    key = "eqlinear";
    auto add = [&](double x) { key.append(reinterpret_cast<const char*>(&x), sizeof x); };
    for (size_t q = 0; q < mapping.size(); ++q) {
      in_row.push_back((int32_t)mapping[q][0]); out_row.push_back((int32_t)mapping[q][1]); rows.push_back((int32_t)mapping[q][3]);
      block.push_back(mapping[q][2]);
      in_order = in_order && mapping[q][2] == (int64_t)q;
      for (int64_t x : mapping[q]) add((double)x);
      add(coeff[q]);
    }
    add(u); add(v); add(I); add(J);
  }
  int64_t paths() const { return (int64_t)rows.size(); }
  fasteq_eqlinear_problem problem(int64_t precision, int64_t batch) const {
    fasteq_eqlinear_problem p{};
    p.precision = (int32_t)precision; p.u = u; p.v = v; p.in_rows = in_rows; p.out_rows = out_rows; p.num_paths = (int32_t)paths();
    p.batch = batch; p.in_row = in_row.data(); p.out_row = out_row.data(); p.rows = rows.data(); p.coeff = coeff.data();
    return p;
  }
};
using Geom = c10::intrusive_ptr<Geometry>;

// forward (a = x) or grad_x (a = grad_out); `keep`: w is a weight whose prepared form may be kept
Tensor eqlinear_apply(const Geometry& g, int64_t precision, const Tensor& w, const Tensor& a, bool dgrad, bool keep) {
  c10::cuda::CUDAGuard guard(a.device());
  const int64_t a_cols = dgrad ? (int64_t)g.out_rows * g.v : (int64_t)g.in_rows * g.u, c_cols = dgrad ? (int64_t)g.in_rows * g.u : (int64_t)g.out_rows * g.v;
  const int64_t batch = a.numel() / a_cols;
  const Tensor ac = a.contiguous();
  Tensor out = at::empty({batch, c_cols}, ac.options());
  const auto p = g.problem(precision, batch);
  cudaStream_t s = stream_of(ac);
  auto ordered = [&] {                 // weight block of path q at index q
    Tensor w3 = w.reshape({g.paths(), g.u, g.v}).contiguous();
    return g.in_order ? w3 : w3.index_select(0, torch::tensor(g.block, torch::kInt64).to(w.device())).contiguous();
  };
  if (precision == kTf32) {
    auto build = [&]() -> Tensor {
      const Tensor w3 = ordered();
      Tensor packed = at::empty({2 * w3.numel()}, w3.options());
      const int rc = core.eqlinear_pack(&p, dgrad, w3.const_data_ptr(), packed.data_ptr(), s);
      if (rc == FASTEQ_UNSUPPORTED) return Tensor();
      check(rc, "fasteq_eqlinear_pack", core.last_cuda_error);
      return packed;
    };
    std::optional<Tensor> packed;
    if (keep) packed = prepared({w}, g.key + (dgrad ? "d" : "f"), build);
    if (!packed) { Tensor t = build(); if (t.defined()) packed = t; }
    if (packed) {
      const int rc = (dgrad ? core.eqlinear_dgrad_packed : core.eqlinear_forward_packed)(&p, packed->const_data_ptr(), ac.const_data_ptr(), out.data_ptr(), s);
      if (rc != FASTEQ_UNSUPPORTED) {
        check(rc, dgrad ? "fasteq_eqlinear_dgrad_packed" : "fasteq_eqlinear_forward_packed", core.last_cuda_error);
        return out;
      }
    }
  }
  const Tensor w3 = ordered();
  check((dgrad ? core.eqlinear_dgrad : core.eqlinear_forward)(&p, w3.const_data_ptr(), ac.const_data_ptr(), out.data_ptr(), s),
        dgrad ? "fasteq_eqlinear_dgrad" : "fasteq_eqlinear_forward", core.last_cuda_error);
  return out;
}

Tensor eqlinear_wgrad(const Geometry& g, int64_t precision, const Tensor& w, const Tensor& x, const Tensor& go) {
  py::gil_scoped_acquire gil;
  return g.wgrad.get()(x, go, precision, x.numel() / ((int64_t)g.in_rows * g.u), w.sizes().vec()).cast<Tensor>();
}

struct EqLinearBackward : torch::autograd::Function<EqLinearBackward> {
  static variable_list forward(AutogradContext* ctx, const Tensor& go, const Tensor& w, const Tensor& x, const Geom& g, int64_t precision, bool need_w, bool need_x) {
    ctx->save_for_backward({go, w, x});
    ctx->saved_data["g"] = capsule(g);
    ctx->saved_data["p"] = precision; ctx->saved_data["w"] = need_w; ctx->saved_data["x"] = need_x;
    ctx->set_materialize_grads(false);
    Tensor dw = need_w ? eqlinear_wgrad(*g, precision, w, x, go) : at::empty({0}, w.options());
    Tensor dx = need_x ? eqlinear_apply(*g, precision, w, go, true, true).view(x.sizes()) : at::empty({0}, x.options());
    return {dw, dx};
  }
  static variable_list backward(AutogradContext* ctx, variable_list gg);
};

struct EqLinear : torch::autograd::Function<EqLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& w, const Tensor& x, const Geom& g, int64_t precision) {
    ctx->save_for_backward({w, x});
    ctx->saved_data["g"] = capsule(g);
    ctx->saved_data["p"] = precision;
    return eqlinear_apply(*g, precision, w, x, false, true);
  }
  static variable_list backward(AutogradContext* ctx, variable_list go) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &w = saved[0], &x = saved[1];
    const bool need_w = ctx->needs_input_grad(0), need_x = ctx->needs_input_grad(1);
    if (!need_w && !need_x) return {Tensor(), Tensor(), Tensor(), Tensor()};
    auto d = EqLinearBackward::apply(go[0].contiguous(), w, x, uncapsule<Geometry>(ctx->saved_data["g"]), ctx->saved_data["p"].toInt(), need_w, need_x);
    return {need_w ? d[0] : Tensor(), need_x ? d[1] : Tensor(), Tensor(), Tensor()};
  }
};

// in grad mode (a third order may follow) from the nodes, else from launches
variable_list EqLinearBackward::backward(AutogradContext* ctx, variable_list gg) {
  const auto saved = ctx->get_saved_variables();
  const Tensor &go = saved[0], &w = saved[1], &x = saved[2];
  const Geom g = uncapsule<Geometry>(ctx->saved_data["g"]);
  const int64_t precision = ctx->saved_data["p"].toInt();
  const Tensor ggw = ctx->saved_data["w"].toBool() ? defined_contiguous(gg[0]) : Tensor();
  const Tensor ggx = ctx->saved_data["x"].toBool() ? defined_contiguous(gg[1]) : Tensor();
  const bool want_go = ctx->needs_input_grad(0), want_w = ctx->needs_input_grad(1), want_x = ctx->needs_input_grad(2);
  const bool nodes = at::GradMode::is_enabled();
  auto forward = [&](const Tensor& b, const Tensor& a, bool weight) {
    return nodes ? Tensor(EqLinear::apply(b, a, g, precision)) : eqlinear_apply(*g, precision, b, a, false, weight);
  };
  Tensor d_go, d_w, d_x;
  if (want_go) {
    if (ggx.defined()) d_go = forward(w, ggx, true);
    if (ggw.defined()) {
      const Tensor t = forward(ggw, x, false);
      d_go = d_go.defined() ? d_go + t : t;
    }
    if (d_go.defined()) d_go = d_go.view(go.sizes());
  }
  if (want_w && ggx.defined()) d_w = nodes ? EqLinearBackward::apply(go, w, ggx, g, precision, true, false)[0] : eqlinear_wgrad(*g, precision, w, ggx, go);
  if (want_x && ggw.defined())
    d_x = nodes ? EqLinearBackward::apply(go, ggw, x, g, precision, false, true)[1] : eqlinear_apply(*g, precision, ggw, go, true, false).view(x.sizes());
  return {d_go, d_w, d_x, Tensor(), Tensor(), Tensor(), Tensor()};
}

Tensor eqlinear(const Geom& g, const Tensor& w, const Tensor& x, int64_t precision) {
  if (!x.is_cuda() || !w.is_cuda()) fail("eqlinear: x and w must be CUDA tensors: fasteq_b200 has no CPU path");
  const int64_t cols = (int64_t)g->in_rows * g->u;
  TORCH_CHECK_VALUE(cols > 0, "eqlinear: the descriptor has no input values (I*U = ", cols, ")");
  TORCH_CHECK_VALUE((x.dim() > 0 && x.size(-1) == cols) || x.numel() % cols == 0, "eqlinear: x has ", x.numel(), " elements, not a multiple of I*U = ", cols);
  TORCH_CHECK_VALUE(w.numel() == g->paths() * g->u * g->v, "eqlinear: w has ", w.numel(), " elements, expected P*U*V = ", g->paths() * g->u * g->v);
  return EqLinear::apply(w, x, g, precision);
}

// ------------------------------------------------------------------------------------------------ dense layer (FP32)
// a [M, K] bt[N, K]^T.  `weight`: the parameter `bt` derives from (undefined: a cotangent, whose parts are not kept)
Tensor gemm(const Tensor& a, const Tensor& bt, const Tensor& weight, bool transposed) {
  c10::cuda::CUDAGuard guard(a.device());
  const Tensor ac = a.contiguous();
  const int64_t M = ac.size(0), K = ac.size(1), N = bt.size(0);
  Tensor out = at::empty({M, N}, ac.options());
  cudaStream_t s = stream_of(ac);
  auto build = [&] {
    const Tensor b = bt.contiguous();
    Tensor split = at::empty({2 * b.numel()}, b.options());
    check(core.gemm_tf32x3_split(b.const_data_ptr(), b.numel(), split.data_ptr(), s), "fasteq_gemm_tf32x3_split", core.last_cuda_error);
    return split;
  };
  std::optional<Tensor> split;
  if (weight.defined()) split = prepared({weight}, transposed ? "dense_t" : "dense", build);
  if (!split) split = build();
  const int rc = core.gemm_tf32x3_presplit(ac.const_data_ptr(), split->const_data_ptr(), out.data_ptr(), M, (int32_t)N, (int32_t)K, s);
  if (rc == FASTEQ_UNSUPPORTED) {      // operand alignment: the FP32 tile kernel of the one-path SO3Linear takes any
    static const int32_t zero = 0, one = 1;
    static const double unit = 1.0;
    fasteq_eqlinear_problem p{};
    p.precision = FASTEQ_EQLIN_FP32; p.u = (int32_t)K; p.v = (int32_t)N; p.in_rows = p.out_rows = p.num_paths = 1; p.batch = M;
    p.in_row = &zero; p.out_row = &zero; p.rows = &one; p.coeff = &unit;
    const Tensor w = bt.t().contiguous();
    check(core.eqlinear_forward(&p, w.const_data_ptr(), ac.const_data_ptr(), out.data_ptr(), s), "fasteq_eqlinear_forward", core.last_cuda_error);
    return out;
  }
  check(rc, "fasteq_gemm_tf32x3", core.last_cuda_error);
  return out;
}

// g [M, N]^T x [M, K] -> [N, K]
Tensor row_product(const Tensor& g, const Tensor& x) {
  c10::cuda::CUDAGuard guard(g.device());
  const Tensor a = g.contiguous(), b = x.contiguous();
  Tensor out = at::empty({a.size(1), b.size(1)}, a.options());
  if (a.size(0) == 0) return out.zero_();
  static const int32_t zero = 0, one = 1;
  static const double unit = 1.0;
  fasteq_eqlinear_problem p{};
  p.precision = FASTEQ_EQLIN_FP32; p.u = (int32_t)a.size(1); p.v = (int32_t)b.size(1); p.in_rows = p.out_rows = p.num_paths = 1; p.batch = a.size(0);
  p.in_row = &zero; p.out_row = &zero; p.rows = &one; p.coeff = &unit;
  int64_t need = 0;
  check(core.eqlinear_wgrad_scratch(&p, a.const_data_ptr(), b.const_data_ptr(), &need), "fasteq_eqlinear_wgrad_scratch", core.last_cuda_error);
  Tensor scratch = at::empty({std::max<int64_t>(need, 16)}, a.options().dtype(at::kByte));
  check(core.eqlinear_wgrad_with(&p, a.const_data_ptr(), b.const_data_ptr(), out.data_ptr(), scratch.data_ptr(), scratch.numel(), stream_of(a)),
        "fasteq_eqlinear_wgrad_with", core.last_cuda_error);
  return out;
}

struct DenseBackward : torch::autograd::Function<DenseBackward> {
  static variable_list forward(AutogradContext* ctx, const Tensor& g, const Tensor& x, const Tensor& weight, bool need_x, bool need_w) {
    ctx->save_for_backward({g, x, weight});
    ctx->saved_data["x"] = need_x; ctx->saved_data["w"] = need_w;
    ctx->set_materialize_grads(false);
    return {need_x ? gemm(g, weight.t(), weight, true) : at::empty({0}, x.options()), need_w ? row_product(g, x) : at::empty({0}, weight.options())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list gg);
};

struct Dense : torch::autograd::Function<Dense> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight) {
    ctx->save_for_backward({x, weight});
    return gemm(x, weight, weight, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list go) {
    const auto saved = ctx->get_saved_variables();
    const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
    if (!need_x && !need_w) return {Tensor(), Tensor()};
    auto d = DenseBackward::apply(go[0].contiguous(), saved[0], saved[1], need_x, need_w);
    return {need_x ? d[0] : Tensor(), need_w ? d[1] : Tensor()};
  }
};

// d_g = ggx W^T + x ggW^T,  d_x = g ggW,  d_W = g^T ggx: in grad mode (a third order may follow) from the nodes, else from launches
variable_list DenseBackward::backward(AutogradContext* ctx, variable_list gg) {
  const auto saved = ctx->get_saved_variables();
  const Tensor &g = saved[0], &x = saved[1], &weight = saved[2];
  const Tensor ggx = ctx->saved_data["x"].toBool() ? defined_contiguous(gg[0]) : Tensor();
  const Tensor ggw = ctx->saved_data["w"].toBool() ? defined_contiguous(gg[1]) : Tensor();
  const bool nodes = at::GradMode::is_enabled();
  auto product = [&](const Tensor& a, const Tensor& bt, const Tensor& w) { return nodes ? Tensor(Dense::apply(a, bt)) : gemm(a, bt, w, false); };
  Tensor d_g, d_x, d_w;
  if (ctx->needs_input_grad(0)) {
    if (ggx.defined()) d_g = product(ggx, weight, weight);
    if (ggw.defined()) {
      const Tensor t = product(x, ggw, Tensor());
      d_g = d_g.defined() ? d_g + t : t;
    }
  }
  if (ctx->needs_input_grad(1) && ggw.defined()) d_x = product(g, ggw.t(), Tensor());
  if (ctx->needs_input_grad(2) && ggx.defined()) d_w = nodes ? DenseBackward::apply(g, ggx, weight, false, true)[1] : row_product(g, ggx);
  return {d_g, d_x, d_w, Tensor(), Tensor()};
}

// ------------------------------------------------------------------------------------------------ SiLU
variable_list silu_run(int order, const Tensor& z, const Tensor& g, const Tensor& h) {
  c10::cuda::CUDAGuard guard(z.device());
  Tensor out0 = at::empty_like(z), out1 = order == 2 ? at::empty_like(z) : Tensor();
  check(core.silu(z.scalar_type() == at::kDouble, order, ptr(z), ptr(g), ptr(h), mptr(out0), mptr(out1), z.numel(), stream_of(z)), "fasteq_silu",
        core.last_cuda_error);
  return {out0, out1};
}

struct SiLUBackward : torch::autograd::Function<SiLUBackward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& g, const Tensor& z) {
    ctx->save_for_backward({g, z});
    return silu_run(1, z, g, Tensor())[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list go) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &g = saved[0], &z = saved[1], &h = go[0];
    if (at::GradMode::is_enabled()) {   // a third order is asked for: the same expressions as torch operations
      const Tensor s = at::sigmoid(z);
      return {h * s * (1 + z * (1 - s)), h * g * s * (1 - s) * (2 + z * (1 - 2 * s))};
    }
    return silu_run(2, z, g, h.contiguous());
  }
};

struct SiLU : torch::autograd::Function<SiLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& z) {
    ctx->save_for_backward({z});
    return silu_run(0, z, Tensor(), Tensor())[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list go) {
    return {SiLUBackward::apply(go[0].contiguous(), ctx->get_saved_variables()[0])};
  }
};

// ------------------------------------------------------------------------------------------------ radial chain
constexpr int64_t kWidth = 64;

std::optional<Tensor> chain_prepared(const std::vector<Tensor>& ws, bool backward, cudaStream_t s) {
  if (ws.size() < 2) return std::nullopt;
  std::vector<Tensor> hidden(ws.begin() + 1, ws.end());
  return prepared(hidden, backward ? "chain_b" : "chain_f", [&] {
    std::vector<const float*> p;
    for (const Tensor& w : hidden) p.push_back(w.const_data_ptr<float>());
    Tensor prep = at::empty({(int64_t)hidden.size() * 2 * kWidth * kWidth}, hidden[0].options());
    check(core.radial_chain_prepare(p.data(), (int32_t)ws.size(), backward, prep.data_ptr<float>(), s), "fasteq_radial_chain_prepare", core.last_cuda_error);
    return prep;
  });
}

// The chain's gradient as differentiable operations, layer by layer: what enters it (the gradient of the chain's value) and the basis may be
// differentiated through in their turn, as where a loss on forces trains other layers behind frozen radial ones.
Tensor chain_gradient(const Tensor& go, const Tensor& basis, const std::vector<Tensor>& ws) {
  variable_list z;
  Tensor h = basis, g = go;
  for (const Tensor& w : ws) {
    z.push_back(Dense::apply(h, w));
    if (z.size() < ws.size()) h = SiLU::apply(z.back());
  }
  for (size_t l = ws.size(); l-- > 0;) g = Dense::apply(SiLUBackward::apply(g, z[l]), ws[l].t());
  return g;
}

struct RadialChain : torch::autograd::Function<RadialChain> {
  static bool takes(const Tensor& basis, const std::vector<Tensor>& ws) {
    if (!basis.is_cuda() || basis.scalar_type() != at::kFloat || basis.dim() != 2 || basis.size(0) == 0) return false;
    if (ws.empty() || ws.size() > 3 || basis.size(1) < 1 || basis.size(1) > 16) return false;
    for (size_t i = 0; i < ws.size(); ++i) {
      const Tensor& w = ws[i];
      if (w.scalar_type() != at::kFloat || !w.is_cuda() || (at::GradMode::is_enabled() && w.requires_grad()) || w.dim() != 2 || w.size(0) != kWidth ||
          w.size(1) != (i ? kWidth : basis.size(1)))
        return false;
    }
    return true;
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& basis, at::TensorList weights) {
    c10::cuda::CUDAGuard guard(basis.device());
    std::vector<Tensor> ws;
    std::vector<const float*> hidden;
    for (const Tensor& w : weights) ws.push_back(w.contiguous());
    for (size_t i = 1; i < ws.size(); ++i) hidden.push_back(ws[i].const_data_ptr<float>());
    hidden.push_back(nullptr);
    const int64_t E = basis.size(0), nb = basis.size(1), L = (int64_t)ws.size();
    Tensor out = at::empty({E, kWidth}, basis.options()), deriv = at::empty({std::max<int64_t>(L - 1, 1), E, kWidth}, basis.options());
    cudaStream_t s = stream_of(basis);
    const auto prep = chain_prepared(ws, false, s);
    check(core.radial_chain_forward(basis.const_data_ptr<float>(), E, (int32_t)nb, ws[0].const_data_ptr<float>(), hidden.data(),
                                    prep ? prep->const_data_ptr<float>() : nullptr, (int32_t)L, out.data_ptr<float>(), deriv.data_ptr<float>(), s),
          "fasteq_radial_chain_forward", core.last_cuda_error);
    variable_list keep = {basis, deriv};
    keep.insert(keep.end(), ws.begin(), ws.end());
    ctx->save_for_backward(keep);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list go) {
    auto saved = ctx->get_saved_variables();
    std::vector<Tensor> ws(saved.begin() + 2, saved.end());
    variable_list grads(1 + ws.size());
    if (!ctx->needs_input_grad(0)) return grads;
    const Tensor& basis = saved[0];
    c10::cuda::CUDAGuard guard(basis.device());
    const Tensor g = go[0].contiguous();
    if (at::GradMode::is_enabled()) {
      grads[0] = chain_gradient(g, basis, ws);
      return grads;
    }
    std::vector<const float*> hidden;
    for (size_t i = 1; i < ws.size(); ++i) hidden.push_back(ws[i].const_data_ptr<float>());
    hidden.push_back(nullptr);
    Tensor gb = at::empty_like(basis);
    cudaStream_t s = stream_of(basis);
    const auto prep = chain_prepared(ws, true, s);
    check(core.radial_chain_backward(g.const_data_ptr<float>(), saved[1].const_data_ptr<float>(), basis.const_data_ptr<float>(), basis.size(0),
                                     (int32_t)basis.size(1), ws[0].const_data_ptr<float>(), hidden.data(), prep ? prep->const_data_ptr<float>() : nullptr,
                                     (int32_t)ws.size(), gb.data_ptr<float>(), s),
          "fasteq_radial_chain_backward", core.last_cuda_error);
    grads[0] = gb;
    return grads;
  }
};

}  // namespace

void bind_layers(py::module_& m) {
  py::class_<Geometry, Geom>(m, "Geometry")
      .def(py::init([](std::vector<std::array<int64_t, 4>> mapping, std::vector<double> coeff, int u, int v, int I, int J, py::object wgrad) {
        return c10::make_intrusive<Geometry>(std::move(mapping), std::move(coeff), u, v, I, J, std::move(wgrad));
      }));
  m.def("eqlinear", &eqlinear);
  m.def("dense", [](const Tensor& x, const Tensor& weight) -> Tensor { return Dense::apply(x, weight); });
  m.def("silu", [](const Tensor& z) -> Tensor { return SiLU::apply(z); });
  m.def("eqlinear_launch", [](const Geom& g, const Tensor& w, const Tensor& a, int64_t precision, bool dgrad) {
    at::AutoGradMode no_grad(false);
    return eqlinear_apply(*g, precision, w, a, dgrad, true);
  });
  m.def("radial_chain_takes", &RadialChain::takes);
  m.def("radial_chain", [](const Tensor& basis, std::vector<Tensor> weights) -> std::optional<Tensor> {
    if (!RadialChain::takes(basis, weights)) return std::nullopt;
    return RadialChain::apply(basis.contiguous(), at::TensorList(weights));
  });
}

}  // namespace front
