// Edge geometry, the radius graph and SymmetricContraction's inference path.
#include "front.h"
#include <pybind11/numpy.h>

namespace front {
namespace {

Tensor int32_contiguous(const Tensor& t) { return (t.scalar_type() == at::kInt ? t : t.to(at::kInt)).contiguous(); }
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kDouble ? 1 : 0; }

// what Python's once_differentiable does: a second differentiation is an error, not a zero
variable_list once(variable_list grads, const variable_list& inputs) {
  if (!at::GradMode::is_enabled()) return grads;
  bool any = false;
  for (const Tensor& t : inputs) any = any || (t.defined() && t.requires_grad());
  if (!any) return grads;
  variable_list live;
  for (Tensor& t : grads) if (t.defined()) live.push_back(t);
  auto refuse = std::make_shared<torch::autograd::DelayedError>("trying to differentiate twice a function that was marked with @once_differentiable",
                                                                (int64_t)live.size());
  for (Tensor& t : live) t = t.detach().requires_grad_(true);
  live = (*refuse)(std::move(live));
  size_t k = 0;
  for (Tensor& t : grads) if (t.defined()) t = live[k++];
  return grads;
}

struct EdgeGeometry : torch::autograd::Function<EdgeGeometry> {
  static variable_list forward(AutogradContext* ctx, const Tensor& pos_, const Tensor& src_, const Tensor& dst_, const Tensor& shift_, double r_max,
                               int64_t n_basis, int64_t p) {
    c10::cuda::CUDAGuard guard(pos_.device());
    const Tensor pos = pos_.contiguous(), shift = shift_.to(pos.scalar_type()).contiguous(), src = int32_contiguous(src_), dst = int32_contiguous(dst_);
    const int64_t E = src.numel();
    Tensor vec = at::empty({E, 3}, pos.options()), basis = at::empty({E, n_basis}, pos.options());
    check(core.edge_geometry_forward(dtype_code(pos), ptr(pos), src.const_data_ptr<int32_t>(), dst.const_data_ptr<int32_t>(), ptr(shift), E, pos.size(0),
                                     r_max, (int32_t)n_basis, (int32_t)p, mptr(vec), mptr(basis), stream_of(pos)),
          "fasteq_edge_geometry_forward", core.last_cuda_error);
    ctx->save_for_backward({pos, src, dst, shift});
    ctx->saved_data["r"] = r_max; ctx->saved_data["n"] = n_basis; ctx->saved_data["p"] = p;
    ctx->set_materialize_grads(false);
    return {vec, basis};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    variable_list grads(7);
    if (!ctx->needs_input_grad(0) || (!g[0].defined() && !g[1].defined())) return grads;
    const auto saved = ctx->get_saved_variables();
    const Tensor &pos = saved[0], &src = saved[1], &dst = saved[2], &shift = saved[3];
    {
      at::AutoGradMode no_grad(false);
      c10::cuda::CUDAGuard guard(pos.device());
      const Tensor gv = defined_contiguous(g[0]), gb = defined_contiguous(g[1]);
      Tensor g_pos = at::empty_like(pos);
      check(core.edge_geometry_backward(dtype_code(pos), ptr(pos), src.const_data_ptr<int32_t>(), dst.const_data_ptr<int32_t>(), ptr(shift), ptr(gv), ptr(gb),
                                        src.numel(), pos.size(0), ctx->saved_data["r"].toDouble(), (int32_t)ctx->saved_data["n"].toInt(),
                                        (int32_t)ctx->saved_data["p"].toInt(), mptr(g_pos), stream_of(pos)),
            "fasteq_edge_geometry_backward", core.last_cuda_error);
      grads[0] = g_pos;
    }
    return once(std::move(grads), {g[0], g[1], pos});
  }
};

// (sender, receiver, shift, CSR offsets, largest degree) of the radius graph; `box` is host data [S, 3].  One host synchronisation.
py::tuple radius_graph(const Tensor& pos, const Tensor& atom_struct, py::array_t<double, py::array::c_style | py::array::forcecast> box, double cutoff,
                       int64_t most) {
  c10::cuda::CUDAGuard guard(pos.device());
  const int64_t N = pos.size(0);
  const Tensor p64 = pos.detach().to(at::kDouble).contiguous(), st = atom_struct.to(pos.device(), at::kInt).contiguous();
  fasteq_nl_problem prob{};
  prob.n_atoms = N; prob.n_structs = (int32_t)box.shape(0); prob.cutoff = cutoff;
  prob.pos = p64.const_data_ptr<double>(); prob.atom_struct = st.const_data_ptr<int32_t>(); prob.box = box.data();
  int64_t bytes = 0;
  check(core.neighbors_work_bytes(&prob, &bytes), "fasteq_neighbors_work_bytes", core.last_cuda_error);
  const auto ints = p64.options().dtype(at::kInt);
  Tensor work = at::empty({bytes}, p64.options().dtype(at::kByte)), counts = at::empty({N + 2}, ints);     // offsets, then the largest degree
  int32_t* seg = counts.data_ptr<int32_t>();
  cudaStream_t s = stream_of(p64);
  C10_CUDA_CHECK(cudaMemsetAsync(seg + N + 1, 0, sizeof(int32_t), s));
  check(core.neighbors_count(&prob, work.data_ptr(), bytes, seg, seg + N + 1, s), "fasteq_neighbors_count", core.last_cuda_error);
  int32_t got[2];
  {
    py::gil_scoped_release nogil;
    C10_CUDA_CHECK(cudaMemcpyAsync(got, seg + N, sizeof got, cudaMemcpyDeviceToHost, s));
    C10_CUDA_CHECK(cudaStreamSynchronize(s));
  }
  if (got[1] > most)
    throw std::runtime_error("radius_graph: an atom has " + std::to_string(got[1]) + " neighbours, more than the " + std::to_string(most) + " the builder sorts");
  const int64_t E = got[0];
  Tensor src = at::empty({E}, ints), dst = at::empty({E}, ints), shift = at::empty({E, 3}, p64.options());
  if (E > 0)
    check(core.neighbors_fill(&prob, work.data_ptr(), bytes, seg, src.data_ptr<int32_t>(), dst.data_ptr<int32_t>(), shift.data_ptr<double>(), s),
          "fasteq_neighbors_fill", core.last_cuda_error);
  return py::make_tuple(src, dst, shift, counts.narrow(0, 0, N + 1), (int64_t)got[1]);
}

// ------------------------------------------------------------------------------------------------ SymmetricContraction
struct StcModule { decltype(&fasteq_stc_forward) forward = nullptr; decltype(&fasteq_stc_backward) backward = nullptr; decltype(&fasteq_last_cuda_error) error = nullptr; };

struct Contraction : torch::CustomClassHolder {
  int64_t u, x1_segs, x0_segs, out_segs;
  PyKeep load;                 // (direction, odd address) -> {name: address}
  PyKeep general;              // (grad_out, x1, x0, species, needs x1, needs x0) -> (grad_x1, grad_x0): weight gradients, second order
  std::mutex lock;
  StcModule modules[2][2];     // [forward, backward][packed, odd addresses]
  Contraction(int64_t u_, int64_t a, int64_t d, int64_t o, py::object l, py::object g)
      : u(u_), x1_segs(a), x0_segs(d), out_segs(o), load(std::move(l)), general(std::move(g)) {}
  StcModule module(bool backward, bool odd) {
    {
      std::lock_guard<std::mutex> g(lock);
      if (modules[backward][odd].forward) return modules[backward][odd];
    }
    StcModule m;
    {
      py::gil_scoped_acquire gil;
      auto d = load.get()(backward ? "bwd" : "fwd", odd).cast<std::unordered_map<std::string, uint64_t>>();
      m.forward = reinterpret_cast<decltype(m.forward)>(d.at("fasteq_stc_forward"));
      m.backward = reinterpret_cast<decltype(m.backward)>(d.at("fasteq_stc_backward"));
      m.error = reinterpret_cast<decltype(m.error)>(d.at("fasteq_last_cuda_error"));
    }
    std::lock_guard<std::mutex> g(lock);
    return modules[backward][odd] = m;
  }
};
using Stc = c10::intrusive_ptr<Contraction>;

bool odd_address(std::initializer_list<Tensor> ts) {
  for (const Tensor& t : ts) if (reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 8) return true;
  return false;
}

struct SymmetricContraction : torch::autograd::Function<SymmetricContraction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x1, const Tensor& x0, const Tensor& i0, const Stc& c) {
    c10::cuda::CUDAGuard guard(x1.device());
    const Tensor x1c = x1.contiguous(), x0c = x0.contiguous(), species = int32_contiguous(i0);
    const int64_t B = x1c.size(0);
    Tensor out = at::empty({B, c->out_segs * c->u}, x1c.options());
    const StcModule m = c->module(false, odd_address({x1c, x0c}));
    check(m.forward(ptr(x1c), ptr(x0c), species.const_data_ptr<int32_t>(), B, x0c.size(0), mptr(out), stream_of(x1c)), "fasteq_stc_forward", m.error);
    ctx->save_for_backward({x1, x0, species});
    ctx->saved_data["c"] = capsule(c);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list go) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x1 = saved[0], &x0 = saved[1], &species = saved[2];
    const Stc c = uncapsule<Contraction>(ctx->saved_data["c"]);
    const bool need_x1 = ctx->needs_input_grad(0), need_x0 = ctx->needs_input_grad(1);
    variable_list grads(4);
    if (!need_x1 && !need_x0) return grads;
    const Tensor g = go[0].contiguous(), x1c = x1.contiguous(), x0c = x0.contiguous();
    if (need_x0 || at::GradMode::is_enabled()) {
      py::gil_scoped_acquire gil;
      py::tuple d = c->general.get()(g, x1c, x0c, species, need_x1, need_x0);
      if (need_x1) grads[0] = d[0].cast<Tensor>();
      if (need_x0) grads[1] = d[1].cast<Tensor>();
      return grads;
    }
    c10::cuda::CUDAGuard guard(x1c.device());
    Tensor gx1 = at::empty_like(x1c);
    const StcModule m = c->module(true, odd_address({g, x1c, x0c}));
    check(m.backward(ptr(g), ptr(x1c), ptr(x0c), species.const_data_ptr<int32_t>(), x1c.size(0), x0c.size(0), mptr(gx1), nullptr, stream_of(x1c)),
          "fasteq_stc_backward", m.error);
    grads[0] = gx1;
    return grads;
  }
};

}  // namespace

void bind_edges(py::module_& m) {
  m.def("edge_geometry", [](const Tensor& pos, const Tensor& src, const Tensor& dst, const Tensor& shift, double r_max, int64_t n_basis, int64_t p) {
    auto out = EdgeGeometry::apply(pos, src, dst, shift, r_max, n_basis, p);
    return py::make_tuple(out[0], out[1]);
  });
  m.def("radius_graph", &radius_graph);
  py::class_<Contraction, Stc>(m, "Contraction").def(py::init([](int64_t u, int64_t a, int64_t d, int64_t o, py::object load, py::object general) {
    return c10::make_intrusive<Contraction>(u, a, d, o, std::move(load), std::move(general));
  }));
  m.def("symmetric_contraction", [](const Tensor& x1, const Tensor& x0, const Tensor& i0, const Stc& c) -> Tensor {
    return SymmetricContraction::apply(x1, x0, i0, c);
  });
}

}  // namespace front
