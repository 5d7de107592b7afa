// The tensor-product operator in its usual form: per-edge weights, sender gather, scalar y (or edge vectors), receiver scatter.
#include "front.h"
#include <algorithm>
#include <atomic>
#include <map>

namespace front {
namespace {

using Flags = std::array<bool, 3>;

struct U1DModule : torch::CustomClassHolder {
  decltype(&fasteq_u1d_forward) forward; decltype(&fasteq_u1d_forward_split) forward_split;
  decltype(&fasteq_u1d_backward) backward; decltype(&fasteq_u1d_backward_split) backward_split;
  decltype(&fasteq_u1d_tangent_forward) tangent_forward; decltype(&fasteq_u1d_tangent_backward) tangent_backward;
  decltype(&fasteq_last_cuda_error) error;
  PyKeep object;
};
using Module = c10::intrusive_ptr<U1DModule>;

// One operator signature: extents and the modules loaded for it so far.
struct Signature : torch::CustomClassHolder {
  int64_t u, w_segs, x_segs, y_segs, out_segs;
  bool y_sh;
  PyKeep load;                 // (direction, needs, tangents or None, odd address) -> (module, {name: address}), None: too wide for second-order ones
  std::mutex lock;
  std::unordered_map<int, Module> modules;
  Signature(int64_t u_, int64_t w, int64_t x, int64_t y, int64_t o, bool sh, py::object l)
      : u(u_), w_segs(w), x_segs(x), y_segs(y), out_segs(o), y_sh(sh), load(std::move(l)) {}
  int64_t y_cols() const { return y_sh ? 3 : y_segs; }
  // null where the signature has no second-order modules
  Module module(bool backward, Flags needs, const Flags* tangents, bool odd) {
    int key = backward | odd << 1;
    for (int i = 0; i < 3; ++i) key |= needs[i] << (2 + i) | (tangents && (*tangents)[i]) << (5 + i);
    if (tangents) key |= 1 << 8;
    {
      std::lock_guard<std::mutex> g(lock);
      auto hit = modules.find(key);
      if (hit != modules.end()) return hit->second;
    }
    auto m = c10::make_intrusive<U1DModule>();
    {
      py::gil_scoped_acquire gil;
      py::object loaded = load.get()(backward ? "bwd" : "fwd", needs, tangents ? py::cast(*tangents) : py::none(), odd);
      if (loaded.is_none()) return Module();
      py::tuple got = loaded;
      auto d = got[1].cast<std::unordered_map<std::string, uint64_t>>();
#define F(name) m->name = reinterpret_cast<decltype(m->name)>(d.at("fasteq_u1d_" #name));
      F(forward) F(forward_split) F(backward) F(backward_split) F(tangent_forward) F(tangent_backward)
#undef F
      m->error = reinterpret_cast<decltype(m->error)>(d.at("fasteq_last_cuda_error"));
      m->object.p = py::object(got[0]).release().ptr();
    }
    std::lock_guard<std::mutex> g(lock);
    return modules.emplace(key, m).first->second;
  }
};
using Sig = c10::intrusive_ptr<Signature>;

// Receiver-sorted view of a scatter index with the partitions its launches use.  Every kernel that builds a part of it leaves an event
// behind; a launch on another stream waits for those first.
struct Plan : torch::CustomClassHolder {
  struct Shares { Tensor part; int32_t n = 0; bool split = false; };
  Tensor seg_ptr, perm;
  int64_t n_rows, n_edges;
  PyKeep rule;                 // module -> (pipelines, whether their shares cut receivers)
  std::mutex lock;
  std::map<std::pair<int64_t, bool>, Tensor> parts;
  std::unordered_map<U1DModule*, std::pair<Module, Shares>> shares;
  std::vector<std::pair<cudaStream_t, std::shared_ptr<at::cuda::CUDAEvent>>> built;
  std::set<cudaStream_t> ordered;      // streams already behind every event in `built`
  uint64_t marks = 0;                  // changes of `built`

  Plan(Tensor s, std::optional<Tensor> p, int64_t rows, int64_t edges, py::object r)
      : seg_ptr(std::move(s)), n_rows(rows), n_edges(edges), rule(std::move(r)) {
    if (p) perm = *p;
  }
  // `publish` (under the lock) makes what the current stream has just been told to build visible; the event behind it comes first
  template <typename Publish> void mark(Publish publish) {
    const auto cur = c10::cuda::getCurrentCUDAStream(seg_ptr.device().index());
    auto e = std::make_shared<at::cuda::CUDAEvent>();
    e->record(cur);
    std::lock_guard<std::mutex> g(lock);
    publish();
    built.erase(std::remove_if(built.begin(), built.end(), [&](const auto& b) { return b.first == cur.stream(); }), built.end());
    built.emplace_back(cur.stream(), std::move(e));
    ordered.clear();
    ++marks;
  }
  void mark_built() { if (!capturing()) mark([] {}); }
  // A stream counts as ordered once its waits are issued: another thread may launch on it at any moment.
  void order_current_stream() {
    const auto cur = c10::cuda::getCurrentCUDAStream(seg_ptr.device().index());
    std::vector<std::shared_ptr<at::cuda::CUDAEvent>> wait;
    std::vector<Tensor> read;
    uint64_t seen;
    {
      std::lock_guard<std::mutex> g(lock);
      if (built.empty() || ordered.count(cur.stream())) return;
      if (capturing()) return;
      for (const auto& b : built) if (b.first != cur.stream()) wait.push_back(b.second);
      if (!wait.empty()) {
        // a reader on a stream other than the building one: tell the allocator, so that an evicted plan's buffers are not handed out again
        // while this stream still reads them
        read.push_back(seg_ptr);
        if (perm.defined()) read.push_back(perm);
        for (const auto& p : parts) read.push_back(p.second);
      }
      seen = marks;
    }
    for (const auto& e : wait) e->block(cur);
    for (const Tensor& t : read) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), cur);
    std::lock_guard<std::mutex> g(lock);
    if (seen == marks) ordered.insert(cur.stream());     // otherwise something was built meanwhile: the next call waits for that too
  }
  // first row of each share [1, n + 1]; with `split` shares are cut between edges and a second row holds their first edges.  One that
  // a capture needs first belongs to that capture: its kernel has not run and its memory is the graph's, so the plan does not keep it
  Tensor partition(int64_t n, bool split) {
    {
      std::lock_guard<std::mutex> g(lock);
      auto hit = parts.find({n, split});
      if (hit != parts.end()) return hit->second;
    }
    c10::cuda::CUDAGuard guard(seg_ptr.device());
    order_current_stream();
    Tensor p = at::empty({split ? 2 : 1, n + 1}, seg_ptr.options());
    int32_t* d = p.data_ptr<int32_t>();
    cudaStream_t s = stream_of(p);
    if (split) check(core.graph_partition_edges(seg_ptr.const_data_ptr<int32_t>(), n_rows, n_edges, (int32_t)n, d, d + n + 1, s), "fasteq_graph_partition_edges", core.last_cuda_error);
    else check(core.graph_partition(seg_ptr.const_data_ptr<int32_t>(), n_rows, n_edges, (int32_t)n, d, s), "fasteq_graph_partition", core.last_cuda_error);
    if (!capturing()) mark([&] { p = parts.emplace(std::make_pair(n, split), p).first->second; });     // another thread's, if it was first
    return p;
  }
  Shares shares_of(const Module& m) {
    {
      std::lock_guard<std::mutex> g(lock);
      auto hit = shares.find(m.get());
      if (hit != shares.end()) return hit->second.second;
    }
    Shares s;
    {
      py::gil_scoped_acquire gil;
      py::tuple got = rule.get()(m->object.get());
      s.n = got[0].cast<int32_t>(); s.split = got[1].cast<bool>();
    }
    s.part = partition(s.n, s.split);
    if (capturing()) return s;
    std::lock_guard<std::mutex> g(lock);
    shares.emplace(m.get(), std::make_pair(m, s));
    return s;
  }
};
using PlanPtr = c10::intrusive_ptr<Plan>;
std::atomic<int> recording{0};
PyObject* record_plan = nullptr;     // enters a Python plan into the lists of record_plans

struct Call : torch::CustomClassHolder {
  Sig sig;
  PlanPtr plan;
  Tensor src;
  int64_t x_rows;
  PyKeep graph;                // the Python plan
};
using CallPtr = c10::intrusive_ptr<Call>;

// the launch's graph record; returns the address of the shares' first edges when they cut receivers
const int32_t* graph_of(const Call& c, const Module& m, fasteq_u1d_graph* g, Plan::Shares* s) {
  *s = c.plan->shares_of(m);
  c.plan->order_current_stream();
  if (recording.load() > 0) {
    py::gil_scoped_acquire gil;
    const py::handle record = record_plan;
    record(c.graph.get());
  }
  *g = {};
  g->n_edges = c.plan->n_edges; g->n_out_rows = c.plan->n_rows; g->x_rows = c.x_rows; g->y_rows = c.plan->n_edges;
  g->x_index = c.src.const_data_ptr<int32_t>();
  g->seg_ptr = c.plan->seg_ptr.const_data_ptr<int32_t>();
  g->perm = c.plan->perm.defined() ? c.plan->perm.const_data_ptr<int32_t>() : nullptr;
  g->n_parts = s->n;
  g->part_ptr = s->part.const_data_ptr<int32_t>();
  return s->split ? g->part_ptr + s->n + 1 : nullptr;
}

bool odd(std::initializer_list<Tensor> ts) {
  for (const Tensor& t : ts) if (t.defined() && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 8) return true;
  return false;
}

// `t`, `has`: tangents of w, x and y.  Undefined where the signature has no second-order modules.
Tensor forward_launch(const Call& c, const Tensor& w, const Tensor& x, const Tensor& y, const Tensor* t = nullptr, const Flags* has = nullptr) {
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t cols = c.sig->out_segs * c.sig->u;
  Tensor out = at::empty({c.plan->n_rows, cols}, x.options());
  const Module m = c.sig->module(false, {false, false, false}, has, odd({w, x, y, out}) || (t && odd({t[0], t[1], t[2]})));
  if (!m) return Tensor();
  fasteq_u1d_graph g;
  Plan::Shares s;
  const int32_t* edge = graph_of(c, m, &g, &s);
  Tensor carry;
  if (edge) carry = at::empty({s.n, cols}, x.options());
  cudaStream_t st = stream_of(x);
  if (t) check(m->tangent_forward(&g, edge, mptr(carry), ptr(w), ptr(x), ptr(y), ptr(t[0]), ptr(t[1]), ptr(t[2]), mptr(out), st), "fasteq_u1d_tangent_forward", m->error);
  else if (edge) check(m->forward_split(&g, edge, mptr(carry), ptr(w), ptr(x), ptr(y), mptr(out), st), "fasteq_u1d_forward_split", m->error);
  else check(m->forward(&g, ptr(w), ptr(x), ptr(y), mptr(out), st), "fasteq_u1d_forward", m->error);
  return out;
}

// empty where the signature has no second-order modules
variable_list backward_launch(const Call& c, const Tensor& go, const Tensor& w, const Tensor& x, const Tensor& y, Flags needs, const Tensor* t = nullptr,
                              const Flags* has = nullptr) {
  c10::cuda::CUDAGuard guard(x.device());
  variable_list d = {needs[0] ? at::empty_like(w) : Tensor(), needs[1] ? at::empty_like(x) : Tensor(), needs[2] ? at::empty_like(y) : Tensor()};
  const Module m = c.sig->module(true, needs, has, odd({go, w, x, y, d[0], d[1], d[2]}) || (t && odd({t[0], t[1], t[2]})));
  if (!m) return {};
  fasteq_u1d_graph g;
  Plan::Shares s;
  const int32_t* edge = graph_of(c, m, &g, &s);
  cudaStream_t st = stream_of(x);
  if (t) check(m->tangent_backward(&g, edge, ptr(go), ptr(w), ptr(x), ptr(y), ptr(t[0]), ptr(t[1]), ptr(t[2]), mptr(d[0]), mptr(d[1]), mptr(d[2]), st),
               "fasteq_u1d_tangent_backward", m->error);
  else if (edge) check(m->backward_split(&g, edge, ptr(go), ptr(w), ptr(x), ptr(y), mptr(d[0]), mptr(d[1]), mptr(d[2]), st), "fasteq_u1d_backward_split", m->error);
  else check(m->backward(&g, ptr(go), ptr(w), ptr(x), ptr(y), mptr(d[0]), mptr(d[1]), mptr(d[2]), st), "fasteq_u1d_backward", m->error);
  return d;
}

struct TensorProductBackward : torch::autograd::Function<TensorProductBackward> {
  static variable_list forward(AutogradContext* ctx, const Tensor& go, const Tensor& w, const Tensor& x, const Tensor& y, const CallPtr& c, Flags needs) {
    auto d = backward_launch(*c, go, w, x, y, needs);
    ctx->save_for_backward({go, w, x, y});
    ctx->saved_data["c"] = capsule(c);
    ctx->saved_data["n"] = (int64_t)(needs[0] | needs[1] << 1 | needs[2] << 2);
    ctx->set_materialize_grads(false);
    for (int i = 0; i < 3; ++i) if (!needs[i]) d[i] = at::empty({0}, x.options());
    return d;
  }
  static variable_list backward(AutogradContext* ctx, variable_list gg);
};

struct TensorProduct : torch::autograd::Function<TensorProduct> {
  static Tensor forward(AutogradContext* ctx, const Tensor& w, const Tensor& x, const Tensor& y, const CallPtr& c) {
    ctx->save_for_backward({w, x, y});
    ctx->saved_data["c"] = capsule(c);
    return forward_launch(*c, w, x, y);
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &w = saved[0], &x = saved[1], &y = saved[2];
    const CallPtr c = uncapsule<Call>(ctx->saved_data["c"]);
    const Flags needs = {ctx->needs_input_grad(0), ctx->needs_input_grad(1), ctx->needs_input_grad(2)};
    if (!needs[0] && !needs[1] && !needs[2]) return variable_list(4);
    const Tensor go = gout[0].contiguous();
    variable_list d;
    if (c->sig->y_sh) {
      // not trilinear in the edge vector: the second-order kernels do not apply
      if (at::GradMode::is_enabled() && (go.requires_grad() || w.requires_grad() || x.requires_grad() || y.requires_grad()))
        throw std::runtime_error("fast_uniform1d_jit: no second-order gradient with in-kernel spherical harmonics; pass the harmonics as the y operand instead");
      d = backward_launch(*c, go, w, x, y, needs);
    } else {
      d = TensorProductBackward::apply(go, w, x, y, c, needs);
    }
    for (int i = 0; i < 3; ++i) if (!needs[i]) d[i] = Tensor();
    d.resize(4);
    return d;
  }
};

// The gradients of <go, F(w', x, y) + F(w, x', y) + F(w, x, y')> from first-order nodes, an operand in its tangent's place.
// `wants`: of go, w, x, y
variable_list second_order_composed(const CallPtr& c, const Tensor& go, const Tensor (&operands)[3], const Tensor (&t)[3], const bool (&wants)[4]) {
  variable_list out(6);
  auto add = [](Tensor& sum, const Tensor& v) { sum = sum.defined() ? sum + v : v; };
  for (int i = 0; i < 3; ++i) {
    if (!t[i].defined()) continue;
    Tensor o[3] = {operands[0], operands[1], operands[2]};
    o[i] = t[i];
    if (wants[0]) add(out[0], TensorProduct::apply(o[0], o[1], o[2], c));
    for (int k = 0; k < 3; ++k) {
      if (k == i || !wants[1 + k]) continue;
      Flags only{};
      only[k] = true;
      add(out[1 + k], TensorProductBackward::apply(go, o[0], o[1], o[2], c, only)[k]);
    }
  }
  return out;
}

// of <go, F(w', x, y) + F(w, x', y) + F(w, x, y')>: one pass over the edges for grad_out's gradient, one for the operands', where the
// signature has modules for that and no third order may follow (grad mode)
variable_list TensorProductBackward::backward(AutogradContext* ctx, variable_list gg) {
  const auto saved = ctx->get_saved_variables();
  const CallPtr c = uncapsule<Call>(ctx->saved_data["c"]);
  const int64_t needed = ctx->saved_data["n"].toInt();
  Tensor t[3];
  Flags has{};
  for (int i = 0; i < 3; ++i) {
    if ((needed >> i & 1) && gg[i].defined()) t[i] = gg[i].contiguous();
    has[i] = t[i].defined();
  }
  variable_list out(6);
  if (!has[0] && !has[1] && !has[2]) return out;
  const Tensor &go = saved[0], &w = saved[1], &x = saved[2], &y = saved[3];
  const bool wants[4] = {ctx->needs_input_grad(0), ctx->needs_input_grad(1), ctx->needs_input_grad(2), ctx->needs_input_grad(3)};
  if (at::GradMode::is_enabled()) return second_order_composed(c, go, {w, x, y}, t, wants);
  if (wants[0]) {
    out[0] = forward_launch(*c, w, x, y, t, &has);
    if (!out[0].defined()) return second_order_composed(c, go, {w, x, y}, t, wants);
  }
  // a gradient needs a tangent on another operand
  const Flags needs = {wants[1] && (has[1] || has[2]), wants[2] && (has[0] || has[2]), wants[3] && (has[0] || has[1])};
  if (needs[0] || needs[1] || needs[2]) {
    auto d = backward_launch(*c, go, w, x, y, needs, t, &has);
    if (d.empty()) return second_order_composed(c, go, {w, x, y}, t, wants);
    for (int i = 0; i < 3; ++i) out[1 + i] = d[i];
  }
  return out;
}

}  // namespace

void bind_u1d(py::module_& m) {
  py::class_<Signature, Sig>(m, "Signature").def(py::init([](int64_t u, int64_t w, int64_t x, int64_t y, int64_t o, bool sh, py::object load) {
    return c10::make_intrusive<Signature>(u, w, x, y, o, sh, std::move(load));
  }));
  py::class_<Plan, PlanPtr>(m, "Plan")
      .def(py::init([](Tensor seg, std::optional<Tensor> perm, int64_t rows, int64_t edges, py::object rule) {
        return c10::make_intrusive<Plan>(std::move(seg), std::move(perm), rows, edges, std::move(rule));
      }))
      .def("mark_built", &Plan::mark_built)
      .def("order_current_stream", &Plan::order_current_stream)
      .def("partition", &Plan::partition)
      .def("parts", [](Plan& p) {
        std::lock_guard<std::mutex> g(p.lock);
        return p.parts;
      });
  m.def("u1d_on_record", [](py::object f) { Py_XDECREF(record_plan); record_plan = f.release().ptr(); });
  m.def("u1d_recording", [](int by) { recording += by; });
  // None: an operand this form does not take (the general path says what is wrong with it, or takes it)
  m.def("u1d", [](const Tensor& w, const Tensor& x, const Tensor& y, const Tensor& src, const Sig& sig, const PlanPtr& plan, py::object graph) -> std::optional<Tensor> {
    const int64_t E = plan->n_edges, u = sig->u;
    for (const Tensor* t : {&w, &x, &y})
      if (!t->is_cuda() || !t->is_contiguous() || t->dim() < 2 || t->scalar_type() != x.scalar_type() || t->device() != x.device()) return std::nullopt;
    if (E == 0 || plan->n_rows == 0 || w.numel() != E * sig->w_segs * u || x.numel() != plan->n_rows * sig->x_segs * u || y.numel() != E * sig->y_cols() ||
        (sig->y_sh && y.size(-1) != 3) || !src.is_cuda() || src.numel() != E)
      return std::nullopt;
    auto c = c10::make_intrusive<Call>();
    c->sig = sig; c->plan = plan; c->x_rows = plan->n_rows;
    c->graph.p = graph.release().ptr();
    c->src = (src.scalar_type() == at::kInt ? src : src.to(at::kInt)).contiguous();
    return TensorProduct::apply(w, x, y, c);
  });
}

}  // namespace front
