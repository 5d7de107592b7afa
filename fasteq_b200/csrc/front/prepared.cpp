// Cache of prepared (split / packed) weight forms for the tensor-core kernels, shared by the SO3Linear, dense and radial-chain
// operators.  Keyed on the weight tensors' storage address, version, type, extents and strides, so that an in-place update, a new tensor or
// another view from the same address (a transposed weight) is another entry; an entry keeps the weights' storages alive (through
// detached aliases: a parameter object can be given another storage, `module.double()` or `p.data = ...`) so the address cannot be
// reused while it exists.  An entry remembers the stream it was built on and an event recorded behind the build: a later call on
// another stream waits for that event (and tells the allocator about the new reader) before it uses the entry.  Plays the part of
// the reference's plan LRU
// (fasteq/ops/auto_schedule/eqlinear_plan.py:38-41, :81-100, :167-187).
//
// Inside CUDA-graph capture a prepared form would be baked into the graph and go stale when the weights change, so the cache is bypassed
// there unless the caller declares the weights frozen.
#include "front.h"

namespace front {
namespace {

struct Entry {
  std::string key;
  std::vector<Tensor> weights;
  Tensor value;
  std::shared_ptr<at::cuda::CUDAEvent> built;
  std::set<cudaStream_t> ordered;      // streams already behind the build
};

constexpr int64_t kDefaultBudget = 256LL << 20;
// Nothing that may take the GIL happens under it (an entry's tensors may carry Python objects, whose release does; so do hooks on
// stream waits): a thread that holds the GIL may be waiting for it.
std::mutex lock;
std::list<Entry> entries;              // most recently used first
std::unordered_map<std::string, std::list<Entry>::iterator> index_of;
int64_t bytes = 0, budget = kDefaultBudget;
int frozen = 0;

// moves an entry to `dropped`, which lets it go after the lock
void drop(std::list<Entry>::iterator e, std::list<Entry>& dropped) {
  bytes -= e->value.nbytes();
  index_of.erase(e->key);
  dropped.splice(dropped.end(), entries, e);
}

void append(std::string& key, int64_t v) { key.append(reinterpret_cast<const char*>(&v), sizeof v); }

}  // namespace

std::optional<Tensor> prepared(const std::vector<Tensor>& weights, const std::string& tag, const std::function<Tensor()>& build) {
  std::string key = tag;
  append(key, weights[0].device().index());
  for (const Tensor& w : weights) {
    append(key, (int64_t)w.const_data_ptr()); append(key, w._version()); append(key, (int64_t)w.scalar_type()); append(key, w.dim());
    for (int64_t n : w.sizes()) append(key, n);
    for (int64_t n : w.strides()) append(key, n);
  }
  const bool in_capture = capturing();
  {
    std::unique_lock<std::mutex> g(lock);
    if (budget <= 0 || (in_capture && !frozen)) return std::nullopt;
    auto hit = index_of.find(key);
    if (hit != index_of.end()) {
      entries.splice(entries.begin(), entries, hit->second);
      const Entry& e = entries.front();
      Tensor value = e.value;
      if (!in_capture) {
        const auto cur = c10::cuda::getCurrentCUDAStream(value.device().index());
        if (!e.ordered.count(cur.stream())) {
          const auto built = e.built;
          g.unlock();
          built->block(cur);
          c10::cuda::CUDACachingAllocator::recordStream(value.storage().data_ptr(), cur);
          g.lock();
          hit = index_of.find(key);
          if (hit != index_of.end() && hit->second->built == built) hit->second->ordered.insert(cur.stream());   // once the wait is issued
          g.unlock();
        }
      }
      return value;
    }
    if (in_capture) return std::nullopt;             // nothing persistent may be allocated inside a capture
  }
  Tensor value = build();
  if (!value.defined()) return std::nullopt;
  auto cur = c10::cuda::getCurrentCUDAStream(value.device().index());
  std::list<Entry> fresh(1), dropped;
  Entry& e = fresh.front();
  e.key = key; e.value = value; e.ordered.insert(cur.stream());
  for (const Tensor& w : weights) e.weights.push_back(w.detach());
  e.built = std::make_shared<at::cuda::CUDAEvent>();
  e.built->record(cur);
  {
    std::lock_guard<std::mutex> g(lock);
    auto hit = index_of.find(key);                    // another thread may have built it meanwhile
    if (hit != index_of.end()) drop(hit->second, dropped);
    while (!entries.empty() && bytes + (int64_t)value.nbytes() > budget) drop(std::prev(entries.end()), dropped);
    entries.splice(entries.begin(), fresh);
    index_of[key] = entries.begin();
    bytes += value.nbytes();
  }
  return value;
}

void bind_prepared(py::module_& m) {
  auto clear = [] {
    std::list<Entry> dropped;
    std::lock_guard<std::mutex> g(lock);
    dropped.swap(entries);
    index_of.clear(); bytes = 0;
  };
  m.def("prepared_clear", clear);
  m.def("prepared_set_budget", [clear](std::optional<int64_t> most) {
    { std::lock_guard<std::mutex> g(lock); budget = most.value_or(kDefaultBudget); }
    if (most && *most <= 0) clear();
  });
  m.def("prepared_freeze", [](int by) { std::lock_guard<std::mutex> g(lock); frozen += by; });
  m.def("prepared_snapshot", [] {
    std::vector<Tensor> out;
    std::lock_guard<std::mutex> g(lock);
    for (const Entry& e : entries) out.push_back(e.value);
    return out;
  });
}

}  // namespace front
