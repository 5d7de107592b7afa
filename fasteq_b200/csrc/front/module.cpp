#include "front.h"

namespace front {

Core core;
static PyObject* raised = nullptr;

void fail(const std::string& message) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(raised, message.c_str());
  throw py::error_already_set();
}

void check(int rc, const char* what, decltype(&fasteq_last_cuda_error) last_error) {
  if (rc == FASTEQ_OK) return;
  static const char* names[] = {"ok", "unsupported", "invalid argument", "CUDA error", "internal error", "device fault"};
  std::string detail;
  if (rc == FASTEQ_CUDA_ERROR && last_error) detail = std::string(": ") + last_error();
  fail(std::string(what) + " failed with status " + std::to_string(rc) + " (" + (rc > 0 && rc < 6 ? names[rc] : "?") + ")" + detail);
}

}  // namespace front

PYBIND11_MODULE(fasteq_front, m) {
  using namespace front;
  // addresses of the core library's functions, and the exception its failures are raised as
  m.def("bind_core", [](std::unordered_map<std::string, uint64_t> at, py::object failure) {
#define F(name) core.name = reinterpret_cast<decltype(core.name)>(at.at("fasteq_" #name));
    F(eqlinear_pack) F(eqlinear_forward) F(eqlinear_dgrad) F(eqlinear_forward_packed) F(eqlinear_dgrad_packed)
    F(eqlinear_wgrad_scratch) F(eqlinear_wgrad_with) F(gemm_tf32x3_split) F(gemm_tf32x3_presplit)
    F(radial_chain_prepare) F(radial_chain_forward) F(radial_chain_backward) F(edge_geometry_forward) F(edge_geometry_backward)
    F(silu) F(neighbors_work_bytes) F(neighbors_count) F(neighbors_fill) F(graph_partition) F(graph_partition_edges) F(last_cuda_error)
#undef F
    raised = failure.release().ptr();
  });
  bind_prepared(m);
  bind_layers(m);
  bind_edges(m);
  bind_u1d(m);
}
