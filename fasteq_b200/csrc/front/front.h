// Host path of the operators in native code: shape checks, output allocation, prepared weights, launches and autograd nodes.  In Python an
// operator's forward and backward took 60 to 90 us between them, several times what its kernels take on a small system; here about 10.
// The kernels stay behind the C interface of include/fasteq_b200.h: this extension is handed the addresses of its functions.
// What is rare stays in Python (modules that have to be compiled, graph plans that have to be built, orders and operand forms these
// nodes do not take) and is called back from here.
#pragma once
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <functional>
#include <list>
#include <mutex>
#include <optional>
#include <set>
#include <string>
#include <unordered_map>
#include <vector>
#include "fasteq_b200.h"

namespace front {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// the C interface of the core library
struct Core {
#define F(name) decltype(&fasteq_##name) name = nullptr;
  F(eqlinear_pack) F(eqlinear_forward) F(eqlinear_dgrad) F(eqlinear_forward_packed) F(eqlinear_dgrad_packed)
  F(eqlinear_wgrad_scratch) F(eqlinear_wgrad_with) F(gemm_tf32x3_split) F(gemm_tf32x3_presplit)
  F(radial_chain_prepare) F(radial_chain_forward) F(radial_chain_backward) F(edge_geometry_forward) F(edge_geometry_backward)
  F(silu) F(neighbors_work_bytes) F(neighbors_count) F(neighbors_fill) F(graph_partition) F(graph_partition_edges) F(last_cuda_error)
#undef F
};
extern Core core;

// Raises the Python layer's error.  It travels as the Python error itself: a C++ type would reach the caller of a backward, whose nodes run
// on autograd's threads, as a plain RuntimeError.
[[noreturn]] void fail(const std::string& message);
void check(int rc, const char* what, decltype(&fasteq_last_cuda_error) last_error = nullptr);

// A Python object held by something autograd may free on a thread without the GIL.
struct PyKeep {
  PyObject* p = nullptr;
  PyKeep() = default;
  explicit PyKeep(py::object o) : p(o.release().ptr()) {}
  PyKeep(const PyKeep&) = delete;
  PyKeep& operator=(const PyKeep&) = delete;
  ~PyKeep() {
    if (p && Py_IsInitialized()) { py::gil_scoped_acquire gil; Py_DECREF(p); }
  }
  py::handle get() const { return py::handle(p); }
};

inline cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
inline bool capturing() { return at::cuda::currentStreamCaptureStatusMayInitCtx() != at::cuda::CaptureStatus::None; }
inline Tensor defined_contiguous(const Tensor& t) { return t.defined() ? t.contiguous() : t; }
inline const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
inline void* mptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// Prepared (split / packed) forms of weights, see prepared.cpp
std::optional<Tensor> prepared(const std::vector<Tensor>& weights, const std::string& tag, const std::function<Tensor()>& build);

// keeps a C++ object in an autograd node
template <typename T> c10::IValue capsule(const c10::intrusive_ptr<T>& p) { return c10::IValue::make_capsule(p); }
template <typename T> c10::intrusive_ptr<T> uncapsule(const c10::IValue& v) {
  return c10::static_intrusive_pointer_cast<T>(v.toCapsule());
}

void bind_prepared(py::module_& m);
void bind_layers(py::module_& m);
void bind_edges(py::module_& m);
void bind_u1d(py::module_& m);

}  // namespace front
