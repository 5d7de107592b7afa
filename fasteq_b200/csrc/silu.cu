// SiLU with its first and second derivative, for the radial MLP of a training step: autograd composes the second backward
// of torch's silu from about a dozen elementwise launches per layer; here each order is one pass.
//   y = z / (1 + exp(-z))                    s = 1 / (1 + exp(-z))
//   dz = g s'(z)       silu'  = s (1 + z (1 - s))
//   second order, for a cotangent h of dz:  d_g = h silu',  d_z = h g silu''   with silu'' = s (1 - s) (2 + z (1 - 2 s))
// Bound: memory (two to five streams); 16-byte accesses where every operand allows them.
// Roundings are kept few: y is one quotient (z s rounds once more: 4.5e-8 instead of 4.0e-8 of root mean square relative to y on normal
// z in FP32), and a cotangent meets s before the rest of the slope does
// (5.34e-8, against 5.38e-8 the other way round and 5.34e-8 for torch's backward).
#include <cstdint>
#include <cuda_runtime.h>
#include "fasteq_b200.h"
#include "core_common.h"
#include "fasteq_device.cuh"

using namespace fasteq;

namespace {

template <typename T> __device__ __forceinline__ T sigmoid(T z) { return T(1) / (T(1) + exp(-z)); }
// g silu'(z)
template <typename T> __device__ __forceinline__ T times_slope(T g, T z, T s) { return (g * s) * (T(1) + z * (T(1) - s)); }

// ORDER 0: out0 = silu(z).  1: out0 = g silu'(z).  2: out0 = h silu'(z), out1 = h g silu''(z).  V values per access.
template <typename T, int ORDER, int V>
__global__ void __launch_bounds__(256) silu_kernel(const T* __restrict__ z, const T* __restrict__ g, const T* __restrict__ h,
                                                   T* __restrict__ out0, T* __restrict__ out1, long long n) {
  let_next_kernel_begin();
  struct alignas(sizeof(T) * V) Pack { T v[V]; };
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n / V) {
    const Pack pz = reinterpret_cast<const Pack*>(z)[i];
    Pack pg{}, ph{}, o0, o1;
    if (ORDER >= 1) pg = reinterpret_cast<const Pack*>(g)[i];
    if (ORDER >= 2) ph = reinterpret_cast<const Pack*>(h)[i];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const T zv = pz.v[k], s = sigmoid(zv);
      if (ORDER == 0) o0.v[k] = zv / (T(1) + exp(-zv));
      if (ORDER == 1) o0.v[k] = times_slope(pg.v[k], zv, s);
      if (ORDER == 2) {
        o0.v[k] = times_slope(ph.v[k], zv, s);
        o1.v[k] = ph.v[k] * pg.v[k] * (s * (T(1) - s) * (T(2) + zv * (T(1) - T(2) * s)));
      }
    }
    reinterpret_cast<Pack*>(out0)[i] = o0;
    if (ORDER == 2) reinterpret_cast<Pack*>(out1)[i] = o1;
  }
}

template <typename T, int ORDER>
int launch(const void* z, const void* g, const void* h, void* out0, void* out1, int64_t n, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const uintptr_t all = reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(h) |
                        reinterpret_cast<uintptr_t>(out0) | reinterpret_cast<uintptr_t>(out1);
  const bool wide = n % V == 0 && (all & 15u) == 0;
  const long long blocks = ((wide ? n / V : n) + 255) / 256;
  if (blocks > 0x7fffffffLL) return FASTEQ_UNSUPPORTED;
  const unsigned grid = (unsigned)blocks;
  if (wide) silu_kernel<T, ORDER, V><<<grid, 256, 0, s>>>((const T*)z, (const T*)g, (const T*)h, (T*)out0, (T*)out1, n);
  else      silu_kernel<T, ORDER, 1><<<grid, 256, 0, s>>>((const T*)z, (const T*)g, (const T*)h, (T*)out0, (T*)out1, n);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

template <typename T>
int dispatch(int order, const void* z, const void* g, const void* h, void* out0, void* out1, int64_t n, cudaStream_t s) {
  switch (order) {
    case 0: return launch<T, 0>(z, nullptr, nullptr, out0, nullptr, n, s);
    case 1: return launch<T, 1>(z, g, nullptr, out0, nullptr, n, s);
    default: return launch<T, 2>(z, g, h, out0, out1, n, s);
  }
}

}  // namespace

extern "C" int fasteq_silu(int32_t dtype, int32_t order, const void* z, const void* g, const void* h, void* out0, void* out1, int64_t n,
                           fasteq_stream_t stream) {
  if (n < 0 || order < 0 || order > 2) return FASTEQ_INVALID;
  if (n == 0) return FASTEQ_OK;
  if (!z || !out0 || (order >= 1 && !g) || (order == 2 && (!h || !out1))) return FASTEQ_INVALID;
  if (dtype == 0) return dispatch<float>(order, z, g, h, out0, out1, n, (cudaStream_t)stream);
  if (dtype == 1) return dispatch<double>(order, z, g, h, out0, out1, n, (cudaStream_t)stream);
  return FASTEQ_INVALID;
}
