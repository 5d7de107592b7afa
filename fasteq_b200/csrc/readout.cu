// Per-atom scalar readout: e[n] = e_in[n] + sum_c h[n, c] w[c] over the first C of D columns (the scalar segment of an ir_mul
// row), and its gradient dh[n, c] = g[n] w[c] for c < C, 0 beyond.  As elementwise operations these were a multiply, a row
// reduction and an add forward and a multiply, a fill and a copy backward: launches of 2 us each that a small system waits
// for one after the other.  Bound: latency (a few rows) or the rows' bytes; one warp per node.
#include <cstdint>
#include <cuda_runtime.h>
#include "fasteq_b200.h"
#include "core_common.h"
#include "fasteq_device.cuh"

using namespace fasteq;

namespace {

template <typename T>
__global__ void __launch_bounds__(256) readout_fwd_kernel(const T* __restrict__ h, const T* __restrict__ w, const T* __restrict__ e_in,
                                                          T* __restrict__ e, long long n, int c_count, long long d) {
  let_next_kernel_begin();
  const long long node = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (node >= n) return;
  const T* row = h + (size_t)node * d;
  T s = T(0);
#pragma unroll 4
  for (int c = lane; c < c_count; c += 32) s += row[c] * w[c];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) e[node] = e_in ? e_in[node] + s : s;
}

template <typename T>
__global__ void __launch_bounds__(256) readout_bwd_kernel(const T* __restrict__ g, const T* __restrict__ w, T* __restrict__ gh, long long n,
                                                          int c_count, long long d) {
  let_next_kernel_begin();
  const long long node = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (node >= n) return;
  const T gv = g[node];
  T* row = gh + (size_t)node * d;
#pragma unroll 4
  for (long long c = threadIdx.x & 31; c < d; c += 32) row[c] = c < c_count ? gv * w[c] : T(0);
}

template <typename T>
int run(bool backward, const void* a, const void* w, const void* e_in, void* out, long long n, int c_count, long long d, cudaStream_t s) {
  const long long blocks = (n + 7) / 8;
  if (blocks > 0x7fffffffLL) return FASTEQ_UNSUPPORTED;
  if (backward) readout_bwd_kernel<T><<<(unsigned)blocks, 256, 0, s>>>((const T*)a, (const T*)w, (T*)out, n, c_count, d);
  else readout_fwd_kernel<T><<<(unsigned)blocks, 256, 0, s>>>((const T*)a, (const T*)w, (const T*)e_in, (T*)out, n, c_count, d);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

int dispatch(int dtype, bool backward, const void* a, const void* w, const void* e_in, void* out, int64_t n, int32_t c_count, int64_t d,
             fasteq_stream_t stream) {
  if (n < 0 || c_count < 0 || d < c_count) return FASTEQ_INVALID;
  if (n == 0 || (backward && d == 0)) return FASTEQ_OK;
  if (!out || (c_count > 0 && (!a || !w))) return FASTEQ_INVALID;
  if (dtype == 0) return run<float>(backward, a, w, e_in, out, n, c_count, d, (cudaStream_t)stream);
  if (dtype == 1) return run<double>(backward, a, w, e_in, out, n, c_count, d, (cudaStream_t)stream);
  return FASTEQ_INVALID;
}

}  // namespace

extern "C" int fasteq_readout_forward(int32_t dtype, const void* h, const void* w, const void* e_in, void* e, int64_t n, int32_t c_count,
                                      int64_t d, fasteq_stream_t stream) {
  return dispatch(dtype, false, h, w, e_in, e, n, c_count, d, stream);
}

extern "C" int fasteq_readout_backward(int32_t dtype, const void* g, const void* w, void* gh, int64_t n, int32_t c_count, int64_t d,
                                       fasteq_stream_t stream) {
  return dispatch(dtype, true, g, w, nullptr, gh, n, c_count, d, stream);
}
