// libfasteq_b200_core: graph utilities and status reporting behind the C ABI of
// include/fasteq_b200.h.  (Spherical harmonics and SO3Linear entry points live in
// their own translation units of the same library.)
#include <cstdio>
#include <cstdint>
#include <algorithm>
#include <cuda_runtime.h>
#include "fasteq_b200.h"
#include "core_common.h"

namespace fasteq {
thread_local char g_cuda_err[256] = "";
int cuda_fail(cudaError_t e) {
  snprintf(g_cuda_err, sizeof(g_cuda_err), "%s", cudaGetErrorString(e));
  return FASTEQ_CUDA_ERROR;
}
}  // namespace fasteq
using namespace fasteq;

extern "C" const char* fasteq_status_string(int s) {
  switch (s) {
    case FASTEQ_OK: return "ok";
    case FASTEQ_UNSUPPORTED: return "unsupported shape or mode";
    case FASTEQ_INVALID: return "invalid argument";
    case FASTEQ_CUDA_ERROR: return "CUDA runtime error";
    case FASTEQ_INTERNAL: return "internal error";
    case FASTEQ_DEVICE_FAULT: return "device-side fault (wait timeout or index out of range)";
    default: return "unknown status";
  }
}
extern "C" const char* fasteq_last_cuda_error(void) { return g_cuda_err; }
extern "C" int fasteq_core_abi_version(void) { return FASTEQ_ABI_VERSION; }

// ---------------------------------------------------------------- sortedness
__global__ void check_sorted_kernel(const int* __restrict__ dst, long long n, int* flag) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  int bad = 0;
  for (; i + 1 < n; i += stride) bad |= (dst[i] > dst[i + 1]);
  if (bad) atomicExch(flag, 0);
}
__global__ void set_flag_kernel(int* flag, int v) { *flag = v; }

extern "C" int fasteq_graph_check_sorted(const int32_t* dst, int64_t n, int32_t* flag, fasteq_stream_t stream) {
  if (!flag || n < 0 || (n > 0 && !dst)) return FASTEQ_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  set_flag_kernel<<<1, 1, 0, s>>>(flag, 1);
  if (n > 1) {
    long long blocks = (n + 255) / 256;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
      sms = 128;
    if (blocks > (long long)sms * 8) blocks = (long long)sms * 8;     // grid-stride loop: eight resident CTAs per SM
    check_sorted_kernel<<<(int)blocks, 256, 0, s>>>(dst, n, flag);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// ---------------------------------------------------------------- order and degrees in one go
// result[0] <- 1 if some edge comes before a smaller one, counts[r] <- edges of row r.  Equal indices of a warp are added as
// one (runs of a sorted index; a receiver that has most edges).
__global__ void __launch_bounds__(256) survey_kernel(const int* __restrict__ dst, long long n, long long n_rows, int* result, int* counts) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  int bad = 0;
  for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n; i0 += stride) {
    const long long i = i0 + lane;
    const int v = i < n ? dst[i] : -1;
    if (i + 1 < n) bad |= v > dst[i + 1];
    const unsigned same = __match_any_sync(0xffffffffu, v);
    if (v >= 0 && v < n_rows && lane == __ffs(same) - 1) atomicAdd(&counts[v], __popc(same));
  }
  if (bad) atomicExch(result, 1);
}

__global__ void __launch_bounds__(256) max_count_kernel(const int* __restrict__ counts, long long n_rows, int* result) {
  int most = 0;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += (long long)gridDim.x * blockDim.x)
    most = counts[r] > most ? counts[r] : most;
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(result, most);
}

extern "C" int fasteq_graph_survey(const int32_t* dst, int64_t n_edges, int64_t n_rows, int32_t* result, fasteq_stream_t stream) {
  if (!result || n_edges < 0 || n_rows < 0 || (n_edges > 0 && !dst)) return FASTEQ_INVALID;
  if (n_edges > 0x7fffffffLL || n_rows >= 0x7fffffffLL) return FASTEQ_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(result, 0, (size_t)(2 + n_rows) * sizeof(int), s);
  if (e != cudaSuccess) return cuda_fail(e);
  if (n_edges > 0 && n_rows > 0) {
    const long long wave = 148 * 8;                     // grid-stride loops: a wave of resident CTAs
    survey_kernel<<<(unsigned)std::min<long long>((n_edges + 255) / 256, wave), 256, 0, s>>>(dst, n_edges, n_rows, result, result + 2);
    max_count_kernel<<<(unsigned)std::min<long long>((n_rows + 255) / 256, wave), 256, 0, s>>>(result + 2, n_rows, result + 1);
  }
  e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// ---------------------------------------------------------------- CSR offsets
// seg_ptr[r] = lower_bound(dst, r): one thread per row, binary search over the sorted index.
__global__ void build_csr_kernel(const int* __restrict__ dst, long long n_edges, long long n_rows, int* __restrict__ seg_ptr) {
  long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r > n_rows) return;
  long long lo = 0, hi = n_edges;
  while (lo < hi) {
    long long mid = (lo + hi) >> 1;
    if ((long long)dst[mid] < r) lo = mid + 1; else hi = mid;
  }
  seg_ptr[r] = (int)lo;
}

extern "C" int fasteq_graph_build_csr(const int32_t* dst, int64_t n_edges, int64_t n_rows, int32_t* seg_ptr,
                                      fasteq_stream_t stream) {
  if (!seg_ptr || n_edges < 0 || n_rows < 0 || (n_edges > 0 && !dst)) return FASTEQ_INVALID;
  if (n_edges > 0x7fffffffLL || n_rows >= 0x7fffffffLL) return FASTEQ_UNSUPPORTED;
  const long long n = n_rows + 1;
  build_csr_kernel<<<(int)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(dst, n_edges, n_rows, seg_ptr);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// ---------------------------------------------------------------- nodes by species
// A node's place in a stable order by species is the number of smaller species plus that of equal ones before it: one
// comparison per pair of nodes, the species of all nodes in shared memory.  Bound by issue (n / 4 loads and 2 n instructions per
// warp, a warp per scheduler).  torch's stable sort took 15 to 20 us of the summed backward of 200 to 3,000 nodes: 33 -> 14 us at 200,
// 79 -> 72 at 3,000, 177 -> 167 at 8,000.
constexpr int ORDER_MAX = 8192;

__global__ void __launch_bounds__(128) species_order_kernel(const int* __restrict__ species, int n, long long* __restrict__ order,
                                                            int* __restrict__ species_sorted) {
  __shared__ __align__(16) int all[ORDER_MAX];
  const int padded = (n + 31) & ~31;
  for (int j = threadIdx.x; j < padded; j += 128) all[j] = j < n ? species[j] : 0x7fffffff;
  __syncthreads();
  const int i = blockIdx.x * 128 + threadIdx.x, warp_first = i & ~31;
  if (warp_first >= n) return;
  const int mine = all[i < padded ? i : 0];
  int place = 0;
#pragma unroll 4
  for (int j = 0; j < warp_first; j += 4) {
    const int4 v = *reinterpret_cast<const int4*>(all + j);
    place += (v.x <= mine) + (v.y <= mine) + (v.z <= mine) + (v.w <= mine);
  }
  for (int j = warp_first; j < warp_first + 32; ++j) place += all[j] < mine || (all[j] == mine && j < i);
#pragma unroll 4
  for (int j = warp_first + 32; j < padded; j += 4) {
    const int4 v = *reinterpret_cast<const int4*>(all + j);
    place += (v.x < mine) + (v.y < mine) + (v.z < mine) + (v.w < mine);
  }
  if (i < n) { order[place] = i; species_sorted[place] = mine; }
}

extern "C" int fasteq_order_by_species(const int32_t* species, int64_t n, int64_t* order, int32_t* species_sorted, fasteq_stream_t stream) {
  if (n < 0 || (n > 0 && (!species || !order || !species_sorted))) return FASTEQ_INVALID;
  if (n > ORDER_MAX) return FASTEQ_UNSUPPORTED;
  if (n == 0) return FASTEQ_OK;
  species_order_kernel<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(species, (int)n, (long long*)order, species_sorted);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// ---------------------------------------------------------------- partition
__global__ void partition_kernel(const int* __restrict__ seg_ptr, long long n_rows, long long n_edges, int n_parts,
                                 int* __restrict__ part_ptr) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > n_parts) return;
  if (p == n_parts) { part_ptr[p] = (int)n_rows; return; }
  // Work of a segment = its edges + 1 (an empty receiver still costs a row store).
  const long long total = n_edges + n_rows;
  const long long target = total * p / n_parts;
  long long lo = 0, hi = n_rows;
  while (lo < hi) {
    long long mid = (lo + hi) >> 1;
    if ((long long)seg_ptr[mid] + mid < target) lo = mid + 1; else hi = mid;
  }
  part_ptr[p] = (int)lo;
}

extern "C" int fasteq_graph_partition(const int32_t* seg_ptr, int64_t n_rows, int64_t n_edges, int32_t n_parts,
                                      int32_t* part_ptr, fasteq_stream_t stream) {
  if (!seg_ptr || !part_ptr || n_parts < 1 || n_rows < 0 || n_edges < 0) return FASTEQ_INVALID;
  partition_kernel<<<(n_parts + 1 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(seg_ptr, n_rows, n_edges, n_parts, part_ptr);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// The same shares cut between edges: boundary p lies `target` units along the rows laid out as (edges, 1), inside a row's
// edges where it falls there.  part_ptr[p] is the row it falls in, part_edge[p] the edge.
__global__ void partition_edges_kernel(const int* __restrict__ seg_ptr, long long n_rows, long long n_edges, int n_parts,
                                       int* __restrict__ part_ptr, int* __restrict__ part_edge) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > n_parts) return;
  if (p == n_parts) { part_ptr[p] = (int)n_rows; part_edge[p] = (int)n_edges; return; }
  const long long target = (n_edges + n_rows) * p / n_parts;
  long long lo = 0, hi = n_rows;                       // the first row that ends beyond the target
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if ((long long)seg_ptr[mid + 1] + mid + 1 <= target) lo = mid + 1; else hi = mid;
  }
  if (lo == n_rows) { part_ptr[p] = (int)n_rows; part_edge[p] = (int)n_edges; return; }
  const long long first = seg_ptr[lo], end = seg_ptr[lo + 1], edge = first + (target - first - lo);
  const bool done = end > first && edge >= end;        // only the row's own unit is left of it
  part_ptr[p] = (int)(done ? lo + 1 : lo);
  part_edge[p] = (int)(done ? end : edge);
}

extern "C" int fasteq_graph_partition_edges(const int32_t* seg_ptr, int64_t n_rows, int64_t n_edges, int32_t n_parts,
                                            int32_t* part_ptr, int32_t* part_edge, fasteq_stream_t stream) {
  if (!seg_ptr || !part_ptr || !part_edge || n_parts < 1 || n_rows < 0 || n_edges < 0) return FASTEQ_INVALID;
  partition_edges_kernel<<<(n_parts + 1 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(seg_ptr, n_rows, n_edges, n_parts, part_ptr, part_edge);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}
