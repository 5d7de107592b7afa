// Hidden layers of the radial MLP (width 64, SiLU) as ONE kernel per direction, so that the per-edge
// activations between the layers never leave the SM:
//
//   forward : b [E, nb] --W1 (CUDA cores)--> h1 = silu(z1) --W2 (tcgen05)--> h2 = silu(z2) --W3--> h3
//             writes h_L [E, 64] and d_l = silu'(z_l) for the tensor-core layers (kept for the backward)
//   backward: g = dE/dh_L;  g <- W_l^T (g * d_l) for l = L..2 (tcgen05);  gz1 = g * silu'(z1) with z1
//             recomputed from b;  dE/db = W1^T gz1  [E, nb]
//
// The radial network of MACE / NequIP models is a small bias-free MLP on the radial basis
// (.../nequip/nn/embedding/_edge.py:174-189 feeds it; the reference leaves the MLP to torch); here its
// 64 x 64 layers run as 3xTF32 tensor-core products (same split as gemm_tf32x3.cu) chained through
// shared memory and TMEM.
//
// One persistent CTA per SM holds two groups of eight worker warps; each walks its own tiles of 128 edges, so that one group's
// activation arithmetic runs while the tensor core works on the other's layer, without an order between them.  The A operand
// never touches shared memory: a worker splits its values and writes them to tensor memory (lane = row, one column per
// K element), where the MMA reads them; through shared memory a layer cost 64 KB of writes and 96 KB of operand reads per tile.
//   warps 0-1   : issue the tcgen05.mma of a group's layer when its eight workers have written the operand; warp 0 first
//                 loads the pre-split hidden weights (TMA, SWIZZLE_128B), which stay resident
//   warps 2-17  : workers; a thread owns half a row of its group's tile (TMEM lane = row, 32 of the 64 columns).  Rows of
//                 [E, 64] tensors enter and leave through per-warp 32 x 32 swizzled slabs and tiled TMA
//                 loads / stores, so that global traffic is made of full 128-byte lines.
// What bounds it: neither memory (DRAM at 35 / 44 % forward / backward, ncu) nor issue (half the slots) but the chain of a tile - operand, MMA
// (24 x 33 clocks and the round trip), activation, twice - of which two are in flight; a third does not fit tensor memory
// (192 columns each).  Three layers of 64 behind 8 basis functions, forward / backward: 640,000 edges 211 / 245 -> 173 / 169 us (eight
// workers alternating between two tiles, operand in shared memory, dE/db zero-filled and added to -> this), 9,984 edges 11.3 / 13.9 -> 8.9 / 8.1 us.
// The next tile's first layer beside the last MMA was slower (180 / 200 us: spills at the 96 registers of 18 warps).
// Every mbarrier wait is bounded; a timeout sets a status word and the kernel drains.
#include <cstdio>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>
#include "fasteq_b200.h"
#include "core_common.h"
#include "fasteq_device.cuh"
#include "gemm_tf32x3.h"
#include "tcgen05_util.cuh"
#include "launch.cuh"

namespace fasteq {
namespace chain {

using namespace fasteq::tc;

constexpr int H = 64;                 // hidden width
constexpr int BM = 128, BK = 32;
constexpr int GROUPS = 2;             // tiles in flight per CTA
constexpr int N_WORKERS = 8;          // worker warps of a group
constexpr int NT = 32 * GROUPS * (1 + N_WORKERS);
constexpr int GROUP_COLUMNS = 3 * H;  // tensor memory of a group: accumulator, operand hi, operand lo
constexpr int TMEM_COLUMNS = 512;     // power of two above GROUPS * GROUP_COLUMNS
constexpr int MAX_TC = 2;             // tensor-core layers (hidden layers after the first)
constexpr int W_LAYER_BYTES = 2 * 2 * H * BK * 4;    // [kb][hi | lo] of a 64 x 64 matrix: 32 KB
constexpr int SLAB_BYTES = 32 * 128;                 // 32 rows x 32 FP32 columns
constexpr int MAX_NB = 16;
constexpr int EXCHANGE_BYTES = GROUPS * 4 * 32 * MAX_NB * 4;   // backward: dE/db of the right half-rows on its way to the left ones
constexpr int SMEM_BYTES = MAX_TC * W_LAYER_BYTES + GROUPS * N_WORKERS * 2 * SLAB_BYTES + H * MAX_NB * 4 + EXCHANGE_BYTES +
                           1024 /* barriers */ + 1024 /* alignment */;

struct Args {
  const float* basis;      // [M, nb]
  const float* w1;         // [H, nb]
  float* grad_basis;       // backward: dE/db [M, nb]
  long long M;
  int nb, n_tc;
  bool rows_in_vectors;    // nb fills the padded row and basis / grad_basis start on 16 bytes: float4 accesses
};

__device__ __forceinline__ void silu_and_derivative(float z, float& h, float& d) {
  const float s = __fdividef(1.0f, 1.0f + __expf(-z));
  h = z * s;
  d = s * (1.0f + z * (1.0f - s));
}

// Loads from addresses known when the kernel begins: volatile, so that no compiler moves them ahead of wait_for_previous_kernel()
__device__ __forceinline__ float load_after_wait(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 load4_after_wait(const float* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// 16-byte chunk c of row r of a 128-byte-row tile sits at chunk position c ^ (r & 7) (SWIZZLE_128B)
__device__ __forceinline__ float4* swz(unsigned char* tile, int r, int c) {
  return reinterpret_cast<float4*>(tile + r * 128 + ((c ^ (r & 7)) << 4));
}

__device__ __forceinline__ void tma_store_block(const CUtensorMap* map, int col0, long long row0, int z, const void* slab) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
               ::"l"(map), "r"(col0), "r"((int)row0), "r"(z), "r"(smem_u32(slab)) : "memory");
}

// tmW: prepared weights; tmIO0 / tmIO1: forward = (h_L out, derivatives out), backward = (dE/dh_L in, derivatives in),
// all [z][M][64] FP32 with 32 x 32 boxes
template <int NB, bool BWD>
__global__ void __launch_bounds__(NT, 1)
radial_chain_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmIO0,
                    const __grid_constant__ CUtensorMap tmIO1, const __grid_constant__ Args a, int* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* w_base = smem;                                   // [MAX_TC][kb][hi 8 KB | lo 8 KB]
  unsigned char* slab_base = smem + MAX_TC * W_LAYER_BYTES;       // [16 warps][2][4 KB]
  float* w1s = reinterpret_cast<float*>(slab_base + GROUPS * N_WORKERS * 2 * SLAB_BYTES);   // [H][NB], zero padded
  float4* exchange = reinterpret_cast<float4*>(w1s + H * MAX_NB);  // [group][quarter][NB / 4][lane]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(exchange) + EXCHANGE_BYTES);
  uint64_t* w_full = bars;                      // 1
  uint64_t* a_ready = bars + 1;                 // [groups] the eight worker warps have written the group's operand
  uint64_t* z_full = bars + 1 + GROUPS;         // [groups] the group's accumulator is complete
  uint64_t* slab_full = bars + 1 + 2 * GROUPS;  // [16 warps][2] backward: a TMA load has landed in the slab
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(slab_full + 2 * GROUPS * N_WORKERS);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_rows = (int)a.M, n_tiles = (int)((a.M + BM - 1) / BM);   // row numbers up to n_rows + BM fit (checked by the caller)
  const int step = GROUPS * (int)gridDim.x;     // a group's tiles: blockIdx.x + group * gridDim.x, + step, ...
  const int n_tc = a.n_tc;

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int g = 0; g < GROUPS; ++g) { mbar_init(&a_ready[g], N_WORKERS); mbar_init(&z_full[g], 1); }
    for (int i = 0; i < 2 * GROUPS * N_WORKERS; ++i) mbar_init(&slab_full[i], 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLUMNS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  wait_for_previous_kernel();
  for (int i = threadIdx.x; i < H * NB; i += NT) {
    const int j = i / NB, k = i % NB;
    w1s[i] = k < a.nb ? load_after_wait(a.w1 + j * a.nb + k) : 0.f;
  }
  __syncthreads();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < GROUPS) {
    // ------------------------------------------------------------------ MMA issue, one warp per group
    if (n_tc > 0) {
      if (warp == 0 && lane == 0) {
        mbar_arrive_expect_tx(w_full, (uint32_t)(n_tc * W_LAYER_BYTES));
        for (int l = 0; l < n_tc; ++l)
          for (int kb = 0; kb < 2; ++kb)
            for (int hl = 0; hl < 2; ++hl)
              tma_load_3d(w_base + l * W_LAYER_BYTES + kb * (2 * H * BK * 4) + hl * (H * BK * 4), &tmW, kb * BK, 0, l * 2 + hl, w_full);
      }
      __syncwarp();
      const int group = (int)uniform((uint32_t)warp);
      const uint32_t idesc = idesc_tf32_m128(H), tmem_d = uniform(tmem_base) + (uint32_t)(group * GROUP_COLUMNS);
      const uint32_t a_hi = tmem_d + H, a_lo = tmem_d + 2 * H;
      const uint64_t w0 = make_desc(uniform(smem_u32(w_base)));
      mbar_wait(w_full, 0u, status);
      tc_fence_after();
      uint32_t cnt = 0u;
      for (int t = (int)blockIdx.x + group * (int)gridDim.x; t < n_tiles; t += step) {
        for (int s = 0; s < n_tc; ++s) {
          mbar_wait(&a_ready[group], cnt & 1u, status);
          ++cnt;
          __syncwarp();
          tc_fence_after();
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
            const uint64_t b_hi = desc_at(w0, (uint32_t)(s * W_LAYER_BYTES + kb * (2 * H * BK * 4))), b_lo = desc_at(b_hi, H * BK * 4);
#pragma unroll
            for (int kk = 0; kk < BK / 8; ++kk) {
              const uint32_t off = kk * 32, col = (uint32_t)(kb * BK + kk * 8);
              warp_mma_tf32_a_tmem(tmem_d, a_lo + col, desc_at(b_hi, off), idesc, (kb | kk) ? 1u : 0u);
              warp_mma_tf32_a_tmem(tmem_d, a_hi + col, desc_at(b_lo, off), idesc, 1u);
              warp_mma_tf32_a_tmem(tmem_d, a_hi + col, desc_at(b_hi, off), idesc, 1u);
            }
          }
          warp_mma_commit(&z_full[group]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ workers
    const int group = (warp - GROUPS) / N_WORKERS;
    const int wk = (warp - GROUPS) % N_WORKERS;       // 0..7 within the group
    const int half = wk >> 2;                         // which 32 of the 64 columns
    const int quarter = warp & 3;                     // the TMEM lanes this warp may read
    const uint32_t tmem_lane = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(group * GROUP_COLUMNS + half * 32);
    unsigned char* slab0 = slab_base + (warp - GROUPS) * 2 * SLAB_BYTES;
    uint64_t* full = &slab_full[2 * (warp - GROUPS)];
    uint32_t n_full[2] = {0u, 0u}, n_z = 0u, n_store = 0u;
    const int col0 = half * 32;

    // ---- backward: tiled TMA loads of [32 rows x 32 columns] blocks into this warp's two slabs: dE/dh_L in slab 0, the top and then
    // the lower derivative in slab 1.  Every block is requested as soon as its slab has been read, one phase before it is needed.
    auto request = [&](int which, const CUtensorMap* map, int z, int row0) {
      fence_async_smem();                 // earlier generic reads of the slab precede the async write
      __syncwarp();
      if (lane == 0) {
        mbar_arrive_expect_tx(&full[which], SLAB_BYTES);
        tma_load_3d(slab0 + which * SLAB_BYTES, map, col0, row0, z, &full[which]);
      }
    };
    auto landed = [&](int which) { mbar_wait(&full[which], n_full[which] & 1u, status); ++n_full[which]; };
    auto load_basis = [&](float (&bb)[NB], int row0, bool exists) {
      const long long r = row0 + lane;
      const bool mine = exists && r < n_rows;
      if (a.rows_in_vectors) {
#pragma unroll
        for (int k = 0; k < NB; k += 4) {
          const float4 q = mine ? load4_after_wait(a.basis + r * NB + k) : make_float4(0.f, 0.f, 0.f, 0.f);
          bb[k] = q.x; bb[k + 1] = q.y; bb[k + 2] = q.z; bb[k + 3] = q.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < NB; ++k) bb[k] = (mine && k < a.nb) ? load_after_wait(a.basis + r * a.nb + k) : 0.f;
      }
    };
    auto first_layer = [&](const float (&bb)[NB], int j, float& h, float& d) {
      float z = 0.f;
#pragma unroll
      for (int k = 0; k < NB; ++k) z = fmaf(w1s[(col0 + j) * NB + k], bb[k], z);
      silu_and_derivative(z, h, d);
    };
    // ---- forward: one 32 x 32 block leaves through the slabs (alternating) as a tiled TMA store
    auto begin_store = [&]() {
      if (lane == 0) bulk_wait_read<1>();     // the slab used two stores ago has been read
      __syncwarp();
      return slab0 + (n_store & 1u) * SLAB_BYTES;
    };
    auto end_store = [&](const unsigned char* sl, const CUtensorMap* map, int z, int row0) {
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (row0 < n_rows) tma_store_block(map, col0, row0, z, sl);
        bulk_commit();
      }
      ++n_store;
    };

    float b[NB], v[32];
    int t = (int)blockIdx.x + group * (int)gridDim.x;
    if (t < n_tiles) {
      const int row0 = t * BM + quarter * 32;
      if (!BWD) {
        load_basis(b, row0, true);
      } else {
        request(0, &tmIO0, 0, row0);
        if (n_tc > 0) request(1, &tmIO1, n_tc - 1, row0);
      }
    }
    for (; t < n_tiles; t += step) {
      const int row0 = t * BM + quarter * 32;
      const bool has_next = t + step < n_tiles;
      const int next_row0 = has_next ? row0 + step * BM : row0;

      // the operand of the first tensor-core layer (or, without one, the final vector)
      if (!BWD) {
#pragma unroll
        for (int j = 0; j < 32; ++j) { float d; first_layer(b, j, v[j], d); }
        load_basis(b, next_row0, has_next);
      } else {
        load_basis(b, row0, true);
        landed(0);
        if (n_tc > 0) landed(1);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          float4 gv = *swz(slab0, lane, c);
          if (n_tc > 0) {
            const float4 dv = *swz(slab0 + SLAB_BYTES, lane, c);
            gv.x *= dv.x; gv.y *= dv.y; gv.z *= dv.z; gv.w *= dv.w;
          }
          v[4 * c] = gv.x; v[4 * c + 1] = gv.y; v[4 * c + 2] = gv.z; v[4 * c + 3] = gv.w;
        }
        if (n_tc > 1) request(1, &tmIO1, n_tc - 2, row0);
        else if (n_tc > 0 && has_next) request(1, &tmIO1, n_tc - 1, next_row0);
        if (has_next) request(0, &tmIO0, 0, next_row0);
      }

      for (int s = 0; s < n_tc; ++s) {
        // operand of layer s -> tensor memory; the accumulator of the layer before has been read by this thread
        {
          uint32_t part[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float hi, lo;
            split_tf32(v[j], hi, lo);
            part[j] = __float_as_uint(hi);
            v[j] = lo;
          }
          tmem_st_32_begin(tmem_lane + H, part);
#pragma unroll
          for (int j = 0; j < 32; ++j) part[j] = __float_as_uint(v[j]);
          tmem_st_32(tmem_lane + 2 * H, part);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_ready[group]);
        uint32_t r[32];
        mbar_wait(&z_full[group], n_z & 1u, status);
        ++n_z;
        tc_fence_after();
        tmem_ld_32(tmem_lane, r);
        if (!BWD) {
          unsigned char* sl = begin_store();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            float4 d;
            silu_and_derivative(__uint_as_float(r[4 * c]), v[4 * c], d.x);
            silu_and_derivative(__uint_as_float(r[4 * c + 1]), v[4 * c + 1], d.y);
            silu_and_derivative(__uint_as_float(r[4 * c + 2]), v[4 * c + 2], d.z);
            silu_and_derivative(__uint_as_float(r[4 * c + 3]), v[4 * c + 3], d.w);
            *swz(sl, lane, c) = d;
          }
          end_store(sl, &tmIO1, s, row0);
        } else {
          const bool more = s + 1 < n_tc;      // multiply by the derivative of the layer below (n_tc <= 2: s == 0)
          if (more) landed(1);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            float4 dv = make_float4(1.f, 1.f, 1.f, 1.f);
            if (more) dv = *swz(slab0 + SLAB_BYTES, lane, c);
            v[4 * c] = __uint_as_float(r[4 * c]) * dv.x; v[4 * c + 1] = __uint_as_float(r[4 * c + 1]) * dv.y;
            v[4 * c + 2] = __uint_as_float(r[4 * c + 2]) * dv.z; v[4 * c + 3] = __uint_as_float(r[4 * c + 3]) * dv.w;
          }
          if (more && has_next) request(1, &tmIO1, n_tc - 1, next_row0);
        }
      }

      if (!BWD) {
        unsigned char* sl = begin_store();
#pragma unroll
        for (int c = 0; c < 8; ++c) *swz(sl, lane, c) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        end_store(sl, &tmIO0, 0, row0);
      } else {
        float gb[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) gb[k] = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float h, d;
          first_layer(b, j, h, d);
          const float gz = v[j] * d;
#pragma unroll
          for (int k = 0; k < NB; ++k) gb[k] = fmaf(gz, w1s[(col0 + j) * NB + k], gb[k]);
        }
        // the two half-rows of an edge meet: the right one's sums go through shared memory to the left one's thread
        float4* ex = exchange + (group * 4 + quarter) * (MAX_NB / 4) * 32 + lane;
        const int pair_barrier = 1 + group * 4 + quarter;
        if (half == 1) {
#pragma unroll
          for (int k = 0; k < NB; k += 4) ex[(k / 4) * 32] = make_float4(gb[k], gb[k + 1], gb[k + 2], gb[k + 3]);
        }
        named_barrier_sync(pair_barrier, 64);      // written
        const long long row = row0 + lane;
        if (half == 0) {
#pragma unroll
          for (int k = 0; k < NB; k += 4) {
            const float4 q = ex[(k / 4) * 32];
            const float4 sum = make_float4(gb[k] + q.x, gb[k + 1] + q.y, gb[k + 2] + q.z, gb[k + 3] + q.w);
            if (row < n_rows) {
              float* out = a.grad_basis + row * a.nb + k;
              if (a.rows_in_vectors) {
                *reinterpret_cast<float4*>(out) = sum;
              } else {
                if (k < a.nb) out[0] = sum.x;
                if (k + 1 < a.nb) out[1] = sum.y;
                if (k + 2 < a.nb) out[2] = sum.z;
                if (k + 3 < a.nb) out[3] = sum.w;
              }
            }
          }
        }
        named_barrier_sync(pair_barrier, 64);      // read: the next tile may write
      }
    }
    if (!BWD && lane == 0) bulk_wait_read<0>();   // the slabs must outlive their stores
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLUMNS);
  }
}

// prepared[l][hi | lo][r][c] = split(transpose ? W_l[c][r] : W_l[r][c]) for up to MAX_TC 64 x 64 matrices
__global__ void prepare_weights_kernel(const float* __restrict__ w0, const float* __restrict__ w1, int n, bool transpose,
                                       float* __restrict__ prepared) {
  const int total = n * H * H;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int l = i / (H * H), r = (i / H) % H, c = i % H;
    const float* w = l == 0 ? w0 : w1;
    const float v = transpose ? w[c * H + r] : w[r * H + c];
    float hi, lo;
    tc::split_tf32(v, hi, lo);
    prepared[(size_t)(l * 2) * H * H + r * H + c] = hi;
    prepared[(size_t)(l * 2 + 1) * H * H + r * H + c] = lo;
  }
}

__device__ int g_chain_status;

int device_status(int* code) {
  int v = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_chain_status, sizeof(int));
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaMemcpyToSymbol(g_chain_status, &zero, sizeof(int));
  if (e != cudaSuccess) return cuda_fail(e);
  *code = v;
  return FASTEQ_OK;
}

template <int NB, bool BWD>
static int launch_nb(const CUtensorMap& tmw, const CUtensorMap& io0, const CUtensorMap& io1, const Args& a, cudaStream_t s) {
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_chain_status);
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaFuncSetAttribute(radial_chain_kernel<NB, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  if (e != cudaSuccess) return cuda_fail(e);
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return cuda_fail(e);
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return cuda_fail(e);
  const long long n_tiles = (a.M + BM - 1) / BM;
  const unsigned grid = (unsigned)(n_tiles < sms ? n_tiles : sms);
  e = launch_dependent(radial_chain_kernel<NB, BWD>, grid, NT, SMEM_BYTES, s, tmw, io0, io1, a, st);
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

static int prepare(const float* const* w_hidden, int n_tc, bool bwd, float* prepared, cudaStream_t s) {
  if (n_tc < 1) return FASTEQ_OK;
  if (n_tc > MAX_TC) return FASTEQ_UNSUPPORTED;
  if (!w_hidden || !prepared) return FASTEQ_INVALID;
  for (int l = 0; l < n_tc; ++l)
    if (!w_hidden[l]) return FASTEQ_INVALID;
  // forward uses W_2, W_3 in order; backward uses W_L^T first
  const float* first = bwd ? w_hidden[n_tc - 1] : w_hidden[0];
  const float* second = n_tc > 1 ? (bwd ? w_hidden[0] : w_hidden[1]) : first;
  prepare_weights_kernel<<<n_tc * 4, 256, 0, s>>>(first, second, n_tc, bwd, prepared);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// io0: forward h_L out / backward dE/dh_L in, [M, 64]; io1: derivatives [n_tc, M, 64] (out / in)
template <bool BWD>
static int run(Args a, const float* const* w_hidden, const float* prepared_in, const float* io0, const float* io1, cudaStream_t s) {
  if (a.M < 0 || a.nb < 1) return FASTEQ_INVALID;
  if (a.nb > MAX_NB || a.n_tc < 0 || a.n_tc > MAX_TC || a.M > 0x7fffffffLL - BM) return FASTEQ_UNSUPPORTED;
  if (a.M == 0) return FASTEQ_OK;
  if (!a.basis || !a.w1 || !io0 || (a.n_tc > 0 && ((!w_hidden && !prepared_in) || !io1)) || (BWD && !a.grad_basis)) return FASTEQ_INVALID;
  if ((reinterpret_cast<uintptr_t>(io0) | reinterpret_cast<uintptr_t>(io1) | reinterpret_cast<uintptr_t>(prepared_in)) & 15u)
    return FASTEQ_UNSUPPORTED;
  a.rows_in_vectors = (a.nb == 8 || a.nb == MAX_NB) &&
                      !((reinterpret_cast<uintptr_t>(a.basis) | reinterpret_cast<uintptr_t>(a.grad_basis)) & 15u);
  cudaError_t e;
  float* tmp = nullptr;
  alignas(64) CUtensorMap tmw, tm0, tm1;
  const int n_alloc = a.n_tc > 0 ? a.n_tc : 1;
  int rc = FASTEQ_OK;
  if (!prepared_in || a.n_tc == 0) {
    e = cudaMallocAsync((void**)&tmp, (size_t)n_alloc * 2 * H * H * sizeof(float), s);
    if (e != cudaSuccess) return cuda_fail(e);
    if (a.n_tc > 0) rc = prepare(w_hidden, a.n_tc, BWD, tmp, s);
  }
  const float* prepared = tmp ? tmp : prepared_in;
  if (rc == FASTEQ_OK)
    rc = tc::make_map(&tmw, prepared, (uint64_t)H, (uint64_t)H, (uint64_t)n_alloc * 2, (uint64_t)H, (uint64_t)H * H, BK, H, 1);
  if (rc == FASTEQ_OK) rc = tc::make_map(&tm0, io0, (uint64_t)H, (uint64_t)a.M, 1, (uint64_t)H, (uint64_t)a.M * H, 32, 32, 1);
  if (rc == FASTEQ_OK)
    rc = tc::make_map(&tm1, a.n_tc > 0 ? io1 : io0, (uint64_t)H, (uint64_t)a.M, (uint64_t)n_alloc, (uint64_t)H, (uint64_t)a.M * H, 32, 32, 1);
  if (rc == FASTEQ_OK) rc = a.nb <= 8 ? launch_nb<8, BWD>(tmw, tm0, tm1, a, s) : launch_nb<16, BWD>(tmw, tm0, tm1, a, s);
  if (tmp) cudaFreeAsync(tmp, s);
  return rc;
}

}  // namespace chain
}  // namespace fasteq

extern "C" int fasteq_radial_chain_forward(const float* basis, int64_t n_edges, int32_t n_basis, const float* w_first,
                                           const float* const* w_hidden, const float* prepared, int32_t n_hidden, float* out,
                                           float* deriv, fasteq_stream_t stream) {
  if (n_hidden < 1) return FASTEQ_INVALID;
  fasteq::chain::Args a{};
  a.basis = basis; a.w1 = w_first; a.M = n_edges; a.nb = n_basis; a.n_tc = n_hidden - 1;
  return fasteq::chain::run<false>(a, w_hidden, prepared, out, deriv, (cudaStream_t)stream);
}

extern "C" int fasteq_radial_chain_backward(const float* grad_out, const float* deriv, const float* basis, int64_t n_edges,
                                            int32_t n_basis, const float* w_first, const float* const* w_hidden,
                                            const float* prepared, int32_t n_hidden, float* grad_basis, fasteq_stream_t stream) {
  if (n_hidden < 1) return FASTEQ_INVALID;
  fasteq::chain::Args a{};
  a.basis = basis; a.w1 = w_first; a.grad_basis = grad_basis; a.M = n_edges; a.nb = n_basis; a.n_tc = n_hidden - 1;
  return fasteq::chain::run<true>(a, w_hidden, prepared, grad_out, deriv, (cudaStream_t)stream);
}

extern "C" int fasteq_radial_chain_prepare(const float* const* w_hidden, int32_t n_hidden, int32_t backward, float* prepared,
                                           fasteq_stream_t stream) {
  if (n_hidden < 1) return FASTEQ_INVALID;
  return fasteq::chain::prepare(w_hidden, n_hidden - 1, backward != 0, prepared, (cudaStream_t)stream);
}
