// 3xTF32 grouped GEMM on the sm_100a tensor cores (tcgen05 + TMEM + TMA), used for the dense
// contractions of the path: SO3Linear forward / grad_x and the radial MLP layers.
//
//   C[b, c_row(item), n] = sum_{segments s of item} sum_k A[b, a_row(s), k] * Bt[w(s), n, k]
//
// A is a [M, rows_a, K] FP32 tensor (K contiguous), Bt a [P, N, K] FP32 tensor (K contiguous), C a
// [M, rows_c, N] FP32 tensor.  A plain GEMM is the case rows_a = rows_c = P = 1.
//
// Precision: each FP32 operand v is split into hi = v with the 13 low mantissa bits cleared (exact in
// TF32) and lo = v - hi (exact in FP32); the kernel accumulates hi*hi + hi*lo + lo*hi in FP32, which
// keeps the relative error near 2^-21 (the reference's tf32x3 scheme,
// fasteq/cuda/src/eqlinear/backends/tf32/shape_plan.cu:109-113: three MMAs, no lo*lo term).
//
// Structure of one CTA (persistent: one CTA per SM walks 128 x BN output tiles round-robin, the rings and the TMEM
// accumulators - two of 64 columns or one of 128 - carry over from tile to tile so that loads, splits, MMAs and stores of
// neighbouring tiles overlap):
//   warps 0, 10  : TMA producers -- 3-D tiled loads (SWIZZLE_128B) of the raw A k-blocks (0) and of the weights' (10)
//   warp 1       : allocates TMEM, issues tcgen05.mma (kind::tf32, M = 128, N = BN and 2 BN, K = 8) as a whole warp that elects a lane,
//                  releases ring stages and signals the epilogue with tcgen05.commit
//   warps 2..5   : split each raw A k-block into hi / lo parts in tensor memory (thread = row = TMEM
//                  lane, tcgen05.st), from where the MMAs take their A operand
//   warps 6..9   : read a finished accumulator with tcgen05.ld and store the tile through swizzled
//                  staging slabs and TMA stores
// Every mbarrier wait is bounded (about two seconds), after which a status word is set and the
// waiter falls through; TMEM is always released before the CTA ends.  Single-CTA copies only, no clusters.
#include <algorithm>
#include <cstdio>
#include <cstdint>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include "fasteq_b200.h"
#include "core_common.h"
#include "fasteq_device.cuh"
#include "gemm_tf32x3.h"
#include "tcgen05_util.cuh"
#include "launch.cuh"

namespace fasteq {
namespace tc {

constexpr int BM = 128, BK = 32;
constexpr int NT = 192;     // A-stationary kernel: 6 warps
constexpr int NT_P = 352;   // persistent grouped kernel: 11 warps

constexpr int ITEM_TABLE = 768;       // entries of the table from item to group (see decode_tile)

template <int BN> struct Cfg {
  static constexpr int A_BYTES = BM * BK * 4;          // 16 KB
  static constexpr int B_BYTES = BN * BK * 4;
  // raw A and the weights' hi | lo tiles each have their own ring: A comes from HBM and is free again once split, the weights come from
  // L2 and stay until the MMAs have read them.  Together they fill 192 KB.  Measured: 6 + 3 stages at 128 columns 85.0 us where 4 + 4 take 82.7
  // (12,288 nodes, see below), 17.8 -> 18.4 at 1,536; 6 + 6 at 64 columns 9.4 us where 8 + 4 take 9.0 (192 nodes).
  static constexpr int A_STAGES = (BN <= 64) ? 8 : 4, B_STAGES = 4;
  static constexpr int RING_BYTES = A_STAGES * A_BYTES + B_STAGES * 2 * B_BYTES;
  static constexpr int SLOTS = 4;                       // split A: 4 x 64 tensor-memory columns
  static constexpr int ACCUMULATORS = 256 / (2 * BN);   // in the other 256: two tiles of 64 columns, one of 128
  static constexpr int STORE_BYTES = 4 * 2 * 4096;     // per epilogue warp: two 32 x 32 FP32 slabs for the TMA stores
  static constexpr int BARRIER_BYTES = (2 * (A_STAGES + B_STAGES + SLOTS + ACCUMULATORS) + 1) * 8;
  static constexpr int SMEM_BYTES = RING_BYTES + STORE_BYTES + BARRIER_BYTES + ITEM_TABLE + 1024 /* alignment slack */;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
};

// one output tile of the persistent loop
struct Tile {
  int g, t, seg0, n_kb, n0;
  long long m0;
};

// Every role of the CTA decodes every tile, in line with its other work: a short tile (K = 64: two k-blocks) spent more on three
// 64-bit divisions and a walk over up to 64 groups than on its MMAs.  Hence 32-bit divisions where the tile count allows
// and a shared-memory table from item to group (`item_g`, null when there are more items than it holds).
//
// Order of the tiles.  With many rounds of tiles the items of a row tile follow one another, turned by one from row tile to row tile (a CTA's
// stride through them then meets long and short items alike): neighbouring CTAs read neighbouring rows of the same entries, whole DRAM
// pages, and different weights.  With items outermost they read 128 bytes out of every entry, and the same weights at once: 12,288 nodes
// (see below) 90.2 -> 85.0 us, 20,011 nodes 142.9 -> 131.8 (6 + 3 stages).  Up to four rounds (`m_tiles` > 0, else 0) items stay outermost: the short ones, which
// come last, fill the last round (1,536 nodes 18.4 us, the other way 19.1).
__device__ __forceinline__ Tile decode_tile(const TcTable& tab, const unsigned char* item_g, long long tile, int m_tiles, int n_tiles,
                                            int kb_per_seg, int BN) {
  Tile r;
  int mx, ny, z;
  if (m_tiles > 0) {
    const unsigned t32 = (unsigned)tile, rest = t32 / (unsigned)m_tiles;
    mx = (int)(t32 - rest * (unsigned)m_tiles);
    z = (int)(rest / (unsigned)n_tiles);
    ny = (int)(rest - (unsigned)z * (unsigned)n_tiles);
  } else if (tile <= 0xffffffffLL) {
    const unsigned t32 = (unsigned)tile, rest = t32 / (unsigned)n_tiles, m = rest / (unsigned)tab.n_items;
    ny = (int)(t32 - rest * (unsigned)n_tiles);
    mx = (int)m;
    z = (int)((rest - m * (unsigned)tab.n_items + m % (unsigned)tab.n_items) % (unsigned)tab.n_items);
  } else {
    const long long rest = tile / n_tiles, m = rest / tab.n_items;
    ny = (int)(tile % n_tiles); mx = (int)m; z = (int)((rest - m * tab.n_items + m) % tab.n_items);
  }
  int g = 0;
  if (item_g) g = item_g[z];
  else while (g + 1 < tab.n_groups && z >= tab.item_first[g + 1]) ++g;
  r.g = g; r.t = z - tab.item_first[g];
  r.seg0 = tab.group_first[g];
  r.n_kb = (tab.group_first[g + 1] - r.seg0) * kb_per_seg;
  r.m0 = (long long)mx * BM; r.n0 = ny * BN;
  return r;
}

// Shared memory bounds a k-block: TMA fills, the split's reads and the MMAs' operand reads share its 128 bytes per clock.  With the
// split A in tensor memory (thread = row = TMEM lane, tcgen05.st) that is 112 KB at 128 columns, 875 clocks beside 773 of MMAs; split in
// place in shared memory it was 176 KB.  SO3Linear after the tensor product (40 rows of 128 channels to 16): 12,288 nodes 112.7 -> 95.5 us a
// direction, 1,536 nodes 21.0 -> 17.9; with the two rings and the order of tiles above 82.7 (4.3 TB/s of features) and 17.8.  A second set of
// split warps on alternate k-blocks changes nothing (93.3 where 90.2).
// The price at 128 columns is a single accumulator (256 columns with its cross terms): the epilogue takes it to registers whole and
// hands it back before it stores.
template <int BN>
__global__ void __launch_bounds__(NT_P, 1)
gemm_tf32x3_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBhi,
                   const __grid_constant__ CUtensorMap tmBlo, const __grid_constant__ CUtensorMap tmC,
                   const __grid_constant__ TcTable tab, long long M, int N, int K, long long n_tiles_total, int m_tiles,
                   int n_tiles, int* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using C_ = Cfg<BN>;
  constexpr int A_STAGES = C_::A_STAGES, B_STAGES = C_::B_STAGES, SLOTS = C_::SLOTS, ACC = C_::ACCUMULATORS;
  constexpr uint32_t TMEM_COLS = 512, TMEM_A = 256;
  static_assert(ACC * 2 * BN == (int)TMEM_A && SLOTS * 2 * BK <= 256, "tensor memory: accumulators + A ring");
  unsigned char* b_base = smem + A_STAGES * C_::A_BYTES;
  unsigned char* store_base = smem + C_::RING_BYTES;               // [4 warps][2 slabs][32 rows x 128 B]
  uint64_t* bars = reinterpret_cast<uint64_t*>(store_base + C_::STORE_BYTES);
  uint64_t* a_full = bars;                   // [A_STAGES] TMA landed
  uint64_t* a_empty = a_full + A_STAGES;     // [A_STAGES] the four split warps have read it
  uint64_t* b_full = a_empty + A_STAGES;     // [B_STAGES] TMA landed
  uint64_t* b_empty = b_full + B_STAGES;     // [B_STAGES] MMAs have read it
  uint64_t* full_split = b_empty + B_STAGES; // [SLOTS] hi / lo parts ready
  uint64_t* slot_empty = full_split + SLOTS; // [SLOTS] MMAs have consumed the split A
  uint64_t* acc_full = slot_empty + SLOTS;   // [ACC] accumulator complete
  uint64_t* acc_empty = acc_full + ACC;      // [ACC] accumulator read back by the four epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + ACC);

  unsigned char* item_table = reinterpret_cast<unsigned char*>(bars) + C_::BARRIER_BYTES;
  const unsigned char* item_g = tab.n_items <= ITEM_TABLE ? item_table : nullptr;
  if (item_g) {
    for (int z = threadIdx.x; z < tab.n_items; z += NT_P) {
      int g = 0;
      while (g + 1 < tab.n_groups && z >= tab.item_first[g + 1]) ++g;
      item_table[z] = (unsigned char)g;
    }
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kb_per_seg = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < A_STAGES; ++s) { mbar_init(&a_full[s], 1); mbar_init(&a_empty[s], 4); }
    for (int s = 0; s < B_STAGES; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < SLOTS; ++s) { mbar_init(&full_split[s], 4); mbar_init(&slot_empty[s], 1); }
    for (int b = 0; b < ACC; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  wait_for_previous_kernel();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_a = tmem_base + TMEM_A;     // [SLOTS][hi 32 columns | lo 32 columns]

  if (warp == 0 || warp == 10) {
    // ------------------------------------------------------------------ TMA producers: warp 0 of A, warp 10 of the weights
    if (lane == 0) {
      int it = 0;
      for (long long tile = blockIdx.x; tile < n_tiles_total; tile += gridDim.x) {
        const Tile tl = decode_tile(tab, item_g, tile, m_tiles, n_tiles, kb_per_seg, BN);
        // each tile starts its walk over the k-blocks at a different one, so that the CTAs do not all fetch the same
        // weight lines from L2 at the same moment (the terms of a sum are the same, their order depends on the tile)
        const int kb_start = (int)(tile % tl.n_kb);
        int seg = tl.seg0 + kb_start / kb_per_seg, k_in = kb_start % kb_per_seg;
        for (int kbi = 0; kbi < tl.n_kb; ++kbi, ++it) {
          if (warp == 0) {
            const int s = it % A_STAGES;
            mbar_wait(&a_empty[s], ((it / A_STAGES) & 1u) ^ 1u, status);
            mbar_arrive_expect_tx(&a_full[s], (uint32_t)C_::A_BYTES);
            tma_load_3d(smem + (size_t)s * C_::A_BYTES, &tmA, k_in * BK, tab.path_a_row[seg] + tl.t, (int)tl.m0, &a_full[s]);
          } else {
            const int s = it % B_STAGES;
            unsigned char* st = b_base + (size_t)s * (2 * C_::B_BYTES);
            mbar_wait(&b_empty[s], ((it / B_STAGES) & 1u) ^ 1u, status);
            mbar_arrive_expect_tx(&b_full[s], (uint32_t)(2 * C_::B_BYTES));
            tma_load_3d(st, &tmBhi, k_in * BK, tl.n0, tab.path_w[seg], &b_full[s]);
            tma_load_3d(st + C_::B_BYTES, &tmBlo, k_in * BK, tl.n0, tab.path_w[seg], &b_full[s]);
          }
          if (++k_in == kb_per_seg) { k_in = 0; ++seg; }
          if (seg == tl.seg0 + tl.n_kb / kb_per_seg) seg = tl.seg0;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (whole warp, one elected lane)
    // instruction descriptors: D = F32, A = B = TF32, both K-major, M = 128; N = 2 BN for the product of
    // A_hi with the stacked [B_hi; B_lo] tile, N = BN for A_lo x B_hi
    const uint32_t idesc2 = idesc_tf32_m128(2 * BN), idesc1 = idesc_tf32_m128(BN);
    const uint32_t tm = uniform(tmem_base), ring = uniform(smem_u32(b_base));
    const uint64_t desc0 = make_desc(ring);
    int it = 0;
    uint32_t lt = 0;
    for (long long tile = blockIdx.x; tile < n_tiles_total; tile += gridDim.x, ++lt) {
      const int n_kb = (int)uniform((uint32_t)decode_tile(tab, item_g, tile, m_tiles, n_tiles, kb_per_seg, BN).n_kb);
      const uint32_t buf = lt % ACC;
      mbar_wait(&acc_empty[buf], ((lt / ACC) & 1u) ^ 1u, status);
      tc_fence_after();
      // columns [0, BN): hi x hi;  [BN, 2 BN): hi x lo + lo x hi (small terms, kept apart so that their
      // sum is not absorbed one rounding at a time into the large accumulator)
      const uint32_t tmem_d = tm + buf * (uint32_t)(2 * BN);
      for (int kb = 0; kb < n_kb; ++kb, ++it) {
        const int s = it % B_STAGES, slot = it % SLOTS;
        mbar_wait(&b_full[s], (it / B_STAGES) & 1u, status);
        mbar_wait(&full_split[slot], (it / SLOTS) & 1u, status);
        __syncwarp();
        tc_fence_after();
        const uint64_t b_hi = desc_at(desc0, (uint32_t)(s * 2 * C_::B_BYTES));    // B_hi tile, B_lo tile right behind it
        const uint32_t ta = tm + TMEM_A + (uint32_t)(slot * 2 * BK);
#pragma unroll
        for (int kk = 0; kk < BK / 8; ++kk) {
          const uint32_t off = kk * 32;   // 8 TF32 values = 32 bytes along K inside the 128-byte swizzle row
          warp_mma_tf32_a_tmem(tmem_d, ta + kk * 8, desc_at(b_hi, off), idesc2, (kb | kk) ? 1u : 0u);
          warp_mma_tf32_a_tmem(tmem_d + (uint32_t)BN, ta + (uint32_t)(BK + kk * 8), desc_at(b_hi, off), idesc1, 1u);
        }
        warp_mma_commit(&b_empty[s]);          // the stage may be refilled once these MMAs have read it
        warp_mma_commit(&slot_empty[slot]);
      }
      warp_mma_commit(&acc_full[buf]);
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ split raw tiles into hi / lo
    // thread = row of the tile = its TMEM lane; 16-byte chunk j of row r sits at chunk position j ^ (r & 7)
    const int row = (warp & 3) * 32 + lane;
    int it = 0;
    for (long long tile = blockIdx.x; tile < n_tiles_total; tile += gridDim.x) {
      const Tile tl = decode_tile(tab, item_g, tile, m_tiles, n_tiles, kb_per_seg, BN);
      for (int kb = 0; kb < tl.n_kb; ++kb, ++it) {
        const int s = it % A_STAGES, slot = it % SLOTS;
        mbar_wait(&a_full[s], (it / A_STAGES) & 1u, status);
        const unsigned char* st = smem + (size_t)s * C_::A_BYTES;
        uint32_t hi[32], lo[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(st + row * 128 + ((j ^ (row & 7)) << 4));
          const float part[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float h, l;
            split_tf32(part[c], h, l);
            hi[4 * j + c] = __float_as_uint(h);
            lo[4 * j + c] = __float_as_uint(l);
          }
        }
        fence_async_smem();                 // these reads precede the TMA write that refills the stage
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_empty[s]);
        mbar_wait(&slot_empty[slot], ((it / SLOTS) & 1u) ^ 1u, status);
        const uint32_t ta = tmem_a + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(slot * 2 * BK);
        tc_fence_after();
        tmem_st_32_begin(ta, hi);
        tmem_st_32(ta + (uint32_t)BK, lo);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_split[slot]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 6..9)
    // TMEM lane = tile row; warp w may touch lanes 32 * (w % 4) .. + 31
    const int quarter = warp & 3;
    // registers -> swizzled staging slab of this warp -> one 32 x 32 TMA store per column chunk
    unsigned char* slab = store_base + (size_t)quarter * 2 * 4096;
    uint32_t lt = 0;
    int chunk_no = 0;
    for (long long tile = blockIdx.x; tile < n_tiles_total; tile += gridDim.x, ++lt) {
      const Tile tl = decode_tile(tab, item_g, tile, m_tiles, n_tiles, kb_per_seg, BN);
      const uint32_t buf = lt % ACC;
      mbar_wait(&acc_full[buf], (lt / ACC) & 1u, status);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int c_row = tab.group_c_row[tl.g] + tl.t;
      float sum[BN];
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32], q[32];
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * (uint32_t)(2 * BN) + (uint32_t)(c * 32);
        tmem_ld_32(taddr, r);                      // hi x hi
        tmem_ld_32(taddr + (uint32_t)BN, q);       // hi x lo + lo x hi
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[c * 32 + j] = __uint_as_float(r[j]) + __uint_as_float(q[j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
#pragma unroll
      for (int c = 0; c < BN / 32; ++c, ++chunk_no) {
        unsigned char* sl = slab + (size_t)(chunk_no & 1) * 4096;
        if (lane == 0) bulk_wait_read<1>();     // the slab used two chunks ago has been read by its store
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          *reinterpret_cast<float4*>(sl + lane * 128 + ((j ^ (lane & 7)) << 4)) =
              make_float4(sum[c * 32 + 4 * j], sum[c * 32 + 4 * j + 1], sum[c * 32 + 4 * j + 2], sum[c * 32 + 4 * j + 3]);
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int col0 = tl.n0 + c * 32;
          const long long row0 = tl.m0 + quarter * 32;
          if (col0 < N && row0 < M) {
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
                         ::"l"(&tmC), "r"(col0), "r"(c_row), "r"((int)row0), "r"(smem_u32(sl)) : "memory");
          }
          bulk_commit();
        }
      }
    }
    if (lane == 0) bulk_wait_read<0>();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------
// Long, narrow plain product (N <= 64: the gradient of the wide radial layer's input, [E, weight_numel] to 64): two 128-row tiles of A to a
// CTA.  With one tile the four stages of the grouped kernel cover 64 KB of A while a load takes 1.7 us to arrive, and as many bytes of
// weights (hi and lo, 16 KB per k-block) as of A come through L2.  Two tiles share a weight k-block and have 128 KB of A in flight.
// Tensor memory: tile t accumulates in columns 128 t (hi x hi) and 128 t + 64 (cross terms), single-buffered; the split A in two slots of
// [tile][hi 32 | lo 32] from column 256.
//   warp 0: TMA producer   warp 1: MMA issue   warps 2-5, 6-9: split of tile 0, 1   warps 10-13: accumulator read-back and TMA stores
// Items are pairs of tiles as long as there are whole rounds of them for all SMs, then single tiles.  The sums are those of the grouped
// kernel.  Measured at 64 columns, grouped kernel -> this one: [320,000, 1280] 408 -> 320 us (5.1 TB/s), [320,000, 1920] 566 -> 477,
// [534,914, 512] 267 -> 223, [40,000, 256] 32.7 -> 15.2.
constexpr int LK_BN = 64, LK_STAGES = 4, LK_SLOTS = 2, NT_LK = 448;
struct LkCfg {
  static constexpr int A_BYTES = BM * BK * 4, B_BYTES = LK_BN * BK * 4;
  static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;      // A tiles 0 and 1, B hi and lo
  static constexpr int STORE_BYTES = 4 * 2 * 4096;
  static constexpr int SMEM_BYTES = LK_STAGES * STAGE_BYTES + STORE_BYTES + 1024 + 1024;
  static constexpr uint32_t TMEM_A = 256, SLOT_COLS = 128;
};

__global__ void __launch_bounds__(NT_LK, 1)
gemm_tf32x3_longk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBhi,
                         const __grid_constant__ CUtensorMap tmBlo, const __grid_constant__ CUtensorMap tmC, long long M, int N, int n_kb,
                         int n_pairs, int n_items, int* status) {
  using C_ = LkCfg;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* store_base = smem + LK_STAGES * C_::STAGE_BYTES;
  uint64_t* full_raw = reinterpret_cast<uint64_t*>(store_base + C_::STORE_BYTES);   // [STAGES] TMA landed
  uint64_t* empty = full_raw + LK_STAGES;        // [STAGES] the MMAs have read B (and the split warps A before them)
  uint64_t* full_split = empty + LK_STAGES;      // [SLOTS] both tiles' parts are in tensor memory
  uint64_t* slot_empty = full_split + LK_SLOTS;  // [SLOTS] the MMAs have read them
  uint64_t* acc_full = slot_empty + LK_SLOTS;    // 1
  uint64_t* acc_empty = acc_full + 1;            // [2 tiles]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < LK_STAGES; ++s) { mbar_init(&full_raw[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < LK_SLOTS; ++s) { mbar_init(&full_split[s], 8); mbar_init(&slot_empty[s], 1); }
    mbar_init(acc_full, 1);
    for (int t = 0; t < 2; ++t) mbar_init(&acc_empty[t], 4);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  wait_for_previous_kernel();
  const uint32_t tmem = *tmem_slot;
  // item -> first tile and number of tiles
  auto first_tile = [&](int item) { return item < n_pairs ? 2 * item : n_pairs + item; };
  auto tiles_of = [&](int item) { return item < n_pairs ? 2 : 1; };

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int tile = first_tile(item), nt = tiles_of(item), start = tile % n_kb;    // staggered: not all CTAs ask for the same weights at once
        for (int kbi = 0; kbi < n_kb; ++kbi, ++it) {
          const int kb = kbi + start < n_kb ? kbi + start : kbi + start - n_kb, s = it % LK_STAGES;
          mbar_wait(&empty[s], ((it / LK_STAGES) & 1u) ^ 1u, status);
          unsigned char* st = smem + (size_t)s * C_::STAGE_BYTES;
          mbar_arrive_expect_tx(&full_raw[s], (uint32_t)(nt * C_::A_BYTES + 2 * C_::B_BYTES));
          for (int t = 0; t < nt; ++t) tma_load_3d(st + t * C_::A_BYTES, &tmA, kb * BK, 0, (tile + t) * BM, &full_raw[s]);
          tma_load_3d(st + 2 * C_::A_BYTES, &tmBhi, kb * BK, 0, 0, &full_raw[s]);
          tma_load_3d(st + 2 * C_::A_BYTES + C_::B_BYTES, &tmBlo, kb * BK, 0, 0, &full_raw[s]);
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc2 = idesc_tf32_m128(2 * LK_BN), idesc1 = idesc_tf32_m128(LK_BN), tm = uniform(tmem);
    const uint64_t desc0 = make_desc(uniform(smem_u32(smem)) + 2 * C_::A_BYTES);
    int it = 0;
    uint32_t n = 0;                              // items done
    for (int item = blockIdx.x; item < n_items; item += gridDim.x, ++n) {
      const bool two = tiles_of(item) == 2;
      mbar_wait(&acc_empty[0], (n & 1u) ^ 1u, status);      // the accumulators have been read back
      mbar_wait(&acc_empty[1], (n & 1u) ^ 1u, status);
      for (int kb = 0; kb < n_kb; ++kb, ++it) {
        const int s = it % LK_STAGES, slot = it % LK_SLOTS;
        mbar_wait(&full_split[slot], (it / LK_SLOTS) & 1u, status);
        __syncwarp();
        tc_fence_after();
        const uint64_t b = desc_at(desc0, (uint32_t)(s * C_::STAGE_BYTES));
        const uint32_t ta = tm + C_::TMEM_A + (uint32_t)(slot * C_::SLOT_COLS);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (t == 1 && !two) break;
#pragma unroll
          for (int kk = 0; kk < BK / 8; ++kk) {
            warp_mma_tf32_a_tmem(tm + t * 2 * LK_BN, ta + (uint32_t)(t * 2 * BK + kk * 8), desc_at(b, kk * 32), idesc2, (kb | kk) ? 1u : 0u);
            warp_mma_tf32_a_tmem(tm + t * 2 * LK_BN + LK_BN, ta + (uint32_t)(t * 2 * BK + BK + kk * 8), desc_at(b, kk * 32), idesc1, 1u);
          }
        }
        warp_mma_commit(&empty[s]);
        warp_mma_commit(&slot_empty[slot]);
      }
      warp_mma_commit(acc_full);
    }
  } else if (warp < 10) {
    // thread = row of the tile = its TMEM lane; 16-byte chunk j of row r sits at chunk position j ^ (r & 7)
    const int t = (warp - 2) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    int it = 0;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      const bool live = t < tiles_of(item);
      for (int kb = 0; kb < n_kb; ++kb, ++it) {
        const int s = it % LK_STAGES, slot = it % LK_SLOTS;
        mbar_wait(&slot_empty[slot], ((it / LK_SLOTS) & 1u) ^ 1u, status);
        if (live) {
          mbar_wait(&full_raw[s], (it / LK_STAGES) & 1u, status);
          tc_fence_after();
          const unsigned char* a = smem + (size_t)s * C_::STAGE_BYTES + t * C_::A_BYTES + row * 128;
          uint32_t hi_bits[32], lo_bits[32];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(a + ((j ^ (row & 7)) << 4));
            float4 h, l;
            split_tf32(v.x, h.x, l.x); split_tf32(v.y, h.y, l.y); split_tf32(v.z, h.z, l.z); split_tf32(v.w, h.w, l.w);
            hi_bits[4 * j] = __float_as_uint(h.x); hi_bits[4 * j + 1] = __float_as_uint(h.y);
            hi_bits[4 * j + 2] = __float_as_uint(h.z); hi_bits[4 * j + 3] = __float_as_uint(h.w);
            lo_bits[4 * j] = __float_as_uint(l.x); lo_bits[4 * j + 1] = __float_as_uint(l.y);
            lo_bits[4 * j + 2] = __float_as_uint(l.z); lo_bits[4 * j + 3] = __float_as_uint(l.w);
          }
          const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + C_::TMEM_A + (uint32_t)(slot * C_::SLOT_COLS + t * 2 * BK);
          tmem_st_32(ta, hi_bits);
          tmem_st_32(ta + (uint32_t)BK, lo_bits);
          tc_fence_before();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_split[slot]);
      }
    }
  } else {
    const int quarter = warp & 3;
    unsigned char* slab = store_base + (size_t)quarter * 2 * 4096;
    uint32_t n = 0;
    int chunk_no = 0;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x, ++n) {
      mbar_wait(acc_full, n & 1u, status);
      tc_fence_after();
      for (int t = 0; t < 2; ++t) {
        if (t < tiles_of(item)) {
          const long long row0 = (long long)(first_tile(item) + t) * BM + quarter * 32;
#pragma unroll 1
          for (int c = 0; c < LK_BN / 32; ++c, ++chunk_no) {
            uint32_t r[32], q[32];
            const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(t * 2 * LK_BN + c * 32);
            tmem_ld_32(taddr, r);                      // hi x hi
            tmem_ld_32(taddr + (uint32_t)LK_BN, q);    // hi x lo + lo x hi
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(q[j]));
            unsigned char* sl = slab + (size_t)(chunk_no & 1) * 4096;
            if (lane == 0) bulk_wait_read<1>();        // the slab used two chunks ago has been read by its store
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(sl + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                  make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (c * 32 < N && row0 < M)
                asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
                             ::"l"(&tmC), "r"(c * 32), "r"(0), "r"((int)row0), "r"(smem_u32(sl)) : "memory");
              bulk_commit();
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[t]);     // (a tile the item does not have counts as read)
      }
    }
    if (lane == 0) bulk_wait_read<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------------------------------------------------------
// "A-stationary" variant for a shallow, wide layer (K <= 128, many N tiles: the last layer of the radial
// MLP, 64 -> weight_numel).  One CTA owns a 128-row block of A, loads and splits it once, then walks
// all N tiles: pre-split weight tiles (hi / lo arrays prepared once per call) stream through a ring,
// two TMEM accumulators alternate so that the MMAs of tile n+1 overlap the stores of tile n.
constexpr int AS_BN = 128, AS_RING = 4, AS_MAX_KB = 4;

template <int KB>
struct AsCfg {
  static constexpr int A_BYTES = BM * BK * 4;
  static constexpr int B_BYTES = AS_BN * BK * 4;
  static constexpr int RING = (KB <= 2) ? AS_RING : 2;
  static constexpr int STORE_BYTES = 4 * 2 * 4096;    // per epilogue warp: two 32 x 32 FP32 slabs for the TMA stores
  static constexpr int SMEM_BYTES = KB * 2 * A_BYTES + RING * 2 * B_BYTES + STORE_BYTES + 1024 + 1024;
};

template <int KB>
__global__ void __launch_bounds__(NT, 1)
gemm_tf32x3_as_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBhi,
                      const __grid_constant__ CUtensorMap tmBlo, const __grid_constant__ CUtensorMap tmC, long long M, int N, int K,
                      int* status) {
  using C_ = AsCfg<KB>;
  constexpr int RING = C_::RING;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* a_base = smem;                                   // [KB][hi 16 KB | lo 16 KB]
  unsigned char* b_base = smem + KB * 2 * C_::A_BYTES;            // [RING][hi 16 KB | lo 16 KB]
  unsigned char* store_base = b_base + RING * 2 * C_::B_BYTES;    // [4 warps][2 slabs][32 rows x 128 B], 1024-aligned
  uint64_t* bars = reinterpret_cast<uint64_t*>(store_base + C_::STORE_BYTES);
  uint64_t* a_full = bars;            // 1
  uint64_t* a_split = bars + 1;       // 4 warps
  uint64_t* b_full = bars + 2;        // [RING]
  uint64_t* b_empty = b_full + RING;  // [RING]
  uint64_t* acc_full = b_empty + RING;   // [2]
  uint64_t* acc_empty = acc_full + 2;    // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long m0 = (long long)blockIdx.x * BM;
  const int n_tiles = (N + AS_BN - 1) / AS_BN;
  const int n_kb = (K + BK - 1) / BK;            // <= KB

  if (threadIdx.x == 0) {
    mbar_init(a_full, 1); mbar_init(a_split, 4);
    for (int s = 0; s < RING; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(a_full, (uint32_t)(n_kb * C_::A_BYTES));
      for (int kb = 0; kb < n_kb; ++kb) tma_load_3d(a_base + (size_t)kb * 2 * C_::A_BYTES, &tmA, kb * BK, 0, (int)m0, a_full);
      int it = 0;
      for (int nt = 0; nt < n_tiles; ++nt) {
        for (int kb = 0; kb < n_kb; ++kb, ++it) {
          const int s = it % RING;
          mbar_wait(&b_empty[s], ((it / RING) & 1u) ^ 1u, status);
          unsigned char* st = b_base + (size_t)s * 2 * C_::B_BYTES;
          mbar_arrive_expect_tx(&b_full[s], (uint32_t)(2 * C_::B_BYTES));
          tma_load_3d(st, &tmBhi, kb * BK, nt * AS_BN, 0, &b_full[s]);
          tma_load_3d(st + C_::B_BYTES, &tmBlo, kb * BK, nt * AS_BN, 0, &b_full[s]);
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = idesc_tf32_m128(AS_BN), tm = uniform(tmem_base);
    const uint64_t a0 = make_desc(uniform(smem_u32(a_base))), b0 = make_desc(uniform(smem_u32(b_base)));
    mbar_wait(a_split, 0u, status);
    tc_fence_after();
    int it = 0;
    for (int nt = 0; nt < n_tiles; ++nt) {
      const int buf = nt & 1;
      mbar_wait(&acc_empty[buf], (((uint32_t)nt >> 1) & 1u) ^ 1u, status);
      tc_fence_after();
      const uint32_t tmem_d = tm + (uint32_t)(buf * AS_BN);
      for (int kb = 0; kb < n_kb; ++kb, ++it) {
        const int s = it % RING;
        mbar_wait(&b_full[s], (it / RING) & 1u, status);
        __syncwarp();
        tc_fence_after();
        const uint64_t a_hi = desc_at(a0, (uint32_t)(kb * 2 * C_::A_BYTES)), a_lo = desc_at(a_hi, C_::A_BYTES);
        const uint64_t b_hi = desc_at(b0, (uint32_t)(s * 2 * C_::B_BYTES)), b_lo = desc_at(b_hi, C_::B_BYTES);
#pragma unroll
        for (int kk = 0; kk < BK / 8; ++kk) {
          const uint32_t off = kk * 32;
          warp_mma_tf32(tmem_d, desc_at(a_lo, off), desc_at(b_hi, off), idesc, (kb | kk) ? 1u : 0u);
          warp_mma_tf32(tmem_d, desc_at(a_hi, off), desc_at(b_lo, off), idesc, 1u);
          warp_mma_tf32(tmem_d, desc_at(a_hi, off), desc_at(b_hi, off), idesc, 1u);
        }
        warp_mma_commit(&b_empty[s]);
      }
      warp_mma_commit(&acc_full[buf]);
    }
  } else {
    const int tid = threadIdx.x - 64;
    mbar_wait(a_full, 0u, status);
    for (int kb = 0; kb < n_kb; ++kb) {
      float4* hi = reinterpret_cast<float4*>(a_base + (size_t)kb * 2 * C_::A_BYTES);
      float4* lo = reinterpret_cast<float4*>(a_base + (size_t)kb * 2 * C_::A_BYTES + C_::A_BYTES);
#pragma unroll
      for (int i = 0; i < C_::A_BYTES / 16 / 128; ++i) {
        const float4 v = hi[tid + i * 128];
        float4 h, l;
        h.x = __uint_as_float(__float_as_uint(v.x) & 0xffffe000u); l.x = v.x - h.x;
        h.y = __uint_as_float(__float_as_uint(v.y) & 0xffffe000u); l.y = v.y - h.y;
        h.z = __uint_as_float(__float_as_uint(v.z) & 0xffffe000u); l.z = v.z - h.z;
        h.w = __uint_as_float(__float_as_uint(v.w) & 0xffffe000u); l.w = v.w - h.w;
        hi[tid + i * 128] = h; lo[tid + i * 128] = l;
      }
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(a_split);
    const int quarter = warp & 3;
    // this warp's 32 rows leave through its own pair of staging slabs: registers -> swizzled shared
    // memory -> one 32 x 32 TMA store per column chunk (full 128-byte lines, clipped at the edges of C)
    unsigned char* slab = store_base + (size_t)quarter * 2 * 4096;
    int chunk_no = 0;
    for (int nt = 0; nt < n_tiles; ++nt) {
      const int buf = nt & 1;
      mbar_wait(&acc_full[buf], ((uint32_t)nt >> 1) & 1u, status);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int c = 0; c < AS_BN / 32; ++c, ++chunk_no) {
        uint32_t r[32];
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * AS_BN + c * 32);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
              "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
              "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        unsigned char* sl = slab + (size_t)(chunk_no & 1) * 4096;
        // the slab used two chunks ago must have been read by its store
        if (lane == 0) bulk_wait_read<1>();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          // SWIZZLE_128B: 16-byte chunk j of row `lane` sits at chunk position j ^ (lane & 7)
          *reinterpret_cast<float4*>(sl + lane * 128 + ((j ^ (lane & 7)) << 4)) =
              make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int col0 = nt * AS_BN + c * 32;
          const long long row0 = m0 + quarter * 32;
          if (col0 < N && row0 < M) {
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
                         ::"l"(&tmC), "r"(col0), "r"((int)row0), "r"(0), "r"(smem_u32(sl)) : "memory");
          }
          bulk_commit();
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
    if (lane == 0) bulk_wait_read<0>();   // the staging slabs must outlive their stores
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(256u) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------
// Persistent form of the A-stationary kernel for K <= 64: one CTA per SM walks row blocks round-robin, and the
// A block lives in TENSOR MEMORY.  Shared-memory bandwidth is the busiest resource of this shape (every
// 128 x 128 x 8 TF32 MMA with both operands in shared memory reads 8 KB), so four warps split each raw A block
// (thread = row = TMEM lane) into hi / lo and write both with tcgen05.st; the MMAs then take A from tensor memory
// and only the weight tile from shared memory.  A is double buffered (raw tile in shared memory and hi / lo in
// tensor memory) and the two accumulators alternate across block boundaries, so the load / split prologue and
// the store tail of a block hide behind its neighbours' MMAs.
//   warp 0: TMA producer (A blocks, weight tiles)   warp 1: tcgen05.mma issue   warps 2-5: hi / lo split of A
//   warps 6-9: accumulator read-back and TMA stores
// Tensor memory (512 columns): accumulators [0, 256); A buffer b at 256 + 128 b: hi [0, 64), lo [64, 128).
// Writing the accumulator rows straight from registers (32-byte st.global per thread) instead of staging them
// for TMA stores was measured slower: row-scattered sectors cost more than the staging.
constexpr int NT_ASP = 320;

struct AspCfg {
  static constexpr int KB = 2;
  static constexpr int A_BYTES = BM * BK * 4;
  static constexpr int A_BUF = KB * A_BYTES;             // raw FP32 block, [KB][16 KB]
  static constexpr int B_BYTES = AS_BN * BK * 4;
  static constexpr int RING = 4;
  static constexpr int STORE_BYTES = 4 * 2 * 4096;
  static constexpr int SMEM_BYTES = 2 * A_BUF + RING * 2 * B_BYTES + STORE_BYTES + 1024 + 1024;
  static constexpr uint32_t TMEM_COLS = 512, TMEM_A0 = 256, TMEM_A_STRIDE = 128, TMEM_A_LO = 64;
};

__global__ void __launch_bounds__(NT_ASP, 1)
gemm_tf32x3_asp_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBhi,
                       const __grid_constant__ CUtensorMap tmBlo, const __grid_constant__ CUtensorMap tmC, long long M, int N, int K,
                       int m_blocks, int col_shares, int* status) {
  using C_ = AspCfg;
  constexpr int RING = C_::RING;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* a_base = smem;                                   // [2 buffers][KB][raw 16 KB]
  unsigned char* b_base = smem + 2 * C_::A_BUF;                   // [RING][hi 16 KB | lo 16 KB]
  unsigned char* store_base = b_base + RING * 2 * C_::B_BYTES;    // [4 warps][2 slabs][32 rows x 128 B]
  uint64_t* bars = reinterpret_cast<uint64_t*>(store_base + C_::STORE_BYTES);
  uint64_t* a_full = bars;              // [2] raw A block landed
  uint64_t* a_split = bars + 2;         // [2] hi / lo are in tensor memory (four split warps)
  uint64_t* a_raw_empty = bars + 4;     // [2] the split warps have read the raw block
  uint64_t* a_tmem_empty = bars + 6;    // [2] the MMAs of the block have completed
  uint64_t* b_full = bars + 8;          // [RING]
  uint64_t* b_empty = b_full + RING;    // [RING]
  uint64_t* acc_full = b_empty + RING;  // [2]
  uint64_t* acc_empty = acc_full + 2;   // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // an item is a row block, or where there are few of those a share of its weight tiles
  const int all_tiles = (N + AS_BN - 1) / AS_BN, n_items = m_blocks * col_shares;
  const int n_kb = (K + BK - 1) / BK;            // <= KB
  const int first = (int)blockIdx.x, stride = (int)gridDim.x;
  struct Item { int blk, nt0, n_tiles; };
  auto item_of = [&](int item) {
    if (col_shares == 1) return Item{item, 0, all_tiles};
    const int blk = item / col_shares, share = item - blk * col_shares, nt0 = all_tiles * share / col_shares;
    return Item{blk, nt0, all_tiles * (share + 1) / col_shares - nt0};
  };

  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&a_full[b], 1); mbar_init(&a_split[b], 4); mbar_init(&a_raw_empty[b], 4); mbar_init(&a_tmem_empty[b], 1);
      mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4);
    }
    for (int s = 0; s < RING; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, C_::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  wait_for_previous_kernel();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      auto load_a = [&](int j, int blk) {
        const int buf = j & 1;
        mbar_wait(&a_raw_empty[buf], (((uint32_t)j >> 1) & 1u) ^ 1u, status);
        unsigned char* dst = a_base + (size_t)buf * C_::A_BUF;
        mbar_arrive_expect_tx(&a_full[buf], (uint32_t)(n_kb * C_::A_BYTES));
        for (int kb = 0; kb < n_kb; ++kb) tma_load_3d(dst + (size_t)kb * C_::A_BYTES, &tmA, kb * BK, 0, blk * BM, &a_full[buf]);
      };
      if (first < n_items) load_a(0, item_of(first).blk);
      int it = 0;
      for (int j = 0, item = first; item < n_items; ++j, item += stride) {
        const Item im = item_of(item);
        bool next_pending = item + stride < n_items;
        int local = 0;
        for (int nti = 0; nti < im.n_tiles; ++nti) {
          const int nt = im.nt0 + (nti + im.blk) % im.n_tiles;     // staggered walk over the weight tiles (see the epilogue)
          for (int kb = 0; kb < n_kb; ++kb, ++it, ++local) {
            // the next A block is requested once this block's first weight tiles are on their way
            if (next_pending && local == 2) { load_a(j + 1, item_of(item + stride).blk); next_pending = false; }
            const int s = it % RING;
            mbar_wait(&b_empty[s], ((it / RING) & 1u) ^ 1u, status);
            unsigned char* st = b_base + (size_t)s * 2 * C_::B_BYTES;
            mbar_arrive_expect_tx(&b_full[s], (uint32_t)(2 * C_::B_BYTES));
            tma_load_3d(st, &tmBhi, kb * BK, nt * AS_BN, 0, &b_full[s]);
            tma_load_3d(st + C_::B_BYTES, &tmBlo, kb * BK, nt * AS_BN, 0, &b_full[s]);
          }
        }
        if (next_pending) load_a(j + 1, item_of(item + stride).blk);
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = idesc_tf32_m128(AS_BN), tm = uniform(tmem_base);
    const uint64_t desc0 = make_desc(uniform(smem_u32(b_base)));
    int it = 0;
    uint32_t t = 0;
    for (int j = 0, item = first; item < n_items; ++j, item += stride) {
      const int abuf = j & 1, n_tiles = item_of(item).n_tiles;
      mbar_wait(&a_split[abuf], ((uint32_t)j >> 1) & 1u, status);
      tc_fence_after();
      const uint32_t a_hi0 = tm + C_::TMEM_A0 + (uint32_t)abuf * C_::TMEM_A_STRIDE, a_lo0 = a_hi0 + C_::TMEM_A_LO;
      for (int nt = 0; nt < n_tiles; ++nt, ++t) {
        const uint32_t buf = t & 1u;
        mbar_wait(&acc_empty[buf], ((t >> 1) & 1u) ^ 1u, status);
        tc_fence_after();
        const uint32_t tmem_d = tm + buf * AS_BN;
        for (int kb = 0; kb < n_kb; ++kb, ++it) {
          const int s = it % RING;
          mbar_wait(&b_full[s], (it / RING) & 1u, status);
          __syncwarp();
          tc_fence_after();
          const uint64_t b_hi = desc_at(desc0, (uint32_t)(s * 2 * C_::B_BYTES)), b_lo = desc_at(b_hi, C_::B_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / 8; ++kk) {
            const uint32_t off = kk * 32, col = (uint32_t)(kb * BK + kk * 8);
            warp_mma_tf32_a_tmem(tmem_d, a_lo0 + col, desc_at(b_hi, off), idesc, (kb | kk) ? 1u : 0u);
            warp_mma_tf32_a_tmem(tmem_d, a_hi0 + col, desc_at(b_lo, off), idesc, 1u);
            warp_mma_tf32_a_tmem(tmem_d, a_hi0 + col, desc_at(b_hi, off), idesc, 1u);
          }
          warp_mma_commit(&b_empty[s]);
        }
        warp_mma_commit(&acc_full[buf]);
      }
      warp_mma_commit(&a_tmem_empty[abuf]);
    }
  } else if (warp < 6) {
    // thread = row of the block = its TMEM lane; 16-byte chunk q of row r sits at chunk position q ^ (r & 7)
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    for (int j = 0, item = first; item < n_items; ++j, item += stride) {
      const int abuf = j & 1;
      mbar_wait(&a_full[abuf], ((uint32_t)j >> 1) & 1u, status);
      mbar_wait(&a_tmem_empty[abuf], (((uint32_t)j >> 1) & 1u) ^ 1u, status);
      tc_fence_after();
      const uint32_t t_hi = tmem_base + ((uint32_t)(quarter * 32) << 16) + C_::TMEM_A0 + (uint32_t)abuf * C_::TMEM_A_STRIDE;
      for (int kb = 0; kb < n_kb; ++kb) {
        const unsigned char* tile = a_base + (size_t)abuf * C_::A_BUF + (size_t)kb * C_::A_BYTES;
        uint32_t hi_bits[32], lo_bits[32];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 v = *reinterpret_cast<const float4*>(tile + row * 128 + ((q ^ (row & 7)) << 4));
          float4 h, l;
          split_tf32(v.x, h.x, l.x); split_tf32(v.y, h.y, l.y); split_tf32(v.z, h.z, l.z); split_tf32(v.w, h.w, l.w);
          hi_bits[4 * q] = __float_as_uint(h.x); hi_bits[4 * q + 1] = __float_as_uint(h.y);
          hi_bits[4 * q + 2] = __float_as_uint(h.z); hi_bits[4 * q + 3] = __float_as_uint(h.w);
          lo_bits[4 * q] = __float_as_uint(l.x); lo_bits[4 * q + 1] = __float_as_uint(l.y);
          lo_bits[4 * q + 2] = __float_as_uint(l.z); lo_bits[4 * q + 3] = __float_as_uint(l.w);
        }
        tmem_st_32(t_hi + (uint32_t)(kb * BK), hi_bits);
        tmem_st_32(t_hi + C_::TMEM_A_LO + (uint32_t)(kb * BK), lo_bits);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(&a_split[abuf]); mbar_arrive(&a_raw_empty[abuf]); }
    }
  } else {
    const int quarter = warp & 3;
    unsigned char* slab = store_base + (size_t)quarter * 2 * 4096;
    int chunk_no = 0;
    uint32_t t = 0;
    for (int item = first; item < n_items; item += stride) {
      const Item im = item_of(item);
      const long long row0 = (long long)im.blk * BM + quarter * 32;
      for (int nti = 0; nti < im.n_tiles; ++nti, ++t) {
        // row block b starts at weight tile b mod n_tiles: the CTAs do not all fetch the same weight lines from L2
        // at the same moment
        const int nt = im.nt0 + (nti + im.blk) % im.n_tiles;
        const uint32_t buf = t & 1u;
        mbar_wait(&acc_full[buf], (t >> 1) & 1u, status);
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < AS_BN / 32; ++c, ++chunk_no) {
          uint32_t r[32];
          tmem_ld_32(tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * AS_BN + (uint32_t)(c * 32), r);
          unsigned char* sl = slab + (size_t)(chunk_no & 1) * 4096;
          if (lane == 0) bulk_wait_read<1>();     // the slab used two chunks ago has been read by its store
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            // SWIZZLE_128B: 16-byte chunk q of row `lane` sits at chunk position q ^ (lane & 7)
            *reinterpret_cast<float4*>(sl + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int col0 = nt * AS_BN + c * 32;
            if (col0 < N && row0 < M) {
              asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
                           ::"l"(&tmC), "r"(col0), "r"((int)row0), "r"(0), "r"(smem_u32(sl)) : "memory");
            }
            bulk_commit();
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
    }
    if (lane == 0) bulk_wait_read<0>();   // the staging slabs must outlive their stores
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C_::TMEM_COLS);
  }
}

__global__ void split_weights_kernel(const float* __restrict__ w, float* __restrict__ hi, float* __restrict__ lo, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = w[i];
    const float h = __uint_as_float(__float_as_uint(v) & 0xffffe000u);
    hi[i] = h; lo[i] = v - h;
  }
}

// --------------------------------------------------------------------------------- host side
__device__ int g_tc_status;

static PFN_cuTensorMapEncodeTiled get_encode() {
  static PFN_cuTensorMapEncodeTiled fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(p);
  }
  return fn;
}

static int encode_map(CUtensorMap* m, const float* base, const cuuint64_t (&dims)[3], const cuuint64_t (&strides)[2], const cuuint32_t (&box)[3],
                      CUtensorMapSwizzle swizzle) {
  PFN_cuTensorMapEncodeTiled enc = get_encode();
  if (!enc) return FASTEQ_INTERNAL;
  const cuuint32_t es[3] = {1, 1, 1};
  auto encode = [&] {
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // a thread whose first CUDA work this is (autograd's, with all its memory from the cache) has a device but no context yet:
    // setting the device binds it, also while a stream is captured
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaSetDevice(dev);
    if (e != cudaSuccess) return cuda_fail(e);
    r = encode();
  }
  if (r != CUDA_SUCCESS) {
    snprintf(g_cuda_err, sizeof(g_cuda_err), "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return FASTEQ_CUDA_ERROR;
  }
  return FASTEQ_OK;
}

// 3-D FP32 tensor [d2][d1][d0] (d0 contiguous), box [b2][b1][b0], 128-byte swizzle, zero fill outside
int make_map(CUtensorMap* m, const float* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t stride1_elems,
                    uint64_t stride2_elems, uint32_t b0, uint32_t b1, uint32_t b2) {
  return encode_map(m, base, {d0, d1, d2}, {stride1_elems * 4, stride2_elems * 4}, {b0, b1, b2}, CU_TENSOR_MAP_SWIZZLE_128B);
}

int make_map_rows(CUtensorMap* m, const float* base, int width, int rows, long long batch, int box_width, int box_batch) {
  return encode_map(m, base, {(cuuint64_t)width, (cuuint64_t)rows, (cuuint64_t)batch}, {(cuuint64_t)width * 4, (cuuint64_t)rows * width * 4},
                    {(cuuint32_t)box_width, 1u, (cuuint32_t)box_batch}, CU_TENSOR_MAP_SWIZZLE_NONE);
}

bool supported(long long M, int a_rows, int K, int P, int N, int c_rows, const void* A, const void* Bt, const void* C) {
  if (M < 1 || K < 4 || N < 4 || (K % 4) || (N % 4)) return false;                 // 16-byte global strides
  if (M > 0x7fffffffLL) return false;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(Bt) | reinterpret_cast<uintptr_t>(C)) & 15u) return false;
  if ((long long)a_rows * K > (1LL << 36) || (long long)N * K > (1LL << 36)) return false;
  return true;
}

static int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  return n;
}

template <int BN>
static int launch_bn(const TcTable& tab, const CUtensorMap& ma, const CUtensorMap& mbh, const CUtensorMap& mbl, const CUtensorMap& mc,
                     long long M, int N, int K, cudaStream_t s) {
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_tc_status);
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaFuncSetAttribute(gemm_tf32x3_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::SMEM_BYTES);
  if (e != cudaSuccess) return cuda_fail(e);
  const long long m_tiles = (M + BM - 1) / BM;
  const int n_tiles = (N + BN - 1) / BN;
  const long long total = m_tiles * n_tiles * tab.n_items;
  const int sms = sm_count();
  if (sms < 1) return FASTEQ_CUDA_ERROR;
  const unsigned grid = (unsigned)(total < sms ? total : sms);     // one persistent CTA per SM
  e = launch_dependent(gemm_tf32x3_kernel<BN>, grid, NT_P, Cfg<BN>::SMEM_BYTES, s, ma, mbh, mbl, mc, tab, M, N, K, total, total > 4LL * sms ? 0 : (int)m_tiles, n_tiles, st);
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// From here on two row tiles share the weights' k-blocks (see gemm_tf32x3_longk_kernel), and from 2 tiles to an SM on:
// fewer would leave SMs idle in pairs.  Measured from 256 columns up; below, an SM's tiles are mostly fill and drain either way.
constexpr int LONG_K = 256;

static int launch_long_k(const CUtensorMap& ma, const CUtensorMap& mbh, const CUtensorMap& mbl, const CUtensorMap& mc, long long M, int N, int K,
                         int sms, cudaStream_t s) {
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_tc_status);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_tf32x3_longk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LkCfg::SMEM_BYTES);
  if (e != cudaSuccess) return cuda_fail(e);
  const long long tiles = (M + BM - 1) / BM;
  const int n_pairs = (int)(tiles / (2 * sms) * sms), n_items = (int)(tiles - n_pairs);
  e = launch_dependent(gemm_tf32x3_longk_kernel, (unsigned)(n_items < sms ? n_items : sms), NT_LK, LkCfg::SMEM_BYTES, s, ma, mbh, mbl, mc, M, N,
                       (K + BK - 1) / BK, n_pairs, n_items, st);
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// Bt_hi / Bt_lo: the [P, N, K] weight blocks already split into their TF32 parts (split_weights / the
// SO3Linear packing kernel do it once per call; the blocks are tiny next to A)
int launch(const TcTable& tab, const float* A, long long M, int a_rows, int K, const float* Bt_hi, const float* Bt_lo, int P, int N,
           float* C, int c_rows, cudaStream_t s) {
  if (tab.n_items < 1 || tab.n_items > 65535) return FASTEQ_UNSUPPORTED;
  const int sms = sm_count();
  if (sms < 1) return FASTEQ_CUDA_ERROR;
  // 64-column tiles where they fit one wave: a tile's time is that of its k-blocks one after the other, and half a tile's are shorter
  // (half the weights, half the MMAs): the eleven launches of a one-cell MACE step at 192 nodes, with the carries beside the forward,
  // 362 -> 344 us for the step.
  const long long tiles64 = ((M + BM - 1) / BM) * ((N + 63) / 64) * tab.n_items;
  const int BN = N <= 64 || tiles64 <= sms ? 64 : 128;
  alignas(64) CUtensorMap ma, mbh, mbl, mc;
  int rc = make_map(&ma, A, (uint64_t)K, (uint64_t)a_rows, (uint64_t)M, (uint64_t)K, (uint64_t)a_rows * K, BK, 1, BM);
  if (rc != FASTEQ_OK) return rc;
  rc = make_map(&mbh, Bt_hi, (uint64_t)K, (uint64_t)N, (uint64_t)P, (uint64_t)K, (uint64_t)N * K, BK, (uint32_t)BN, 1);
  if (rc != FASTEQ_OK) return rc;
  rc = make_map(&mbl, Bt_lo, (uint64_t)K, (uint64_t)N, (uint64_t)P, (uint64_t)K, (uint64_t)N * K, BK, (uint32_t)BN, 1);
  if (rc != FASTEQ_OK) return rc;
  rc = make_map(&mc, C, (uint64_t)N, (uint64_t)c_rows, (uint64_t)M, (uint64_t)N, (uint64_t)c_rows * N, 32, 1, 32);
  if (rc != FASTEQ_OK) return rc;
  if (N <= 64 && a_rows == 1 && c_rows == 1 && P == 1 && K >= LONG_K && M >= 2LL * sms * BM) return launch_long_k(ma, mbh, mbl, mc, M, N, K, sms, s);
  return BN == 64 ? launch_bn<64>(tab, ma, mbh, mbl, mc, M, N, K, s) : launch_bn<128>(tab, ma, mbh, mbl, mc, M, N, K, s);
}

// hi / lo parts of n contiguous FP32 values into split[0 .. n) and split[n .. 2n)
int split_weights(const float* w, long long n, float* split, cudaStream_t s) {
  split_weights_kernel<<<(unsigned)((n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024), 256, 0, s>>>(w, split, split + n, n);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

template <int KB>
static int launch_as_kb(const CUtensorMap& ma, const CUtensorMap& mbh, const CUtensorMap& mbl, const CUtensorMap& mc, long long M, int N,
                        int K, cudaStream_t s) {
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_tc_status);
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaFuncSetAttribute(gemm_tf32x3_as_kernel<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, AsCfg<KB>::SMEM_BYTES);
  if (e != cudaSuccess) return cuda_fail(e);
  gemm_tf32x3_as_kernel<KB><<<(unsigned)((M + BM - 1) / BM), NT, AsCfg<KB>::SMEM_BYTES, s>>>(ma, mbh, mbl, mc, M, N, K, st);
  e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

static int launch_as_persistent(const CUtensorMap& ma, const CUtensorMap& mbh, const CUtensorMap& mbl, const CUtensorMap& mc, long long M,
                                int N, int K, cudaStream_t s) {
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_tc_status);
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaFuncSetAttribute(gemm_tf32x3_asp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AspCfg::SMEM_BYTES);
  if (e != cudaSuccess) return cuda_fail(e);
  const long long m_blocks = (M + BM - 1) / BM;
  const int sms = sm_count();
  if (sms < 1) return FASTEQ_CUDA_ERROR;
  // Few row blocks leave SMs idle, or one more block to some of them: then a block's weight tiles are shared out, as far as the longest
  // CTA (tiles, and about one for each share's block of A) gets shorter.  [10,000, 64] to 1280 columns, 79 blocks: 21.7 -> 15.1 us; 100 rows 18.7 -> 5.3,
  // 4,000 20.9 -> 9.0, 20,000 39.9 -> 29.9, 40,000 56.1 -> 46.4, 80,000 unchanged.
  const int n_tiles = (N + AS_BN - 1) / AS_BN;
  int col_shares = 1;
  auto longest = [&](long long shares) { return ((m_blocks * shares + sms - 1) / sms) * ((n_tiles + shares - 1) / shares + 1); };
  for (int c = 2; m_blocks <= 4LL * sms && c <= n_tiles; ++c) if (longest(c) < longest(col_shares)) col_shares = c;
  const long long items = m_blocks * col_shares;
  const unsigned grid = (unsigned)(items < sms ? items : sms);     // one persistent CTA per SM
  e = launch_dependent(gemm_tf32x3_asp_kernel, grid, NT_ASP, AspCfg::SMEM_BYTES, s, ma, mbh, mbl, mc, M, N, K, (int)m_blocks, col_shares, st);
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}

// plain C[M, N] = A[M, K] @ Bt[N, K]^T with K <= 128 and several N tiles
// `split`: hi / lo parts of Bt (2 * N * K floats)
int launch_a_stationary(const float* A, long long M, int K, const float* split, int N, float* C, cudaStream_t s) {
  const long long nw = (long long)N * K;
  alignas(64) CUtensorMap ma, mbh, mbl, mc;
  int rc = make_map(&ma, A, (uint64_t)K, 1, (uint64_t)M, (uint64_t)K, (uint64_t)K, BK, 1, BM);
  if (rc == FASTEQ_OK) rc = make_map(&mc, C, (uint64_t)N, (uint64_t)M, 1, (uint64_t)N, (uint64_t)N * M, 32, 32, 1);
  if (rc == FASTEQ_OK) rc = make_map(&mbh, split, (uint64_t)K, (uint64_t)N, 1, (uint64_t)K, (uint64_t)N * K, BK, AS_BN, 1);
  if (rc == FASTEQ_OK) rc = make_map(&mbl, split + nw, (uint64_t)K, (uint64_t)N, 1, (uint64_t)K, (uint64_t)N * K, BK, AS_BN, 1);
  if (rc == FASTEQ_OK) {
    const int kb = (K + BK - 1) / BK;
    rc = kb <= 2 ? launch_as_persistent(ma, mbh, mbl, mc, M, N, K, s) : launch_as_kb<4>(ma, mbh, mbl, mc, M, N, K, s);
  }
  return rc;
}

// C = A @ Bt^T with Bt given raw (split into a temporary) or already split
int dense(const float* A, const float* Bt, const float* split_in, float* C, long long M, int N, int K, cudaStream_t s) {
  if (M < 0 || N < 1 || K < 1) return FASTEQ_INVALID;
  if (M == 0) return FASTEQ_OK;
  if (!A || (!Bt && !split_in) || !C) return FASTEQ_INVALID;
  if (!supported(M, 1, K, 1, N, 1, A, split_in ? split_in : Bt, C)) return FASTEQ_UNSUPPORTED;
  const long long nw = (long long)N * K;
  float* tmp = nullptr;
  int rc = FASTEQ_OK;
  if (!split_in) {
    cudaError_t e = cudaMallocAsync((void**)&tmp, (size_t)nw * 2 * sizeof(float), s);
    if (e != cudaSuccess) return cuda_fail(e);
    rc = split_weights(Bt, nw, tmp, s);
  }
  const float* split = split_in ? split_in : tmp;
  if (rc == FASTEQ_OK) {
    if (K <= 128 && N >= 256) {
      rc = launch_a_stationary(A, M, K, split, N, C, s);
    } else {
      TcTable tab{};
      tab.n_groups = 1; tab.n_items = 1; tab.group_c_row[0] = 0; tab.group_first[0] = 0; tab.group_first[1] = 1;
      tab.item_first[0] = 0; tab.item_first[1] = 1; tab.path_a_row[0] = 0; tab.path_w[0] = 0;
      rc = launch(tab, A, M, 1, K, split, split + nw, 1, N, C, 1, s);
    }
  }
  if (tmp) cudaFreeAsync(tmp, s);
  return rc;
}

cudaError_t status_word(int** word) { return cudaGetSymbolAddress((void**)word, g_tc_status); }

int device_status(int* code) {
  int v = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int));
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int));
  if (e != cudaSuccess) return cuda_fail(e);
  *code = v;
  return FASTEQ_OK;
}

}  // namespace tc
}  // namespace fasteq

// C[M, N] = A[M, K] @ Bt[N, K]^T, FP32 data, 3xTF32 tensor-core arithmetic (a layer of the radial MLP:
// Bt is torch's [out_features, in_features] weight).  K and N multiples of 4, 16-byte aligned pointers.
extern "C" int fasteq_gemm_tf32x3(const void* A, const void* Bt, void* C, int64_t M, int32_t N, int32_t K,
                                  fasteq_stream_t stream) {
  return fasteq::tc::dense((const float*)A, (const float*)Bt, nullptr, (float*)C, M, N, K, (cudaStream_t)stream);
}

// The two TF32 parts of a weight matrix, prepared once for many fasteq_gemm_tf32x3_presplit calls.
extern "C" int fasteq_gemm_tf32x3_split(const void* Bt, int64_t n_elems, void* split, fasteq_stream_t stream) {
  if (n_elems < 0 || (n_elems > 0 && (!Bt || !split))) return FASTEQ_INVALID;
  if (n_elems == 0) return FASTEQ_OK;
  return fasteq::tc::split_weights((const float*)Bt, n_elems, (float*)split, (cudaStream_t)stream);
}

extern "C" int fasteq_gemm_tf32x3_presplit(const void* A, const void* split, void* C, int64_t M, int32_t N, int32_t K,
                                           fasteq_stream_t stream) {
  if (!split && M > 0) return FASTEQ_INVALID;
  return fasteq::tc::dense((const float*)A, nullptr, (const float*)split, (float*)C, M, N, K, (cudaStream_t)stream);
}

extern "C" int fasteq_tensorcore_device_status(int32_t* code) {
  if (!code) return FASTEQ_INVALID;
  int a = 0, b = 0;
  int rc = fasteq::tc::device_status(&a);
  if (rc != FASTEQ_OK) return rc;
  rc = fasteq::chain::device_status(&b);
  if (rc != FASTEQ_OK) return rc;
  *code = a ? a : b;
  return FASTEQ_OK;
}
