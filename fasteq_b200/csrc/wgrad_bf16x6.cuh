// FP32 weight gradient on the tensor cores: per path X^T G over batch * rows, FP32 operands as three bf16 parts each.
//
// v = v1 + v2 + v3 with every part the nearest bf16 of what is left is exact (8 + 8 + 8 significand bits), and
// v1 w1 + v1 w2 + v2 w1 + v2 w2 + v1 w3 + v3 w1 leaves out terms of 2^-27 v w: the products are better than FP32's.  What limits the
// accuracy is the tensor core's accumulation, which truncates: 2^-24 or so per K step, toward zero.  Hence chunks of 32 rows, two K
// steps at full magnitude (the small products go first), each added to registers with ordinary rounding, 16 chunks to a
// second-level sum in shared memory.  Two TF32 parts would need lo x lo and TF32 runs at half the rate: no cheaper, less exact.
// What the truncation costs on average, 0.75 x 2^-24 of a sum, the reduction multiplies back in, with the coefficient and in one rounding.
//
// One CTA of 18 warps per SM takes a share of one path's chunks, 32 batch
// entries of one irrep row each, and a 128 x TN tile:
//   warp 17     TMA loads of both operands' chunks, [32][channels], up to three ahead; entries and channels beyond the ends come as zeros
//   warps 0-3   M operand, thread = channel = TMEM lane: split, packed in pairs of rows, tcgen05.st
//   warps 4-7   N operand, thread = channel: the same into K-major bf16 tiles (64-byte swizzle), 16 bytes at a time
//   warp 16     issues the twelve 128 x TN x 16 MMAs of a chunk
//   warps 8-15  add finished chunks (two accumulators alternate) to their registers and store the tile
// so no operand needs a transpose pass: the contraction index is the row, which is the K axis of both register packings.
// Bound: the way of a chunk through split, MMA and drain: at TN = 128 and 12,288 nodes one of a chunk's twelve MMAs ends every 158 clocks, of which the
// tensor cores are busy for 66 and issue for half (ncu).  Measured
// with the reduction, against 8 x 8 register tiles on the FP32 pipe: the 128-channel SO3Linear after the tensor product at
// 12,288 nodes 365 -> 117 us, at 512 nodes 28 -> 22; [80000, 64]^T [80000, 1280] 309 -> 149; [80000, 128]^T [80000, 128] 65 -> 31; at
// 200 rows 18.6 -> 14.4.  Errors against FP64 (2-norm, 1e-8; FP32 chunks of 32 rows, this without the gain, this) at 160, 2,000
// and 100,003 rows of 128 x 128: normal operands 11.3, 7.3, 6.8; 12.8, 9.4, 9.1; 16.8, 13.7, 13.5; of one sign, where the losses do not cancel, 5.5, 6.6, 4.8;
// 5.4, 7.4, 7.4; 4.4, 6.8, 4.6 (where the gain is less than half a step of the result it rounds away).
// About 13 us are the launch, the first chunk's way through the roles and the reduction.
// Range: a third part reaches 24 bits below its operand, and bf16's smallest numbers are 2^-133.  Operands are therefore split 2^24 times as
// large, which holds every FP32 number in three parts and keeps every product's parts above FP32's smallest; the stored sums are scaled
// back.  Sums that are not finite then (an infinite or NaN operand, one above 2^104, sums above 2^80) the CTA recomputes in FP32.
#pragma once
#include "tcgen05_util.cuh"

namespace fasteq {
namespace wg {

constexpr int TM = 128, ROWS = 32, RAW = 3, STAGES = 2, THREADS = 18 * 32, OUTER = 16;
constexpr double GAIN = 1.0 + 4.5e-8;
constexpr float SCALE = 16777216.f, UNSCALE = 1.f / (SCALE * SCALE);
constexpr int A_COLS = 3 * ROWS / 2;                       // TMEM columns of one M-operand stage: three parts, two rows per column
__host__ __device__ constexpr int b_part(int tn) { return tn * ROWS * 2; }
__host__ __device__ constexpr int smem_bytes(int tn) { return 1024 + STAGES * 3 * b_part(tn) + RAW * ROWS * (TM + tn) * 4 + TM * tn * 4 + 256; }

// K-major bf16 tile with rows of 64 bytes, SWIZZLE_64B: 16-byte chunk j of row n at chunk position j ^ ((n >> 1) & 3)
__device__ __forceinline__ uint64_t desc_sw64(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;           // eight rows
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;                    // SWIZZLE_64B
  return d;
}
// D = F32, A = B = BF16, both K-major, M = 128
__device__ __forceinline__ uint32_t idesc_bf16_m128(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void tmem_st_8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// nearest bf16 of two values, `lo` in the low half
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ void split_pair(float2 v, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  const float2 minus = make_float2(-1.f, -1.f);
  v = vmul(v, make_float2(SCALE, SCALE));
  p1 = bf16_pair(v.x, v.y);
  v = vfma(make_float2(__uint_as_float(p1 << 16), __uint_as_float(p1 & 0xffff0000u)), minus, v);
  p2 = bf16_pair(v.x, v.y);
  v = vfma(make_float2(__uint_as_float(p2 << 16), __uint_as_float(p2 & 0xffff0000u)), minus, v);
  p3 = bf16_pair(v.x, v.y);
}
// 16 accumulator columns of this thread's lane, then wait
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace wg
}  // namespace fasteq
