// split_mma.cuh — f32 products on mma.sync for the recurrences of prompts (recurrence_chunked.cu, delta_chunked.cu): operands in three
// bf16 pieces, six products.  Why three pieces, and why hi.hi is summed apart, stands in recurrence_chunked.cu.
#pragma once

#include "recurrence.cuh"

namespace nvllm {
namespace split {

__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }

__device__ __forceinline__ bool far_off(uint32_t bits, int lo, int hi) {   // not zero and outside [2^lo, 2^hi)
  return bits != 0u && (bits < (static_cast<uint32_t>(127 + lo) << 23) || bits >= (static_cast<uint32_t>(127 + hi) << 23));
}
// (x0, x1) -> three bf16 pairs, hi + mid + lo = x to 2^-25 of it
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(x0, x1);
  x0 -= bf16_lo(hi);
  x1 -= bf16_hi(hi);
  mid = pack_bf16x2(x0, x1);
  lo = pack_bf16x2(x0 - bf16_lo(mid), x1 - bf16_hi(mid));
}
// The same of x0 + e0 and x1 + e1, the second parts some ulps of the first at the most.
__device__ __forceinline__ void split3(float x0, float x1, float e0, float e1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(x0, x1);
  x0 -= bf16_lo(hi);
  x1 -= bf16_hi(hi);
  mid = pack_bf16x2(x0, x1);
  lo = pack_bf16x2((x0 - bf16_lo(mid)) + e0, (x1 - bf16_hi(mid)) + e1);
}
// a + b = result + err (Knuth 1969)
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float s = a + b, t = s - a;
  err = (a - (s - t)) + (b - t);
  return s;
}
// (not volatile: the compiler may interleave independent accumulators)
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <int M, int N>
__device__ __forceinline__ void zero(float (&d)[M][N][4]) {
#pragma unroll
  for (int m = 0; m < M; ++m)
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) d[m][n][i] = 0.f;
}
// The six products of M tiles (16 x 16) of A with N tiles (16 x 8) of B (a[tile][piece], b[piece][tile][half]): hi.hi into dh, the others into
// dl.  An accumulator comes up again after M x N others at the least: dependent ones are about four issues apart.
template <int M, int N>
__device__ __forceinline__ void mma6(float (&dh)[M][N][4], float (&dl)[M][N][4], const uint32_t (&a)[M][3][4], const uint32_t (&b)[3][N][2]) {
  constexpr int order[6][2] = {{2, 0}, {0, 2}, {0, 0}, {1, 1}, {1, 0}, {0, 1}};
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int n = 0; n < N; ++n) mma(i == 2 ? dh[m][n] : dl[m][n], a[m][order[i][0]], b[order[i][1]][n][0], b[order[i][1]][n][1]);
}

// hi.hi and the other products together.  mma.sync cuts off where an addition rounds, always towards zero: measured, sums of hi.hi come out 0.16 (normal
// values) to 0.59 (values over 14 octaves) times 2^-24 too small, over the recurrences' chunks 0.36 on the average.  That mean is put back here,
// beside the small products, where it can be represented.  It is a mean and no bound: a single sum may miss up to 2^-23 of itself.
__device__ __forceinline__ float small_part(float hh, float rest) { return fmaf(hh, 0.36f * 5.9604645e-8f, rest); }
__device__ __forceinline__ float join(float hh, float rest) { return hh + small_part(hh, rest); }

}  // namespace split
}  // namespace nvllm
