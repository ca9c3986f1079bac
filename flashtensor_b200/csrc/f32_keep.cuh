// f32 arithmetic that keeps subnormal values, which the build's flags flush elsewhere, and the scales of the folded
// output projection (linattn32.cu writes it, linear_f32.cu applies it).
#pragma once
#include <cstdint>

namespace asuka {

__device__ __forceinline__ float mul_keep(float a, float b) {
  float y;
  asm("mul.rn.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}
__device__ __forceinline__ float fma_keep(float a, float b, float c) {
  float y;
  asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
__device__ __forceinline__ float add_keep(float a, float b) {
  float y;
  asm("add.rn.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}

// The folded weights of an output column are sums of 32 products of M' with a head's part of a row of the output
// projection.  M' grows with the values over the queries and the row may be of any size, so the product can leave f32's
// range where (Q M') w_o^T stays in it.  A head's 32 weights are therefore brought to a largest magnitude of 2^-8 to 2^-7 by
// a power of two first: 32 products with a finite M' are finite then, and with products that keep their subnormal bits
// what a folded weight loses at the lower end is below 2^-141 of the weights' size, less than the 2^-126 at which M'
// itself is flushed.  (Weights beyond 2^119 are scaled by 2^-126, not less.)  The exponents (1 to 245) travel with the folded
// weights; the projection brings the heads of a column to the scale of its largest and takes that out of its sums again.
// Bits of the scale's exponent from those of the largest magnitude; the inverse's are 254 less this.
__device__ __forceinline__ uint32_t fold_scale_exponent(uint32_t max_bits) {
  const int e = static_cast<int>(max_bits >> 23);
  return e == 255 ? 127u : static_cast<uint32_t>(max(1, 246 - max(e, 1)));
}

// largest magnitude of a head's 32 weights, as bits, in each of the eight neighbouring lanes with four of them each
__device__ __forceinline__ uint32_t head_max_bits(const float4& v) {
  uint32_t m = max(max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu),
                   max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

}  // namespace asuka
