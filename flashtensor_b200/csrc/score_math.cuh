// Arithmetic that the column passes and the fused Keyformer pass share: hardware exponential and logarithm,
// the seeded noise generator, the record of an expired wait.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace asuka {
namespace {

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
__device__ __forceinline__ float lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Seeded Keyformer noise: one bijective 32-bit mix ("lowbias32") per logit.
//   head_key = hash(seed_lo ^ hash((b*H + h) ^ seed_hi));  word = hash(((q << 16) ^ kv) ^ head_key)
//   u = ((word >> 9) + 0.5) * 2^-23 in (0,1);  exp_rand = -ln(u);  noise g = -ln(exp_rand) ~ Gumbel(0,1)
__device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}
__device__ __forceinline__ uint32_t seeded_head_key(uint64_t seed, uint32_t bh) {
  return hash_u32(static_cast<uint32_t>(seed) ^ hash_u32(bh ^ static_cast<uint32_t>(seed >> 32)));
}
// log2(exp_rand) of two logits less kSeededLg2Unit, from their words after the first xor-shift of the mix.
// The passes that use it are bound by what they issue beside three MUFU operations per logit (logarithm of u,
// logarithm of exp_rand, exponential), hence: the first xor-shift is one LOP3 per logit (the words of a thread's
// neighbouring logits differ in their low bits only), the last one and the conversion to a float in [1, 2) are two
// shifts and a LOP3, the f32 arithmetic is packed, and the factor ln 2 of exp_rand, a constant after the second
// logarithm, is left to the row statistic.  17 instructions where the plain restatement takes 25: B2 H32 S1501,
// row pass 114 -> 88 us, column pass 107 -> 82, whole case 275 -> 217.
constexpr float kSeededLg2Unit = -0.52876637294489779f;  // log2(ln 2)
__device__ __forceinline__ float2 seeded_lg2_exp_rand2(uint32_t x0, uint32_t x1) {
  auto word = [](uint32_t x) {
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    return __uint_as_float(((x >> 9) ^ (x >> 25)) | 0x3f800000u);
  };
  const float2 u = __fadd2_rn(make_float2(word(x0), word(x1)), make_float2(-1.0f + 5.9604645e-8f, -1.0f + 5.9604645e-8f));  // exact
  // -log2(u): the hardware log2 has a fixed ABSOLUTE error, useless for u next to 1 (where the
  // large, row-dominating Gumbel values come from); there use the series in d = 1 - u (exact)
  const float2 d = __ffma2_rn(u, make_float2(-1.f, -1.f), make_float2(1.f, 1.f));
  float2 series = __ffma2_rn(d, make_float2(0.48089835f, 0.48089835f), make_float2(0.72134752f, 0.72134752f));
  series = __ffma2_rn(d, series, make_float2(1.44269504f, 1.44269504f));
  series = __fmul2_rn(d, series);
  const float e0 = -lg2(u.x), e1 = -lg2(u.y);
  return make_float2(lg2(d.x < 0.015625f ? series.x : e0), lg2(d.y < 0.015625f ? series.y : e1));
}

__device__ __forceinline__ void record_timeout(uint32_t* status, uint32_t site) {
  atomicAdd(&status[0], 1u);
  status[1] = site;
}

}  // namespace
}  // namespace asuka
