// Division by a number that a launch fixes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace asuka {

// x / d by a multiplication while x * d < 2^32 (the caller's matter), else as it is
struct FastDiv {
  uint32_t d, magic;  // magic 0: divide
  __device__ __forceinline__ int div(int x) const {
    return static_cast<int>(magic != 0 ? __umulhi(static_cast<uint32_t>(x), magic) : static_cast<uint32_t>(x) / d);
  }
};
inline FastDiv fast_div(int d, long long x_max) {
  FastDiv f;
  f.d = static_cast<uint32_t>(d);
  f.magic = d > 1 && x_max * d < (1ll << 32) ? static_cast<uint32_t>((1ull << 32) / f.d + 1) : 0u;
  return f;
}

}  // namespace asuka
