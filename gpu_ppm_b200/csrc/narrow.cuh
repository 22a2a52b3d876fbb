// FP64 to FP32 on the integer pipe, for the tensor-core fold's flux rows.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace ppm {

// The bits of the FP32 value nearest to the double of words hi and lo (ties to even) where that is a normal number, or
// the double is zero or subnormal; ok is left alone then and cleared otherwise.  On the integer pipe, which has room in
// the fold: the conversion instruction runs on the special-function pipe, 35 % of whose issue the kernel took (12 %
// with this).
__host__ __device__ __forceinline__ uint32_t narrow_bits(uint32_t hi, uint32_t lo, bool& ok) {
  const uint32_t mag = hi & 0x7fffffffu;
  uint32_t t = (hi << 3) | (lo >> 29);  // 23 bits of the significand under 9 of the exponent
  // round up when the 29 bits below are above half, or half and t is odd; exponent bias 1023 -> 127
  const uint32_t rest = (lo << 3) | (t & 1u);
  t += 0x40000000u + (rest > 0x80000000u ? 1u : 0u);
  if (mag < 0x00100000u) t = 0;
  ok = ok && (mag < 0x00100000u || mag - 0x38100000u < 0x0fe00000u);
  return (t & 0x7fffffffu) | (hi & 0x80000000u);
}

}  // namespace ppm
