// Host check of narrow_bits (csrc/narrow.cuh) against the host's FP64 to FP32 conversion: random significands at every
// exponent, the 29 bits below FP32's at, next to and between their halves, both signs.  Where the result is a normal
// FP32 number (or overflows to infinity by rounding), or the double is zero or subnormal, the bits are equal and ok
// stays; ok is cleared for the other results (FP32 subnormals, overflow, infinities and NaN).
// Built and run by tests/test_narrow.py; prints "<cases> <mismatches>".
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "narrow.cuh"

int main() {
  std::mt19937_64 rng(11);
  long long cases = 0, bad = 0;
  const uint64_t low[] = {0, 1, 0x0fffffff, 0x10000000, 0x10000001, 0x1fffffff};
  for (uint64_t e = 0; e < 2048; ++e)
    for (int k = 0; k < 200; ++k) {
      uint64_t m = rng() & 0xfffffffffffffull;
      if (k % 4 == 0) m |= 0xfffffe0000000ull;  // rounds up into the exponent
      if (k % 4 != 3) m = (m & ~0x1fffffffull) | low[rng() % 6];
      const uint64_t bits = ((rng() & 1) << 63) | (e << 52) | m;
      double d;
      std::memcpy(&d, &bits, 8);
      const float f = (float)d;
      uint32_t want;
      std::memcpy(&want, &f, 4);
      bool ok = true;
      const uint32_t got = ppm::narrow_bits((uint32_t)(bits >> 32), (uint32_t)bits, ok);
      const double mag = std::fabs(d);
      const bool meant = mag < DBL_MIN || (mag >= (double)FLT_MIN && mag < 2.0 * std::ldexp(1.0, 127));
      ++cases;
      if (ok != meant || (meant && got != want)) ++bad;
    }
  std::printf("%lld %lld\n", cases, bad);
  return bad != 0;
}
