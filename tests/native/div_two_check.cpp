// Host check of the short division sequence (drot::div_rn_two) for divisors
// that pass drot::div_two_step_exact, against IEEE float division.
// Prints: divisors tried, divisors that pass, mismatches.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "drot_math.cuh"

static float from_bits(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }

int main() {
  uint64_t s = 0x9e3779b97f4a7c15ull;
  long tried = 0, pass = 0, bad = 0;
  for (int k = 0; k < 60; ++k) {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    // kappa = 1 + 2 r with r spread over [1e-6, 10], the last ones anywhere in [1, 2)
    const float b = k < 40 ? (float)(1.0 + 2.0 * std::pow(10.0, -6.0 + 7.0 * k / 39.0))
                           : from_bits(0x3f800000u | (uint32_t)(s & 0x7fffffu));
    const float y = (float)(1.0 / (double)b);
    ++tried;
    if (!drot::div_two_step_exact(b, y)) continue;
    ++pass;
    for (uint32_t m = 0; m < (1u << 23); ++m) {
      const float a = from_bits(0x3f800000u | m);
      if (drot::div_rn_two(a, b, y) != a / b) ++bad;
    }
    for (int i = 0; i < (1 << 18); ++i) {
      s ^= s << 13; s ^= s >> 7; s ^= s << 17;
      const uint32_t e = 37u + (uint32_t)(s % 120u);  // biased exponent of 2^-90 .. 2^30
      const float a = from_bits((e << 23) | (uint32_t)((s >> 20) & 0x7fffffu));
      if (drot::div_rn_two(a, b, y) != a / b) ++bad;
    }
    if (drot::div_rn_two(0.0f, b, y) != 0.0f) ++bad;
  }
  std::printf("%ld %ld %ld\n", tried, pass, bad);
  return bad ? 1 : 0;
}
