// Compares adc_ottawa_gb300/csrc/divide.h with the host's division (compiled
// and run by tests/test_divide.py): argv[1] random operand pairs of several
// kinds, each with a reciprocal estimate off by up to +-2^-21.  Prints the
// number of differing bit patterns.
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "divide.h"

static uint64_t state = 88172645463325252ull;
static uint64_t next() {
  state ^= state << 13; state ^= state >> 7; state ^= state << 17;
  return state;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    const uint64_t frac = 0xfffffffffffffull;
    uint64_t a = next() & frac, b = next() & frac;
    const int kind = (int)(next() % 8);
    if (kind == 1) a = b + (next() % 9) - 4;                       // quotient next to 1
    if (kind == 2) b = frac - next() % 4;                          // divisor next to 2
    if (kind == 3) b = next() % 4;                                 // divisor next to 1
    if (kind == 4) a = frac - next() % 4;
    if (kind == 5) a &= ~((1ull << (next() % 52)) - 1), b &= ~((1ull << (next() % 52)) - 1);   // short operands
    a &= frac;
    b &= frac;
    uint64_t ea = 1023 + (int)(next() % 81) - 40, eb = 1023 + (int)(next() % 81) - 40;
    if (kind == 6) { ea = next() % 2048; eb = next() % 2048; }     // the whole range, specials included
    const double x = adcgpu::div_double((ea << 52) | a | (next() & (1ull << 63)));
    double y = adcgpu::div_double((eb << 52) | b | (next() & (1ull << 63)));
    if (kind == 7) {                                               // quotient next to a midpoint: x = RN((q + half ulp) y)
      const double q = adcgpu::div_double((1023ull << 52) | (next() & frac));
      const long double m = (long double)q + 0x1p-53L;
      const double xx = (double)(m * (long double)y);
      const double e = ((float)(int)(next() % 3) - 1.0f) * 0x1p-21f;
      const double z = xx / y, w = adcgpu::div_rn(xx, y, (float)e);
      bad += adcgpu::div_bits(z) != adcgpu::div_bits(w);
      continue;
    }
    const float err = ((float)(next() % 2001) - 1000.0f) * (0x1p-21f / 1000.0f);
    const double z = x / y, w = adcgpu::div_rn(x, y, err);
    if (z != z) { bad += w == w; continue; }
    bad += adcgpu::div_bits(z) != adcgpu::div_bits(w);
  }
  printf("%ld\n", bad);
  return 0;
}
