// CPU check of df2d_any (p3g_arith.cuh): hi + lo in binary64 for pairs of every
// magnitude, bit for bit the sum of the two widened words.  Built and run by
// tests/test_spectrum_widening.py.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../p3dfft_gb300/csrc/p3g_arith.cuh"

static int failures = 0;
static void check(float hi, float lo) {
  const double want = (double)hi + (double)lo, got = p3g::df2d_any(hi, lo);
  if (p3g::d2u(got) == p3g::d2u(want)) return;
  if (failures++ < 20) std::printf("FAIL %a + %a: %a, not %a\n", (double)hi, (double)lo, got, want);
}

int main() {
  std::mt19937_64 rng(2024);
  std::uniform_real_distribution<double> u(1.0, 2.0);
  // the low word from the size of the high word's last bits down to nothing
  for (int e = -149; e <= 127; ++e)
    for (int i = 0; i < 4000; ++i) {
      const float hi = std::ldexp((float)u(rng) * (1.0f - 0x1p-24f), e);
      const float lo = std::ldexp((float)(u(rng) - 1.5), e - 20 - (int)(rng() % 40));
      check(hi, lo);
      check(hi, -lo);
      check(hi, 0.0f);
      check(std::ldexp(1.0f, e), lo);  // a power of two: a negative low word changes the binade
      check(std::ldexp(1.0f, e), -lo);
    }
  check(0.0f, 0.0f);
  check(INFINITY, 0.0f);
  if (!std::isnan(p3g::df2d_any(NAN, 0.0f))) ++failures;
  std::printf("%d failures\n", failures);
  return failures ? 1 : 0;
}
