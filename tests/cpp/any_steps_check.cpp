// Compares run_steps_any (steps.h) with the sample-by-sample loop it replaces:
// random and halfway step sizes (dt at half a spacing of t, where sums round to
// even), steps of the order of the spacing and below it, runs across powers of
// two, caps and step budgets.  Prints one summary line; status 1 on a mismatch.
#include <cstdint>
#include <cstdio>
#include <random>

#include "steps.h"

using namespace aloha;

int main() {
  std::mt19937_64 rng(20260709u);
  std::uniform_real_distribution<float> u01(0.0f, 1.0f);
  long runs = 0, steps = 0, halfway = 0, crossings = 0, mismatches = 0;
  for (int i = 0; i < 400000; ++i) {
    const int e = (int)(u01(rng) * 26.0f) - 2;
    float t = ldexpf(1.0f + u01(rng), e);
    if (i % 5 == 0) t = ldexpf(2.0f, e) - ldexpf(u01(rng) * 64.0f, e - 8);  // just below a power of two
    if (i % 97 == 0) t = 0.0f;
    const float spacing = ldexpf(1.0f, e - 23);
    float dt;
    switch (i % 4) {
      case 0: dt = 0.05f + 2.0f * u01(rng); break;
      case 1: dt = spacing * ((float)(int)(u01(rng) * 4000.0f) + 0.5f); ++halfway; break;  // ties
      case 2: dt = spacing * (0.2f + 8.0f * u01(rng)); break;
      default: dt = i % 8 == 3 ? 0.3f : 0.1f; break;
    }
    const float tb = t + dt * (u01(rng) * (i % 3 == 0 ? 400.0f : 40.0f) - 2.0f);
    const uint32_t n0 = (uint32_t)(u01(rng) * 50.0f);
    const uint32_t cap = n0 + (i % 7 == 0 ? (uint32_t)(u01(rng) * 30.0f) : 2000u);
    const uint32_t budget = i % 6 == 0 ? (uint32_t)(u01(rng) * 40.0f) : 0xffffffffu;
    float a = t, b = t;
    uint32_t na = n0, nb = n0, ka = 0;
    while (ka < budget && a < tb && na < cap) {
      ++na;
      a = a + dt;
      ++ka;
    }
    const uint32_t kb = run_steps_any(b, nb, tb, cap, dt, budget);
    ++runs;
    steps += ka;
    if ((float_bits(t) >> 23) != (float_bits(a) >> 23)) ++crossings;
    if (ka != kb || na != nb || float_bits(a) != float_bits(b)) {
      if (mismatches++ < 5)
        std::printf("t %a dt %a tb %a n %u cap %u budget %u: loop %u %a, jump %u %a\n", t, dt, tb, n0, cap, budget, ka, a,
                    kb, b);
    }
  }
  std::printf("runs %ld steps %ld halfway %ld crossings %ld mismatches %ld\n", runs, steps, halfway, crossings, mismatches);
  return mismatches == 0 && crossings > 10000 ? 0 : 1;
}
