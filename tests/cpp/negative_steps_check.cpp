// Compares run_steps_any (steps.h) with the sample-by-sample loop it replaces
// from negative ray parameters, which a march reaches with constant jitters of
// 10^7 steps and more (the first sample rounds below the brick's entry), where
// the float spacing gets finer as t rises: random starts, and whole marches from
// first_sample_t.  Prints one summary line; status 1 on a mismatch.
#include <cstdint>
#include <cstdio>
#include <random>

#include "steps.h"

using namespace aloha;

int main() {
  std::mt19937_64 rng(20261205u);
  std::uniform_real_distribution<float> u01(0.0f, 1.0f);
  long runs = 0, negative = 0, crossed = 0, mismatches = 0;
  auto compare = [&](float t, float tb, uint32_t cap, float dt, uint32_t budget) {
    float a = t, b = t;
    uint32_t na = 0, nb = 0, ka = 0;
    while (ka < budget && a < tb && na < cap) {
      ++na;
      a = a + dt;
      ++ka;
    }
    const uint32_t kb = run_steps_any(b, nb, tb, cap, dt, budget);
    ++runs;
    negative += t < 0.0f;
    crossed += t < 0.0f && a > 0.0f;
    if (ka != kb || na != nb || float_bits(a) != float_bits(b))
      if (mismatches++ < 5)
        std::printf("t %a dt %a tb %a cap %u budget %u: loop %u %a, jump %u %a\n", t, dt, tb, cap, budget, ka, a, kb, b);
  };
  for (int i = 0; i < 200000; ++i) {
    const int e = (int)(u01(rng) * 16.0f) - 4;
    const float t = i % 50 == 0 ? -0.0f : -ldexpf(1.0f + u01(rng), e);
    const float dt = i % 4 == 0 ? 0.3f : 0.05f + 2.0f * u01(rng);
    const float tb = t + dt * (u01(rng) * (i % 3 == 0 ? 900.0f : 60.0f) - 2.0f);
    compare(t, tb, i % 7 == 0 ? (uint32_t)(u01(rng) * 30.0f) : 5000u, dt, i % 6 == 0 ? (uint32_t)(u01(rng) * 40.0f) : 0xffffffffu);
  }
  compare(first_sample_t(0.0f, 0.3f, 462550464.0f), 9.0f, 5000u, 0.3f, 0xffffffffu);
  compare(first_sample_t(0.0f, 0.971369f, 69312904.0f), 24.0f, 5000u, 0.971369f, 0xffffffffu);
  for (int i = 0; i < 300000; ++i) {
    const float lower = i % 2 ? 0.0f : u01(rng) * 300.0f, dt = i % 3 ? 0.05f + 2.0f * u01(rng) : 0.3f;
    const float ils = ldexpf(1.0f + u01(rng), 10 + (int)(u01(rng) * 26.0f)) * (i % 5 ? 1.0f : -1.0f);
    const float t1 = lower + u01(rng) * 60.0f, t = first_sample_t(lower, dt, ils);
    if (t > -1e4f) compare(t, t1, march_cap(lower, t1, dt), dt, 0xffffffffu);
  }
  std::printf("runs %ld negative %ld crossed %ld mismatches %ld\n", runs, negative, crossed, mismatches);
  return mismatches == 0 && crossed > 50000 ? 0 : 1;
}
