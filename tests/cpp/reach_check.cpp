// Compares the passes of the macrocell codes (reach.h) with the definition, the
// Chebyshev distance to the nearest cell of the other kind in the brick, on
// random grids of all thin and odd shapes.  Prints one summary line; status 1 on
// a mismatch.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "reach.h"

using namespace aloha;

int main() {
  std::mt19937_64 rng(5u);
  long cells = 0, mismatches = 0, seen[kMaxReach + 1] = {};
  constexpr int W = kMaxReach - 1;
  for (int round = 0; round < 300; ++round) {
    int n[3];
    for (int& d : n) d = 1 + (int)(rng() % (round % 3 == 0 ? 4 : 21));
    const int spikes = (int)(rng() % 7);
    const bool invert = rng() & 1;
    std::vector<uint8_t> full((size_t)n[0] * n[1] * n[2], invert);
    for (int k = 0; k < spikes; ++k) full[rng() % full.size()] = !invert;
    if (round % 5 == 0)
      for (auto& f : full) f = rng() & 1;
    auto id = [&](int x, int y, int z) { return ((size_t)z * n[1] + y) * n[0] + x; };
    std::vector<int> a(full.size()), b(full.size());  // sign-extended code bytes
    for (size_t i = 0; i < full.size(); ++i) {  // x, with a row's neighbours in memory around it
      uint32_t window = 0;
      for (int d = -W; d <= W; ++d) {
        const long j = (long)i + d;
        if (j >= 0 && j < (long)full.size() && full[j]) window |= 1u << (W + d);
      }
      a[i] = (int8_t)((full[i] ? kCellFull : 0) | row_reach(window, (int)(i % n[0]), n[0]));
    }
    for (int axis = 1; axis < 3; ++axis) {
      for (int z = 0; z < n[2]; ++z)
        for (int y = 0; y < n[1]; ++y)
          for (int x = 0; x < n[0]; ++x) {
            int s[2 * W + 1];
            for (int d = -W; d <= W; ++d)
              s[W + d] = axis == 1 ? a[id(x, std::min(std::max(y + d, 0), n[1] - 1), z)]
                                   : a[id(x, y, std::min(std::max(z + d, 0), n[2] - 1))];
            b[id(x, y, z)] = (int8_t)axis_code(s + W);
          }
      a.swap(b);
    }
    for (int z = 0; z < n[2]; ++z)
      for (int y = 0; y < n[1]; ++y)
        for (int x = 0; x < n[0]; ++x) {
          int want = kMaxReach;
          for (int k = std::max(0, z - W); k <= std::min(n[2] - 1, z + W); ++k)
            for (int j = std::max(0, y - W); j <= std::min(n[1] - 1, y + W); ++j)
              for (int i = std::max(0, x - W); i <= std::min(n[0] - 1, x + W); ++i)
                if (full[id(i, j, k)] != full[id(x, y, z)])
                  want = std::min(want, std::max(std::abs(i - x), std::max(std::abs(j - y), std::abs(k - z))));
          const int got = a[id(x, y, z)] & 0xff;
          ++cells;
          ++seen[want];
          if (got != ((full[id(x, y, z)] ? kCellFull : 0) | want)) ++mismatches;
        }
  }
  bool all = true;
  for (int r = 1; r <= kMaxReach; ++r) all = all && seen[r] > 100;
  std::printf("cells %ld mismatches %ld\n", cells, mismatches);
  return mismatches == 0 && all ? 0 : 1;
}
