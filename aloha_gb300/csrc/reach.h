// reach.h -- the macrocell codes' reach, one axis at a time (host and device).
//
// A cell's reach is the Chebyshev distance to the nearest cell of the other kind
// in its brick, at most kMaxReach.  It is separable: over y and z, the smallest
// max(step, reach there) with a cell of the other kind counting 0, from the
// reach along x.  Host-compilable so that the CPU tests can compare the passes
// with the definition.
#pragma once

#include "steps.h"

namespace aloha {

constexpr int kMaxReach = 8;
constexpr int kCellFull = 0x80;  // the kind bit of a code byte

// The reach along x of the cell at x of a row of `row` cells: bit kMaxReach - 1 +
// d of `window` is set if the cell d to its right is full.
ALOHA_HD int row_reach(uint32_t window, int x, int row) {
  constexpr int W = kMaxReach - 1;
  constexpr uint32_t side = (1u << W) - 1u;
  const uint32_t other = (window >> W) & 1u ? ~window : window;
  const int to_left = x < W ? x : W, to_right = row - 1 - x < W ? row - 1 - x : W;
  const uint32_t left = other & side & ~((1u << (W - to_left)) - 1u);  // distance d at bit W - d
  const uint32_t right = (other >> (W + 1)) & ((1u << to_right) - 1u);  // ... at bit d - 1
#ifdef __CUDA_ARCH__
  const int l = left ? W - 31 + __clz((int)left) : kMaxReach, r = right ? __ffs((int)right) : kMaxReach;
#else
  const int l = left ? W - 31 + __builtin_clz(left) : kMaxReach, r = right ? __builtin_ffs((int)right) : kMaxReach;
#endif
  return l < r ? l : r;
}

// One pass along another axis: the code of the cell whose code byte, sign-
// extended, is s[0], from its neighbours' up to kMaxReach - 1 away (indices
// clamped to the brick: a repeated edge cell is farther than the cell itself,
// so it takes nothing away).  Relative to the cell's kind, a code of the other
// kind is negative, so the step is the larger.
ALOHA_HD int axis_code(const int* s) {
  const int kind = s[0] & ~(kCellFull - 1);
  int reach = s[0] ^ kind;
  int least = reach;  // of the cells up to j away (the smallest max(j, there) is that of max(j, least))
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int j = 1; j < kMaxReach; ++j) {
    const int a = s[-j] ^ kind, b = s[j] ^ kind, ab = a < b ? a : b;
    least = ab < least ? ab : least;
    const int d = least > j ? least : j;
    reach = d < reach ? d : reach;
  }
  return kind | reach;
}

}  // namespace aloha
