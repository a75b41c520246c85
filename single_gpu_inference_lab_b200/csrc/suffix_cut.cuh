// How the fused shared-prefix kernel cuts a request's own tokens (csrc/shared_prefix_fused.cuh) into pieces, one
// warp each.  A rule of the request alone: the kernel and the merge kernel behind it work it out for themselves.
// Plain arithmetic, the same on host and device.
#pragma once

#include <stdint.h>

#include "loner_split.cuh"  // PFD_HOST_DEVICE

namespace pfd {

constexpr int kSuffixPairs = 2;  // page pairs to a piece, at least

struct SuffixCut {
  int32_t pieces, pairs;  // pieces, and page pairs to each (the last may have fewer)
};

// `pairs` page pairs in at most `slots` pieces.
PFD_HOST_DEVICE SuffixCut suffix_cut(int pairs, int slots) {
  SuffixCut c = {0, 0};
  if (pairs <= 0) return c;
  const int most = (pairs - 1) / kSuffixPairs + 1;
  const int n = slots < 1 ? 1 : most < slots ? most : slots;
  c.pairs = (pairs - 1) / n + 1;
  c.pieces = (pairs - 1) / c.pairs + 1;
  return c;
}

}  // namespace pfd
