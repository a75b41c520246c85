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

// Own tokens of a request of `seq_len` tokens that attends from `kv0` on, all behind its prefix (`splits` > 0: as many
// splits of `split_size`, the caller's bound on them) or its whole context (`splits` 0); never past the `cols` pages that a
// row of the block table is known to have.  Less than it has: a broken bound, which the caller of this reports.
PFD_HOST_DEVICE int own_length(int seq_len, int kv0, int cols, int splits, int split_size) {
  const int64_t row = static_cast<int64_t>(cols) * 16 - kv0;
  const int64_t bound = splits > 0 ? static_cast<int64_t>(splits) * split_size : row;
  const int64_t most = bound < row ? bound : row;
  const int64_t has = static_cast<int64_t>(seq_len) - kv0;
  const int64_t live = has < most ? has : most;
  return live > 0 ? static_cast<int>(live) : 0;
}

}  // namespace pfd
