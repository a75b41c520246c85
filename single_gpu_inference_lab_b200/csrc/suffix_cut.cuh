// How the fused shared-prefix kernel cuts a request's own tokens (csrc/shared_prefix_fused.cuh) into pieces, one
// warp each.  A rule of the request alone: the kernel and the merge kernel behind it work it out for themselves.
// And which calls it takes.
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

// What the host knows of a shared-prefix call: bounds, where the lengths and the groups are on the device.
struct FusedShape {
  int64_t batch, group, kv_heads;  // requests, query heads to a kv head, kv heads
  int64_t chunks;                  // prefix chunks of the longest prefix, at most
  int64_t slots;                   // slots for own tokens behind them
  int64_t own;                     // tokens behind a prefix, at most
  int64_t alone;                   // tokens of a request in no group, at most; 0: there is none
  bool grouped;                    // prefixes may differ, so that `own` is the shortest one's
};

// Calls that the fused kernel takes from the two kernels (the dense pass, then split-KV work behind it).  Its four warps
// per SM for own tokens, one to a piece, have the dense tiles' time for them, where the split-KV kernel's twelve share a
// split by four and run on SMs that have no tile.  In us: the tiles allow 9 for each round of them and 12 for the part
// of the SMs that has one in a single round; taking a piece up costs 2.8, a page pair of the longest piece 1.2, and of
// the average warp's share 1.0 (requests have half of their bound on average, in groups behind unequal prefixes
// less).  Apart from that, a page pair of a request in no group costs 1.35, since the slots that bound its pieces are few where
// its context is long.
// Measured on 1110 shapes: 16 + 2, 28 + 4, 32 + 8, 8 + 1, 8 + 8 and 32 + 16 heads, 8 .. 256 requests, prefixes of 256 .. 8192, 16 ..
// 2048 own tokens, up to all requests in no group, of up to 65536 tokens.  The fused kernel takes 714 of them; 46 are more than
// 2 % slower with it and 60 of the others more than 2 % faster.  us, two kernels / fused:
//   taken: 64 x 4096 + 512, 16 + 2 heads 17.5 / 15.6, 32 + 8 43.3 / 36.2; two groups 27.2 / 17.9, and 8 requests in none 29.9 / 20.8
//   not taken: 64 x 1024 + 512, 8 + 8 heads 18.8 / 25.7, 32 + 8 23.1 / 27.3; 16 x 2048 + 2048, 16 + 2 16.7 / 22.1;
//     64 x 4096 + 512 and one request in no group of 16384 tokens 23.9 / 33.2, of 65536 46.8 / 103; 4 of 4096 beside 60 x 256 + 16 26.1 / 66.3
//   taken, and slower: how many requests are in no group only the device knows.  64 x 4096 + 512, 16 + 2 heads, 32 of them in none
//     32.2 / 34.4, 48 37.7 / 47.4, all 51.9 / 51.6; all of 32 + 8 133 / 153 (with max_prefix_len left at max_seq_len 35.3 / 33.7,
//     41.9 / 40.6, 53.3 / 47.4 and 147 / 153)
inline bool fused_pays(const FusedShape& s, int64_t sms) {
  const auto up = [](int64_t x, int64_t by) { return (x + by - 1) / by; };
  const int64_t tiles = up(s.batch * s.group, 128) * s.chunks * s.kv_heads, warps = 4 * sms;
  const int64_t pairs = up(s.own, 32), half = pairs / (2 * kSuffixPairs);
  const int64_t pieces = half < 1 ? 1 : half < s.slots ? half : s.slots;
  const double allowed = 9.0 * static_cast<double>(up(tiles, sms)) + 12.0 * static_cast<double>(tiles) / static_cast<double>(sms);
  const double longest = static_cast<double>(up(pairs, s.slots)) * (s.grouped ? 0.75 : 1.0);
  const double share = 0.5 * static_cast<double>(s.batch * pairs * s.kv_heads) / static_cast<double>(warps);
  const double turns = static_cast<double>(up(s.batch * s.kv_heads * pieces, warps));
  const double alone = static_cast<double>(up(up(s.alone, 32), s.chunks + s.slots));
  return 2.8 * turns + 1.2 * longest + share <= allowed && 1.35 * alone <= allowed;
}

// Registers a thread that a block of the fused kernel is launched with.  Its warps hand them from one another
// (shared_prefix_fused.cuh): launched with any other number the ones that want more would wait for ever.
constexpr int kFusedRegs = 96;

// Calls that the fused kernel takes, if the compiler gave it `built_regs` registers a thread.
inline bool fused_takes(const FusedShape& s, int64_t sms, int built_regs) {
  return (built_regs + 7) / 8 * 8 == kFusedRegs && fused_pays(s, sms);
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
