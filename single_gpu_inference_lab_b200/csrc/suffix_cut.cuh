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

// Calls that the fused kernel takes from the two kernels (the dense pass, then split-KV work behind or beside it).  In
// us, roughly: the tiles allow its four warps per SM for own tokens 9 for each round of them and 12 for the part of the SMs
// that has one in a single round, and the two kernels need 1.5 more for each wave of split-KV CTAs; a warp's turn costs 1, a
// page pair of the average warp's share 1, of the longest piece 1 (0.4 in groups behind unequal prefixes, where few are
// that long), and looking through 32 requests 0.4, twice that where the ones in no group come first.
// Where every request has a prefix, the two kernels side by side on the same SMs are as fast while a single round of
// tiles is all there is, or hardly any own tokens: the fused kernel takes what has more.  Where some may be in no group,
// they run one behind the other, and a page pair of such a request costs 1.35, since the slots that bound its pieces are
// few where its context is long.
// Measured on 5880 shapes, each on cold caches in the form that the two kernels take by themselves: 8 + 1, 8 + 8, 16 + 2, 28 + 4,
// 32 + 8 and 32 + 16 heads, 8 .. 256 requests, prefixes of 256 .. 8192, 16 .. 2048 own tokens, one prefix, or up to four groups
// with none to all of the requests outside.  us, two kernels / fused:
//   one prefix, taken: 64 x 4096 + 512, 32 + 8 heads 36.6 / 36.4; 128 x 8192 + 512, 16 + 2 50.9 / 48.4; 256 x 4096 + 128, 32 + 16 130 / 87.0
//     not taken: 64 x 4096 + 512, 16 + 2 15.6 / 16.4; 16 x 8192 + 1024, 16 + 2 14.6 / 17.4
//     of 2400 such shapes (and groups that hold every request) 450 are taken, 58 of them more than 2 % slower so, 318 faster
//   two groups, 64 x 4096 + 512, 16 + 2, taken: 23.3 / 19.5, with 8 requests in none 28.2 / 23.3, with 32 34.1 / 35.6
//     256 x 4096 + 16, 28 + 4, one group and 32 in none 107 / 92.4, two and 128 173 / 181
//     not taken: 256 x 256 + 128, 16 + 2, 32 in none 22.8 / 25.9
//     one group, 64 x 4096 + 512, 16 + 2, taken: 21.8 / 18.7
//     of 2718 with less than half of the requests in none 1109 are taken, 282 slower so, 742 faster (0.5 instead of 0.55: 1020, 273 and 673)
//   taken, and slower: 64 x 4096 + 2048, 16 + 2, two groups and 8 requests in none 35.7 / 43.5.  How many are in none only
//     the device knows: of 372 calls with all of them in none 168 are taken, 95 slower so, 256 x 4096 + 16, 28 + 4
//     213 / 297 the worst
inline bool fused_pays(const FusedShape& s, int64_t sms) {
  const auto up = [](int64_t x, int64_t by) { return (x + by - 1) / by; };
  const int64_t tiles = up(s.batch * s.group, 128) * s.chunks * s.kv_heads, warps = 4 * sms;
  const int64_t pairs = up(s.own, 32), half = pairs / (2 * kSuffixPairs);
  const int64_t pieces = half < 1 ? 1 : half < s.slots ? half : s.slots;
  const int64_t splits = s.slots < up(pairs, kSuffixPairs) ? s.slots : up(pairs, kSuffixPairs);  // (of 64 tokens or more, as measured)
  const double waves = static_cast<double>(s.batch * s.kv_heads * splits) / static_cast<double>(3 * sms);
  const double allowed = 9.0 * static_cast<double>(up(tiles, sms)) + 12.0 * static_cast<double>(tiles) / static_cast<double>(sms) + 1.5 * waves;
  const double longest = static_cast<double>(up(pairs, s.slots));
  const double share = 0.5 * static_cast<double>(s.batch * pairs * s.kv_heads) / static_cast<double>(warps);
  const double scan = 0.4 * static_cast<double>(up(s.batch, 32) * (s.grouped ? 2 : 1));
  const double own = static_cast<double>(up(s.batch * s.kv_heads * pieces, warps)) + share + scan;
  if (s.alone == 0) return tiles > sms && share >= 0.6 && own + longest <= 0.45 * allowed;
  const double alone = static_cast<double>(up(up(s.alone, 32), s.chunks + s.slots));
  return own + 0.4 * longest <= 0.5 * allowed && (alone <= 5.0 || 1.35 * alone <= 0.55 * allowed);
}

// Registers a thread that a block of the fused kernel is launched with.  Its warps hand them from one another
// (shared_prefix_fused.cuh): launched with any other number the ones that want more would wait for ever.
constexpr int kFusedRegs = 96;

// Calls that the fused kernel takes, if the compiler gave it `built_regs()` registers a thread, which is asked only of a
// call that would take it: the answer loads the kernel.
template <typename Registers>
inline bool fused_takes(const FusedShape& s, int64_t sms, Registers&& built_regs) {
  return fused_pays(s, sms) && (built_regs() + 7) / 8 * 8 == kFusedRegs;
}

// Own tokens of a request of `seq_len` tokens that attends from `kv0` on, all behind its prefix (`splits` > 0: as many
// splits of `split_size`, the caller's bound on them) or its whole context (`splits` 0); never past the `cols` pages that a
// row of the block table is known to have.  Less than it has: a broken bound, which the caller of this reports.
PFD_HOST_DEVICE int own_length(int seq_len, int kv0, int cols, int splits, int split_size) {
  constexpr int kMost = 0x7fffffff;  // (32 bits: every warp of the fused kernel works this out for every request)
  const int row = cols <= kMost / 16 ? cols * 16 : kMost;
  const int len = seq_len < 0 ? 0 : seq_len < row ? seq_len : row;
  int live = len - kv0;
  if (splits > 0) {
    const int64_t bound = static_cast<int64_t>(splits) * split_size;
    live = live < bound ? live : static_cast<int>(bound);
  }
  return live > 0 ? live : 0;
}

}  // namespace pfd
