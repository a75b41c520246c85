// How a grouped shared-prefix decode cuts up the requests that are in no group.  They have CTAs of their
// own, which take (request, kv head, split) items in turns; how many such requests there are only the
// device knows.  Plain arithmetic, the same on host and device; a split's first token, number x size,
// is always below the bound on the lengths, so nothing here or in the kernels leaves 32 bits.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define PFD_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PFD_HOST_DEVICE inline
#endif

namespace pfd {

constexpr int kLonerSplit = 256;  // tokens to an item, at least (two page pairs for each of four warps)

struct LonerGrid {
  int32_t rows;     // grid rows of CTAs in front of the batch's; 0: such requests have no CTAs of their own
  int32_t least;    // tokens to a split, at least: as many as the requests' slots make necessary
  int32_t share;    // tokens of one such request, as long as any, for each of those CTAs
  int32_t longest;  // bound on the lengths, in whole pages
};

// One wave of CTAs (three to an SM) in grid rows of ns x kv_heads; `slots`: partials a request has room for.
inline LonerGrid loner_grid(int64_t max_seq_len, int64_t slots, int64_t ns, int64_t kv_heads, int64_t sms) {
  const auto up = [](int64_t x, int64_t to) { return (x + to - 1) / to * to; };
  const auto most = [](int64_t x, int64_t y) { return x > y ? x : y; };
  const auto least = [](int64_t x, int64_t y) { return x < y ? x : y; };
  LonerGrid g;
  g.rows = static_cast<int32_t>((3 * sms + ns * kv_heads - 1) / (ns * kv_heads));
  g.longest = static_cast<int32_t>(least(up(max_seq_len, 16), INT32_MAX & ~15));
  g.least = static_cast<int32_t>(most(least(up((max_seq_len + slots - 1) / slots, 16), INT32_MAX & ~15), kLonerSplit));
  g.share = static_cast<int32_t>(least(max_seq_len * kv_heads / (g.rows * ns * kv_heads), 1 << 19));
  return g;
}

// Tokens to a split when `loners` requests of at most 2048 are in no group: as many items as the CTAs can
// take at once, no smaller than the slots allow, none longer than a request can be.
PFD_HOST_DEVICE int loner_split_size(const LonerGrid& g, int loners) {
  const int even = (loners * g.share + 63) & ~63;
  const int size = even < g.longest ? even : g.longest;
  return size > g.least ? size : g.least;
}

// Splits of a request of the greatest length: no item beyond them can have work.
PFD_HOST_DEVICE int loner_split_count(const LonerGrid& g, int size) {
  return g.longest > size ? (g.longest - 1) / size + 1 : 1;
}

}  // namespace pfd
