// Shared-prefix decode in one kernel in front of the merge, sm_100a: a persistent CTA per SM whose first
// sixteen warps take tiles of the dense prefix pass (dense_tile: tcgen05 on 128 rows x 256 prefix tokens)
// while its last four take pieces of the requests' own tokens -- the suffixes behind a prefix, the whole
// context of a request in no group -- with the step of the balanced kernel (bal_step).
//
// What bounds it: latencies.  The dense tiles of a batch of 64 are one chain of some 8 us on 128 of the
// SMs (block table, operands, MMA, softmax, MMA, stores), and the suffixes' 8 MB a layer are 1.3 us of memory
// time in chains of 5 us.  As kernels of their own they cost the layer two grid completions in a row in
// front of the merge, and the second of them started on what the first left free.  Here one grid
// completes, and the tiles of all groups are one list, so that a batch whose groups' prefixes differ
// takes as many rounds as it has tiles for the SMs.  (Side by side on the same SMs the two kernels are as fast
// where a single round is all there is; fused_pays.)  A layer of 64 requests, two groups and eight requests in none, 16 + 2
// heads: 23.3 us with it, 28.2 with the two.  Of a launch's 23 us the tensor cores work 11 %, and DRAM 15 %.
//
// Registers: 640 threads at 96 are what the block is launched with; the dense warps hand back 16 each
// (setmaxnreg) and the four others take 64 more, 4 x 80 + 160 = 5 x 96 per 128 threads.  Both spill a little
// (108 bytes stored and 188 loaded a thread, over both parts).
// Shared memory: the dense pass's 160 KB and a ring of two 8 KiB stages for each of the four warps.  No second CTA fits
// beside it, so that the 512 columns of TMEM, which every CTA takes before it knows whether it has a tile, are always
// free; a CTA of another kernel that held some would be waited for.
#pragma once

#include "paged_decode_balanced.cuh"
#include "shared_prefix_dense.cuh"

namespace pfd {

constexpr int kFusedSuffixWarps = 4;
constexpr int kFusedStages = 2;
constexpr int kFusedThreads = kDenseThreads + 32 * kFusedSuffixWarps;
constexpr uint32_t kFusedStage = 4 * kPage * 128;
constexpr int kFusedSmem = 1024 + DenseLayout::kBytes + kFusedSuffixWarps * kFusedStages * (kFusedStage + 8) + 32;

// Tile number `t` of the prefix pass; false behind the last one.  All groups' tiles are one list: by group,
// then chunk and kv head, the 128-row tiles that share those K and V side by side.
__device__ __forceinline__ bool fused_tile(const KernelParams& p, const PrefixParams& pp, int t, PrefixTile& tile) {
  const int B = pp.groups_batch, G = pp.max_groups;
  int first = 0, members = 0, prefix_len = 0;
  bool found = false;
  const auto take = [&](int begin, int end, int len) {  // a group's rows and prefix: is tile t among its own?
    const int chunks = (len + kPrefixChunk - 1) / kPrefixChunk;
    const int tiles = ((end - begin) * p.group + kPrefixRows - 1) / kPrefixRows * chunks * p.num_kv_heads;
    if (t < tiles) { found = true; first = begin; members = end - begin; prefix_len = len; }
    else t -= tiles;
  };
  if (pp.groups == nullptr) {
    take(0, pp.batch, pp.prefix_len);
  } else {
    const int32_t* offs = pp.groups + groups_offsets_off(B);
    const int32_t* lens = pp.groups + groups_prefix_off(B, G);
    const auto usable = [&](int len) { return min(len & ~15, pp.prefix_len); };  // (pp.prefix_len: the cap)
    // Up to 8 groups: all offsets and prefix lengths in one round trip (offsets of unused groups equal the
    // total, i.e. no tiles).
    constexpr int kFast = 8;
    if (G <= kFast) {
      int o[kFast + 1], pl[kFast];
#pragma unroll
      for (int i = 0; i <= kFast; ++i) o[i] = offs[min(i, G)];
#pragma unroll
      for (int i = 0; i < kFast; ++i) pl[i] = lens[min(i, G - 1)];
#pragma unroll
      for (int i = 0; i < kFast; ++i)
        if (!found && o[i + 1] > o[i]) take(o[i], o[i + 1], usable(pl[i]));
    } else {
      const int n_groups = min(pp.groups[3], G);
      for (int g = 0; g < n_groups && !found; ++g) take(offs[g], offs[g + 1], usable(lens[g]));
    }
  }
  if (!found) return false;
  const int row_tiles = (members * p.group + kPrefixRows - 1) / kPrefixRows;
  tile.mtile = t % row_tiles;
  tile.kvh = t / row_tiles % p.num_kv_heads;
  tile.chunk = t / row_tiles / p.num_kv_heads;
  tile.prefix_len = prefix_len;
  tile.n_req = members;
  tile.req_list = pp.groups != nullptr ? pp.groups + groups_rows_off(B, G) + first : nullptr;
  tile.page_row = tile.req_list != nullptr ? tile.req_list[0] : 0;  // any member's row names the prefix pages
  return true;
}

// The four last warps of a CTA: each takes pieces (request, part of its tokens, kv head) of the list by request, one
// a turn of all such warps of the grid.  A piece is an item of one warp: no barrier, no merge with
// other warps.  The warp finds its pieces itself, 32 requests at a time, one per lane.
template <bool QBF16>
__device__ __forceinline__ void suffix_pieces(const KernelParams& p, const TmaParams& tp, const CUtensorMap& tmap_k,
                                              const CUtensorMap& tmap_v, uint32_t ring, uint32_t bars, int warp, int lane) {
  constexpr int D = 128;
  const int i = lane >> 2, j = lane & 3;
  const int B = p.batch, hkv = p.num_kv_heads;
  const uint32_t my_ring = ring + warp * kFusedStages * kFusedStage;
  const uint32_t my_bars = bars + warp * kFusedStages * 8;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < kFusedStages; ++s) mbar_init(my_bars + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();

  uint32_t k_off[2][2], v_off[4];
#pragma unroll
  for (int half = 0; half < 2; ++half)
#pragma unroll
    for (int l = 0; l < 2; ++l) k_off[half][l] = bal_chunk<D>(half * 8 + rho(i), j + 4 * l);
#pragma unroll
  for (int r = 0; r < 4; ++r) v_off[r] = bal_chunk<D>(bal_v_row<D>(j, r), i);

  // Neighbouring warps of a CTA take two heads of the same tokens (adjacent in memory); the CTAs without a dense
  // tile, which are the last ones, take the first pieces.
  const int side = hkv % 2 == 0 ? 2 : 1;
  const int first = (warp / side * (int)gridDim.x + (int)(gridDim.x - 1 - blockIdx.x)) * side + warp % side;
  const int warps = kFusedSuffixWarps * (int)gridDim.x;
  // The list begins with the requests in no group, whose pieces are the longest, and every other turn runs
  // backwards: the warps with the longest pieces of one turn get the shortest of the next, or none (64
  // requests, two groups, 8 in none, eight layers: at most 8 instead of 10 page pairs to a warp, 207 -> 192 us).
  const int rounds = (B + 31) / 32, in_none = p.row_kv_start != nullptr ? rounds : 0;
  int round = -1;
  // 32 requests, one per lane: their tokens and pieces, and the pieces up to and including the lane's
  int before = 0, total = 0, incl = 0;
  OwnTokens own{};
  SuffixCut cut{};
  int s = 0, parity = 0;  // the ring's next stage, and its barrier's phase
  const uint64_t policy = l2_policy_evict_first();
  bool ok = true;
#pragma unroll 1
  for (int turn = 0; ok; ++turn) {
    const int rank = turn * warps + (turn & 1 ? warps - 1 - first : first);
    const int piece = rank / hkv, kvh = rank - piece * hkv;
#pragma unroll 1
    while (piece >= before + total) {
      before += total;
      if (++round >= rounds + in_none) return;
      own = OwnTokens{};
      cut = SuffixCut{};
      const int r = (round < in_none ? round : round - in_none) * 32 + lane;
      if (r < B) {
        own = own_tokens(p, r);
        if (in_none == 0 || (own.kv0 == 0) == (round < in_none)) cut = own_cut(own);
      }
      incl = cut.pieces;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += x;
      }
      total = __shfl_sync(0xffffffffu, incl, 31);
    }
    const int at = __ffs(__ballot_sync(0xffffffffu, incl > piece - before)) - 1;
    const int b = (round < in_none ? round : round - in_none) * 32 + at;
    const int part = piece - before - __shfl_sync(0xffffffffu, incl - cut.pieces, at);
    const int pairs = __shfl_sync(0xffffffffu, cut.pairs, at);
    const int kv0 = __shfl_sync(0xffffffffu, own.kv0, at);
    const int end = kv0 + __shfl_sync(0xffffffffu, own.live, at);
    const int slot = __shfl_sync(0xffffffffu, own.slot0, at) + part;
    const int lo = kv0 + part * pairs * 2 * kPage;
    const int hi = min(lo + pairs * 2 * kPage, end);

    const int page_first = lo / kPage, page_last = (hi - 1) / kPage;
    const int n = (page_last - page_first + 2) / 2;
    const auto fetch = [&](int t) -> int32_t {  // page ids of pairs t .. t + 15, one page per lane
      const int pg = page_first + 2 * t + lane;
      return pg <= page_last ? p.block_table[(int64_t)b * p.bt_stride_b + pg] : -1;
    };
    int32_t ids = fetch(0), ids_next = n > 16 ? fetch(16) : -1;
    int ids_base = 0;
    const auto fire = [&](int t, int s) {  // pair t into stage s; all lanes call, lane 0 issues
      const int32_t phys0 = __shfl_sync(0xffffffffu, ids, (2 * (t - ids_base)) & 31);
      const int32_t phys1 = __shfl_sync(0xffffffffu, ids, (2 * (t - ids_base) + 1) & 31);
      if (lane == 0) {
        const uint32_t bar = my_bars + 8 * s, dst = my_ring + s * kFusedStage;
        mbar_expect_tx(bar, phys1 >= 0 ? kFusedStage : kFusedStage / 2);
        const int c1 = tp.head_is_dim1 ? kvh : 0, c2 = tp.head_is_dim1 ? 0 : kvh;
        tma_load_tile(dst, &tmap_k, bar, c1, c2, phys0, policy);
        tma_load_tile(dst + 2 * kPage * D, &tmap_v, bar, c1, c2, phys0, policy);
        if (phys1 >= 0) {
          tma_load_tile(dst + kPage * D, &tmap_k, bar, c1, c2, phys1, policy);
          tma_load_tile(dst + 3 * kPage * D, &tmap_v, bar, c1, c2, phys1, policy);
        }
      }
    };
#pragma unroll
    for (int t = 0; t < kFusedStages; ++t)
      if (t < n) fire(t, (s + t) % kFusedStages);

    const float ks = p.k_scale_ph ? p.k_scale_ph[kvh] : p.k_scale;
    const float vs = p.v_scale_ph ? p.v_scale_ph[kvh] : p.v_scale;
    const float scale_signed = ks * p.sm_scale * kLog2e;
    const uint32_t q_flip = scale_signed < 0.f ? 0x80008000u : 0u;  // (see paged_decode_fp8_chunk_kernel)
    uint32_t qb[1][D / 16][2];
    bal_load_q<QBF16, 1, D>(qb, p, b, kvh, i, j);
#pragma unroll
    for (int f = 0; f < D / 16; ++f) { qb[0][f][0] ^= q_flip; qb[0][f][1] ^= q_flip; }
    BalState<1, D> st;
    bal_reset<1, D>(st);
    int t = 0;
#pragma unroll 1
    for (; t < n; ++t) {
      if (!mbar_wait_bounded(my_bars + 8 * s, parity, tp.wait_limit_ns)) { ok = false; break; }
      bal_step<1, D>(st, my_ring + s * kFusedStage, k_off, v_off, qb, fabsf(scale_signed), lo + t * 2 * kPage, lo, hi, i, j);
      __syncwarp();  // all reads of the stage fed MMAs above: hand it back to TMA
      const int tn = t + kFusedStages;
      if (tn < n) {
        if ((tn & 15) == 0) {
          ids = ids_next;
          ids_base = tn;
          ids_next = fetch(tn + 16);
        }
        if (lane == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        fire(tn, s);
      }
      if (++s == kFusedStages) { s = 0; parity ^= 1; }
    }
    if (!ok) {
      // a copy never landed: record it; give the copies still in flight a bounded chance to land
      if (lane == 0) {
        atomicExch(tp.status, kErrTmaTimeout);
        for (int u = t + 1; u < min(n, t + kFusedStages); ++u) {
          if (++s == kFusedStages) { s = 0; parity ^= 1; }
          mbar_wait_bounded(my_bars + 8 * s, parity, tp.wait_limit_ns);
        }
      }
      break;
    }
    if (lane == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the next piece's copies reuse the ring
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float l = st.l[0][c];
      l += __shfl_xor_sync(0xffffffffu, l, 4);
      l += __shfl_xor_sync(0xffffffffu, l, 8);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      const int head = 2 * j + c;
      if (head >= p.group) continue;
      const int64_t r = (int64_t)b * p.partial_stride_b + (int64_t)(kvh * p.group + head) * p.partial_stride_h +
                        (int64_t)slot * p.partial_stride_s;
      float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.partial_output) + r * D + (D / 8) * i);
#pragma unroll
      for (int f = 0; f < D / 32; ++f)
        dst[f] = make_float4(st.o[0][2 * f][c] * vs, st.o[0][2 * f][2 + c] * vs, st.o[0][2 * f + 1][c] * vs,
                             st.o[0][2 * f + 1][2 + c] * vs);
      if (i == 0) {
        p.partial_max[r] = st.m[0][c] * kLn2;
        p.partial_sum[r] = l;
      }
    }
  }
}

// grid: one CTA per SM; block: kFusedThreads.  For at most 8 query heads per kv head and caches that TMA can describe.
template <bool QBF16>
__global__ void __launch_bounds__(kFusedThreads, 1)
shared_prefix_fused_kernel(const KernelParams p, const TmaParams tp, const PrefixParams pp,
                           const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t ring = base + DenseLayout::kBytes;
  const uint32_t suffix_bars = ring + kFusedSuffixWarps * kFusedStages * kFusedStage;
  const uint32_t bars = suffix_bars + kFusedSuffixWarps * kFusedStages * 8;  // two mbarriers of the dense warps
  const uint32_t tslot = bars + 16;                                          // TMEM base address
  const volatile uint32_t* tslot_ptr = reinterpret_cast<volatile uint32_t*>(gen + (tslot - base));
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  // A programmatic dependent of whatever precedes it: nothing is read before that has completed.  The merge
  // kernel behind reads the lengths before its own wait and is let in only then.
  if (t >= kDenseThreads) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
    if (t == kDenseThreads) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_k)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_v)) : "memory");
    }
    pdl_wait();
    pdl_launch_dependents();
    suffix_pieces<QBF16>(p, tp, tmap_k, tmap_v, ring, suffix_bars, warp - kDenseThreads / 32, lane);
    return;
  }
  asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
  if (t == 0) {
    mbar_init(bars, 1);
    mbar_init(bars + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(tslot, 512);
  pdl_wait();
  pdl_launch_dependents();
  bool ok = true;
  int turns = 0;
  PrefixTile tile;
#pragma unroll 1
  for (int at = blockIdx.x; fused_tile(p, pp, at, tile); at += gridDim.x, ++turns)
    ok = dense_tile<QBF16>(p, pp, tile, gen, base, bars, tslot_ptr, turns & 1) && ok;
  if (!ok && t == 0) atomicExch(pp.status, kErrUmmaTimeout);
  // A request that has more tokens than the caller's bounds say is reported, not silently cut.  Here, by warps whose CTA
  // has the fewest tiles: in the other warps' search for pieces it cost a layer of 64 requests 0.2 us of 23.6.
  if (p.row_kv_start != nullptr && blockIdx.x == gridDim.x - 1)
    for (int r = t; r < p.batch; r += kDenseThreads)
      if (own_tokens(p, r).cut_off) atomicExch(pp.status, kErrSuffixBound);
  __syncwarp();
  if (warp == 0) tmem_dealloc(*tslot_ptr, 512);
}

}  // namespace pfd
