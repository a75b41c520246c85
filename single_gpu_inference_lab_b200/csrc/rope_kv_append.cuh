// The producer step in front of decode attention: rotary embedding of the new tokens' Q and K
// (in place), then K and V written into the paged cache at the slots the engine assigned --
// into fp16 / bf16 caches as they are, into FP8-e4m3 caches divided by a per-(layer, kv head)
// scale.  Same call as the reference's fused operator (integrations/vllm/l20_rope_kv.py:256-328,
// kernels :26-253), which refuses quantised caches (:273-274).
//
// The arithmetic is written so that a CPU restatement in torch reproduces
// it bit for bit: products and the sum of the rotation are rounded separately (no fused
// multiply-add), the rotated value is rounded to the model's 16-bit type first (that is what
// stays in `key` / `query`), and the FP8 value is that rounded number divided by the scale in
// fp32, saturated to +-448 and rounded to nearest even.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace pfd {

struct RopeParams {
  void* query;        // [T, Hq, D], rotated in place
  void* key;          // [T, Hkv, D], rotated in place
  const void* value;  // [T, Hkv, D]
  const int64_t* positions;     // [T]
  const void* cos_sin_cache;    // [max_position, rotary_dim]: cos of the rotary_dim / 2 frequencies, then sin
  const int64_t* slot_mapping;  // [T]: block * block_size + offset, negative = do not store
  void* key_cache;              // logical [blocks, block_size, Hkv, D]
  void* value_cache;
  const float* k_scale_ph;  // FP8 caches: per kv head, or the scalars below
  const float* v_scale_ph;
  float k_scale, v_scale;
  int64_t q_stride_t, q_stride_h, k_stride_t, k_stride_h, v_stride_t, v_stride_h;  // elements
  int64_t kc_stride_block, kc_stride_token, kc_stride_head;                          // elements of the cache
  int64_t vc_stride_block, vc_stride_token, vc_stride_head;
  int64_t cs_stride;  // elements between rows of cos_sin_cache
  int32_t num_tokens, num_q_heads, num_kv_heads, head_dim, rotary_dim, block_size;
  int32_t is_neox;       // 1: pairs (i, i + rotary_dim / 2); 0: pairs (2i, 2i + 1)
  int32_t cos_sin_f32;   // 1: cos_sin_cache is float32, 0: it has the query's type
  int32_t cache_fp8;     // 1: e4m3 caches, 0: caches of the query's type
  // log2 of block_size, of the 16-byte chunks of a head and of its rotation tasks, -1 where that is no power of two
  int32_t block_shift, chunk_shift, task_shift;
  unsigned long long neg_zeros;  // two floats -0 (see f2_mul)
};

template <bool BF16>
__device__ __forceinline__ float load16(const void* p, int64_t i) {
  if constexpr (BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  else return __half2float(reinterpret_cast<const __half*>(p)[i]);
}
template <bool BF16>
__device__ __forceinline__ float round16(float x) {  // x rounded to the 16-bit type, as a float
  if constexpr (BF16) return __bfloat162float(__float2bfloat16_rn(x));
  else return __half2float(__float2half_rn(x));
}
template <bool BF16>
__device__ __forceinline__ void store16(void* p, int64_t i, float x) {
  if constexpr (BF16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(x);
  else reinterpret_cast<__half*>(p)[i] = __float2half_rn(x);
}
__device__ __forceinline__ uint8_t to_e4m3(float x, float scale) {
  // x / scale in fp32 (IEEE division), saturate-to-finite, round to nearest even
  const float y = __fdiv_rn(x, scale);
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.f), "f"(y));
  return static_cast<uint8_t>(r & 0xffu);
}

// One CTA per token, element by element: whatever the kernel below does not take.
template <bool BF16>
__global__ void __launch_bounds__(256) rope_quant_append_kernel(const RopeParams p) {
  // lets a kernel launched behind this one as a programmatic dependent become resident while this
  // one runs (the decode kernels, which wait for its completion before they touch what it writes)
  asm volatile("griddepcontrol.launch_dependents;");
  const int t = blockIdx.x;
  const int64_t pos = p.positions[t];
  const int64_t slot = p.slot_mapping[t];
  const int half = p.rotary_dim / 2;
  const int D = p.head_dim;
  const auto cs = [&](int f, bool sine) -> float {
    const int64_t i = pos * p.cs_stride + (sine ? half : 0) + f;
    return p.cos_sin_f32 ? reinterpret_cast<const float*>(p.cos_sin_cache)[i] : load16<BF16>(p.cos_sin_cache, i);
  };
  const int64_t block = slot >= 0 ? slot / p.block_size : 0;
  const int64_t offset = slot >= 0 ? slot % p.block_size : 0;

  // rotation pairs of the Q heads and of the K heads: one (head, frequency) per thread-iteration
  const int heads = p.num_q_heads + p.num_kv_heads;
  for (int e = threadIdx.x; e < heads * half; e += blockDim.x) {
    const int head = e / half, f = e % half;
    const bool is_q = head < p.num_q_heads;
    const int h = is_q ? head : head - p.num_q_heads;
    void* base = is_q ? p.query : p.key;
    const int64_t row = is_q ? (int64_t)t * p.q_stride_t + (int64_t)h * p.q_stride_h
                             : (int64_t)t * p.k_stride_t + (int64_t)h * p.k_stride_h;
    const int d1 = p.is_neox ? f : 2 * f, d2 = p.is_neox ? f + half : 2 * f + 1;
    const float x1 = load16<BF16>(base, row + d1), x2 = load16<BF16>(base, row + d2);
    const float c = cs(f, false), s = cs(f, true);
    const float y1 = round16<BF16>(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)));
    const float y2 = round16<BF16>(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, s)));
    store16<BF16>(base, row + d1, y1);
    store16<BF16>(base, row + d2, y2);
    if (!is_q && slot >= 0) {
      const int64_t dst = block * p.kc_stride_block + offset * p.kc_stride_token + (int64_t)h * p.kc_stride_head;
      if (p.cache_fp8) {
        const float sc = p.k_scale_ph ? p.k_scale_ph[h] : p.k_scale;
        reinterpret_cast<uint8_t*>(p.key_cache)[dst + d1] = to_e4m3(y1, sc);
        reinterpret_cast<uint8_t*>(p.key_cache)[dst + d2] = to_e4m3(y2, sc);
      } else {
        store16<BF16>(p.key_cache, dst + d1, y1);
        store16<BF16>(p.key_cache, dst + d2, y2);
      }
    }
  }
  if (slot < 0) return;
  // the part of K behind rotary_dim (not rotated), and V
  for (int e = threadIdx.x; e < p.num_kv_heads * D; e += blockDim.x) {
    const int h = e / D, d = e % D;
    const int64_t kdst = block * p.kc_stride_block + offset * p.kc_stride_token + (int64_t)h * p.kc_stride_head + d;
    const int64_t vdst = block * p.vc_stride_block + offset * p.vc_stride_token + (int64_t)h * p.vc_stride_head + d;
    const float v = load16<BF16>(p.value, (int64_t)t * p.v_stride_t + (int64_t)h * p.v_stride_h + d);
    if (p.cache_fp8) {
      reinterpret_cast<uint8_t*>(p.value_cache)[vdst] = to_e4m3(v, p.v_scale_ph ? p.v_scale_ph[h] : p.v_scale);
    } else {
      store16<BF16>(p.value_cache, vdst, v);
    }
    if (d >= p.rotary_dim) {
      const float k = load16<BF16>(p.key, (int64_t)t * p.k_stride_t + (int64_t)h * p.k_stride_h + d);
      if (p.cache_fp8) reinterpret_cast<uint8_t*>(p.key_cache)[kdst] = to_e4m3(k, p.k_scale_ph ? p.k_scale_ph[h] : p.k_scale);
      else store16<BF16>(p.key_cache, kdst, k);
    }
  }
}

// ---- rows of 16-byte chunks ------------------------------------------------------------------
// Both pairings, whole or partial rotation, rotary_dim a multiple of 16, head_dim of 8, every row
// 16-byte aligned.  A rotation task is 16 elements of one head with their eight cosines and sines:
// elements f .. f + 7 and f + half .. f + half + 7 (NeoX) or 2f .. 2f + 15 (interleaved), two
// 16-byte loads and two 16-byte stores either way, and for a K head two stores into the cache
// (8 bytes each as e4m3).  A copy task is eight elements of V, or of the part of K behind rotary_dim,
// on their way to the cache.
//
// TPT threads share a token.  A thread keeps its eight frequencies for all the heads it takes, so
// the cosines and sines are fetched and converted once per thread and not once per head, and it
// requests its next head before it works on the one it has.  What bounds a prefill chunk is the
// instructions between a load and its store as much as memory: with one warp to a token, the
// packed arithmetic below, shifts for the index divisions and no division per quantised value, 8192
// tokens of 28 + 4 heads of 128 with an FP8 cache (155 MB) take 28.4 us, 5.4 TB/s; a task per
// thread, scalar arithmetic and a division per value took 36.0 us.  4096 tokens of 32 + 8 heads,
// interleaved over half the head, 16-bit cache: 13.2 us (41.2 us element by element); a decode
// step's 64 tokens of 16 + 2 heads: 2.9 us (4.3 us).
// Element by element the arithmetic is that of the kernel above, so the results are the same bits.

// Two floats in one register pair and the packed arithmetic of sm_100 on them: one instruction for two
// products or sums, each rounded as the scalar one is (and, like those under this build's flags,
// with denormals as zeros).  A product is written a * b + (-0), which is its rounded value, sign of zero
// included, with the -0 from a kernel argument: a packed multiplication in front of a packed sum is fused
// into one rounding by the assembler, .rn or not, and the results would be other bits.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2_pack(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f2_split(F2 x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b, F2 neg_zeros) {
  F2 r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg_zeros));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) { F2 r; asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { F2 r; asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

template <bool BF16>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  else return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {  // rounded to the 16-bit type
  if constexpr (BF16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}
__device__ __forceinline__ uint4 load16B(const void* base, int64_t i) {  // 8 consecutive 16-bit elements, 16-byte aligned
  return *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + i);
}
__device__ __forceinline__ void store16B(void* base, int64_t i, const uint4& v) {
  *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(base) + i) = v;
}

// x / scale as e4m3, two at a time, without dividing each: y = x * inv (inv = 1 / scale, rounded) is
// within 2^-23 of the quotient, relatively, and the rounded quotient within 2^-24 of it.  So where
// y (1 - 2^-21) and y (1 + 2^-21) round to the same e4m3 value, the rounded quotient does too;
// where they do not (a value in some hundred thousand) the division decides.  For a power of two y is
// the quotient, and so are both bounds.  `fast` is false for scales whose reciprocal or products
// could leave the normal range.
struct E4m3Scale {
  float scale, inv, down, up;
  bool fast;
};
__device__ __forceinline__ E4m3Scale e4m3_scale(float scale) {
  const bool exact = (__float_as_uint(scale) & 0x007fffffu) == 0u;
  return E4m3Scale{scale, __frcp_rn(scale), exact ? 1.f : 1.f - 0x1p-21f, exact ? 1.f : 1.f + 0x1p-21f,
                   scale > 0x1p-90f && scale < 0x1p90f};
}
__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi) {  // the first operand lands in the upper byte
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
template <bool BF16>
__device__ __forceinline__ uint32_t to_e4m3x2(uint32_t w, const E4m3Scale& s) {
  const float2 x = unpack2<BF16>(w);
  const float y0 = __fmul_rn(x.x, s.inv), y1 = __fmul_rn(x.y, s.inv);
  uint32_t r = cvt_e4m3x2(__fmul_rn(y0, s.down), __fmul_rn(y1, s.down));
  if (!s.fast || r != cvt_e4m3x2(__fmul_rn(y0, s.up), __fmul_rn(y1, s.up))) r = cvt_e4m3x2(__fdiv_rn(x.x, s.scale), __fdiv_rn(x.y, s.scale));
  return r;
}
template <bool BF16>
__device__ __forceinline__ void store8_e4m3(void* cache, int64_t i, const uint4& raw, const E4m3Scale& s) {
  const uint32_t lo = to_e4m3x2<BF16>(raw.x, s) | (to_e4m3x2<BF16>(raw.y, s) << 16);
  const uint32_t hi = to_e4m3x2<BF16>(raw.z, s) | (to_e4m3x2<BF16>(raw.w, s) << 16);
  *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(cache) + i) = make_uint2(lo, hi);
}
// eight consecutive values of a cos_sin_cache row
template <bool BF16>
__device__ __forceinline__ void load_cs8(const RopeParams& p, int64_t i, float (&v)[8]) {
  if (p.cos_sin_f32) {
    const float4* cp = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.cos_sin_cache) + i);
    const float4 a = cp[0], b = cp[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 raw = load16B(p.cos_sin_cache, i);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = unpack2<BF16>(w[k]);
      v[2 * k] = x.x; v[2 * k + 1] = x.y;
    }
  }
}

// x / d for x >= 0, a shift where d is a power of two (shift >= 0; the same in all threads): an integer
// division costs a thread more than the arithmetic of one rotation task.
template <typename T>
__device__ __forceinline__ T quotient(T x, int d, int shift) { return shift >= 0 ? x >> shift : x / d; }

constexpr int kRopeThreads = 256;
constexpr int kRopeMinCtas = 4;
template <bool BF16, bool NEOX, int TPT>
__global__ void __launch_bounds__(kRopeThreads, kRopeMinCtas) rope_quant_append_vec_kernel(const RopeParams p) {
  // Launched as a programmatic dependent itself: nothing is read before the kernel in front has
  // completed.  Only then are dependents let in, so that one which reads the step's metadata before its
  // own wait (PFD_FLAG_EARLY_METADATA) finds whatever ran in front of this kernel complete.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const int t = (int)blockIdx.x * (kRopeThreads / TPT) + (int)threadIdx.x / TPT;
  if (t >= p.num_tokens) return;
  const int tid = threadIdx.x % TPT;
  const int64_t pos = p.positions[t];
  const int64_t slot = p.slot_mapping[t];
  const int D = p.head_dim, half = p.rotary_dim / 2;
  const int heads = p.num_q_heads + p.num_kv_heads;
  const int64_t block = slot >= 0 ? quotient(slot, p.block_size, p.block_shift) : 0;
  const int64_t offset = slot >= 0 ? slot - block * p.block_size : 0;
  const int64_t kc_row = block * p.kc_stride_block + offset * p.kc_stride_token;
  const int64_t vc_row = block * p.vc_stride_block + offset * p.vc_stride_token;

  // copy tasks: the V heads, then the tails of the K heads
  const int v_chunks = D / 8, tail_chunks = (D - p.rotary_dim) / 8;
  const int n_v = p.num_kv_heads * v_chunks;
  const int n_copy = slot >= 0 ? n_v + p.num_kv_heads * tail_chunks : 0;
  const auto copy_load = [&](int e) -> uint4 {
    if (e < n_v) {
      const int h = quotient(e, v_chunks, p.chunk_shift), d = (e - h * v_chunks) * 8;
      return load16B(p.value, (int64_t)t * p.v_stride_t + (int64_t)h * p.v_stride_h + d);
    }
    const int h = (e - n_v) / tail_chunks, d = p.rotary_dim + (e - n_v - h * tail_chunks) * 8;
    return load16B(p.key, (int64_t)t * p.k_stride_t + (int64_t)h * p.k_stride_h + d);
  };
  const auto copy_store = [&](int e, const uint4& raw) {
    const bool is_v = e < n_v;
    const int q = is_v ? e : e - n_v, per = is_v ? v_chunks : tail_chunks;
    const int h = is_v ? quotient(q, per, p.chunk_shift) : q / per, d = (is_v ? 0 : p.rotary_dim) + (q - h * per) * 8;
    void* cache = is_v ? p.value_cache : p.key_cache;
    const int64_t dst = is_v ? vc_row + (int64_t)h * p.vc_stride_head + d : kc_row + (int64_t)h * p.kc_stride_head + d;
    if (p.cache_fp8) {
      const float* ph = is_v ? p.v_scale_ph : p.k_scale_ph;
      store8_e4m3<BF16>(cache, dst, raw, e4m3_scale(ph ? ph[h] : (is_v ? p.v_scale : p.k_scale)));
    } else {
      store16B(cache, dst, raw);
    }
  };
  // the first batch is requested here and stored behind the rotation
  constexpr int CB = TPT >= 128 ? 1 : 2;
  uint4 cp[CB];
  const auto copy_request = [&](int e0) {
#pragma unroll
    for (int u = 0; u < CB; ++u)
      if (e0 + u * TPT < n_copy) cp[u] = copy_load(e0 + u * TPT);
  };
  copy_request(tid);

  const int per_head = half / 8;           // rotation tasks per head; at most TPT (the launch checks)
  const int lanes = quotient(TPT, per_head, p.task_shift);  // heads the token's threads take side by side
  const int hs = quotient(tid, per_head, p.task_shift), f = (tid - hs * per_head) * 8;
  if (hs < lanes) {
    const int d1 = NEOX ? f : 2 * f, d2 = NEOX ? f + half : 2 * f + 8;  // first elements of the task's two chunks
    const F2 nz = p.neg_zeros;
    F2 c2[8], s2[8];  // NeoX: frequencies (2k, 2k + 1), four of each; interleaved: (cos, cos) and (-sin, sin) of one
    {
      float c[8], sn[8];
      load_cs8<BF16>(p, pos * p.cs_stride + f, c);
      load_cs8<BF16>(p, pos * p.cs_stride + half + f, sn);
#pragma unroll
      for (int k = 0; k < (NEOX ? 4 : 8); ++k) {
        c2[k] = NEOX ? f2_pack(c[(2 * k) & 7], c[(2 * k + 1) & 7]) : f2_pack(c[k], c[k]);
        s2[k] = NEOX ? f2_pack(sn[(2 * k) & 7], sn[(2 * k + 1) & 7]) : f2_pack(-sn[k], sn[k]);
      }
    }
    const auto row_of = [&](int head) -> uint16_t* {
      const bool is_q = head < p.num_q_heads;
      const int64_t row = is_q ? (int64_t)t * p.q_stride_t + (int64_t)head * p.q_stride_h
                               : (int64_t)t * p.k_stride_t + (int64_t)(head - p.num_q_heads) * p.k_stride_h;
      return reinterpret_cast<uint16_t*>(is_q ? p.query : p.key) + row;
    };
    uint4 n1, n2;
    const auto request = [&](int head) {
      if (head < heads) {
        const uint16_t* row = row_of(head);
        n1 = load16B(row, d1);
        n2 = load16B(row, d2);
      }
    };
    request(hs);
    for (int head = hs; head < heads; head += lanes) {
      const uint4 r1 = n1, r2 = n2;
      request(head + lanes);
      uint32_t w[8] = {r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z, r2.w};
#pragma unroll
      for (int k = 0; k < (NEOX ? 4 : 8); ++k) {
        const float2 x = unpack2<BF16>(w[k]);
        if constexpr (NEOX) {  // frequencies 2k, 2k + 1: first halves in word k, second halves in word 4 + k
          const float2 z = unpack2<BF16>(w[4 + k]);
          const F2 a = f2_pack(x.x, x.y), b = f2_pack(z.x, z.y);
          const float2 ya = f2_split(f2_sub(f2_mul(a, c2[k], nz), f2_mul(b, s2[k], nz)));
          const float2 yb = f2_split(f2_add(f2_mul(b, c2[k], nz), f2_mul(a, s2[k], nz)));
          w[k] = pack2<BF16>(ya.x, ya.y);
          w[4 + k] = pack2<BF16>(yb.x, yb.y);
        } else {  // frequency k: its pair is word k
          const float2 y = f2_split(f2_add(f2_mul(f2_pack(x.x, x.y), c2[k], nz), f2_mul(f2_pack(x.y, x.x), s2[k], nz)));
          w[k] = pack2<BF16>(y.x, y.y);
        }
      }
      const uint4 wa = make_uint4(w[0], w[1], w[2], w[3]), wb = make_uint4(w[4], w[5], w[6], w[7]);
      uint16_t* row = row_of(head);
      store16B(row, d1, wa);
      store16B(row, d2, wb);
      if (head >= p.num_q_heads && slot >= 0) {
        const int h = head - p.num_q_heads;
        const int64_t dst = kc_row + (int64_t)h * p.kc_stride_head;
        if (p.cache_fp8) {
          const E4m3Scale sc = e4m3_scale(p.k_scale_ph ? p.k_scale_ph[h] : p.k_scale);
          store8_e4m3<BF16>(p.key_cache, dst + d1, wa, sc);  // (what stays in `key`, quantised)
          store8_e4m3<BF16>(p.key_cache, dst + d2, wb, sc);
        } else {
          store16B(p.key_cache, dst + d1, wa);
          store16B(p.key_cache, dst + d2, wb);
        }
      }
    }
  }
  for (int e0 = tid; e0 < n_copy; e0 += CB * TPT) {
    uint4 now[CB];
#pragma unroll
    for (int u = 0; u < CB; ++u) now[u] = cp[u];
    copy_request(e0 + CB * TPT);
#pragma unroll
    for (int u = 0; u < CB; ++u)
      if (e0 + u * TPT < n_copy) copy_store(e0 + u * TPT, now[u]);
  }
}

}  // namespace pfd
