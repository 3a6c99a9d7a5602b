// Selection of the smallest scores of a row by one block (coarse.cu, coarse_tc.cu).
#pragma once

#include "topk.cuh"

namespace cuvs_b200 {

// Sorts the first n2 (a power of two) keys ascending; the whole block calls it after a barrier.
__device__ __forceinline__ void block_sort_keys(uint64_t* keys, uint32_t n2)
{
  for (uint32_t size = 2; size <= n2; size <<= 1) {
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = threadIdx.x; i < n2 / 2; i += blockDim.x) {
        const uint32_t lo = 2 * i - (i & (stride - 1));
        const uint32_t hi = lo + stride;
        const bool up     = (lo & size) == 0;
        const uint64_t a = keys[lo], b = keys[hi];
        if ((a > b) == up) {
          keys[lo] = b;
          keys[hi] = a;
        }
      }
      __syncthreads();
    }
  }
}

// The exact `want` smallest (score, position) of a row of scores, written in ascending order, by a block of kThreads; where
// the row has fewer the rest of the result is empty (score NaN).
//
// First way: every thread keeps the kTops smallest scores of its strided part of the row; at least `want` scores are at or
// below the want-th smallest of the kThreads * kTops kept ones, and few others are (expected 1.2 `want` at 64 of 256,
// 1.4 at 128; 1.1 at 1,000 of 1,024 x 2), so two reads of the row find them all: keys (score, position) into shared
// memory, one sort.  A radix select reads the row five times, and its first histogram is one bucket's serial atomics
// (scores share their exponent): 252 us against 111 us for 64 of 4,000 scores in 10,000 rows, 280 against 85 us for 1,000 of
// 15,000 in 500 rows.
// Second way (more ties at the threshold than the buffer holds): radix select on the order-preserving image of the score
// (4 passes of 8 bits), one gather pass, then the sort.
// `load` reads scores: with __ldg, or plainly where the same kernel wrote them.  vec4: the row starts on a 16-byte boundary.
// `s_keys`: `cap` keys (select_cap), at least as many as a power of two that `want` fits.  Entered and left after a barrier.
struct select_mem {
  uint32_t hist[256];
  uint32_t prefix, remaining, count, eq_taken;
};
template <uint32_t kThreads, uint32_t kTops, typename Load>
__device__ __forceinline__ void select_row(const float* row, uint32_t len, bool vec4, uint32_t want, uint32_t cap, uint64_t* s_keys, select_mem& mem,
                                           Load&& load, uint32_t* out_idx, float* out_scores)
{
  const uint32_t tid = threadIdx.x;
  const uint32_t n4  = vec4 ? len / 4 : 0u;
  // every score of the row with its position
  auto for_row = [&](auto&& fn) {
    const float4* r4 = reinterpret_cast<const float4*>(row);
#pragma unroll 4
    for (uint32_t i = tid; i < n4; i += kThreads) {
      const float4 v = load(r4 + i);
      fn(float_to_ordered(v.x), 4 * i);
      fn(float_to_ordered(v.y), 4 * i + 1);
      fn(float_to_ordered(v.z), 4 * i + 2);
      fn(float_to_ordered(v.w), 4 * i + 3);
    }
#pragma unroll 4
    for (uint32_t i = 4 * n4 + tid; i < len; i += kThreads) { fn(float_to_ordered(load(row + i)), i); }
  };

  uint32_t n_sort = 0;
  {
    uint32_t best[kTops];
#pragma unroll
    for (uint32_t i = 0; i < kTops; i++) { best[i] = 0xFFFFFFFFu; }
    for_row([&](uint32_t o, uint32_t) {
#pragma unroll
      for (uint32_t i = kTops - 1; i > 0; i--) { best[i] = min(best[i], max(best[i - 1], o)); }
      best[0] = min(best[0], o);
    });
    // 24 bits of the want-th smallest of the kept scores, rounded up
    uint32_t lo = 0;
    for (int bit = 31; bit >= 8; bit--) {
      const uint32_t c = lo | (1u << bit);
      uint32_t n       = 0;
#pragma unroll
      for (uint32_t i = 0; i < kTops; i++) { n += uint32_t(__syncthreads_count(best[i] < c)); }
      if (n < want) { lo = c; }
    }
    const uint32_t T = lo | 0xFFu;
    if (tid == 0) { mem.count = 0; }
    __syncthreads();
    if (best[0] <= T) {  // (a thread whose smallest score is above the threshold has nothing)
      for_row([&](uint32_t o, uint32_t l) {
        if (o <= T) {
          const uint32_t slot = atomicAdd(&mem.count, 1u);
          if (slot < cap) { s_keys[slot] = (uint64_t(o) << 32) | l; }
        }
      });
    }
    __syncthreads();
    const uint32_t n = mem.count;
    if (n <= cap) {
      n_sort = 64;
      while (n_sort < n || n_sort < want) { n_sort <<= 1; }
      for (uint32_t i = n + tid; i < n_sort; i += kThreads) { s_keys[i] = kEmptyKey; }
    }
    __syncthreads();
  }
  if (n_sort == 0) {
    n_sort = 64;
    while (n_sort < want) { n_sort <<= 1; }
    if (tid == 0) {
      mem.prefix    = 0;
      mem.remaining = want;
    }
    // radix select: after the passes mem.prefix is the ordered image T of the want-th smallest score
    for (int pass = 0; pass < 4; pass++) {
      const int shift = 24 - 8 * pass;
      if (tid < 256) { mem.hist[tid] = 0; }
      __syncthreads();
      const uint32_t prefix = mem.prefix;
      const uint32_t mask   = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
      for_row([&](uint32_t o, uint32_t) {
        if ((o & mask) == prefix) { atomicAdd(&mem.hist[(o >> shift) & 0xFFu], 1u); }
      });
      __syncthreads();
      if (tid < 32) {
        uint32_t d, left;
        find_digit(mem.hist, mem.remaining, d, left);
        if (tid == 0) {
          mem.prefix    = prefix | (d << shift);
          mem.remaining = left;  // how many elements are wanted among those sharing the new prefix
        }
      }
      __syncthreads();
    }
    const uint32_t T       = mem.prefix;
    const uint32_t want_eq = mem.remaining;  // elements equal to T that belong to the selection
    if (tid == 0) {
      mem.count    = 0;
      mem.eq_taken = 0;
    }
    for (uint32_t i = tid; i < n_sort; i += kThreads) { s_keys[i] = kEmptyKey; }
    __syncthreads();
    // gather: everything below T, plus the want_eq lowest positions equal to T
    for (uint32_t base = 0; base < len; base += kThreads) {
      const uint32_t l = base + tid;
      uint32_t o       = 0xFFFFFFFFu;
      if (l < len) { o = float_to_ordered(load(row + l)); }
      if (l < len && o < T) { s_keys[atomicAdd(&mem.count, 1u)] = (uint64_t(o) << 32) | l; }
      // ties at T are taken in order: ballot keeps order inside a warp, warps take turns
      const bool eq = l < len && o == T;
      if (__syncthreads_or(eq)) {
        for (uint32_t w = 0; w < kThreads / 32; w++) {
          if ((tid >> 5) == w) {
            const unsigned m = __ballot_sync(kFullMask, eq);
            if (m) {
              const uint32_t start = mem.eq_taken;
              const uint32_t rank  = start + __popc(m & ((1u << (tid & 31)) - 1u));
              if (eq && rank < want_eq) { s_keys[atomicAdd(&mem.count, 1u)] = (uint64_t(o) << 32) | l; }
              __syncwarp();
              if ((tid & 31) == 0) { mem.eq_taken = start + __popc(m); }
            }
          }
          __syncthreads();
        }
      }
    }
    __syncthreads();
  }
  if (n_sort == 64) {
    if (tid < 32) {
      uint64_t a0 = s_keys[tid], a1 = s_keys[tid + 32];
      warp_sort64<uint64_t, false>(a0, a1);
      s_keys[tid]      = a0;
      s_keys[tid + 32] = a1;
    }
    __syncthreads();
  } else {
    block_sort_keys(s_keys, n_sort);
  }
  for (uint32_t p = tid; p < want; p += kThreads) {
    const uint64_t key = s_keys[p];
    out_idx[p]         = uint32_t(key);
    if (out_scores) { out_scores[p] = ordered_to_float(uint32_t(key >> 32)); }
  }
}

// Keys of shared memory that leave room beyond `want` (a power of two, as the sort needs).
inline uint32_t select_cap(uint32_t want)
{
  uint32_t cap = 64;
  while (cap < want + (want <= 1024 ? want / 2 : want / 4) || (want <= 160 && cap < 3 * want)) { cap <<= 1; }
  return cap;
}

}  // namespace cuvs_b200
