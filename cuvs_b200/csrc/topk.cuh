// Warp-level top-k on 64-bit keys.
//
// A candidate is one 64-bit key: (order-preserving image of the fp32 score) << 32 | 32-bit payload.
// Smaller key = better candidate; equal scores order by payload, so every selection in the search
// path is a total order and the results do not depend on scheduling.
//
// warp_topk<KPL> keeps the 32*KPL smallest keys seen so far, sorted ascending across the warp:
// position p lives in register a[p / 32] of lane p % 32.  A few candidates are inserted one by
// one (a warp-wide shift); many at once are merged as a sorted batch (bitonic networks).  Callers
// pre-filter against kth() so that, after warm-up, almost no candidate reaches either path.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace cuvs_b200 {

constexpr uint64_t kEmptyKey    = 0xFFFFFFFFFFFFFFFFull;
constexpr uint32_t kEmptyScore  = 0xFFFFFFFFu;
constexpr unsigned kFullMask    = 0xFFFFFFFFu;

// fp32 -> uint32 such that a < b  <=>  ord(a) < ord(b) for all non-NaN values.
__host__ __device__ __forceinline__ uint32_t float_to_ordered(float f)
{
#ifdef __CUDA_ARCH__
  uint32_t u = __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, 4);
#endif
  return u ^ ((u >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}
__host__ __device__ __forceinline__ float ordered_to_float(uint32_t o)
{
  uint32_t u = o ^ ((o >> 31) ? 0x80000000u : 0xFFFFFFFFu);
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}
__device__ __forceinline__ uint64_t make_key(float score, uint32_t payload)
{
  return (uint64_t(float_to_ordered(score)) << 32) | payload;
}

__device__ __forceinline__ uint64_t shfl_u64(uint64_t v, int src)
{
  uint32_t lo = __shfl_sync(kFullMask, uint32_t(v), src);
  uint32_t hi = __shfl_sync(kFullMask, uint32_t(v >> 32), src);
  return (uint64_t(hi) << 32) | lo;
}
__device__ __forceinline__ uint64_t shfl_up_u64(uint64_t v, int d)
{
  uint32_t lo = __shfl_up_sync(kFullMask, uint32_t(v), d);
  uint32_t hi = __shfl_up_sync(kFullMask, uint32_t(v >> 32), d);
  return (uint64_t(hi) << 32) | lo;
}

template <int KPL>
struct warp_topk {
  uint64_t a[KPL];
  uint64_t kth_;  // warp-uniform: key at position k-1
  int k_;

  __device__ __forceinline__ void init(int k)
  {
#pragma unroll
    for (int r = 0; r < KPL; r++) { a[r] = kEmptyKey; }
    kth_ = kEmptyKey;
    k_   = k;
  }
  __device__ __forceinline__ uint64_t kth() const { return kth_; }

  // Insert a warp-uniform key c with c < kth().
  __device__ __forceinline__ void insert(uint64_t c)
  {
    const int lane = threadIdx.x & 31;
    uint64_t carry = 0;  // key preceding this row (last key of the previous row)
#pragma unroll
    for (int r = 0; r < KPL; r++) {
      const uint64_t cur  = a[r];
      uint64_t prev       = shfl_up_u64(cur, 1);
      const uint64_t last = shfl_u64(cur, 31);
      if (lane == 0) { prev = carry; }
      a[r]  = (cur <= c) ? cur : (prev > c ? prev : c);
      carry = last;
    }
    refresh_kth();
  }
  __device__ __forceinline__ void refresh_kth()
  {
    const int pos = k_ - 1;
    uint64_t mine = a[0];
#pragma unroll
    for (int r = 1; r < KPL; r++) {
      if ((pos >> 5) == r) { mine = a[r]; }
    }
    kth_ = shfl_u64(mine, pos & 31);
  }

  // Bitonic merge step over the 32 lanes of one register: v holds a bitonic sequence -> ascending.
  static __device__ __forceinline__ uint64_t bitonic_finish(uint64_t v)
  {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
      const uint64_t o = shfl_u64(v, lane ^ j);
      v                = ((lane & j) == 0) ? (o < v ? o : v) : (o > v ? o : v);
    }
    return v;
  }

  // Merge a whole batch (one key per lane, kEmptyKey where there is none) into the queue: sort the
  // batch across the warp, then row by row split (row, batch) into the 32 smallest (stay in the
  // row) and the 32 largest (carried to the next row).
  __device__ __forceinline__ void merge_batch(uint64_t b)
  {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        const uint64_t o    = shfl_u64(b, lane ^ j);
        const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
        b                   = keep_min ? (o < b ? o : b) : (o > b ? o : b);
      }
    }
#pragma unroll
    for (int r = 0; r < KPL; r++) {
      const uint64_t rev = shfl_u64(b, 31 - lane);  // descending
      // ascending row against descending batch: element-wise min / max are both bitonic and hold
      // the 32 smallest / 32 largest keys of the union
      const uint64_t lo = a[r] < rev ? a[r] : rev;
      const uint64_t hi = a[r] < rev ? rev : a[r];
      a[r]              = bitonic_finish(lo);
      if (r + 1 < KPL) { b = bitonic_finish(hi); }
    }
    refresh_kth();
  }

  // Offer one key per lane (valid lanes only); keys >= kth() are dropped.
  __device__ __forceinline__ void offer(uint64_t key, bool valid)
  {
    const bool pass = valid && key < kth_;
    unsigned m      = __ballot_sync(kFullMask, pass);
    if (m == 0) { return; }
    if (__popc(m) > 2 + 2 * KPL) {
      merge_batch(pass ? key : kEmptyKey);
      return;
    }
    while (m) {
      int src = __ffs(m) - 1;
      m &= m - 1;
      uint64_t c = shfl_u64(key, src);
      if (c < kth_) { insert(c); }
    }
  }

  // Sorted position of register r on this lane.
  static __device__ __forceinline__ uint32_t position(int r) { return uint32_t(r) * 32u + (threadIdx.x & 31); }

  // Store the first n sorted keys to dst[0..n).
  __device__ __forceinline__ void store(uint64_t* dst, int n) const
  {
#pragma unroll
    for (int r = 0; r < KPL; r++) {
      const int p = int(position(r));
      if (p < n) { dst[p] = a[r]; }
    }
  }
};

// 64 values per warp, value e = r * 32 + lane in register a<r>: full bitonic sort.
template <typename T, bool Desc>
__device__ __forceinline__ void warp_sort64(T& a0, T& a1)
{
  const uint32_t lane = threadIdx.x & 31u;
  auto shfl = [](T v, int j) {
    if constexpr (sizeof(T) == 8) {
      const uint32_t lo = __shfl_xor_sync(kFullMask, uint32_t(v), j);
      const uint32_t hi = __shfl_xor_sync(kFullMask, uint32_t(uint64_t(v) >> 32), j);
      return T((uint64_t(hi) << 32) | lo);
    } else {
      return T(__shfl_xor_sync(kFullMask, v, j));
    }
  };
#pragma unroll
  for (uint32_t k = 2; k <= 64; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      if (j == 32) {  // k == 64: partner is the other register of the same lane, ascending block
        const T lo = a0 < a1 ? a0 : a1, hi = a0 < a1 ? a1 : a0;
        a0 = Desc ? hi : lo;
        a1 = Desc ? lo : hi;
      } else {
        const T o0 = shfl(a0, int(j)), o1 = shfl(a1, int(j));
        // value index e = r * 32 + lane; block direction from bit k of e (k == 64: one block)
        const bool up0 = ((lane & k) == 0) || k >= 32;         // r = 0: bit 5 of e is 0
        const bool up1 = k == 64 || (k < 32 && (lane & k) == 0);  // r = 1: bit 5 of e is 1
        const bool low = (lane & j) == 0;
        const bool min0 = (low == up0) != Desc, min1 = (low == up1) != Desc;
        a0 = min0 ? (a0 < o0 ? a0 : o0) : (a0 < o0 ? o0 : a0);
        a1 = min1 ? (a1 < o1 ? a1 : o1) : (a1 < o1 ? o1 : a1);
      }
    }
  }
}

// The digit (0..255) at which the running count of `hist` reaches `rem`, and how many of that digit are wanted; one whole
// warp calls it.  Fewer than `rem` in all: false, digit 255 and `left` = rem.
__device__ __forceinline__ bool find_digit(const uint32_t* hist, uint32_t rem, uint32_t& digit, uint32_t& left)
{
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t c[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    c[i] = hist[lane * 8u + i];
    sum += c[i];
  }
  uint32_t inc = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(kFullMask, inc, d);
    if (lane >= uint32_t(d)) { inc += o; }
  }
  const unsigned reach = __ballot_sync(kFullMask, inc >= rem);
  digit = 255u;
  left  = rem;
  if (reach == 0u) { return false; }
  const int src = __ffs(reach) - 1;
  uint32_t d = lane * 8u, r = rem - (inc - sum);
#pragma unroll
  for (int i = 0; i < 7; i++) {
    if (d == lane * 8u + i && c[i] < r) {
      r -= c[i];
      d++;
    }
  }
  digit = __shfl_sync(kFullMask, d, src);
  left  = __shfl_sync(kFullMask, r, src);
  return true;
}

}  // namespace cuvs_b200
