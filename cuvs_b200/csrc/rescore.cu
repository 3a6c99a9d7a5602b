// The exact pass of the fine search: bounds from the tensor-core pass (filter_scan.cu), exact scores of the
// rows that the bounds leave, top-k, ids and distances -- one launch.
//
// Bounds.  A unit (eight rows of a list) carries the smallest approximate score v of its rows.  With m >= |d| + |r|
// (L2; d the difference to the list centre, r a row's decoded residual) the score that the reference's
// arithmetic gives a row with approximation v lies in [lo(v), hi(v)]:
//   sqrt(t) in [sqrt(v - w) - e1 m - e0, sqrt(v + w) + e1 m + e0], w = kappa m^2 + e2   (t: the real distance)
//       e1: operands rounded to half precision; kappa: fp32 accumulation; e0, e2: half-precision underflow of components and of |r|^2
//       (rows far shorter than the longest, whose |r|^2 sets the scale)
//   lo = t_lo (1 - delta_lo) - eta,  hi = t_hi (1 + delta_hi) + eta
//       delta, eta: what rounding table entries and partial sums does to a sum of non-negative terms
// and for inner products t is within ip_gemm |q| rmax of v, the score within ip_lut |q| (rmax + |c|) + eta of t.
// Both ends grow with v, and units do not share rows: with V the k-th smallest value of a query's units, at least k
// rows have a score <= B, the largest hi(V) over its pairs.  A row whose lo exceeds B is not among the k best.  So:
// find V and B, score every row of the units with lo <= B exactly as the reference does (one fp32 chain per
// subspace, one rounding to the table type, entries summed in subspace order in the internal type), keep keys
// (score, sample index) at or below B, sort, emit the first k.  Results do not depend on how the bounds were
// computed.  After a time-out of the tensor-core pass (error word) every row is scored.  Units of rows that do not
// count (beyond the list, filtered out) carry a huge value; where too few others exist they may be listed, and
// their rows are dropped there.
//
// What bounds it: gathers from the fp32 codebook (one 8-byte look-up per code for two dimensions per subspace);
// it sits in shared memory once per CTA and thread groups of 32 to 256 take one query at a time.
#include "common.hpp"
#include "filter_scan.hpp"
#include "packed.cuh"
#include "scan.cuh"
#include "search_internal.hpp"
#include "tc_ptx.cuh"
#include "topk.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace cuvs::neighbors::ivf_pq {

using namespace cuvs_b200;

namespace {

__device__ __forceinline__ float sqrt_approx(float x)
{
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Bound of a query's norm from its square; below 1e-15 squares may have underflowed and products may: no bounds then.
__device__ __forceinline__ float query_norm(float square) { return square >= 1e-30f ? sqrtf(square) * 1.00001f : INFINITY; }

// lo of a unit's value v in a pair with norm `norm` (a NaN compares as "cannot be ruled out").
template <bool kIP>
__device__ __forceinline__ float unit_lo(const rescore_params& p, float v, float norm, float qn)
{
  if (v == INFINITY) { return -INFINITY; }  // a pair without bounds
  if constexpr (kIP) {
    if (!(qn * (p.rmax + norm) < p.sum_limit)) { return -INFINITY; }  // entries may be -inf
    return v + (p.cosine ? 1.0f : 0.0f) - (qn * (p.rmax * p.ip_gemm + (p.rmax + norm) * p.ip_lut) + p.eta);
  } else {
    if (norm < 0.0f && p.saturates) { return -INFINITY; }
    const float vp = fmaxf(v, 0.0f);
    const float m  = 2.0f * fabsf(norm) + sqrt_approx(vp);
    const float a  = fmaxf(sqrt_approx(fmaxf(vp - __fmaf_rn(p.kappa * m, m, p.e2), 0.0f)) - __fmaf_rn(p.e1, m, p.e0), 0.0f);
    return a * a * (1.0f - p.delta_lo) - p.eta;
  }
}
// hi of a value v, +inf where an entry or a sum may leave the range of its type.
template <bool kIP>
__device__ __forceinline__ float unit_hi(const rescore_params& p, float v, float norm, float qn)
{
  float hi;
  if constexpr (kIP) {
    hi = v + (p.cosine ? 1.0f : 0.0f) + (qn * (p.rmax * p.ip_gemm + (p.rmax + norm) * p.ip_lut) + p.eta);
    return qn * (p.rmax + norm) < p.sum_limit ? hi : INFINITY;
  } else {
    const float vp = fmaxf(v, 0.0f);
    const float m  = 2.0f * fabsf(norm) + sqrt_approx(vp);
    const float b  = sqrt_approx(vp + __fmaf_rn(p.kappa * m, m, p.e2)) + __fmaf_rn(p.e1, m, p.e0);
    hi             = b * b * (1.0f + p.delta_hi) + p.eta;
    return norm < 0.0f || !(hi < p.sum_limit) ? INFINITY : hi;
  }
}
// A value that every v with lo(v) <= bound stays below (L2: with x = sqrt(v) and A the distance that the bound allows,
// x <= A + e0 + sqrt(e2) + (e1 + sqrt(kappa)) (2 |d| + x), so 1.05 (A + e0 + sqrt(e2)) + 0.05 |d| exceeds x; one step from there).
template <bool kIP>
__device__ __forceinline__ float value_limit(const rescore_params& p, float bound, float norm, float qn)
{
  if constexpr (kIP) {
    const float w = qn * (p.rmax * p.ip_gemm + (p.rmax + norm) * p.ip_lut) + p.eta;
    const float x = bound - (p.cosine ? 1.0f : 0.0f) + w;
    return x + fabsf(x) * 1e-6f;
  } else {
    const float dn = fabsf(norm);
    const float A  = sqrt_approx((fmaxf(bound, 0.0f) + p.eta) / (1.0f - p.delta_lo)) * 1.00001f;
    const float m  = 2.0f * dn + 1.05f * (A + p.e0 + sqrt_approx(p.e2)) + 0.05f * dn;
    const float x  = A + __fmaf_rn(p.e1, m, p.e0);
    return (x * x + __fmaf_rn(p.kappa * m, m, p.e2)) * 1.00001f;
  }
}

// last entry of the ascending offsets off[0..n] that is <= x
__device__ __forceinline__ uint32_t find_offset(const uint32_t* off, uint32_t n, uint32_t x)
{
  uint32_t lo = 0, hi = n - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (off[mid] <= x) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  return lo;
}

// Shared memory of one thread group.
struct group_mem {
  uint64_t* buf;     // [cap] keys
  uint32_t* rows;    // [2 * threads, with row codes] rows of the query's groups, expanded from units and not scored yet
  uint2* list;       // [list_cap] {unit, value}: from the front the units among the k smallest, from the back the rest
  float* rq;         // [rot_dim]
  uint64_t* row;     // [P] arena row of the probe's list
  uint32_t* goff;    // [P + 1] groups before probe p
  uint32_t* soff;    // [P + 1] samples before probe p
  float* norm;       // [P]
  uint32_t* label;   // [P]
  uint32_t* word;    // [8]
};
constexpr uint32_t kListPerThread   = 4;    // list_cap = kListPerThread * threads of a group
constexpr uint32_t kMaxGroupThreads = 256;  // threads per query
// No bound: every score is kept but NaN (its bits order as 0xFFFFFFFF), which is no result, as in the scan (scan.cuh).  As a
// float a NaN itself, which nothing exceeds.
constexpr uint32_t kNoBound = 0xFFFFFFFEu;
enum { W_KEYS = 0, W_FRONT = 1, W_BACK = 2, W_BOUND = 3, W_VK = 4, W_VMAX = 5, W_NEXT = 6, W_ROWS = 7 };
__host__ __device__ inline uint32_t group_mem_bytes(uint32_t cap, uint32_t list_cap, uint32_t rows_cap, uint32_t n_probes, uint32_t rot_dim)
{
  return round_up<uint32_t>(cap * 8u + list_cap * 8u + rows_cap * 4u + n_probes * 8u + round_up<uint32_t>(rot_dim, 4u) * 4u +
                              (n_probes + 1u) * 8u + n_probes * 8u + 32u, 16u);
}

// One code's contribution in the reference's arithmetic, added to the running score.
template <int LutKind, bool OutHalf, bool IsIP>
__device__ __forceinline__ void add_entry(float entry, float& f, __half& h)
{
  if constexpr (!OutHalf) {
    if constexpr (LutKind == LUT_F32) {
      f = __fadd_rn(f, entry);
    } else if constexpr (LutKind == LUT_F16) {
      f = __fadd_rn(f, __half2float(__float2half_rn(entry)));
    } else {
      // fp8_to_float(fp8_encode(entry)) of a non-negative entry: clamped to the type's range, all but the three
      // upper mantissa bits replaced by half a step; a NaN (a query with NaN components) has code 0x7F, which reads 1.9375
      static_assert(!IsIP, "inner products do not take this path");
      constexpr float kMin = 1.0f / 32768.0f;
      const float kMax     = __uint_as_float(0x3F800000u - (15u << 23) + (255u << 20));  // smallest value of the last code
      const float a        = fminf(fmaxf(entry, kMin), kMax);
      const float read     = __uint_as_float((__float_as_uint(a) & 0xFFF00000u) | 0x00080000u);
      f = __fadd_rn(f, entry == entry ? read : 1.9375f);
    }
  } else {
    if constexpr (LutKind == LUT_F16) {
      h = __hadd(h, __float2half_rn(entry));
    } else {
      h = __hadd(h, fp8_to_half<IsIP>(fp8_encode<IsIP>(entry)));
    }
  }
}
template <bool IsIP>
__device__ __forceinline__ float component(float entry, float q, float c, float pq)
{
  if constexpr (!IsIP) {
    const float diff = __fsub_rn(__fsub_rn(q, c), pq);
    return __fmaf_rn(diff, diff, entry);
  } else {
    return __fmaf_rn(-q, pq, __fsub_rn(entry, __fmul_rn(c, q)));
  }
}

// Codebook loads at [address + constant]; the contents do not change, so they may move freely.
template <uint32_t kOff>
__device__ __forceinline__ void book_ld2(uint32_t a, float* b)
{
  asm("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(b[0]), "=f"(b[1]) : "r"(a), "n"(kOff));
}
template <uint32_t kOff>
__device__ __forceinline__ void book_ld4(uint32_t a, float* b)
{
  asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4+%5];" : "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]) : "r"(a), "n"(kOff));
}

// Exact score of one row: `src` its first 16-byte code piece (the next ones 512 bytes apart), c the rotated centre of
// its list.  Stops early (false) when a partial sum of non-negative terms has passed `bound`.
// kLen 2 or 4 with kBits 8 or 4: straight-line code over a piece; else the general loop.  kSmem: the codebook is in
// shared memory.
template <int LutKind, bool OutHalf, bool IsIP, int kLen, int kBits, bool kSmem>
__device__ __forceinline__ bool score_row(const rescore_params& p, const float* s_book, const float* rq, const float* c,
                                          const uint4* src, float bound, float& f, __half& h)
{
  const uint32_t book = p.book_size;
  uint4 nxt           = __ldg(src);
  uint32_t j          = 0;
  for (uint32_t piece = 0; piece < p.n_pieces; piece++) {
    uint4 v = nxt;
    if (piece + 1 < p.n_pieces) { nxt = __ldg(src + size_t(piece + 1) * 32u); }
    if constexpr (kBits != 0) {
      constexpr uint32_t kCodes = 128u / kBits, kBook = 1u << kBits;
      constexpr uint32_t kStep  = 4u / kLen;  // codes per four components
      const uint32_t w[4]  = {v.x, v.y, v.z, v.w};
      const uint32_t nj    = min(kCodes, p.pq_dim - j);
      const float* rq_j    = rq + j * kLen;
      const float* c_j     = c + j * kLen;
      const uint32_t book_a = kSmem ? smem_addr(s_book) + j * (kBook * kLen * 4u) : 0u;
      const float* book_g   = kSmem ? nullptr : p.pq_centers + size_t(j) * (kLen * kBook);
      auto step = [&](auto ic) {
        constexpr uint32_t i = decltype(ic)::value * kStep;
        const float4 qv = *reinterpret_cast<const float4*>(rq_j + i * kLen);
        const float4 cv = __ldg(reinterpret_cast<const float4*>(c_j + i * kLen));
        const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ca[4] = {cv.x, cv.y, cv.z, cv.w};
        static_for<kStep>([&](auto sc) {
          constexpr uint32_t s = decltype(sc)::value, n = i + s;
          const uint32_t code = kBits == 8 ? __byte_perm(w[n * kBits / 32u], 0u, 0x4440u + (n & 3u))
                                           : (w[n * kBits / 32u] >> ((n * kBits) & 31u)) & (kBook - 1u);
          float b[kLen];
          if constexpr (kSmem) {
            const uint32_t at = book_a + code * (kLen * 4u);
            if constexpr (kLen == 2) {
              book_ld2<n * kBook * kLen * 4u>(at, b);
            } else {
              book_ld4<n * kBook * kLen * 4u>(at, b);
            }
          } else {
#pragma unroll
            for (uint32_t kk = 0; kk < kLen; kk++) { b[kk] = __ldg(book_g + (n * kLen + kk) * kBook + code); }
          }
          float e = 0.0f;
#pragma unroll
          for (uint32_t kk = 0; kk < kLen; kk++) { e = component<IsIP>(e, qa[s * kLen + kk], ca[s * kLen + kk], b[kk]); }
          add_entry<LutKind, OutHalf, IsIP>(e, f, h);
        });
      };
      if (nj == kCodes) {
        static_for<kCodes / kStep>(step);
      } else {
        static_for<kCodes / kStep>([&](auto ic) {
          if (decltype(ic)::value * kStep < nj) { step(ic); }
        });
      }
      j += kCodes;
    } else {
      const uint32_t len = p.pq_len;
      const uint32_t nj  = min(128u / p.pq_bits, p.pq_dim - j);
      for (uint32_t i = 0; i < nj; i++, j++) {
        const uint32_t code = v.x & (book - 1u);
        v.x = __funnelshift_r(v.x, v.y, p.pq_bits);
        v.y = __funnelshift_r(v.y, v.z, p.pq_bits);
        v.z = __funnelshift_r(v.z, v.w, p.pq_bits);
        v.w >>= p.pq_bits;
        float e        = 0.0f;
        const float* b = kSmem ? s_book + (size_t(j) * book + code) * len : p.pq_centers + size_t(j) * len * book + code;
        for (uint32_t kk = 0; kk < len; kk++) {
          e = component<IsIP>(e, rq[j * len + kk], __ldg(c + j * len + kk), kSmem ? b[kk] : __ldg(b + kk * book));
        }
        add_entry<LutKind, OutHalf, IsIP>(e, f, h);
      }
    }
    if constexpr (!IsIP) {
      if ((OutHalf ? __half2float(h) : f) > bound) { return false; }
    }
  }
  return true;
}

template <int LutKind, bool OutHalf, bool IsIP, int kLen, int kBits, bool kSmem, bool kCodes>
__global__ void __launch_bounds__(1024, 1) rescore_kernel(const rescore_params p)
{
  extern __shared__ __align__(16) uint8_t smem[];
  const uint32_t gt = p.group_threads;
  const uint32_t g = threadIdx.x / gt, t = threadIdx.x % gt;
  const uint32_t warp = t >> 5, lane = t & 31u;
  const uint32_t P = p.n_probes, k = p.k;
  auto sync = [&]() {
    if (gt == 32u) {
      __syncwarp();
    } else {
      group_bar(int(g), int(gt));
    }
  };
  group_mem s;
  {
    uint8_t* b = smem + p.book_bytes + size_t(g) * p.group_bytes;
    s.buf      = reinterpret_cast<uint64_t*>(b);
    s.list     = reinterpret_cast<uint2*>(s.buf + p.cap);
    s.rows     = reinterpret_cast<uint32_t*>(s.list + p.list_cap);
    s.rq       = reinterpret_cast<float*>(s.rows + (kCodes ? 2u * gt : 0u));
    s.row      = reinterpret_cast<uint64_t*>(s.rq + round_up<uint32_t>(p.rot_dim, 4u));
    s.goff     = reinterpret_cast<uint32_t*>(s.row + P);
    s.soff     = s.goff + P + 1;
    s.norm     = reinterpret_cast<float*>(s.soff + P + 1);
    s.label    = reinterpret_cast<uint32_t*>(s.norm + P);
    s.word     = s.label + P;
  }
  // codebook of a subspace: global layout [len][book]; the copy in shared memory is [book][len]
  const float* s_book = reinterpret_cast<const float*>(smem);
  if constexpr (kSmem) {
    const uint32_t len = kLen > 0 ? uint32_t(kLen) : p.pq_len, book = p.book_size;
    float* dst         = reinterpret_cast<float*>(smem);
    const uint32_t n   = p.pq_dim * book * len;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      const uint32_t e = i % book, jk = i / book, kk = jk % len, j = jk / len;
      dst[(j * book + e) * len + kk] = __ldg(p.pq_centers + i);
    }
  }
  __syncthreads();
  chain_begin();  // (the codebook is the index's: copied while the kernel before this one ends)
  const bool all          = *p.error != 0u;
  if (all && blockIdx.x == 0 && threadIdx.x == 0) { count_timeout(p.timeouts); }
  const uint32_t n_groups = blockDim.x / gt;

  // the first query of a group by its number, the next ones from a counter (claimed one ahead)
  for (uint32_t q = blockIdx.x * n_groups + g; q < p.n_queries;) {
    sync();  // the previous query's shared memory is free
    if (t == 0) { s.word[W_NEXT] = gridDim.x * n_groups + atomicAdd(p.claim, 1u); }
    for (uint32_t i = t; i < p.rot_dim; i += gt) { s.rq[i] = __ldg(p.rot_q + size_t(q) * p.rot_dim + i); }
    for (uint32_t i = t; i < P; i += gt) {
      const uint32_t label = __ldg(p.probes + size_t(q) * P + i);
      const bool in        = label < p.n_lists;
      s.norm[i]            = __ldg(p.pair_norm + size_t(q) * P + i);
      s.goff[i + 1]        = __ldg(p.group_index + size_t(q) * P + i);
      s.soff[i + 1]        = __ldg(p.chunk_index + size_t(q) * P + i);
      s.label[i]           = in ? label : 0u;
      s.row[i]             = in ? __ldg(p.row_off + label) : 0u;
    }
    if (t == 0) {
      s.goff[0]       = 0;
      s.soff[0]       = 0;
      s.word[W_KEYS]  = 0;
      s.word[W_FRONT] = 0;
      s.word[W_BACK]  = 0;
      s.word[W_ROWS]  = 0;
      s.word[W_BOUND] = kNoBound;
      s.word[W_VK]    = __float_as_uint(-INFINITY);
      s.word[W_VMAX]  = __float_as_uint(INFINITY);
    }
    const uint32_t n_units4 = __ldg(p.group_index + size_t(q) * P + P - 1);
    const float4* units     = p.units + size_t(q) * p.max_groups;
    const auto* codes       = kCodes ? reinterpret_cast<const uint32_t*>(p.row_codes + size_t(q) * p.max_groups) : nullptr;
    const float row_step    = kCodes && IsIP ? p.row_step / __ldg(p.q_scale + q) : 0.0f;

    // ---- V: the k-th smallest value of the units (every thread contributes its two smallest) ----
    float best[2] = {INFINITY, INFINITY};
    if (!all) {
      auto take = [&](const float4& v) {
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int u = 0; u < 4; u++) {
          best[1] = fminf(best[1], fmaxf(best[0], x[u]));
          best[0] = fminf(best[0], x[u]);
        }
      };
      const float4 none = make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
      for (uint32_t gi = t; gi < n_units4; gi += 4 * gt) {
        float4 v[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) { v[i] = gi + i * gt < n_units4 ? __ldg(units + gi + i * gt) : none; }
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) { take(v[i]); }
      }
      if (gt > 32u) {
        uint32_t* top = reinterpret_cast<uint32_t*>(s.buf);  // 2 * gt <= 2 * cap words
        top[t]        = float_to_ordered(best[0]);
        top[gt + t]   = float_to_ordered(best[1]);
      }
    }
    sync();
    float qn = 0.0f;
    if (warp == 0 && !all) {
      if constexpr (IsIP) {
        for (uint32_t i = lane; i < p.rot_dim; i += 32) { qn = __fmaf_rn(s.rq[i], s.rq[i], qn); }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { qn += __shfl_xor_sync(kFullMask, qn, o); }
        qn = query_norm(qn);
      }
      // 22 bits of the k-th smallest, rounded up
      float vk = INFINITY;
      if (k <= 2u * gt) {
        uint32_t lo = 0;  // largest multiple of the step with fewer than k values below it
        auto bisect = [&](auto count) {
          for (int bit = 31; bit >= 10; bit--) {
            const uint32_t c = lo | (1u << bit);
            if (__reduce_add_sync(kFullMask, count(c)) < k) { lo = c; }
          }
        };
        if (gt == 32u) {
          bisect([&](uint32_t c) {
            return (float_to_ordered(best[0]) < c ? 1u : 0u) + (float_to_ordered(best[1]) < c ? 1u : 0u);
          });
        } else {
          const uint32_t* top = reinterpret_cast<const uint32_t*>(s.buf);
          uint32_t v[2 * kMaxGroupThreads / 32];
#pragma unroll
          for (uint32_t i = 0; i < 2 * kMaxGroupThreads / 32; i++) { v[i] = i * 16u < gt ? top[i * 32u + lane] : 0xFFFFFFFFu; }
          bisect([&](uint32_t c) {
            uint32_t n = 0;
#pragma unroll
            for (uint32_t i = 0; i < 2 * kMaxGroupThreads / 32; i++) { n += v[i] < c ? 1u : 0u; }
            return n;
          });
        }
        vk = ordered_to_float(lo | 0x3FFu);
      }
      // B: what k rows with values up to V can score at most; and the value that a unit must not exceed
      if (vk < INFINITY) {
        float hi = -INFINITY, vmax = -INFINITY;
        for (uint32_t i = lane; i < P; i += 32) {
          if (s.goff[i + 1] != s.goff[i]) { hi = fmaxf(hi, unit_hi<IsIP>(p, vk, s.norm[i], qn)); }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { hi = fmaxf(hi, __shfl_xor_sync(kFullMask, hi, o)); }
        if (hi < INFINITY) {
          for (uint32_t i = lane; i < P; i += 32) {
            if (s.goff[i + 1] != s.goff[i]) { vmax = fmaxf(vmax, value_limit<IsIP>(p, hi, s.norm[i], qn)); }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) { vmax = fmaxf(vmax, __shfl_xor_sync(kFullMask, vmax, o)); }
          if (lane == 0) {
            s.word[W_BOUND] = float_to_ordered(hi);
            s.word[W_VK]    = __float_as_uint(vk);
            s.word[W_VMAX]  = __float_as_uint(vmax);
          }
        }
      }
    }
    sync();
    if constexpr (IsIP) {
      if (gt > 32u) {  // (warp 0 has it)
        qn = 0.0f;
        for (uint32_t i = lane; i < p.rot_dim; i += 32) { qn = __fmaf_rn(s.rq[i], s.rq[i], qn); }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { qn += __shfl_xor_sync(kFullMask, qn, o); }
        qn = query_norm(qn);
      }
    }
    const float vk = __uint_as_float(s.word[W_VK]), vmax = __uint_as_float(s.word[W_VMAX]);

    // Sorts the first n2 (a power of two) keys of buf across the group.
    auto sort_keys = [&](uint32_t n2) {
      for (uint32_t size = 2; size <= n2; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
          for (uint32_t i = t; i < n2 / 2; i += gt) {
            const uint32_t lo = 2 * i - (i & (stride - 1));
            const uint32_t hi = lo + stride;
            const bool up     = (lo & size) == 0;
            const uint64_t a = s.buf[lo], b = s.buf[hi];
            if ((a > b) == up) {
              s.buf[lo] = b;
              s.buf[hi] = a;
            }
          }
          sync();
        }
      }
    };
    // Sort the keys, keep the k best; the bound follows.  Entered by the whole group after a barrier; `n_most`,
    // the same in every thread, is an upper bound of the number of keys.
    uint32_t n_most = 0;
    auto compact = [&]() {
      const uint32_t n = s.word[W_KEYS];
      n_most           = min(n, k);
      uint32_t n2      = 64;
      while (n2 < n) { n2 <<= 1; }
      for (uint32_t i = n + t; i < n2; i += gt) { s.buf[i] = kEmptyKey; }
      sync();
      sort_keys(n2);
      if (t == 0) {
        s.word[W_KEYS] = min(n, k);
        if (n >= k) { s.word[W_BOUND] = min(s.word[W_BOUND], uint32_t(s.buf[k - 1] >> 32)); }
      }
      sync();
    };
    // exact scores of the rows of the listed units [first, last).  With row codes, eight threads per unit leave the rows that the
    // bound does not rule out (a unit's value and the row's code bound the row's value from below) and a thread per row scores them:
    // some 350 rows per query of a 64-probe batch with 8-bit tables and k 100, whose whole units are 2,000.
    // Kernels of their own with and without codes, here and in step 1: one for both took 253 against 247 us without codes (777 x 40
    // pairs, half sums) and 1,204 against 1,187 with them (10,000 queries x 50,000 lists).
    auto score_listed = [&](uint32_t first, uint32_t last) {
      uint32_t n_rows = 0;  // rows waiting
      for (uint32_t u0 = first; u0 < last || n_rows > 0;) {
        uint32_t gi, pi, lrow;  // group of the query, its probe, row of that list
        bool valid;
        if constexpr (kCodes) {
          while (u0 < last && n_rows < gt) {
            const uint32_t ui = u0 + t / kUnitRows;
            bool live         = ui < last;
            const uint2 e     = s.list[live ? ui : first];
            gi                = e.x >> 2;
            pi                = find_offset(s.goff, P, gi);
            const uint32_t lr = (e.x & 3u) * kUnitRows + (lane & 7u);
            live              = live && (gi - s.goff[pi]) * 32u + lr < s.soff[pi + 1] - s.soff[pi];
            if (!all && live) {
              float value          = __uint_as_float(e.y);
              const float norm     = s.norm[pi];
              const uint32_t steps = (__ldg(codes + e.x) >> (4u * (lane & 7u))) & 15u;
              if (steps != 0u && value < INFINITY) { value = __fmaf_rd(float(steps), IsIP ? row_step : norm * norm * p.row_step, value); }
              live = !(unit_lo<IsIP>(p, value, norm, qn) > ordered_to_float(s.word[W_BOUND]));
            }
            u0 += gt / kUnitRows;
            const unsigned m = __ballot_sync(kFullMask, live);
            if (m != 0u) {
              uint32_t base = 0;
              if (lane == 0) { base = atomicAdd(&s.word[W_ROWS], uint32_t(__popc(m))); }
              base = __shfl_sync(kFullMask, base, 0);
              if (live) { s.rows[base + __popc(m & ((1u << lane) - 1u))] = (gi << 5) | lr; }
            }
            sync();
            n_rows = s.word[W_ROWS];
            sync();  // everybody has read it before anybody adds to it
          }
          if (n_rows == 0) { break; }
          // (the last ones; fewer than gt are left to wait)
          const uint32_t from = n_rows > gt ? n_rows - gt : 0u;
          valid               = from + t < n_rows;
          const uint32_t row_of = s.rows[valid ? from + t : from];
          n_rows              = from;
          gi                  = row_of >> 5;
          pi                  = find_offset(s.goff, P, gi);
          lrow                = (gi - s.goff[pi]) * 32u + (row_of & 31u);
          if (n_most + gt > p.cap) { compact(); }
        } else {
          if (n_most + gt > p.cap) { compact(); }
          const uint32_t ui = u0 + t / kUnitRows;
          valid             = ui < last;
          const uint2 e     = s.list[valid ? ui : first];
          gi                = e.x >> 2;
          pi                = find_offset(s.goff, P, gi);
          lrow              = (gi - s.goff[pi]) * 32u + (e.x & 3u) * kUnitRows + (lane & 7u);
          valid             = valid && lrow < s.soff[pi + 1] - s.soff[pi];
          if (!all) { valid = valid && !(unit_lo<IsIP>(p, __uint_as_float(e.y), s.norm[pi], qn) > ordered_to_float(s.word[W_BOUND])); }
          u0 += gt / kUnitRows;
        }
        n_most += gt;
        const uint64_t row  = s.row[pi] + lrow;
        const uint32_t b_ord = s.word[W_BOUND];
        const float bound    = ordered_to_float(b_ord);  // NaN: none
        if (kCodes && t == 0) { s.word[W_ROWS] = n_rows; }
        float f  = 0.0f;
        __half h = __ushort_as_half(0);
        if (valid) {
          const uint4* src = reinterpret_cast<const uint4*>(p.codes + ((row & ~uint64_t(31)) * p.n_pieces) * 16u) + (row & 31u);
          const float* c   = p.centers + size_t(s.label[pi]) * p.rot_dim;
          valid = score_row<LutKind, OutHalf, IsIP, kLen, kBits, kSmem>(p, s_book, s.rq, c, src, bound, f, h);
        }
        float score;
        if constexpr (!OutHalf) {
          score = p.cosine ? __fadd_rn(f, 1.0f) : f;
        } else {
          if (p.cosine) { h = __hadd(h, __float2half(1.0f)); }
          score = __half2float(h);
        }
        const uint32_t ord = float_to_ordered(score);
        bool keep          = valid && ord <= b_ord;
        if (keep && p.filter_bits != nullptr) {
          const int64_t id = p.ids[row];
          keep = id >= 0 && uint64_t(id) < p.filter_nbits && ((p.filter_bits[id >> 5] >> (id & 31)) & 1u);
        }
        const unsigned m = __ballot_sync(kFullMask, keep);
        if (m != 0u) {
          uint32_t base = 0;
          if (lane == 0) { base = atomicAdd(&s.word[W_KEYS], uint32_t(__popc(m))); }
          base = __shfl_sync(kFullMask, base, 0);
          if (keep) { s.buf[base + __popc(m & ((1u << lane) - 1u))] = (uint64_t(ord) << 32) | (s.soff[pi] + lrow); }
        }
        sync();
      }
    };

    // ---- list the units up to that value, score their rows ----
    // Units among the k smallest go to the front of the list and are scored first: with wide bounds (8-bit tables,
    // half-precision sums) their exact scores then tighten the bound for the others.
    uint32_t chunk = n_units4;
    for (uint32_t c0 = 0; c0 < n_units4;) {
      const uint32_t c1 = min(n_units4, c0 + chunk);
      auto take = [&](uint32_t gi, const float4& v) {
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
          // (negated: a NaN is taken; +inf stands for a pair without bounds)
          if (all || !(x[u] > vmax) || x[u] == INFINITY) {
            const bool front    = !all && x[u] <= vk;  // (after a time-out the values are anything)
            const uint32_t slot = atomicAdd(&s.word[front ? W_FRONT : W_BACK], 1u);
            if (slot < p.list_cap) {
              s.list[front ? slot : p.list_cap - 1u - slot] = make_uint2((gi << 2) | u, __float_as_uint(x[u]));
            }
          }
        }
      };
      for (uint32_t gi = c0 + t; gi < c1; gi += 4 * gt) {
        float4 v[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
          if (gi + i * gt < c1) { v[i] = __ldg(units + gi + i * gt); }
        }
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
          if (gi + i * gt < c1 && (all || !(min3(v[i].x, v[i].y, fminf(v[i].z, v[i].w)) > vmax) ||
                                   fmaxf(fmaxf(v[i].x, v[i].y), fmaxf(v[i].z, v[i].w)) == INFINITY)) {
            take(gi + i * gt, v[i]);
          }
        }
      }
      sync();
      const uint32_t n_front = s.word[W_FRONT], n_back = s.word[W_BACK];
      sync();  // everybody has read them before anybody resets them
      if (t == 0) {
        s.word[W_FRONT] = 0;
        s.word[W_BACK]  = 0;
      }
      if (n_front + n_back > p.list_cap) {
        chunk = p.list_cap / 4u;  // cannot overflow
        sync();
        continue;
      }
      uint32_t first = 0, last = n_front;
      for (uint32_t phase = 0;; phase++) {
        score_listed(first, last);
        if (phase == 1) { break; }
        first = p.list_cap - n_back;
        last  = p.list_cap;
        if (p.sharpen && n_back > gt / kUnitRows && n_front != 0u) {
          // what the tightened bound still leaves of the rest moves to the front
          compact();
          const float bound = ordered_to_float(s.word[W_BOUND]);
          uint2 mine[kListPerThread];
          uint32_t take = 0;
#pragma unroll
          for (uint32_t i = 0; i < kListPerThread; i++) {
            const uint32_t at = first + i * gt + t;
            mine[i]           = make_uint2(0u, 0u);
            if (at < p.list_cap) {
              mine[i]           = s.list[at];
              const uint32_t pi = find_offset(s.goff, P, mine[i].x >> 2);
              if (!(unit_lo<IsIP>(p, __uint_as_float(mine[i].y), s.norm[pi], qn) > bound)) { take |= 1u << i; }
            }
          }
          sync();
          uint32_t to = take != 0u ? atomicAdd(&s.word[W_FRONT], uint32_t(__popc(take))) : 0u;
#pragma unroll
          for (uint32_t i = 0; i < kListPerThread; i++) {
            if ((take >> i) & 1u) { s.list[to++] = mine[i]; }
          }
          sync();
          first = 0;
          last  = s.word[W_FRONT];
          sync();
          if (t == 0) { s.word[W_FRONT] = 0; }
        }
      }
      sync();
      c0 = c1;
    }

    // ---- the k best: sort, translate, store ----
    const uint32_t n_keys = s.word[W_KEYS];
    auto store = [&](uint32_t i, uint64_t key) {
      int64_t id  = kOutOfBoundsRecord;
      float score = INFINITY;
      if (key != kEmptyKey) {
        const uint32_t sample = uint32_t(key);
        score                 = ordered_to_float(uint32_t(key >> 32));
        const uint32_t pi     = find_offset(s.soff, P, sample);
        id                    = __ldg(p.ids + s.row[pi] + (sample - s.soff[pi]));
      }
      p.neighbors[size_t(q) * k + i] = id;
      p.distances[size_t(q) * k + i] = postprocess_distance(score, p.metric, p.post_scale);
    };
    if (n_keys <= 64u && k <= 64u) {
      if (warp == 0) {
        uint64_t a0 = lane < n_keys ? s.buf[lane] : kEmptyKey, a1 = lane + 32u < n_keys ? s.buf[lane + 32u] : kEmptyKey;
        warp_sort64<uint64_t, false>(a0, a1);
        if (lane < k) { store(lane, a0); }
        if (lane + 32u < k) { store(lane + 32u, a1); }
      }
    } else {
      uint32_t n2 = 64;
      while (n2 < n_keys) { n2 <<= 1; }
      for (uint32_t i = n_keys + t; i < n2; i += gt) { s.buf[i] = kEmptyKey; }
      sync();
      sort_keys(n2);
      for (uint32_t i = t; i < k; i += gt) { store(i, i < n2 ? s.buf[i] : kEmptyKey); }
    }
    q = s.word[W_NEXT];
  }
}

}  // namespace

void launch_rescore(const rescore_params& p, int lut_kind, bool out_half, bool is_ip, int grid, size_t smem,
                    cudaStream_t stream)
{
  auto go = [&](auto kernel) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    launch_chained(kernel, grid, int(p.groups * p.group_threads), smem, stream, p);
    CUDA_TRY(cudaGetLastError());
  };
  // straight-line code for 8- and 4-bit codes of two or four components (whole 16-byte groups of components)
  const bool whole = p.rot_dim % 4 == 0;
  auto shape_home = [&](auto lut, auto oh, auto ip, auto smem_book, auto codes) {
    constexpr int kL   = decltype(lut)::value;
    constexpr bool kOH = decltype(oh)::value, kIP = decltype(ip)::value, kS = decltype(smem_book)::value, kC = decltype(codes)::value;
    if (whole && p.pq_bits == 8 && p.pq_len == 2) {
      go(rescore_kernel<kL, kOH, kIP, 2, 8, kS, kC>);
    } else if (whole && p.pq_bits == 8 && p.pq_len == 4) {
      go(rescore_kernel<kL, kOH, kIP, 4, 8, kS, kC>);
    } else if (whole && p.pq_bits == 4 && p.pq_len == 2) {
      go(rescore_kernel<kL, kOH, kIP, 2, 4, kS, kC>);
    } else {
      go(rescore_kernel<kL, kOH, kIP, 0, 0, kS, kC>);
    }
  };
  auto shape = [&](auto lut, auto oh, auto ip) {
    auto home = [&](auto codes) {
      if (p.book_bytes != 0u) {
        shape_home(lut, oh, ip, std::true_type{}, codes);
      } else {
        shape_home(lut, oh, ip, std::false_type{}, codes);
      }
    };
    if (p.row_codes == nullptr) {
      home(std::false_type{});
    } else {
      home(std::true_type{});
    }
  };
  using std::bool_constant;
  using std::integral_constant;
  if (is_ip) {
    if (lut_kind == LUT_F32) {
      shape(integral_constant<int, LUT_F32>{}, bool_constant<false>{}, bool_constant<true>{});
    } else {
      shape(integral_constant<int, LUT_F16>{}, bool_constant<false>{}, bool_constant<true>{});
    }
  } else if (out_half) {
    if (lut_kind == LUT_F16) {
      shape(integral_constant<int, LUT_F16>{}, bool_constant<true>{}, bool_constant<false>{});
    } else {
      shape(integral_constant<int, LUT_FP8>{}, bool_constant<true>{}, bool_constant<false>{});
    }
  } else if (lut_kind == LUT_F32) {
    shape(integral_constant<int, LUT_F32>{}, bool_constant<false>{}, bool_constant<false>{});
  } else if (lut_kind == LUT_F16) {
    shape(integral_constant<int, LUT_F16>{}, bool_constant<false>{}, bool_constant<false>{});
  } else {
    shape(integral_constant<int, LUT_FP8>{}, bool_constant<false>{}, bool_constant<false>{});
  }
}

filter_plan plan_filter(const raft::resources& res, const index<int64_t>& idx, int lut_kind, bool out_half, bool is_ip,
                        uint32_t k, uint32_t n_probes, uint32_t n_queries, bool row_codes)
{
  filter_plan plan{};
  // Where the bounds say too little the look-up-table scan is the better one: signed sums of coarse entries
  // (inner product with 8-bit tables or half-precision sums) cancel, so their rounding is not small against the
  // differences between scores.  Codebooks per list have no shared operand.
  if (idx.codebook_kind() != codebook_gen::PER_SUBSPACE || (is_ip && (lut_kind == LUT_FP8 || out_half))) { return plan; }
  // The error model counts rounding relative to the terms: codewords whose squares, or products with them, may underflow or
  // overflow fp32 are left to the look-up tables.
  const float rmax = idx.filter_model().rmax;
  if (idx.filter_model().comp_max != 0.0f && !(rmax >= 1e-15f && rmax <= 1e15f)) { return plan; }
  if (k > 128) { return plan; }
  const size_t limit  = size_t(res.smem_optin) - 1024;
  const auto& m       = idx.filter_model();
  const size_t fixed  = m.book.size() * 2 + 256 + 1024;
  const size_t kStageBytes = 48 * 1024;
  uint32_t stages     = 4;
  while (stages > 1 && fixed + stages * kStageBytes > limit) { stages--; }
  if (stages < 2 || fixed + stages * kStageBytes > limit) { return plan; }
  plan.n_stages    = stages;
  plan.filter_smem = fixed + stages * kStageBytes;
  // Threads per query: enough that a thread sees at most about 16 groups of units and that keys and candidate rows
  // spread over the warps; more when there are too few queries to fill the chip.
  const uint64_t avg_groups = ceildiv<uint64_t>(uint64_t(idx.size()) * n_probes, uint64_t(idx.n_lists()) * 32) + n_probes / 2;
  uint32_t gt = k <= 16 ? 32 : (k <= 64 ? 64 : 128);
  while (gt < kMaxGroupThreads && avg_groups > 16ull * gt) { gt <<= 1; }
  while (gt < kMaxGroupThreads && uint64_t(n_queries) * gt < uint64_t(res.sm_count) * 1024) { gt <<= 1; }
  const size_t book = round_up<size_t>(idx.pq_centers_size() * 4, 16);
  const bool few    = n_queries <= uint32_t(res.sm_count);
  uint32_t cap = 128;
  while (cap < 2 * k + gt) { cap <<= 1; }
  plan.cap           = cap;
  plan.list_cap      = kListPerThread * gt;
  plan.group_threads = gt;
  plan.group_bytes   = group_mem_bytes(cap, plan.list_cap, row_codes ? 2 * gt : 0, n_probes, idx.rot_dim());
  // As many groups per CTA as threads and shared memory allow, beside the codebook in shared memory where that leaves at
  // least half of the threads; with fewer queries than SMs, one query per CTA reading the codebook through the caches
  // (a copy would cost more than the look-ups it serves).
  auto groups_in = [&](size_t room) { return uint32_t(std::min<size_t>(1024 / gt, room / plan.group_bytes)); };
  uint32_t groups = !few && book < limit ? groups_in(limit - book) : 0;
  if (groups > 0 && groups * gt >= 512) {
    plan.book_bytes = uint32_t(book);
  } else {
    groups          = few ? std::min<uint32_t>(1, groups_in(limit)) : groups_in(limit);
    plan.book_bytes = 0;
  }
  if (groups == 0) { return plan; }
  groups            = std::min<uint32_t>(groups, std::max<uint32_t>(1, ceildiv(n_queries, uint32_t(res.sm_count))));
  plan.groups       = groups;
  plan.rescore_smem = plan.book_bytes + size_t(groups) * plan.group_bytes;
  plan.use          = true;
  return plan;
}

}  // namespace cuvs::neighbors::ivf_pq
