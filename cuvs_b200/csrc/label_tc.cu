// Nearest list of many rows on the tensor cores, exact: labels[i] = argmin over lists l of (score, l) with the score's
// defining fp32 chain (coarse.cu) -- what k-means steps, extend and transform need.
//
// Reference: kmeans_balanced::predict (cpp/src/cluster/detail/kmeans_balanced.cuh:100-160).
//
// The probe selection of coarse_tc.cu with n_probes = 1 answers the same question, but keeps eight keys of every 64
// lists in global memory and finishes with a block per row: 12 of 23 ms for 1 M rows x 16,384 lists.  For the nearest list
// alone, one maximum per 64 lists is enough:
//   1. operands in half precision (the same 11 significant bits as TF32 at twice the rate), relative to the mean m of the
//      centres: rows (q - m) 2^e, lists (c - m) / cp, with cp the power of two above the largest |c - m|; two more
//      columns carry |c|^2 / 2 - m.c + |m|^2 / 2, so that the accumulator holds F (score + a constant of the row), F = 2^e /
//      cp, within (-0.5, 0.5).  `eps` of a row bounds how far that is from the exact value: the measured norms of what
//      rounding took from row and lists, accumulation, the defining chain's own rounding, the rounding of the keys.
//      Up to 190 dimensions (where both fit shared memory beside three list stages) the row operand comes as two halfs, hi +
//      lo, and two products: its rounding drops out of eps.  The second product is on the critical path: at 96 dimensions the
//      MMA thread issues the 14 products of a tile in about 3,400 clocks, the epilogue needs 2,200.
//   2. label_tc_kernel: a persistent CTA takes a tile of 128 rows against all (or a share) of the lists, 256 at a time.
//      Per row and unit of 64 lists the epilogue finds the largest value as a packed key (value in fixed point, low bits
//      the column: see coarse_tc.cu) and the second largest; across the tiles it keeps, per row and column quarter, the
//      units with the four largest.  Three float additions and three min / max per value; the issue of the MMAs bounds the
//      kernel.
//   3. label_finish_kernel: units within 2 eps of the largest value are looked at.  One such unit whose second value is
//      outside: that is the label.  Several: their lists are rescored with the defining chain.  Units whose second value
//      is inside too go to label_units_kernel, which rescores all 64 lists of them.  If the fourth unit kept is inside,
//      a fifth might be: the row is redone exactly over all lists.
// Every wait is bounded: on a time-out the kernel raises the error word and returns, and all rows are redone.
#include "search_internal.hpp"
#include "tc_ptx.cuh"
#include "topk.cuh"

#include <algorithm>

namespace cuvs::neighbors::ivf_pq {

using namespace cuvs_b200;

namespace {

constexpr uint32_t kRows = 128, kLists = 256, kBlockK = 64, kUnit = 64, kKeep = 4;
constexpr uint32_t kEpiWarps = 16;
constexpr uint32_t kThreads  = (2 + kEpiWarps) * 32;  // warp 0 TMA, warp 1 MMA, warps 2..17 epilogue
constexpr uint32_t kABlock = kRows * kBlockK * 2, kBBlock = kLists * kBlockK * 2;  // 16 and 32 KB
constexpr uint32_t kMaxStages = 6;
constexpr uint32_t kRoom      = 6 * kBBlock;          // shared memory for operands: 192 KB

// Model: words {bits of the largest max(|c - m|^2, 2 |norm column|), of the largest |c|^2 or norm column, of the largest
// squared norm of what rounding took from a list}, the sum of the centres at kMeanAt, the list operand at operand_at(dim).
constexpr uint32_t kMeanAt = 256;
__host__ __device__ __forceinline__ size_t operand_at(uint32_t dim) { return kMeanAt + round_up<size_t>(size_t(dim) * 4, 256); }

__global__ void center_sum_kernel(const float* __restrict__ centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                                  float* __restrict__ sum)
{
  // block (32 dimensions, 8 list lanes); blockIdx.y: a share of the lists
  __shared__ float s_part[8][33];
  const uint32_t k = blockIdx.x * 32u + threadIdx.x;
  float acc        = 0.0f;
  if (k < dim) {
#pragma unroll 8
    for (uint32_t l = blockIdx.y * 8u + threadIdx.y; l < n_lists; l += gridDim.y * 8u) { acc += centers[size_t(l) * dim_ext + k]; }
  }
  s_part[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && k < dim) {
#pragma unroll
    for (uint32_t y = 1; y < 8; y++) { acc += s_part[y][threadIdx.x]; }
    atomicAdd(sum + k, acc);
  }
}

// |c|^2 / 2 - m.c + |m|^2 / 2 of a list, by one warp (any m gives valid results: it only has to be the same everywhere)
__device__ __forceinline__ void list_norms(const float* c, const float* sum, float inv_n, uint32_t dim, float& cc, float& dd, double& norm)
{
  const uint32_t lane = threadIdx.x & 31u;
  double mc = 0.0, mm = 0.0;
  cc = dd = 0.0f;
  for (uint32_t k = lane; k < dim; k += 32) {
    const float m = sum[k] * inv_n, v = c[k], d = v - m;
    mc += double(m) * v;
    mm += double(m) * m;
    cc = __fmaf_rn(v, v, cc);
    dd = __fmaf_rn(d, d, dd);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mc += __shfl_xor_sync(kFullMask, mc, o);
    mm += __shfl_xor_sync(kFullMask, mm, o);
    cc += __shfl_xor_sync(kFullMask, cc, o);
    dd += __shfl_xor_sync(kFullMask, dd, o);
  }
  norm = 0.5 * double(c[dim]) - mc + 0.5 * mm;
}

__global__ void center_stats_kernel(const float* __restrict__ centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                                    const float* __restrict__ sum, uint32_t* __restrict__ words)
{
  const uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (l >= n_lists) { return; }
  const float* c = centers + size_t(l) * dim_ext;
  float cc, dd;
  double norm;
  list_norms(c, sum, 1.0f / float(n_lists), dim, cc, dd, norm);
  if ((threadIdx.x & 31u) == 0) {
    atomicMax(words, __float_as_uint(fmaxf(dd, 2.0f * fabsf(float(norm))) * 1.0001f));
    atomicMax(words + 1, __float_as_uint(fmaxf(cc, fabsf(c[dim])) * 1.0001f));
  }
}

// cp = a power of two above sqrt(largest squared norm); bn = that norm / cp, infinite where no bound holds
__device__ __forceinline__ float center_scale(const uint32_t* words, float& bn)
{
  const float nrm = sqrtf(__uint_as_float(__ldg(words)));
  const int E     = int((__float_as_uint(nrm) >> 23) & 0xFFu);   // nrm in [2^(E-127), 2^(E-126))
  const bool fine = E >= 64 && E <= 190;
  const float cp  = fine ? __uint_as_float(uint32_t(E + 1) << 23) : 1.0f;
  bn              = fine ? nrm / cp * 1.0001f : INFINITY;
  return cp;
}

// One warp per list.
__global__ void center_operand_kernel(const float* __restrict__ centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                                      uint32_t width, const float* __restrict__ sum, uint32_t* __restrict__ words,
                                      __half* __restrict__ out)
{
  const uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
  if (l >= n_lists) { return; }
  float bn, cc, dd;
  const float inv   = 1.0f / center_scale(words, bn);
  const float inv_n = 1.0f / float(n_lists);
  const float* c    = centers + size_t(l) * dim_ext;
  double norm;
  list_norms(c, sum, inv_n, dim, cc, dd, norm);
  const float nf = float(norm * double(inv) * double(inv));
  const float hi = __half2float(__float2half_rn(nf));
  __half* dst    = out + size_t(l) * width;
  float lost     = 0.0f;
  for (uint32_t k = lane; k < width; k += 32) {
    const float v  = k < dim ? (c[k] - sum[k] * inv_n) * inv : (k == dim ? hi : (k == dim + 1 ? nf - hi : 0.0f));
    const __half h = __float2half_rn(v);
    dst[k]         = h;
    if (k < dim) {
      const float d = v - __half2float(h);
      lost          = __fmaf_rn(d, d, lost);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { lost += __shfl_xor_sync(kFullMask, lost, o); }
  if (lane == 0) { atomicMax(words + 2, __float_as_uint(lost * 1.001f)); }
}

// One warp per row: the operand row (kSplit: hi, then lo, `width` halfs each), and eps (infinite: redo the row).
template <bool kSplit>
__global__ void row_operand_kernel(const float* __restrict__ x, uint32_t n_rows, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                                   uint32_t width, const float* __restrict__ sum, const uint32_t* __restrict__ words,
                                   __half* __restrict__ out, float* __restrict__ eps)
{
  const uint32_t r    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  if (r >= n_rows) { return; }
  float bn;
  const float cp    = center_scale(words, bn);
  const float inv_n = 1.0f / float(n_lists);
  const float* q    = x + size_t(r) * dim_ext;
  float ss = 0.0f, qq = 0.0f;
  for (uint32_t k = lane; k < dim; k += 32) {
    const float v = q[k], d = v - sum[k] * inv_n;
    ss = __fmaf_rn(d, d, ss);
    qq = __fmaf_rn(v, v, qq);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ss += __shfl_xor_sync(kFullMask, ss, o);
    qq += __shfl_xor_sync(kFullMask, qq, o);
  }
  const float dn = sqrtf(ss) * 1.0001f, qn = sqrtf(qq) * 1.0001f;
  // 2^e (|q - m| + cp / 2) in [0.25, 0.5)
  const float b     = (dn + 0.5f * cp) * 1.01f;
  const int E       = int((__float_as_uint(b) >> 23) & 0xFFu);
  const bool fine   = E >= 2 && E <= 250;
  const float scale = fine ? __uint_as_float(uint32_t(252 - E) << 23) : 0.0f;
  const float a     = scale * cp;
  __half2* dst      = reinterpret_cast<__half2*>(out + size_t(r) * width * (kSplit ? 2u : 1u));
  float lost        = 0.0f;
  for (uint32_t k2 = lane; k2 < width / 2; k2 += 32) {
    float v[2];
#pragma unroll
    for (uint32_t e = 0; e < 2; e++) {
      const uint32_t k = 2 * k2 + e;
      v[e]             = k < dim ? (q[k] - sum[k] * inv_n) * scale : (k < dim + 2 ? -a : 0.0f);
    }
    const __half2 h = __floats2half2_rn(v[0], v[1]);
    float2 f        = __half22float2(h);
    dst[k2]         = h;
    f               = make_float2(v[0] - f.x, v[1] - f.y);
    if constexpr (kSplit) {
      const __half2 lo     = __floats2half2_rn(f.x, f.y);
      const float2 g       = __half22float2(lo);
      dst[width / 2 + k2] = lo;
      f                    = make_float2(f.x - g.x, f.y - g.y);
    }
    lost = __fmaf_rn(f.x, f.x, lost);
    lost = __fmaf_rn(f.y, f.y, lost);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { lost += __shfl_xor_sync(kFullMask, lost, o); }
  if (lane == 0) {
    const float an = dn * scale, w = float(width);
    const float bl = sqrtf(__uint_as_float(__ldg(words + 2))), cn = sqrtf(__uint_as_float(__ldg(words + 1)));
    const float orig = qn * cn + 0.5f * cn * cn;  // bounds every partial sum of the defining chain
    float e = (sqrtf(lost) * (bn + bl) + an * bl) * 1.01f       // rounding of the operands
              + (w + 24.0f) * (kSplit ? 1.8e-7f : 1.2e-7f)      // accumulation of sums below 0.5 by the tensor core
              + (scale / cp) * orig * (float(dim_ext) + 4.0f) * 1.2e-7f  // the defining chain, and q - m
              + 8.2e-6f;                                        // norm columns, keys
    if (!fine || !(a >= 6.2e-5f)) { e = INFINITY; }
    eps[r] = e;
  }
}

struct label_params {
  uint32_t n_rows, n_lists, k_steps /* of 16 halfs */, k_blocks;
  uint32_t n_tiles, tiles_per_split, n_items, splits;
  uint32_t a_resident, n_stages, products, width;
  uint4* keys;       // [splits, n_rows, 4] largest keys of a column quarter
  uint4* seconds;    // second largest keys of their units
  uint4* lists;      // their lists
  uint32_t* error;
  uint32_t spin_limit, skip_kb;  // tc_wait_limits
};

__global__ void __launch_bounds__(kThreads, 1)
label_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const label_params p)
{
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_a  = smem_u32(smem_raw);
  const uint32_t base_a = (raw_a + 1023u) & ~1023u;
  uint8_t* base_p       = smem_raw + (base_a - raw_a);
  uint64_t* bars        = reinterpret_cast<uint64_t*>(base_p + kRoom);
  const uint32_t bar_full   = smem_u32(bars);
  const uint32_t bar_empty  = bar_full + kMaxStages * 8;
  const uint32_t bar_tfull  = bar_empty + kMaxStages * 8;
  const uint32_t bar_tempty = bar_tfull + 2 * 8;
  const uint32_t bar_afull  = bar_tempty + 2 * 8;
  const uint32_t bar_aempty = bar_afull + 8;
  uint32_t* tmem_slot       = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 6);
  // [row tile, when resident][stages: list block, then row block when not]
  const uint32_t a_bytes    = p.a_resident ? p.products * p.k_blocks * kABlock : 0u;
  const uint32_t stage_size = kBBlock + (p.a_resident ? 0u : kABlock);
  const uint32_t stage_base = base_a + a_bytes;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < p.n_stages; s++) {
      mbar_init(bar_full + s * 8, 1);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (uint32_t a = 0; a < 2; a++) {
      mbar_init(bar_tfull + a * 8, 1);
      mbar_init(bar_tempty + a * 8, kEpiWarps);
    }
    mbar_init(bar_afull, 1);
    mbar_init(bar_aempty, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  bool ok = true;
  // the list tiles of an item
  auto tiles_of = [&](uint32_t item, uint32_t& t0, uint32_t& t1) {
    const uint32_t s = item % p.splits;
    t0               = s * p.tiles_per_split;
    t1               = min(p.n_tiles, t0 + p.tiles_per_split);
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t stage = 0, phase = 0, n_a = 0;
      for (uint32_t item = blockIdx.x; ok && item < p.n_items; item += gridDim.x) {
        const int row0 = int((item / p.splits) * kRows);
        uint32_t t0, t1;
        tiles_of(item, t0, t1);
        if (p.a_resident) {
          if (!mbar_wait(bar_aempty, (n_a & 1u) ^ 1u, p.spin_limit)) {
            ok = false;
            break;
          }
          n_a++;
          mbar_arrive_expect_tx(bar_afull, a_bytes);
          for (uint32_t i = 0; i < p.products; i++) {
            for (uint32_t kb = 0; kb < p.k_blocks; kb++) {
              tma_load_2d(base_a + (i * p.k_blocks + kb) * kABlock, &map_a, bar_afull, int(i * p.width + kb * kBlockK), row0);
            }
          }
        }
        for (uint32_t t = t0; ok && t < t1; t++) {
          for (uint32_t kb = 0; kb < p.k_blocks; kb++) {
            if (!mbar_wait(bar_empty + stage * 8, phase ^ 1u, p.spin_limit)) {
              ok = false;
              break;
            }
            const uint32_t dst = stage_base + stage * stage_size, bar = bar_full + stage * 8;
            // (test only: a block that never comes, so that the wait for it runs out)
            if (kb + 1 != p.skip_kb || t != t0 || item != blockIdx.x) {
              mbar_arrive_expect_tx(bar, stage_size);
              tma_load_2d(dst, &map_b, bar, int(kb * kBlockK), int(t * kLists));
              if (!p.a_resident) { tma_load_2d(dst + kBBlock, &map_a, bar, int(kb * kBlockK), row0); }
            }
            if (++stage == p.n_stages) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      // fp32 accumulate, half x half, both K-major, M = 128, N = 256
      constexpr uint32_t idesc = (1u << 4) | ((kLists >> 3) << 17) | ((kRows >> 4) << 24);
      uint32_t stage = 0, phase = 0, n_a = 0, it = 0;
      for (uint32_t item = blockIdx.x; ok && item < p.n_items; item += gridDim.x) {
        uint32_t t0, t1;
        tiles_of(item, t0, t1);
        if (p.a_resident) {
          if (!mbar_wait(bar_afull, n_a & 1u, p.spin_limit)) {
            ok = false;
            break;
          }
          n_a++;
        }
        for (uint32_t t = t0; ok && t < t1; t++, it++) {
          const uint32_t acc = it & 1u;
          if (!mbar_wait(bar_tempty + acc * 8, ((it >> 1) & 1u) ^ 1u, p.spin_limit)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t tmem_d = tmem_base + acc * kLists;
          for (uint32_t kb = 0; kb < p.k_blocks; kb++) {
            if (!mbar_wait(bar_full + stage * 8, phase, p.spin_limit)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = stage_base + stage * stage_size;
            const uint32_t la = desc_sw128_lo(p.a_resident ? base_a + kb * kABlock : sa + kBBlock);
            const uint32_t lb = desc_sw128_lo(sa);
            const uint32_t nk = p.k_steps - kb * 4u;  // 32 bytes of K (2 descriptor units) per step
            if (kb == 0) {
              tc_mma_f16_lo<false>(tmem_d, la, lb, idesc);
            } else {
              tc_mma_f16_lo<true>(tmem_d, la, lb, idesc);
            }
            auto rest = [&](uint32_t a) {
              if (nk >= 4u) {
                tc_mma_f16_lo<true>(tmem_d, a + 2u, lb + 2u, idesc);
                tc_mma_f16_lo<true>(tmem_d, a + 4u, lb + 4u, idesc);
                tc_mma_f16_lo<true>(tmem_d, a + 6u, lb + 6u, idesc);
              } else {
                if (nk >= 2u) { tc_mma_f16_lo<true>(tmem_d, a + 2u, lb + 2u, idesc); }
                if (nk >= 3u) { tc_mma_f16_lo<true>(tmem_d, a + 4u, lb + 4u, idesc); }
              }
            };
            rest(la);
            if (p.products == 2u) {
              const uint32_t ll = la + p.k_blocks * (kABlock >> 4);
              tc_mma_f16_lo<true>(tmem_d, ll, lb, idesc);
              rest(ll);
            }
            tc_commit(bar_empty + stage * 8);
            if (++stage == p.n_stages) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (ok) { tc_commit(bar_tfull + acc * 8); }
        }
        if (ok && p.a_resident) { tc_commit(bar_aempty); }  // the row tile may be replaced once these MMAs are done
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: thread = row, warp = (lane quarter, 64 columns) ----------------
    const uint32_t quarter = warp & 3u, unit = (warp - 2) >> 2;
    uint32_t it            = 0;
    for (uint32_t item = blockIdx.x; ok && item < p.n_items; item += gridDim.x) {
      uint32_t t0, t1;
      tiles_of(item, t0, t1);
      uint32_t key[kKeep] = {0u, 0u, 0u, 0u}, second[kKeep] = {0u, 0u, 0u, 0u}, list[kKeep] = {0u, 0u, 0u, 0u};
      for (uint32_t t = t0; t < t1; t++, it++) {
        const uint32_t acc = it & 1u;
        if (ok && !mbar_wait(bar_tfull + acc * 8, (it >> 1) & 1u, p.spin_limit)) { ok = false; }
        if (__any_sync(kFullMask, !ok)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t n0 = t * kLists + unit * kUnit;
        uint32_t l0 = 0u, l1 = 0u;
        auto chunk = [&](const uint32_t (&x)[32], auto second, auto full) {
          constexpr uint32_t c = decltype(second)::value ? 32u : 0u;
#pragma unroll
          for (uint32_t e = 0; e < 32; e++) {
            // value rounded to a multiple of 2^-16, + 1.5 + tag 2^-23: bits that sort, low 7 the tag 63 - column
            float f = __fadd_rn(__uint_as_float(x[e]), 192.0f);
            f       = __fadd_rn(f, -192.0f);
            f       = __fadd_rn(f, 1.5f + float(63u - c - e) * 0x1p-23f);
            uint32_t k = __float_as_uint(f);
            if constexpr (!decltype(full)::value) {
              if (n0 + c + e >= p.n_lists) { k = 0u; }
            }
            l1 = max(l1, min(l0, k));
            l0 = max(l0, k);
          }
        };
        // (the second half is on its way while the first is looked at)
        const uint32_t tm = tmem_base + ((quarter * 32u) << 16) + acc * kLists + unit * kUnit;
        uint32_t x0[32], x1[32];
        tmem_ld32(tm, x0);
        tmem_ld32_async(tm + 32u, x1);
        if (n0 + kUnit <= p.n_lists) {
          chunk(x0, std::false_type{}, std::true_type{});
          tmem_ld_wait(x1);
          chunk(x1, std::true_type{}, std::true_type{});
        } else {
          chunk(x0, std::false_type{}, std::false_type{});
          tmem_ld_wait(x1);
          chunk(x1, std::true_type{}, std::false_type{});
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(bar_tempty + acc * 8); }
        if (l0 > key[kKeep - 1]) {
          key[kKeep - 1]    = l0;
          second[kKeep - 1] = l1;
          list[kKeep - 1] = n0 + (63u - (l0 & 127u));
#pragma unroll
          for (int i = int(kKeep) - 1; i > 0; i--) {
            if (key[i] > key[i - 1]) {
              const uint32_t a = key[i], b = list[i], c = second[i];
              key[i]        = key[i - 1];
              list[i]       = list[i - 1];
              second[i]     = second[i - 1];
              key[i - 1]    = a;
              list[i - 1]   = b;
              second[i - 1] = c;
            }
          }
        }
      }
      const uint32_t row = (item / p.splits) * kRows + quarter * 32u + lane;
      if (ok && row < p.n_rows) {
        const size_t at = (size_t(item % p.splits) * p.n_rows + row) * 4u + unit;
        p.keys[at]      = make_uint4(key[0], key[1], key[2], key[3]);
        p.lists[at]     = make_uint4(list[0], list[1], list[2], list[3]);
        p.seconds[at]   = make_uint4(second[0], second[1], second[2], second[3]);
      }
    }
  }
  if (!ok) { atomicExch(p.error, ERR_TIMEOUT); }

  tc_fence_before();
  if (__syncthreads_or(!ok)) {
    // a time-out: give copies and MMAs that are still in flight time to finish before their memory is released
    for (int i = 0; i < 64; i++) { __nanosleep(1000); }
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

__device__ __forceinline__ float key_value(uint32_t key)
{
  return key >= 0x00800000u ? __fadd_rn(__uint_as_float(key & ~127u), -1.5f) : -INFINITY;
}

struct label_records {
  const uint4* keys;
  const uint4* seconds;
  const uint4* lists;
  const float* eps;
  const uint32_t* error;
  uint32_t* timeouts;  // pinned host word: calls with the error word set
  uint32_t splits, n_rows, n_lists;
};

// the defining chain of one list
__device__ __forceinline__ uint64_t exact_key(const float* q, const float* centers, uint32_t list, uint32_t dim_ext, float alpha)
{
  const float4* c = reinterpret_cast<const float4*>(centers + size_t(list) * dim_ext);
  float acc       = 0.0f;
#pragma unroll 4
  for (uint32_t k4 = 0; k4 < dim_ext / 4; k4++) {  // dim_ext is a multiple of 8
    const float4 cv = __ldg(c + k4), qv = __ldg(reinterpret_cast<const float4*>(q) + k4);
    acc             = __fmaf_rn(cv.x, qv.x, acc);
    acc             = __fmaf_rn(cv.y, qv.y, acc);
    acc             = __fmaf_rn(cv.z, qv.z, acc);
    acc             = __fmaf_rn(cv.w, qv.w, acc);
  }
  return make_key(__fmul_rn(alpha, acc), list);
}

// Four lanes per row: lane u reads what column quarter u kept (of every split).  Rows for the other two passes are
// listed: redo[0 .. counts[0]) from the front, whole units from the back (counts[1] of them).
__global__ void __launch_bounds__(256)
label_finish_kernel(const label_records p, const float* __restrict__ x, const float* __restrict__ centers, uint32_t dim_ext,
                    float alpha, uint32_t* __restrict__ labels, uint32_t* __restrict__ redo, uint32_t* __restrict__ counts)
{
  const uint32_t r = (blockIdx.x * 256u + threadIdx.x) >> 2, u = threadIdx.x & 3u;
  const unsigned mask = 0xFu << (threadIdx.x & 28u);
  if (r >= p.n_rows) { return; }
  float top = -INFINITY, out = -INFINITY;  // largest value, largest that bounds units not kept
  for (uint32_t s = 0; s < p.splits; s++) {
    const uint4 k = __ldg(p.keys + (size_t(s) * p.n_rows + r) * 4u + u);
    top           = fmaxf(top, key_value(k.x));
    out           = fmaxf(out, key_value(k.w));
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    top = fmaxf(top, __shfl_xor_sync(mask, top, o));
    out = fmaxf(out, __shfl_xor_sync(mask, out, o));
  }
  const float t = top - 2.0f * __ldg(p.eps + r);
  if (*p.error != 0u && blockIdx.x == 0 && threadIdx.x == 0) { count_timeout(p.timeouts); }
  // (negated: an infinite or undefined bound is not proof)
  if (*p.error != 0u || !(out < t)) {
    if (u == 0) { redo[atomicAdd(counts, 1u)] = r; }
    return;
  }
  uint32_t n = 0, only = 0xFFFFFFFFu;
  bool more  = false;
  for (uint32_t s = 0; s < p.splits; s++) {
    const size_t at = (size_t(s) * p.n_rows + r) * 4u + u;
    const uint4 k   = __ldg(p.keys + at);
    if (key_value(k.x) >= t) {
      const uint4 b = __ldg(p.seconds + at);
      only          = __ldg(&p.lists[at].x);
      n += 1u + (key_value(k.y) >= t ? 1u : 0u) + (key_value(k.z) >= t ? 1u : 0u);
      more = more || key_value(b.x) >= t || (key_value(k.y) >= t && key_value(b.y) >= t) ||
             (key_value(k.z) >= t && key_value(b.z) >= t);
    }
  }
  uint32_t all = n;
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) { all += __shfl_xor_sync(mask, all, o); }
  if (__any_sync(mask, more)) {
    if (u == 0) { redo[p.n_rows - 1u - atomicAdd(counts + 1, 1u)] = r; }
    return;
  }
  if (all == 1u) {
    if (n == 1u) { labels[r] = only; }
    return;
  }
  // each lane rescores its own (rarely more than one)
  uint64_t best = kEmptyKey;
  if (n > 0) {
    for (uint32_t s = 0; s < p.splits; s++) {
      const size_t at      = (size_t(s) * p.n_rows + r) * 4u + u;
      const uint4 k        = __ldg(p.keys + at), l = __ldg(p.lists + at);
      const uint32_t kk[3] = {k.x, k.y, k.z}, ll[3] = {l.x, l.y, l.z};
#pragma unroll
      for (int i = 0; i < 3; i++) {
        if (key_value(kk[i]) < t) { continue; }
        const uint64_t key = exact_key(x + size_t(r) * dim_ext, centers, ll[i], dim_ext, alpha);
        best               = key < best ? key : best;
      }
    }
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    const uint32_t hi = __shfl_xor_sync(mask, uint32_t(best >> 32), o), lo = __shfl_xor_sync(mask, uint32_t(best), o);
    const uint64_t other = (uint64_t(hi) << 32) | lo;
    best                 = other < best ? other : best;
  }
  if (u == 0) { labels[r] = uint32_t(best); }
}

// Rows with units whose second value is within reach: one warp per row rescores every list of such units, and the single
// lists of the others.
__global__ void __launch_bounds__(256)
label_units_kernel(const label_records p, const float* __restrict__ x, const float* __restrict__ centers, uint32_t dim_ext,
                   float alpha, uint32_t* __restrict__ labels, const uint32_t* __restrict__ redo, const uint32_t* __restrict__ counts)
{
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t n    = __ldg(counts + 1);
  for (uint32_t i = (blockIdx.x * 256u + threadIdx.x) >> 5; i < n; i += gridDim.x * 8u) {
    const uint32_t r = redo[p.n_rows - 1u - i];
    const float* q   = x + size_t(r) * dim_ext;
    // lane 4 u + j: unit j of column quarter u
    const uint32_t* keys = reinterpret_cast<const uint32_t*>(p.keys);
    auto at = [&](uint32_t s) { return (size_t(s) * p.n_rows + r) * 16u + (lane & 15u); };
    float top = -INFINITY;
    for (uint32_t s = 0; s < p.splits; s++) { top = fmaxf(top, key_value(__ldg(keys + at(s)))); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { top = fmaxf(top, __shfl_xor_sync(kFullMask, top, o)); }
    const float t = top - 2.0f * __ldg(p.eps + r);
    uint64_t best = kEmptyKey;
    for (uint32_t s = 0; s < p.splits; s++) {
      const bool in       = lane < 16u && key_value(__ldg(keys + at(s))) >= t;
      const bool whole    = in && key_value(__ldg(reinterpret_cast<const uint32_t*>(p.seconds) + at(s))) >= t;
      const uint32_t list = in ? __ldg(reinterpret_cast<const uint32_t*>(p.lists) + at(s)) : 0u;
      if (in && !whole) {
        const uint64_t key = exact_key(q, centers, list, dim_ext, alpha);
        best               = key < best ? key : best;
      }
      unsigned m = __ballot_sync(kFullMask, whole);
      while (m) {
        const uint32_t base = __shfl_sync(kFullMask, list, __ffs(m) - 1) & ~(kUnit - 1u);
        m &= m - 1;
        for (uint32_t l = base + lane; l < min(base + kUnit, p.n_lists); l += 32) {
          const uint64_t key = exact_key(q, centers, l, dim_ext, alpha);
          best               = key < best ? key : best;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const uint64_t other = shfl_u64(best, int(lane) ^ o);
      best                 = other < best ? other : best;
    }
    if (lane == 0) { labels[r] = uint32_t(best); }
  }
}

uint32_t operand_width(uint32_t dim) { return round_up(dim + 2u, 16u); }
uint32_t operand_products(uint32_t dim) { return ceildiv(operand_width(dim), kBlockK) <= 3u ? 2u : 1u; }

}  // namespace

// Below some 16 M products a whole exact pass costs less than these launches; fewer than 256 lists are not one tile.
bool label_tc_usable(uint32_t n_rows, uint32_t n_lists)
{
  return n_lists >= 256 && uint64_t(n_rows) * n_lists >= (1ull << 24);
}

size_t label_model_bytes(uint32_t n_lists, uint32_t dim) { return operand_at(dim) + size_t(n_lists) * operand_width(dim) * 2; }

void prepare_label_model(cudaStream_t stream, const float* centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext, void* model)
{
  auto* words = static_cast<uint32_t*>(model);
  auto* sum   = reinterpret_cast<float*>(static_cast<char*>(model) + kMeanAt);
  auto* b     = reinterpret_cast<__half*>(static_cast<char*>(model) + operand_at(dim));
  CUDA_TRY(cudaMemsetAsync(model, 0, operand_at(dim), stream));
  const uint32_t shares = std::min<uint32_t>(64, ceildiv(n_lists, 64u));
  center_sum_kernel<<<dim3(ceildiv(dim, 32u), shares), dim3(32, 8), 0, stream>>>(centers, n_lists, dim, dim_ext, sum);
  center_stats_kernel<<<ceildiv<uint32_t>(n_lists, 8u), 256, 0, stream>>>(centers, n_lists, dim, dim_ext, sum, words);
  center_operand_kernel<<<ceildiv<uint32_t>(n_lists, 8u), 256, 0, stream>>>(centers, n_lists, dim, dim_ext, operand_width(dim), sum,
                                                                           words, b);
  CUDA_TRY(cudaGetLastError());
}

namespace {
struct label_layout {
  uint32_t splits, tiles_per_split;
  size_t o_a, o_eps, o_keys, o_seconds, o_lists, o_redo, o_words, o_best, total;
};
label_layout layout_for(uint32_t n_rows, uint32_t n_lists, uint32_t dim, int sm_count)
{
  label_layout y{};
  const uint32_t row_tiles = ceildiv(n_rows, kRows), n_tiles = ceildiv(n_lists, kLists);
  // few row tiles: the lists are shared out, so that there are about four items per SM
  y.splits = 1;
  while (y.splits < n_tiles && row_tiles * y.splits < 4u * uint32_t(sm_count) && y.splits < 16) { y.splits <<= 1; }
  y.splits          = std::min(y.splits, n_tiles);
  y.tiles_per_split = ceildiv(n_tiles, y.splits);
  y.splits          = ceildiv(n_tiles, y.tiles_per_split);
  const size_t recs = size_t(y.splits) * n_rows * 4;
  ws_layout lay;
  y.o_a      = lay.add(size_t(n_rows) * operand_width(dim) * operand_products(dim) * 2);
  y.o_eps    = lay.add(size_t(n_rows) * 4);
  y.o_keys   = lay.add(recs * 16);
  y.o_lists  = lay.add(recs * 16);
  y.o_seconds = lay.add(recs * 16);
  y.o_redo   = lay.add(size_t(n_rows) * 4);
  y.o_words  = lay.add(256);
  y.o_best   = lay.add(size_t(n_rows) * 8);
  y.total    = lay.total();
  return y;
}
}  // namespace

size_t label_workspace_bytes(const raft::resources& res, uint32_t n_rows, uint32_t n_lists, uint32_t dim)
{
  return layout_for(n_rows, n_lists, dim, res.sm_count).total;
}

void label_rows_tc(raft::resources& res, const float* centers, const void* model, uint32_t n_lists, uint32_t dim,
                   uint32_t dim_ext, float alpha, const float* x_ext, uint32_t n_rows, uint32_t* labels, void* workspace)
{
  if (n_rows == 0) { return; }
  const label_layout y = layout_for(n_rows, n_lists, dim, res.sm_count);
  const uint32_t width = operand_width(dim);
  char* ws             = static_cast<char*>(workspace);
  auto* a              = reinterpret_cast<__half*>(ws + y.o_a);
  auto* eps            = reinterpret_cast<float*>(ws + y.o_eps);
  auto* words          = reinterpret_cast<uint32_t*>(ws + y.o_words);  // error, rows to redo
  auto* redo           = reinterpret_cast<uint32_t*>(ws + y.o_redo);
  auto* best           = reinterpret_cast<unsigned long long*>(ws + y.o_best);
  const auto* stats    = static_cast<const uint32_t*>(model);
  const auto* sum      = reinterpret_cast<const float*>(static_cast<const char*>(model) + kMeanAt);
  const auto* b        = reinterpret_cast<const __half*>(static_cast<const char*>(model) + operand_at(dim));
  cudaStream_t stream  = res.stream;
  CUDA_TRY(cudaMemsetAsync(words, 0, 12, stream));
  const uint32_t products = operand_products(dim);
  const uint32_t blocks   = ceildiv<uint32_t>(n_rows, 8u);
  if (products == 2) {
    row_operand_kernel<true><<<blocks, 256, 0, stream>>>(x_ext, n_rows, n_lists, dim, dim_ext, width, sum, stats, a, eps);
  } else {
    row_operand_kernel<false><<<blocks, 256, 0, stream>>>(x_ext, n_rows, n_lists, dim, dim_ext, width, sum, stats, a, eps);
  }
  label_params p{};
  p.n_rows          = n_rows;
  p.n_lists         = n_lists;
  p.k_steps         = width / 16;
  p.k_blocks        = ceildiv(width, kBlockK);
  p.n_tiles         = ceildiv(n_lists, kLists);
  p.tiles_per_split = y.tiles_per_split;
  p.splits          = y.splits;
  p.n_items         = ceildiv(n_rows, kRows) * y.splits;
  // the row tile stays in shared memory where that leaves at least three list stages
  const uint32_t a_size = products * p.k_blocks * kABlock;
  p.products   = products;
  p.width      = width;
  p.a_resident = a_size + 3 * kBBlock <= kRoom;
  CUVS_EXPECTS(p.a_resident || products == 1, "internal error: split row operands are resident");
  p.n_stages   = p.a_resident ? std::min(kMaxStages, (kRoom - a_size) / kBBlock) : kRoom / (kABlock + kBBlock);
  p.keys       = reinterpret_cast<uint4*>(ws + y.o_keys);
  p.lists      = reinterpret_cast<uint4*>(ws + y.o_lists);
  p.seconds    = reinterpret_cast<uint4*>(ws + y.o_seconds);
  p.error      = words;
  const wait_limits wl = tc_wait_limits();
  p.spin_limit = wl.spin_limit;
  p.skip_kb    = wl.skip_kb;
  const CUtensorMap ma = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a, n_rows, uint64_t(width) * products, kRows, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  const CUtensorMap mb = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, b, n_lists, width, kLists, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  const size_t smem    = kRoom + 1024 + 256;
  ensure_dynamic_smem(reinterpret_cast<const void*>(label_tc_kernel), smem);
  label_tc_kernel<<<std::min(uint32_t(res.sm_count), p.n_items), kThreads, smem, stream>>>(ma, mb, p);
  const label_records rec{p.keys, p.seconds, p.lists, eps, words, res.pinned + 13, p.splits, n_rows, n_lists};
  label_finish_kernel<<<ceildiv(n_rows, 64u), 256, 0, stream>>>(rec, x_ext, centers, dim_ext, alpha, labels, redo, words + 1);
  label_units_kernel<<<std::min<uint32_t>(uint32_t(res.sm_count) * 8, blocks), 256, 0, stream>>>(rec, x_ext, centers, dim_ext, alpha,
                                                                                               labels, redo, words + 1);
  CUDA_TRY(cudaGetLastError());
  assign_nearest_listed(res, centers, n_lists, dim_ext, alpha, x_ext, n_rows, redo, words + 1, labels, best);
  res.launches += 4;
}

}  // namespace cuvs::neighbors::ivf_pq
