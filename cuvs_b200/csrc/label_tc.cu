// Nearest list of many rows on the tensor cores, exact: labels[i] = argmin over lists l of (score, l) with the score's
// defining fp32 chain (coarse.cu) -- what k-means steps, extend and transform need.  At the end: the nearest lists (probes) of a
// batch of queries, by the same products.
//
// Reference: kmeans_balanced::predict (cpp/src/cluster/detail/kmeans_balanced.cuh:100-160).
//
// For the nearest list alone, one maximum per few lists is enough:
//   1. operands in half precision (the same 11 significant bits as TF32 at twice the rate), relative to the mean m of the
//      centres: rows (q - m) 2^e, lists (c - m) / cp, with cp the power of two above the largest |c - m|, so that products lie
//      within (-0.5, 0.5); the epilogue subtracts the list's norm term |c|^2 / 2 - m.c + |m|^2 / 2 times a factor of the row,
//      which gives F (score + a constant of the row).  The bounds of a row say how far that can be from the exact value: the
//      measured norms of what rounding took from row and lists, accumulation, the defining chain's own rounding, the keys.
//   2. row_list_kernel: a persistent CTA takes a tile of 256 rows against all (or a share) of the lists, 256 at a time: two
//      accumulators of 128 rows, so that a list tile is read once for both and the epilogue of one runs beside the products of
//      the other.  Per row and unit of 8 lists the epilogue finds the largest value (its low bits replaced by the unit's
//      number); across the tiles it keeps, per row and column quarter, the four largest: 1.3 comparisons per value.
//   3. label_finish_kernel looks at the units within 2 eps of the largest value: first their operands' products in fp32, then
//      what is left in ever finer sums, the defining chain last.
//   4. If the fourth unit kept is inside, a fifth might be: such rows (2.7% of 1 M rows x 16,384 lists of 96 dimensions) go
//      through 2 and 3 once more with the lists in eight shares; only what that does not settle is redone exactly over all lists.
// What bounds row_list_kernel: the epilogue.  A 128 x 256 x 96 tile takes 1,260 clocks, 860 with the epilogue left out of a copy
// of the kernel, and its products alone 770.  1,000,003 rows x 16,384 lists x 96 dimensions, all of the labelling: 9.4 ms with two
// products (row operand as two halfs), units of 64 lists whose largest two values were kept with their columns, and 2% of the
// rows redone over all lists; 3.8 ms so.  (One product widens the bounds from 5.2e-5 to 6.5e-5: 2.6 instead of 2.2 lists within
// reach.)
// Every wait is bounded: on a time-out the kernel raises the error word and returns, and all rows are redone.
#include "common.hpp"
#include "packed.cuh"
#include "search_internal.hpp"
#include "tc_ptx.cuh"
#include "topk.cuh"

#include <algorithm>

namespace cuvs::neighbors::ivf_pq {

using namespace cuvs_b200;

namespace {

constexpr uint32_t kRows = 128, kTileRows = 2 * kRows, kLists = 256, kBlockK = 64, kUnit = 8, kKeep = 4;
constexpr uint32_t kUnitsPerTile = 64 / kUnit;        // units of a tile in one column quarter
constexpr uint32_t kSplitTiles   = 64;                // most list tiles of an item: nine bits number its units
constexpr uint32_t kEpiWarps = 16;
constexpr uint32_t kThreads  = (2 + kEpiWarps) * 32;  // warp 0 TMA, warp 1 MMA, warps 2..17 epilogue
constexpr uint32_t kABlock = kRows * kBlockK * 2, kBBlock = kLists * kBlockK * 2;  // 16 and 32 KB
constexpr uint32_t kRoom      = 6 * kBBlock;          // shared memory for operands: 192 KB
constexpr uint32_t kMaxStages = 4;
constexpr uint32_t kNormSlots = 8;                    // list tiles whose norm terms are on hand
constexpr uint32_t kNormBytes = kLists * 4;
constexpr float kNoList       = 1e30f;                // norm term of a list that is not there

// Model: words {bits of the largest max(|c - m|^2, 2 |norm column|), of the largest |c|^2 or norm column, of the largest
// squared norm of what rounding took from a list}, the sum of the centres at kMeanAt, the lists' norm terms at norms_at(dim) (whole
// tiles of them), the list operand behind, and once more by units at unit_operand_at: [units][width / 8][8 lists] 16-byte chunks.
constexpr uint32_t kMeanAt = 256;
__host__ __device__ __forceinline__ size_t norms_at(uint32_t dim) { return kMeanAt + round_up<size_t>(size_t(dim) * 4, 256); }
__host__ __device__ __forceinline__ size_t operand_at(uint32_t n_lists, uint32_t dim)
{
  return norms_at(dim) + size_t(round_up(n_lists, kLists)) * 4;
}

__host__ __device__ __forceinline__ size_t unit_operand_at(uint32_t n_lists, uint32_t dim, uint32_t width)
{
  return operand_at(n_lists, dim) + round_up<size_t>(size_t(n_lists) * width * 2, 256);
}

// The list at a place of the operand that probes are selected from: a fixed shuffle of 0 .. n - 1 (odd multiples and shifted
// exclusive-ors, each a permutation of the numbers of some bits, repeated while it leads beyond n).  A unit's maximum stands for
// 8 to 128 neighbouring places: where neighbouring lists are alike -- a data set stored by cluster or by time, whose evenly taken
// rows k-means starts from, or a model trained in levels -- few units hold all lists that are near, and a value that n_probes
// units reach lies far below that of the n_probes-th list (4,000 lists sorted by component, 64 probes: every query had more
// lists within reach than there is room for).
__device__ __forceinline__ uint32_t list_at(uint32_t place, uint32_t n)
{
  const uint32_t bits = 32u - uint32_t(__clz(int(n - 1u))), shift = max(bits / 2u, 1u);
  const uint32_t mask = bits < 32u ? (1u << bits) - 1u : ~0u;
  do {
    place = (place * 0x9E3779B1u) & mask;
    place ^= place >> shift;
    place = (place * 0x6A09E667u) & mask;
    place ^= place >> shift;
  } while (place >= n);
  return place;
}

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

// weight |c|^2 - m.c + |m|^2 / 2 of a list, by one warp (any m gives valid results: it only has to be the same everywhere)
__device__ __forceinline__ void list_norms(const float* c, const float* sum, float inv_n, uint32_t dim, float weight, float& cc, float& dd,
                                           double& norm)
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
  norm = double(weight) * double(c[dim]) - mc + 0.5 * mm;
}

__global__ void center_stats_kernel(const float* __restrict__ centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                                    float weight, const float* __restrict__ sum, uint32_t* __restrict__ words)
{
  const uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (l >= n_lists) { return; }
  const float* c = centers + size_t(l) * dim_ext;
  float cc, dd;
  double norm;
  list_norms(c, sum, 1.0f / float(n_lists), dim, weight, cc, dd, norm);
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

// One warp per place (of whole tiles: there is nothing in those beyond the last list but their norm terms).  Without `by_unit` the
// lists are shuffled (list_at).
__global__ void center_operand_kernel(const float* __restrict__ centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                                      uint32_t width, float weight, const float* __restrict__ sum, uint32_t* __restrict__ words,
                                      float* __restrict__ norms, __half* __restrict__ out, __half* __restrict__ by_unit)
{
  const uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
  if (l >= n_lists) {
    if (l < round_up(n_lists, kLists) && lane == 0) { norms[l] = kNoList; }
    return;
  }
  float bn, cc, dd;
  const float inv   = 1.0f / center_scale(words, bn);
  const float inv_n = 1.0f / float(n_lists);
  const float* c    = centers + size_t(by_unit != nullptr ? l : list_at(l, n_lists)) * dim_ext;
  double norm;
  list_norms(c, sum, inv_n, dim, weight, cc, dd, norm);
  __half* dst    = out + size_t(l) * width;
  float lost     = 0.0f;
  for (uint32_t k = lane; k < width; k += 32) {
    const float v  = k < dim ? (c[k] - sum[k] * inv_n) * inv : 0.0f;
    const __half h = __float2half_rn(v);
    dst[k]         = h;
    if (by_unit != nullptr) { by_unit[((size_t(l / kUnit) * (width / 8u) + k / 8u) * kUnit + l % kUnit) * 8u + (k & 7u)] = h; }
    const float d  = v - __half2float(h);
    lost           = __fmaf_rn(d, d, lost);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { lost += __shfl_xor_sync(kFullMask, lost, o); }
  if (lane == 0) {
    atomicMax(words + 2, __float_as_uint(lost * 1.001f));
    norms[l] = float(norm * double(inv) * double(inv));
  }
}

// Eight lanes per row: the operand row, the factor of the lists' norm terms, and three bounds: {of a key, of a sum of the half-precision operands in fp32, of the
// defining chain and of any other fp32 sum of its products, the last in units of the chain} (infinite: the row is redone).
// What bounds it: memory (dim_ext floats in, `width` halfs out).  A warp per row spent its time on the arithmetic of the
// bounds: 161 us for 524,288 rows of 96 dimensions.  kRegs: the row stays in registers (width <= 128).
template <bool kRegs>
__global__ void __launch_bounds__(256)
row_operand_kernel(const float* __restrict__ x, uint32_t n_rows, uint32_t n_lists, uint32_t dim, uint32_t dim_ext, uint32_t width,
                   const float* __restrict__ sum, const uint32_t* __restrict__ words, float key_error, __half* __restrict__ out,
                   float* __restrict__ factor, float4* __restrict__ eps, uint4* __restrict__ clear)
{
  chain_begin();
  if (blockIdx.x == 0 && threadIdx.x == 0) { *clear = make_uint4(0u, 0u, 0u, 0u); }  // errors and counts of the kernels behind
  const uint32_t r    = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const uint32_t lane = threadIdx.x & 7u;
  const unsigned mask = 0xFFu << (threadIdx.x & 24u);
  if (r >= n_rows) { return; }
  const float inv_n = 1.0f / float(n_lists);
  const float4* q   = reinterpret_cast<const float4*>(x + size_t(r) * dim_ext);  // dim_ext is a multiple of 8
  constexpr uint32_t kIters = kRegs ? 4u : 1u;
  float4 a4[kIters];
  if constexpr (kRegs) {
#pragma unroll
    for (uint32_t i = 0; i < kIters; i++) {
      const uint32_t k = lane * 4u + i * 32u;
      a4[i]            = k < dim_ext ? __ldg(q + (k >> 2)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  // four components of the row and of its difference to the mean (zero from `dim` on)
  auto load = [&](uint32_t k, uint32_t i, float (&v)[4], float (&d)[4]) {
    float4 a;
    if constexpr (kRegs) {
      a = a4[i];
    } else {
      a = k < dim_ext ? __ldg(q + (k >> 2)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
#pragma unroll
    for (uint32_t e = 0; e < 4; e++) {
      const bool in = k + e < dim;
      v[e]          = in ? v[e] : 0.0f;
      d[e]          = in ? v[e] - __ldg(sum + k + e) * inv_n : 0.0f;
    }
  };
  auto steps = [&](auto&& fn) {
    if constexpr (kRegs) {
#pragma unroll
      for (uint32_t i = 0; i < kIters; i++) { fn(lane * 4u + i * 32u, i); }
    } else {
      for (uint32_t k = lane * 4u; k < width; k += 32u) { fn(k, 0u); }
    }
  };
  float ss = 0.0f, qq = 0.0f;
  steps([&](uint32_t k, uint32_t i) {
    float v[4], d[4];
    load(k, i, v, d);
#pragma unroll
    for (uint32_t e = 0; e < 4; e++) {
      ss = __fmaf_rn(d[e], d[e], ss);
      qq = __fmaf_rn(v[e], v[e], qq);
    }
  });
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    ss += __shfl_xor_sync(mask, ss, o);
    qq += __shfl_xor_sync(mask, qq, o);
  }
  float bn;
  const float cp = center_scale(words, bn);
  const float dn = sqrtf(ss) * 1.0001f, qn = sqrtf(qq) * 1.0001f;
  // 2^e (|q - m| + cp / 2) in [0.25, 0.5)
  const float b     = (dn + 0.5f * cp) * 1.01f;
  const int E       = int((__float_as_uint(b) >> 23) & 0xFFu);
  const bool fine   = E >= 2 && E <= 250;
  const float scale = fine ? __uint_as_float(uint32_t(252 - E) << 23) : 0.0f;
  const float a     = scale * cp;
  float lost        = 0.0f;
  steps([&](uint32_t k, uint32_t i) {
    float v[4], d[4];
    load(k, i, v, d);
#pragma unroll
    for (uint32_t e = 0; e < 4; e++) { d[e] *= scale; }
    const __half2 h0 = __floats2half2_rn(d[0], d[1]), h1 = __floats2half2_rn(d[2], d[3]);
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    d[0] -= f0.x; d[1] -= f0.y; d[2] -= f1.x; d[3] -= f1.y;
#pragma unroll
    for (uint32_t e = 0; e < 4; e++) { lost = __fmaf_rn(d[e], d[e], lost); }
    uint2 w;
    w.x = *reinterpret_cast<const uint32_t*>(&h0);
    w.y = *reinterpret_cast<const uint32_t*>(&h1);
    if (k < width) { *reinterpret_cast<uint2*>(out + size_t(r) * width + k) = w; }  // width is a multiple of 16
  });
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) { lost += __shfl_xor_sync(mask, lost, o); }
  if (lane == 0) {
    const float an = dn * scale, w = float(width);
    const float bl = sqrtf(__uint_as_float(__ldg(words + 2))), cn = sqrtf(__uint_as_float(__ldg(words + 1)));
    const float orig  = qn * cn + 0.5f * cn * cn;  // bounds every partial sum of the defining chain
    const float chain = orig * (float(dim_ext) + 4.0f) * 1.2e-7f;
    float e = (sqrtf(lost) * (bn + bl) + an * bl) * 1.01f  // rounding of the operands
              + (scale / cp) * chain                       // the defining chain, and q - m
              + 0.6e-6f;                                   // norm terms
    if (!fine || !(a >= 6.2e-5f)) { e = INFINITY; }
    // accumulation of sums below 0.5 by the tensor core, and in fp32
    factor[r] = a;
    eps[r] = make_float4(e + (w + 24.0f) * 1.2e-7f + key_error, e + w * 6.1e-8f, chain, 0.0f);
  }
}

// Operand rows and factors of the listed rows, one after the other.  One warp per row at a time.
__global__ void __launch_bounds__(256)
gather_operand_kernel(const __half* __restrict__ a, const float* __restrict__ factor, const uint32_t* __restrict__ rows,
                      const uint32_t* __restrict__ count, uint32_t cap, uint32_t width, __half* __restrict__ out,
                      float* __restrict__ factor_out, unsigned long long* __restrict__ listed)
{
  chain_begin();
  const uint32_t n = min(__ldg(count), cap), lane = threadIdx.x & 31u;
  if (n > 0 && blockIdx.x == 0 && threadIdx.x == 0) { atomicAdd(listed, static_cast<unsigned long long>(n)); }
  for (uint32_t i = (blockIdx.x * 256u + threadIdx.x) >> 5; i < n; i += gridDim.x * 8u) {
    const uint32_t r = __ldg(rows + i);
    const uint4* src = reinterpret_cast<const uint4*>(a + size_t(r) * width);
    uint4* dst       = reinterpret_cast<uint4*>(out + size_t(i) * width);
    for (uint32_t c = lane; c < width / 8u; c += 32u) { dst[c] = __ldg(src + c); }
    if (lane == 0) { factor_out[i] = __ldg(factor + r); }
  }
}

struct label_params {
  uint32_t n_rows;       // rows of the operand (and of `keys`)
  const uint32_t* count; // where given: only so many of them count
  uint32_t k_steps /* of 16 halfs */, k_blocks;
  uint32_t n_tiles, tiles_per_split, splits;
  uint32_t tag_mask;     // low bits of a key: number of the unit among those of an item's column quarter
  const float* norms;    // of the lists, whole tiles
  const float* factor;   // of the rows
  float4* keys;          // kKeys: [splits, n_rows, 4] largest keys of a column quarter
  float* maxima;         // kMaxima: [n_rows, max_stride] largest value of every `unit` (8, 32, 64 or 128) lists
  uint32_t unit, max_stride;
  const float* threshold;  // kEmit: of the rows
  uint32_t* found;         // [n_rows, 2 splits, found_cap] places of the lists whose value reaches it
  uint32_t* n_found;       // [n_rows, 2 splits]
  uint32_t found_cap;
  uint32_t* error;
  uint32_t spin_limit, skip_kb;  // tc_wait_limits
};
// What the epilogue makes of the values
enum row_list_mode { kKeys, kMaxima, kEmit };

// kKB: K blocks of 64 halfs; up to three of both halves of the row tile stay in shared memory beside a ring of kSlots list
// tiles.  0: any number, row blocks stream beside the list blocks.
template <uint32_t kKB, row_list_mode kMode>
__global__ void __launch_bounds__(kThreads, 1)
row_list_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const label_params p)
{
  constexpr bool kResident   = kKB > 0;
  constexpr uint32_t kSlots  = kKB == 1 ? 4u : (kKB == 2 ? 2u : 1u);
  constexpr uint32_t kStages = kResident ? kSlots * kKB : kRoom / (2 * kABlock + kBBlock);
  static_assert(kStages <= kMaxStages && kKB * (2 * kABlock + kSlots * kBBlock) <= kRoom, "shared memory");
  // [row tile, when resident: two halves of kKB blocks][stages: list block, then the two row blocks when not][norm terms]
  constexpr uint32_t kABytes    = kResident ? 2u * kKB * kABlock : 0u;
  constexpr uint32_t kStageSize = kBBlock + (kResident ? 0u : 2u * kABlock);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_a  = smem_u32(smem_raw);
  const uint32_t base_a = (raw_a + 1023u) & ~1023u;
  uint8_t* base_p       = smem_raw + (base_a - raw_a);
  uint64_t* bars        = reinterpret_cast<uint64_t*>(base_p + kRoom + kNormSlots * kNormBytes);
  const uint32_t bar_full   = smem_u32(bars);
  const uint32_t bar_empty  = bar_full + kMaxStages * 8;
  const uint32_t bar_tfull  = bar_empty + kMaxStages * 8;
  const uint32_t bar_tempty = bar_tfull + 2 * 8;
  const uint32_t bar_afull  = bar_tempty + 2 * 8;
  const uint32_t bar_aempty = bar_afull + 8;
  const uint32_t bar_norms  = bar_aempty + 8;
  uint32_t* tmem_slot       = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 6 + kNormSlots);
  const uint32_t stage_base = base_a + kABytes;
  const uint32_t norm_base  = base_a + kRoom;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kStages; s++) {
      mbar_init(bar_full + s * 8, 1);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (uint32_t a = 0; a < 2; a++) {
      mbar_init(bar_tfull + a * 8, 1);
      mbar_init(bar_tempty + a * 8, kEpiWarps / 2);
    }
    mbar_init(bar_afull, 1);
    mbar_init(bar_aempty, 1);
    for (uint32_t s = 0; s < kNormSlots; s++) { mbar_init(bar_norms + s * 8, 1); }
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
  chain_begin();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint32_t n_rows    = p.count != nullptr ? min(__ldg(p.count), p.n_rows) : p.n_rows;
  const uint32_t n_items   = ceildiv(n_rows, kTileRows) * p.splits;
  const uint32_t k_blocks  = kResident ? kKB : p.k_blocks;
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
      uint32_t stage = 0, phase = 0, n_a = 0, it = 0;
      for (uint32_t item = blockIdx.x; ok && item < n_items; item += gridDim.x) {
        const int row0 = int((item / p.splits) * kTileRows);
        uint32_t t0, t1;
        tiles_of(item, t0, t1);
        if constexpr (kResident) {
          if (!mbar_wait(bar_aempty, (n_a & 1u) ^ 1u, p.spin_limit)) {
            ok = false;
            break;
          }
          n_a++;
          mbar_arrive_expect_tx(bar_afull, kABytes);
          for (uint32_t h = 0; h < 2; h++) {
            for (uint32_t kb = 0; kb < kKB; kb++) {
              tma_load_2d(base_a + (h * kKB + kb) * kABlock, &map_a, bar_afull, int(kb * kBlockK), row0 + int(h * kRows));
            }
          }
        }
        for (uint32_t t = t0; ok && t < t1; t++, it++) {
          for (uint32_t kb = 0; kb < k_blocks; kb++) {
            if (!mbar_wait(bar_empty + stage * 8, phase ^ 1u, p.spin_limit)) {
              ok = false;
              break;
            }
            if (kb == 0) {
              // the slot's last reader is kNormSlots tiles back, and the tile of the stage just freed, whose products wait
              // for the epilogue of the one before, at most kSlots
              const uint32_t slot = it % kNormSlots, bar = bar_norms + slot * 8;
              mbar_arrive_expect_tx(bar, kNormBytes);
              bulk_load(norm_base + slot * kNormBytes, p.norms + size_t(t) * kLists, kNormBytes, bar);
            }
            const uint32_t dst = stage_base + stage * kStageSize, bar = bar_full + stage * 8;
            // (test only: a block that never comes, so that the wait for it runs out)
            if (kb + 1 != p.skip_kb || t != t0 || item != blockIdx.x) {
              mbar_arrive_expect_tx(bar, kStageSize);
              tma_load_2d(dst, &map_b, bar, int(kb * kBlockK), int(t * kLists));
              if constexpr (!kResident) {
                tma_load_2d(dst + kBBlock, &map_a, bar, int(kb * kBlockK), row0);
                tma_load_2d(dst + kBBlock + kABlock, &map_a, bar, int(kb * kBlockK), row0 + int(kRows));
              }
            }
            if (++stage == kStages) {
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
    // (the warp goes through the loops as a whole; one lane issues: see elect_one)
    // fp32 accumulate, half x half, both K-major, M = 128, N = 256
    constexpr uint32_t idesc = (1u << 4) | ((kLists >> 3) << 17) | ((kRows >> 4) << 24);
    const uint32_t tmem_d    = __shfl_sync(kFullMask, tmem_base, 0);
    const uint32_t last_k    = p.k_steps - (k_blocks - 1u) * 4u;  // steps of the last K block
    // the steps of one K block (32 bytes of K, 2 descriptor units, each)
    auto block = [&](uint32_t d, uint32_t la, uint32_t lb, auto first, bool last) {
      tc_mma_f16_lo<!decltype(first)::value>(d, la, lb, idesc);
      if (!last || last_k >= 2u) { tc_mma_f16_lo<true>(d, la + 2u, lb + 2u, idesc); }
      if (!last || last_k >= 3u) { tc_mma_f16_lo<true>(d, la + 4u, lb + 4u, idesc); }
      if (!last || last_k >= 4u) { tc_mma_f16_lo<true>(d, la + 6u, lb + 6u, idesc); }
    };
    uint32_t stage = 0, phase = 0, n_a = 0, it = 0;
    for (uint32_t item = blockIdx.x; ok && item < n_items; item += gridDim.x) {
      uint32_t t0, t1;
      tiles_of(item, t0, t1);
      if constexpr (kResident) {
        ok = mbar_wait_warp(bar_afull, n_a & 1u, p.spin_limit);
        if (!ok) { break; }
        n_a++;
      }
      for (uint32_t t = t0; t < t1; t++, it++) {
        const uint32_t t_empty = (it & 1u) ^ 1u;
        if constexpr (kResident) {
          // one half of the rows after the other, both against the list blocks of the tile
          const uint32_t slot = it % kSlots, full = (it / kSlots) & 1u;
          const uint32_t lb   = desc_sw128_lo(stage_base) + slot * (kKB * kBBlock >> 4);
          const uint32_t la   = desc_sw128_lo(base_a);
          auto half = [&](auto hc) {
            constexpr uint32_t h = decltype(hc)::value;
            if (!mbar_wait_warp(bar_tempty + h * 8, t_empty, p.spin_limit)) { return false; }
            bool fine = true;
            static_for<kKB>([&](auto kc) {
              constexpr uint32_t kb = decltype(kc)::value;
              const uint32_t s      = slot * kKB + kb;
              if (h == 0 && fine) { fine = mbar_wait_warp(bar_full + s * 8, full, p.spin_limit); }
              if (!fine) { return; }
              tc_fence_after();
              if (elect_one()) {
                block(tmem_d + h * kLists, la + (h * kKB + kb) * (kABlock >> 4), lb + kb * (kBBlock >> 4),
                      std::integral_constant<bool, kb == 0>{}, kb + 1 == kKB);
                if constexpr (h == 1) { tc_commit(bar_empty + s * 8); }
                if constexpr (kb + 1 == kKB) { tc_commit(bar_tfull + h * 8); }
              }
              __syncwarp();
            });
            return fine;
          };
          ok = half(std::integral_constant<uint32_t, 0>{}) && half(std::integral_constant<uint32_t, 1>{});
          if (!ok) { break; }
        } else {
          for (uint32_t kb = 0; kb < k_blocks; kb++) {
            ok = mbar_wait_warp(bar_full + stage * 8, phase, p.spin_limit);
            if (!ok) { break; }
            const uint32_t sa = stage_base + stage * kStageSize;
            for (uint32_t h = 0; h < 2; h++) {
              if (kb == 0) {
                ok = mbar_wait_warp(bar_tempty + h * 8, t_empty, p.spin_limit);
                if (!ok) { break; }
              }
              tc_fence_after();
              if (elect_one()) {
                const uint32_t la = desc_sw128_lo(sa + kBBlock + h * kABlock), lb = desc_sw128_lo(sa);
                if (kb == 0) {
                  block(tmem_d + h * kLists, la, lb, std::true_type{}, kb + 1 == k_blocks);
                } else {
                  block(tmem_d + h * kLists, la, lb, std::false_type{}, kb + 1 == k_blocks);
                }
                if (kb + 1 == k_blocks) { tc_commit(bar_tfull + h * 8); }
                if (h == 1) { tc_commit(bar_empty + stage * 8); }
              }
              __syncwarp();
            }
            if (!ok) { break; }
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (!ok) { break; }
        }
      }
      // the row tile may be replaced once these MMAs are done
      if (kResident && ok && elect_one()) { tc_commit(bar_aempty); }
      __syncwarp();
    }
  } else {
    // ---------------- epilogue: thread = row, warp = (half of the rows, half of the columns, lane quarter) ----------------
    // (eight warps per accumulator, so that one half's loads run beside the other half's comparisons)
    const uint32_t quarter = warp & 3u, side = ((warp - 2) >> 2) & 1u, h = (warp - 2) >> 3;
    uint32_t it            = 0;
    for (uint32_t item = blockIdx.x; ok && item < n_items; item += gridDim.x) {
      uint32_t t0, t1;
      tiles_of(item, t0, t1);
      const uint32_t row = (item / p.splits) * kTileRows + h * kRows + quarter * 32u + lane;
      const uint64_t neg = dup2(row < n_rows ? -__ldg(p.factor + row) : 0.0f);
      [[maybe_unused]] float key[2][kKeep];  // kKeys: of two column quarters
      if constexpr (kMode == kKeys) {
#pragma unroll
        for (uint32_t c = 0; c < 2; c++) {
#pragma unroll
          for (uint32_t i = 0; i < kKeep; i++) { key[c][i] = -3e38f; }
        }
      }
      // kEmit: this thread's own places (nothing is taken for a row that is not there)
      [[maybe_unused]] float threshold  = INFINITY;
      [[maybe_unused]] uint32_t n_found = 0;
      [[maybe_unused]] const size_t seg = size_t(row) * (2u * p.splits) + (item % p.splits) * 2u + side;
      if constexpr (kMode == kEmit) {
        if (row < n_rows) { threshold = __ldg(p.threshold + row); }
      }
      for (uint32_t t = t0; t < t1; t++, it++) {
        const uint32_t id   = (t - t0) * kUnitsPerTile;
        const uint32_t slot = it % kNormSlots;
        if (ok && !mbar_wait(bar_norms + slot * 8, (it / kNormSlots) & 1u, p.spin_limit)) { ok = false; }
        if (ok && !mbar_wait(bar_tfull + h * 8, it & 1u, p.spin_limit)) { ok = false; }
        if (__any_sync(kFullMask, !ok)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t tm = tmem_base + ((quarter * 32u) << 16) + h * kLists + side * 128u;
        const uint32_t na = norm_base + slot * kNormBytes + side * 512u;
        [[maybe_unused]] float* out = p.maxima;
        if constexpr (kMode == kMaxima) { out += size_t(row) * p.max_stride + (t * kLists + side * 128u) / p.unit; }
        [[maybe_unused]] float wide[4];
        auto chunk = [&](uint32_t (&x)[32], auto cc) {
          constexpr uint32_t c = decltype(cc)::value;
          [[maybe_unused]] float m[4];
          [[maybe_unused]] uint32_t hits = 0;
          static_for<4>([&](auto uc) {
            constexpr uint32_t u = decltype(uc)::value;
            float v[8];
#pragma unroll
            for (uint32_t e = 0; e < 8; e += 4) {
              uint64_t n01, n23;
              lds128(na + (c * 32u + u * 8u + e) * 4u, n01, n23);
              const uint64_t a = fma2(n01, neg, pack2(x[u * 8u + e], x[u * 8u + e + 1]));
              const uint64_t b = fma2(n23, neg, pack2(x[u * 8u + e + 2], x[u * 8u + e + 3]));
              v[e] = lo2(a); v[e + 1] = hi2(a); v[e + 2] = lo2(b); v[e + 3] = hi2(b);
            }
            if constexpr (kMode == kEmit) {
#pragma unroll
              for (uint32_t e = 0; e < 8; e++) {
                if (v[e] >= threshold) { hits |= 1u << (u * 8u + e); }
              }
            } else {
              const float y = fmaxf(max3(max3(max3(v[0], v[1], v[2]), v[3], v[4]), v[5], v[6]), v[7]);
              m[u] = kMode == kKeys ? __uint_as_float((__float_as_uint(y) & ~p.tag_mask) | (id + (c & 1u) * 4u + u)) : y;
            }
          });
          if constexpr (kMode == kEmit) {
            while (hits != 0u) {
              if (n_found < p.found_cap) {
                p.found[seg * p.found_cap + n_found] = t * kLists + side * 128u + c * 32u + uint32_t(__ffs(int(hits))) - 1u;
              }
              n_found++;
              hits &= hits - 1u;
            }
          }
          if constexpr (kMode == kMaxima) {
            if (p.unit == 8u) {
              if (row < n_rows) { *reinterpret_cast<float4*>(out + c * 4u) = make_float4(m[0], m[1], m[2], m[3]); }
            } else {
              wide[c] = fmaxf(max3(m[0], m[1], m[2]), m[3]);
              if (c == 3u && row < n_rows) {
                const float w0 = fmaxf(wide[0], wide[1]), w1 = fmaxf(wide[2], wide[3]);
                if (p.unit == 32u) {
                  *reinterpret_cast<float4*>(out) = make_float4(wide[0], wide[1], wide[2], wide[3]);
                } else if (p.unit == 64u) {
                  *reinterpret_cast<float2*>(out) = make_float2(w0, w1);
                } else {
                  *out = fmaxf(w0, w1);
                }
              }
            }
          }
          if constexpr (kMode == kKeys) {
            // two units at a time into the four largest: the m-th largest of two ordered runs a and b is the maximum over
            // i + j = m of min(a[i - 1], b[j - 1])
            float (&k)[kKeep] = key[c >> 1];
#pragma unroll
            for (uint32_t u = 0; u < 4; u += 2) {
              const float hi = fmaxf(m[u], m[u + 1]), lo = fminf(m[u], m[u + 1]);
              const float k3 = max3(k[3], fminf(k[2], hi), fminf(k[1], lo));
              const float k2 = max3(k[2], fminf(k[1], hi), fminf(k[0], lo));
              const float k1 = max3(k[1], fminf(k[0], hi), lo);
              k[0]           = fmaxf(k[0], hi);
              k[1]           = k1;
              k[2]           = k2;
              k[3]           = k3;
            }
          }
        };
        using std::integral_constant;
        uint32_t x0[32], x1[32];
        tmem_ld32(tm, x0);
        tmem_ld32_async(tm + 32u, x1);
        chunk(x0, integral_constant<uint32_t, 0>{});
        tmem_ld_wait(x1);
        tmem_ld32_async(tm + 64u, x0);
        chunk(x1, integral_constant<uint32_t, 1>{});
        tmem_ld_wait(x0);
        tmem_ld32_async(tm + 96u, x1);
        chunk(x0, integral_constant<uint32_t, 2>{});
        tmem_ld_wait(x1);
        // (the last values are in registers: the accumulator is free)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(bar_tempty + h * 8); }
        chunk(x1, integral_constant<uint32_t, 3>{});
      }
      if (ok && row < n_rows) {
        if constexpr (kMode == kKeys) {
#pragma unroll
          for (uint32_t c = 0; c < 2; c++) {
            p.keys[(size_t(item % p.splits) * p.n_rows + row) * 4u + side * 2u + c] =
              make_float4(key[c][0], key[c][1], key[c][2], key[c][3]);
          }
        }
        if constexpr (kMode == kEmit) { p.n_found[seg] = n_found; }
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

struct finish_params {
  const float* keys;       // [splits, stride, 16]
  const float4* eps;
  const uint32_t* error;
  uint32_t* timeouts;      // pinned host word: passes with the error word set
  uint32_t splits, stride, n_lists, tiles_per_split, tag_mask, width, block_rows;
  uint32_t n_rows;
  const uint32_t* count;   // where given: so many rows (at most n_rows), named by `rows`
  const uint32_t* rows;
  const __half* a;         // operands of all rows, and of all lists by units; factors and norm terms
  const __half* b;
  const float* factor;
  const float* norms;
  const float* x;
  const float* centers;
  uint32_t dim_ext;
  float alpha;
  uint32_t* labels;
  // rows that more units reach than are kept: to `next` while it has room, else to `last`
  uint32_t* next;
  uint32_t* next_count;
  uint32_t next_cap;
  uint32_t* last;
  uint32_t* last_count;
  unsigned long long* best;  // set to "none yet" for rows that go to `last`
};

// acc += a.lo b.lo + a.hi b.hi in fp32 (the halfs widen exactly)
__device__ __forceinline__ float fma_half2(uint32_t a, uint32_t b, float acc)
{
  asm("{\n\t.reg .b16 al, ah, bl, bh;\n\tmov.b32 {al, ah}, %1;\n\tmov.b32 {bl, bh}, %2;\n\t"
      "fma.rn.f32.f16 %0, al, bl, %0;\n\tfma.rn.f32.f16 %0, ah, bh, %0;\n\t}" : "+f"(acc) : "r"(a), "r"(b));
  return acc;
}

// A block per `block_rows` rows (at most kFinishRows), in steps that share the work evenly over its half warps:
//   1. two threads per row: which kept units are within 2 eps of the largest value;
//   2. a half warp per unit: the operands' products of its eight lists in fp32, two lanes per list (that takes the tensor
//      core's accumulation and the keys out of the bound), and which lists are within reach of the row's best one;
//   3. rows with several such lists, a half warp per list: the product summed in fp32 (that takes the rounding of the
//      operands out);
//   4. where that leaves several, a thread per list: the defining chain.
// What bounds it: latency, then L2 -- 8 operand rows per unit, 2.6 units per row on 1 M rows x 16,384 lists of 96 dimensions.
// With a warp, or half a warp, to itself a row's dependent reads took 1.3 and 1.1 ms there.
constexpr uint32_t kFinishRows = 64, kSecondRows = 32, kFinishUnits = 640, kFinishLists = 640;
__device__ __forceinline__ uint32_t half_warp_max(uint32_t v)
{
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) { v = max(v, __shfl_xor_sync(kFullMask, v, o)); }
  return v;
}
__global__ void __launch_bounds__(256, 6)
label_finish_kernel(const finish_params p)
{
  __shared__ uint32_t s_unit[kFinishUnits];        // unit's first list
  __shared__ uint8_t s_unit_row[kFinishUnits];
  __shared__ float s_val[kFinishUnits * kUnit];
  __shared__ uint32_t s_list[kFinishLists];
  __shared__ uint8_t s_list_row[kFinishLists];
  __shared__ float s_sum[kFinishLists];
  __shared__ unsigned long long s_key[kFinishRows];
  __shared__ float4 s_eps[kFinishRows];
  __shared__ uint32_t s_row[kFinishRows], s_best[kFinishRows], s_sum_best[kFinishRows], s_label[kFinishRows], s_n_sum[kFinishRows];
  __shared__ uint32_t s_n_list[kFinishRows], s_redo[kFinishRows], s_count[2];
  chain_begin();
  const uint32_t tid = threadIdx.x, lane = tid & 31u, l16 = lane & 15u, hw = tid >> 4;
  const uint32_t n   = p.count != nullptr ? min(__ldg(p.count), p.n_rows) : p.n_rows;
  const uint32_t w8 = p.width / 8u, n4 = p.dim_ext / 4u;
  const bool failed = *p.error != 0u;
  if (failed && n > 0 && blockIdx.x == 0 && tid == 0) { count_timeout(p.timeouts); }
  for (uint32_t i0 = blockIdx.x * p.block_rows; i0 < n; i0 += gridDim.x * p.block_rows) {
    if (tid < 2) { s_count[tid] = 0u; }
    __syncthreads();
    // ---- 1. units within reach ----
    if (tid < 2u * p.block_rows) {  // (whole warps)
      const uint32_t lr = tid >> 1, side = tid & 1u;  // thread: two column quarters of row lr
      const uint32_t i = min(i0 + lr, n - 1u);
      const uint32_t r = p.rows != nullptr ? __ldg(p.rows + i) : i;
      const float4 e   = __ldg(p.eps + r);
      auto keys_of = [&](uint32_t s, uint32_t c) {
        return __ldg(reinterpret_cast<const float4*>(p.keys) + (size_t(s) * p.stride + i) * 4u + side * 2u + c);
      };
      float top = -INFINITY, out = -INFINITY;  // largest value, largest that bounds units not kept
      for (uint32_t s = 0; s < p.splits; s++) {
        const float4 a = keys_of(s, 0), b = keys_of(s, 1);
        top = max3(top, a.x, b.x);
        out = max3(out, a.w, b.w);
      }
      top           = fmaxf(top, __shfl_xor_sync(kFullMask, top, 1));
      out           = fmaxf(out, __shfl_xor_sync(kFullMask, out, 1));
      const float t = top - 2.0f * e.x;
      // (negated: an infinite or undefined bound is not proof)
      bool redo = failed || !(out < t);
      for (uint32_t s = 0; !redo && s < p.splits; s++) {
#pragma unroll
        for (uint32_t c = 0; c < 2; c++) {
          const float4 a   = keys_of(s, c);
          const float k[3] = {a.x, a.y, a.z};
          const uint32_t m = (k[0] >= t ? 1u : 0u) + (k[1] >= t ? 1u : 0u) + (k[2] >= t ? 1u : 0u);  // (they are in order)
          if (m == 0u || redo) { continue; }
          const uint32_t at = atomicAdd(&s_count[0], m);
          if (at + m > kFinishUnits) { redo = true; }
#pragma unroll
          for (uint32_t j = 0; j < 3; j++) {
            if (j >= m || at + j >= kFinishUnits) { continue; }
            const uint32_t id   = __float_as_uint(k[j]) & p.tag_mask;
            s_unit[at + j]      = (s * p.tiles_per_split + id / kUnitsPerTile) * kLists + (side * 2u + c) * 64u + (id % kUnitsPerTile) * kUnit;
            s_unit_row[at + j]  = uint8_t(lr);
          }
        }
      }
      redo = __shfl_xor_sync(kFullMask, redo ? 1 : 0, 1) != 0 || redo;
      if (side == 0u) {
        s_row[lr]      = r;
        s_eps[lr]      = e;
        s_redo[lr]     = redo ? 1u : 0u;
        s_best[lr]     = 0u;
        s_sum_best[lr] = 0u;
        s_n_list[lr]   = 0u;
        s_n_sum[lr]    = 0u;
        s_key[lr]      = ~0ull;
      }
    }
    __syncthreads();
    // (every entry below this is written; units that had no room are not there: their rows are redone)
    const uint32_t n_units = min(s_count[0], kFinishUnits);
    // ---- 2. their lists ----
    for (uint32_t u0 = 0; u0 < n_units; u0 += 16u) {
      const uint32_t u  = u0 + hw;
      const bool has    = u < n_units;
      const uint32_t lr = has ? s_unit_row[u] : 0u, list0 = has ? s_unit[u] : 0u, list = list0 + (l16 & 7u);
      const bool look   = has && s_redo[lr] == 0u, valid = look && list < p.n_lists;
      float acc = 0.0f, acc1 = 0.0f;
      if (look) {
        // (lanes 0-7 and 8-15: neighbouring 16-byte chunks of the eight lists)
        const uint32_t r = s_row[lr];
        const uint4* av  = reinterpret_cast<const uint4*>(p.a + size_t(r) * p.width);
        const uint4* bv  = reinterpret_cast<const uint4*>(p.b) + size_t(list0 / kUnit) * w8 * kUnit + l16;
#pragma unroll 6
        for (uint32_t c = 0; c < w8; c += 2u) {
          const uint4 ac = __ldg(av + c + (l16 >> 3)), bc = __ldg(bv + c * kUnit);
          acc  = fma_half2(ac.x, bc.x, acc);
          acc1 = fma_half2(ac.y, bc.y, acc1);
          acc  = fma_half2(ac.z, bc.z, acc);
          acc1 = fma_half2(ac.w, bc.w, acc1);
        }
        if (l16 < 8u && valid) { acc1 = __fmaf_rn(__ldg(p.norms + list), -__ldg(p.factor + r), acc1); }
      }
      acc += acc1;
      acc += __shfl_xor_sync(kFullMask, acc, 8);
      const uint32_t mx = half_warp_max(valid ? float_to_ordered(acc) : 0u);
      if (has) {
        if (l16 < 8u) { s_val[u * kUnit + l16] = valid ? acc : -INFINITY; }
        if (l16 == 0u && mx != 0u) { atomicMax(&s_best[lr], mx); }
      }
    }
    __syncthreads();
    for (uint32_t v = tid; v < n_units * kUnit; v += 256u) {
      const uint32_t lr = s_unit_row[v / kUnit];
      if (s_redo[lr] == 0u && s_val[v] >= ordered_to_float(s_best[lr]) - 2.0f * s_eps[lr].y) {
        const uint32_t at = atomicAdd(&s_count[1], 1u), list = s_unit[v / kUnit] + v % kUnit;
        atomicAdd(&s_n_list[lr], 1u);
        s_label[lr] = list;  // (the only one, or another is found below)
        if (at < kFinishLists) {
          s_list[at]     = list;
          s_list_row[at] = uint8_t(lr);
        } else {
          s_n_list[lr] = 1u << 30;  // no room: the row is redone
        }
      }
    }
    __syncthreads();
    const uint32_t n_lists = min(s_count[1], kFinishLists);
    // ---- 3. rows with several ----
    for (uint32_t c0 = 0; c0 < n_lists; c0 += 16u) {
      const uint32_t c  = c0 + hw;
      const uint32_t lr = c < n_lists ? s_list_row[c] : 0u;
      const bool has    = c < n_lists && s_n_list[lr] > 1u;
      if (!__any_sync(kFullMask, has)) { continue; }
      float acc = 0.0f;
      if (has) {
        const float4* x  = reinterpret_cast<const float4*>(p.x + size_t(s_row[lr]) * p.dim_ext);
        const float4* cv = reinterpret_cast<const float4*>(p.centers + size_t(s_list[c]) * p.dim_ext);
#pragma unroll 2
        for (uint32_t k4 = l16; k4 < n4; k4 += 16u) {
          const float4 a = __ldg(cv + k4), b = __ldg(x + k4);
          acc = __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, __fmaf_rn(a.z, b.z, __fmaf_rn(a.w, b.w, acc))));
        }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) { acc += __shfl_xor_sync(kFullMask, acc, o); }
      if (has && l16 == 0u) {
        s_sum[c] = acc;
        atomicMax(&s_sum_best[lr], float_to_ordered(acc));
      }
    }
    __syncthreads();
    auto close = [&](uint32_t c, uint32_t lr) {
      return s_n_list[lr] > 1u && s_sum[c] >= ordered_to_float(s_sum_best[lr]) - 2.0f * s_eps[lr].z;
    };
    for (uint32_t c = tid; c < n_lists; c += 256u) {
      const uint32_t lr = s_list_row[c];
      if (close(c, lr)) {
        atomicAdd(&s_n_sum[lr], 1u);
        s_label[lr] = s_list[c];
      }
    }
    __syncthreads();
    // ---- 4. near ties ----
    for (uint32_t c = tid; c < n_lists; c += 256u) {
      const uint32_t lr = s_list_row[c];
      if (s_n_sum[lr] > 1u && close(c, lr)) {
        atomicMin(&s_key[lr], exact_key(p.x + size_t(s_row[lr]) * p.dim_ext, p.centers, s_list[c], p.dim_ext, p.alpha));
      }
    }
    __syncthreads();
    if (tid < p.block_rows && i0 + tid < n) {
      const uint32_t r = s_row[tid];
      if (s_redo[tid] != 0u || s_n_list[tid] >= (1u << 30)) {
        uint32_t at = p.next_cap;
        if (!failed && p.next_cap > 0) { at = atomicAdd(p.next_count, 1u); }
        if (at < p.next_cap) {
          p.next[at] = r;
        } else {
          p.last[atomicAdd(p.last_count, 1u)] = r;
          p.best[r]                           = ~0ull;
        }
      } else {
        p.labels[r] = s_n_sum[tid] > 1u ? uint32_t(s_key[tid]) : s_label[tid];
      }
    }
    __syncthreads();
  }
}

uint32_t operand_width(uint32_t dim) { return round_up(dim, 16u); }

}  // namespace

// Below some 16 M products a whole exact pass costs less than these launches; fewer than 256 lists are not one tile.
bool label_tc_usable(uint32_t n_rows, uint32_t n_lists)
{
  return n_lists >= 256 && uint64_t(n_rows) * n_lists >= (1ull << 24);
}

size_t label_model_bytes(uint32_t n_lists, uint32_t dim, bool by_units)
{
  return unit_operand_at(n_lists, dim, operand_width(dim)) + (by_units ? size_t(round_up(n_lists, kUnit)) * operand_width(dim) * 2 : 0);
}

void prepare_label_model(cudaStream_t stream, const float* centers, uint32_t n_lists, uint32_t dim, uint32_t dim_ext, float weight,
                         bool by_units, void* model)
{
  auto* words = static_cast<uint32_t*>(model);
  auto* sum   = reinterpret_cast<float*>(static_cast<char*>(model) + kMeanAt);
  auto* norms = reinterpret_cast<float*>(static_cast<char*>(model) + norms_at(dim));
  auto* b     = reinterpret_cast<__half*>(static_cast<char*>(model) + operand_at(n_lists, dim));
  auto* units = by_units ? reinterpret_cast<__half*>(static_cast<char*>(model) + unit_operand_at(n_lists, dim, operand_width(dim))) : nullptr;
  CUDA_TRY(cudaMemsetAsync(model, 0, norms_at(dim), stream));
  const uint32_t shares = std::min<uint32_t>(64, ceildiv(n_lists, 64u));
  center_sum_kernel<<<dim3(ceildiv(dim, 32u), shares), dim3(32, 8), 0, stream>>>(centers, n_lists, dim, dim_ext, sum);
  center_stats_kernel<<<ceildiv<uint32_t>(n_lists, 8u), 256, 0, stream>>>(centers, n_lists, dim, dim_ext, weight, sum, words);
  center_operand_kernel<<<round_up(n_lists, kLists) / 8u, 256, 0, stream>>>(centers, n_lists, dim, dim_ext, operand_width(dim), weight, sum,
                                                                           words, norms, b, units);
  CUDA_TRY(cudaGetLastError());
}

namespace {
template <row_list_mode kMode>
void launch_row_list(const label_params& p, const CUtensorMap& ma, const CUtensorMap& mb, uint32_t items, int sm_count, cudaStream_t stream)
{
  constexpr size_t smem = kRoom + kNormSlots * kNormBytes + 1024 + 256;
  auto go = [&](auto kernel) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    launch_chained(kernel, std::min(uint32_t(sm_count), items), kThreads, smem, stream, ma, mb, p);
    CUDA_TRY(cudaGetLastError());
  };
  switch (p.k_blocks) {
    case 1: go(row_list_kernel<1, kMode>); break;
    case 2: go(row_list_kernel<2, kMode>); break;
    case 3: go(row_list_kernel<3, kMode>); break;
    default: go(row_list_kernel<0, kMode>);
  }
}

// One pass of row_list_kernel over up to `rows` rows: the lists are shared out (`splits`) where row tiles alone do not fill
// the SMs four times, and so that an item has at most kSplitTiles list tiles.
struct label_pass {
  uint32_t splits, tiles_per_split, tag_mask;
  label_pass(uint32_t rows, uint32_t n_lists, uint32_t items)
  {
    const uint32_t row_tiles = ceildiv(rows, kTileRows), n_tiles = ceildiv(n_lists, kLists);
    splits = ceildiv(n_tiles, kSplitTiles);
    while (splits < n_tiles && row_tiles * splits < items && splits < 16) { splits <<= 1; }
    splits          = std::min(splits, n_tiles);
    tiles_per_split = ceildiv(n_tiles, splits);
    splits          = ceildiv(n_tiles, tiles_per_split);
    tag_mask        = 1;
    while (tag_mask < tiles_per_split * kUnitsPerTile) { tag_mask <<= 1; }
    tag_mask--;
  }
};
// Rows whose reach the first pass does not settle go through a second one with the lists in eight shares, whose records keep
// eight times as many units: room for this many rows (what exceeds it is redone by the exact product).  On 300,000 8-bit rows
// against 4,000 lists a tenth of the rows go there.
constexpr uint32_t kSecondShares = 8;
uint32_t second_rows(uint32_t n_rows) { return round_up(std::max(n_rows / 4u, std::min(n_rows, 1024u)), kTileRows); }

struct label_layout {
  label_pass first, second;
  uint32_t cap;
  // (few rows: the first pass has as many shares already)
  bool second_pass() const { return second.splits > first.splits; }
  size_t o_a, o_factor, o_eps, o_keys, o_a2, o_factor2, o_keys2, o_next, o_last, o_words, o_best, total;
  label_layout(uint32_t n_rows, uint32_t n_lists, uint32_t dim, int sm_count)
    : first(n_rows, n_lists, 4u * uint32_t(sm_count)), second(1, n_lists, kSecondShares), cap(second_pass() ? second_rows(n_rows) : 0)
  {
    const size_t row = size_t(operand_width(dim)) * 2;
    ws_layout lay;
    o_a     = lay.add(n_rows * row);
    o_factor = lay.add(size_t(n_rows) * 4);
    o_eps   = lay.add(size_t(n_rows) * 16);
    o_keys  = lay.add(size_t(first.splits) * n_rows * 64);
    o_a2    = lay.add(cap * row);
    o_factor2 = lay.add(size_t(cap) * 4);
    o_keys2 = lay.add(size_t(second.splits) * cap * 64);
    o_next  = lay.add(size_t(cap) * 4);
    o_last  = lay.add(size_t(n_rows) * 4);
    o_words = lay.add(256);
    o_best  = lay.add(size_t(n_rows) * 8);
    total   = lay.total();
  }
};
}  // namespace

size_t label_workspace_bytes(const raft::resources& res, uint32_t n_rows, uint32_t n_lists, uint32_t dim)
{
  return label_layout(n_rows, n_lists, dim, res.sm_count).total;
}

void label_rows_tc(raft::resources& res, const float* centers, const void* model, uint32_t n_lists, uint32_t dim,
                   uint32_t dim_ext, float alpha, const float* x_ext, uint32_t n_rows, uint32_t* labels, void* workspace)
{
  if (n_rows == 0) { return; }
  const label_layout y(n_rows, n_lists, dim, res.sm_count);
  const uint32_t width = operand_width(dim);
  char* ws             = static_cast<char*>(workspace);
  auto* a              = reinterpret_cast<__half*>(ws + y.o_a);
  auto* a2             = reinterpret_cast<__half*>(ws + y.o_a2);
  auto* factor         = reinterpret_cast<float*>(ws + y.o_factor);
  auto* factor2        = reinterpret_cast<float*>(ws + y.o_factor2);
  auto* eps            = reinterpret_cast<float4*>(ws + y.o_eps);
  auto* keys           = reinterpret_cast<float4*>(ws + y.o_keys);
  auto* keys2          = reinterpret_cast<float4*>(ws + y.o_keys2);
  auto* next           = reinterpret_cast<uint32_t*>(ws + y.o_next);
  auto* last           = reinterpret_cast<uint32_t*>(ws + y.o_last);
  auto* best           = reinterpret_cast<unsigned long long*>(ws + y.o_best);
  auto* words          = reinterpret_cast<uint32_t*>(ws + y.o_words);  // errors of the passes, rows in `next` and `last`
  const auto* stats    = static_cast<const uint32_t*>(model);
  const auto* sum      = reinterpret_cast<const float*>(static_cast<const char*>(model) + kMeanAt);
  const auto* norms    = reinterpret_cast<const float*>(static_cast<const char*>(model) + norms_at(dim));
  const auto* b        = reinterpret_cast<const __half*>(static_cast<const char*>(model) + operand_at(n_lists, dim));
  cudaStream_t stream  = res.stream;
  // (a key's low bits number its unit: of a value below 0.5 that takes less than tag_mask + 1 units of 2^-25)
  const float key_error = float(std::max(y.first.tag_mask, y.second.tag_mask) + 1u) * 0x1p-25f;
  auto operand = [&](auto kernel) {
    launch_chained(kernel, ceildiv<uint32_t>(n_rows, 32u), 256, 0, stream, x_ext, n_rows, n_lists, dim, dim_ext, width, sum, stats,
                   key_error, a, factor, eps, reinterpret_cast<uint4*>(words));
  };
  if (width <= 128) {
    operand(row_operand_kernel<true>);
  } else {
    operand(row_operand_kernel<false>);
  }
  label_params p{};
  p.k_steps  = width / 16;
  p.k_blocks = ceildiv(width, kBlockK);
  p.n_tiles  = ceildiv(n_lists, kLists);
  p.norms    = norms;
  const wait_limits wl = tc_wait_limits();
  p.spin_limit = wl.spin_limit;
  p.skip_kb    = wl.skip_kb;
  const CUtensorMap mb = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, b, n_lists, width, kLists, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  finish_params f{};
  f.eps = eps;
  f.timeouts = res.pinned + 13;
  f.n_lists = n_lists;
  f.width = width;
  f.a = a;
  f.b = reinterpret_cast<const __half*>(static_cast<const char*>(model) + unit_operand_at(n_lists, dim, width));
  f.factor = factor;
  f.norms = norms;
  f.x = x_ext;
  f.centers = centers;
  f.dim_ext = dim_ext;
  f.alpha = alpha;
  f.labels = labels;
  f.last = last;
  f.last_count = words + 3;
  f.best = best;
  auto pass = [&](const label_pass& s, const __half* operand, const float* factors, float4* k, uint32_t rows, uint32_t* error, const uint32_t* count,
                  uint32_t block_rows, uint32_t finish_blocks) {
    p.n_rows = f.n_rows = f.stride = rows;
    f.block_rows = block_rows;
    p.count = f.count = count;
    p.splits = f.splits = s.splits;
    p.tiles_per_split = f.tiles_per_split = s.tiles_per_split;
    p.tag_mask = f.tag_mask = s.tag_mask;
    p.keys = k;
    p.factor = factors;
    f.keys = reinterpret_cast<const float*>(k);
    p.error = error;
    f.error = error;
    const CUtensorMap ma = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, operand, rows, width, kRows, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
    const uint32_t items = ceildiv(rows, kTileRows) * s.splits;
    launch_row_list<kKeys>(p, ma, mb, items, res.sm_count, stream);
    launch_chained(label_finish_kernel, finish_blocks, 256, 0, stream, f);
    CUDA_TRY(cudaGetLastError());
  };
  f.next = next;
  f.next_count = words + 2;
  f.next_cap = y.second_pass() ? y.cap : 0;
  pass(y.first, a, factor, keys, n_rows, words, nullptr, kFinishRows, ceildiv(n_rows, kFinishRows));
  res.launches += 3;
  if (y.second_pass()) {
    const uint32_t few = std::min<uint32_t>(uint32_t(res.sm_count) * 8, ceildiv(y.cap, 8u));
    launch_chained(gather_operand_kernel, few, 256, 0, stream, a, factor, next, words + 2, y.cap, width, a2, factor2,
                   res.redo_counts + raft::resources::LABELS_SECOND);
    f.rows = next;
    f.next_cap = 0;
    pass(y.second, a2, factor2, keys2, y.cap, words + 1, words + 2,
         kSecondRows, std::min<uint32_t>(uint32_t(res.sm_count) * 4, ceildiv(y.cap, kSecondRows)));
    res.launches += 3;
  }
  assign_nearest_listed(res, centers, n_lists, dim_ext, alpha, x_ext, n_rows, last, words + 3, labels, best);
}

// ------------------------------------------------------------------------------------------------
// The nearest lists of a batch of queries (search's coarse stage), exact: probes ordered by (score, list), the score being
// the defining fp32 chain.
//
// Two passes of row_list_kernel and no score matrix.  The first writes the largest value of every `unit` lists; the n_probes-th
// largest of a query's maxima, T, is a value that n_probes lists reach, so a wanted list has a value of at least T - 2 eps.
// The second emits the lists that do (some n_probes of them where lists are many).  Those are scored with the defining
// chain and ranked.  Queries that have no bound, or more lists within reach than there is room for, are redone exactly
// over all lists (coarse_tc.cu).
//
// Measured (us, coarse stage): 10,000 queries x 50,000 lists, 20 probes: 553 by candidate keys (coarse_tc.cu) -> 270; 4,000 x
// 12,288, 128 probes: 585 by the exact product and row selection -> 290; 10,000 x 4,000, 64 probes: 436 -> 230.  What is left is the
// exact scores (half), then the two passes.
// ------------------------------------------------------------------------------------------------
namespace {

// A warp per query: a value that at least n_probes of its maxima reach, from twelve halvings of their range, less 2 eps.
template <uint32_t kPer>
__global__ void __launch_bounds__(256)
probe_threshold_kernel(const float* __restrict__ maxima, uint32_t n_units, uint32_t stride, uint32_t n_rows, uint32_t n_probes,
                       const float4* __restrict__ eps, float* __restrict__ threshold, uint32_t* __restrict__ redo,
                       uint32_t* __restrict__ n_redo)
{
  chain_begin();
  const uint32_t r = (blockIdx.x * 256u + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
  if (r >= n_rows) { return; }
  const float4* src = reinterpret_cast<const float4*>(maxima + size_t(r) * stride);  // the stride is a multiple of four
  float v[kPer];
  float lo = INFINITY, hi = -INFINITY;
#pragma unroll
  for (uint32_t i = 0; i < kPer; i += 4) {
    const uint32_t at = i * 8u + lane;
    const float4 x    = at * 4u < n_units ? __ldg(src + at) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
#pragma unroll
    for (uint32_t e = 0; e < 4; e++) {
      // (nothing, or nothing but lists that are not there)
      if (at * 4u + e >= n_units || v[i + e] < -1e20f) { v[i + e] = -INFINITY; }
      hi = fmaxf(hi, v[i + e]);
      lo = v[i + e] > -INFINITY ? fminf(lo, v[i + e]) : lo;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(kFullMask, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(kFullMask, hi, o));
  }
  // (all of them reach the smallest, and there are at least n_probes)
  for (int step = 0; step < 12; step++) {
    const float mid = 0.5f * (lo + hi);
    uint32_t n      = 0;
#pragma unroll
    for (uint32_t i = 0; i < kPer; i++) { n += v[i] >= mid ? 1u : 0u; }
    n = __reduce_add_sync(kFullMask, n);
    if (n >= n_probes) {
      lo = mid;
    } else {
      hi = mid;
    }
  }
  if (lane == 0) {
    float t         = lo - 2.0f * __ldg(eps + r).x;
    const bool fine = t > -INFINITY && t < INFINITY;  // (false for NaN)
    if (!fine) {
      redo[atomicAdd(n_redo, 1u)] = r;
      t                           = INFINITY;
    }
    threshold[r] = t;
  }
}

constexpr uint32_t kMaxSegments   = 64;
constexpr uint32_t kChainCols     = 64;   // columns staged at a time

// A warp per query: the places found, whose lists go 32 at a time through shared memory, one per lane with the defining chain (the next
// columns are on their way while some are used); a list's rank is the number of lists before it.
// What bounds it: L1, which the centres' rows and shared memory share, 69% busy (8,000 queries x 128 probes x 96 dimensions: 123 us; 86% for
// 2,000 x 100 x 768: 181), and the latency of shared memory, whose four or five blocks per SM are few warps.  Bulk copies of a
// lane's own row, 256 bytes each, took as long or longer (768 dimensions: 300 against 250 us).
constexpr uint32_t kProbeWarps = 4, kChainPitch = kChainCols + 4u;
// (a cap that is a multiple of eight, fourteen bytes each: the next warp's rows start on 16)
__host__ __device__ __forceinline__ uint32_t probe_warp_bytes(uint32_t cap)
{
  return (32u * kChainPitch + kChainCols) * 4u + cap * 14u;
}
__global__ void __launch_bounds__(kProbeWarps * 32)
probe_finish_kernel(const uint32_t* __restrict__ found, const uint32_t* __restrict__ n_found, uint32_t segments, uint32_t found_cap,
                    const float* __restrict__ fq, const float* __restrict__ centers, uint32_t n_lists, uint32_t dim_ext,
                    float alpha, uint32_t n_queries, uint32_t n_probes, uint32_t cap, const float* __restrict__ threshold,
                    const uint32_t* __restrict__ error, uint32_t* __restrict__ timeouts, uint32_t* __restrict__ probes,
                    uint32_t* __restrict__ redo, uint32_t* __restrict__ n_redo)
{
  // per warp: [32][kChainPitch] columns, [kChainCols] of the query, [cap] scores (order-preserving), lists, places and ranks
  extern __shared__ __align__(16) uint8_t s_probe[];
  __shared__ uint32_t s_first[kProbeWarps][kMaxSegments];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, q = blockIdx.x * kProbeWarps + warp;
  const uint32_t bytes = probe_warp_bytes(cap);
  float* s_rows  = reinterpret_cast<float*>(s_probe + warp * bytes);
  float* s_query = s_rows + 32u * kChainPitch;
  auto* s_score  = reinterpret_cast<uint32_t*>(s_query + kChainCols);
  uint32_t *s_list = s_score + cap, *s_place = s_list + cap;
  auto* s_rank   = reinterpret_cast<uint16_t*>(s_place + cap);
  chain_begin();
  const bool there      = q < n_queries;
  const uint32_t failed = __ldg(error);
  const float limit     = there ? __ldg(threshold + q) : INFINITY;
  // (at most 64 segments, two per lane)
  uint32_t n_seg[2], sum = 0;
  bool fits = true;
#pragma unroll
  for (uint32_t i = 0; i < 2; i++) {
    n_seg[i] = there && 2u * lane + i < segments ? __ldg(n_found + size_t(q) * segments + 2u * lane + i) : 0u;
    fits     = fits && n_seg[i] <= found_cap;
    n_seg[i] = min(n_seg[i], cap + 1u);
    sum += n_seg[i];
  }
  if (failed != 0u) {  // every query is redone
    if (q == 0 && lane == 0) { count_timeout(timeouts); }
    return;
  }
  if (limit == INFINITY) { return; }  // (listed already)
  uint32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(kFullMask, inc, o);
    if (lane >= uint32_t(o)) { inc += x; }
  }
  const uint32_t n = __shfl_sync(kFullMask, inc, 31);
  if (!__all_sync(kFullMask, fits) || n > cap || n < n_probes) {
    if (lane == 0) { redo[atomicAdd(n_redo, 1u)] = q; }
    return;
  }
  s_first[warp][2u * lane]      = inc - sum;
  s_first[warp][2u * lane + 1u] = inc - n_seg[1];
  __syncwarp();
  for (uint32_t i = lane; i < n; i += 32u) {
    // the last segment that starts at or before i (an empty one starts where the next does)
    uint32_t seg = 0;
#pragma unroll
    for (uint32_t step = kMaxSegments / 2u; step > 0; step >>= 1) { seg += s_first[warp][seg + step] <= i ? step : 0u; }
    s_list[i] = list_at(__ldg(found + (size_t(q) * segments + seg) * found_cap + (i - s_first[warp][seg])), n_lists);
  }
  __syncwarp();
  // sixteen lanes per row; step: (32 lists, kChainCols columns)
  float4 v[16], x;
  auto load = [&](uint32_t c0, uint32_t k0) {
    const uint32_t k4 = k0 / 4u + (lane & 15u);
    const bool in     = k4 < dim_ext / 4u;
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) {
      const uint32_t c = c0 + 2u * i + (lane >> 4);
      if (in && c < n) { v[i] = __ldg(reinterpret_cast<const float4*>(centers + size_t(s_list[c]) * dim_ext) + k4); }
    }
    if (in && lane < 16u) { x = __ldg(reinterpret_cast<const float4*>(fq + size_t(q) * dim_ext) + k4); }
  };
  load(0, 0);
  float acc = 0.0f;
  for (uint32_t c0 = 0, k0 = 0; c0 < n;) {
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) {
      *reinterpret_cast<float4*>(s_rows + (2u * i + (lane >> 4)) * kChainPitch + (lane & 15u) * 4u) = v[i];
    }
    if (lane < 16u) { *reinterpret_cast<float4*>(s_query + lane * 4u) = x; }
    __syncwarp();
    const uint32_t kn = min(kChainCols, dim_ext - k0) / 4u;  // dim_ext is a multiple of 8
    uint32_t next_c = c0, next_k = k0 + kChainCols;
    if (next_k >= dim_ext) {
      next_k = 0;
      next_c += 32u;
    }
    if (next_c < n) { load(next_c, next_k); }
    const float* mine = s_rows + lane * kChainPitch;
#pragma unroll 4
    for (uint32_t k = 0; k < kn; k++) {
      const float4 c = *reinterpret_cast<const float4*>(mine + k * 4u);
      const float4 y = *reinterpret_cast<const float4*>(s_query + k * 4u);
      acc = __fmaf_rn(c.x, y.x, acc);
      acc = __fmaf_rn(c.y, y.y, acc);
      acc = __fmaf_rn(c.z, y.z, acc);
      acc = __fmaf_rn(c.w, y.w, acc);
    }
    if (next_k == 0) {
      if (c0 + lane < n) { s_score[c0 + lane] = float_to_ordered(__fmul_rn(alpha, acc)); }
      acc = 0.0f;
    }
    c0 = next_c;
    k0 = next_k;
    __syncwarp();
  }
  // the rank by score, four lists of a lane at a time
  if (lane < 3u && n + lane < cap) { s_score[n + lane] = 0xFFFFFFFFu; }  // (read below in fours)
  __syncwarp();
  for (uint32_t c0 = 0; c0 < n; c0 += 128u) {
    uint32_t mine[4], rank[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) { mine[i] = c0 + i * 32u + lane < n ? s_score[c0 + i * 32u + lane] : 0u; }
    for (uint32_t o = 0; o < n; o += 4) {
      const uint4 y = *reinterpret_cast<const uint4*>(s_score + o);
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) {
        rank[i] += (y.x < mine[i] ? 1u : 0u) + (y.y < mine[i] ? 1u : 0u);
        rank[i] += (y.z < mine[i] ? 1u : 0u) + (y.w < mine[i] ? 1u : 0u);
      }
    }
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
      const uint32_t c = c0 + i * 32u + lane;
      if (c < n) {
        s_place[rank[i]] = c;
        s_rank[c]        = uint16_t(rank[i]);
      }
    }
  }
  __syncwarp();
  // Lists of equal score met at one place: then the order is by (score, list).  For each of them the warp counts the lists of
  // equal score before it.  (Among 350 scores of fp32 two are often equal, and more so where all are large.  When every lane
  // ranked its lists anew by both: 4,000 queries x 4,096 lists x 256 probes, 512 against 214 us for a whole selection; with centres
  // around a common offset of ten times their spread, 1,193 against 248.)
  constexpr uint32_t kMet = 1u << 31;
  bool tied = false;
  for (uint32_t c = lane; c < n; c += 32u) { tied = tied || s_place[s_rank[c]] != c; }
  if (__any_sync(kFullMask, tied)) {
    for (uint32_t c = lane; c < n; c += 32u) {
      if ((s_place[s_rank[c]] & ~kMet) != c) { atomicOr(s_place + s_rank[c], kMet); }
    }
    __syncwarp();
    for (uint32_t c0 = 0; c0 < n; c0 += 32u) {
      const uint32_t c = c0 + lane;
      const bool met   = c < n && (s_place[s_rank[c]] & kMet) != 0u;
      uint32_t rank    = c < n ? s_rank[c] : n_probes;
      for (unsigned left = __ballot_sync(kFullMask, met); left != 0u; left &= left - 1u) {
        const uint32_t one   = uint32_t(__ffs(int(left))) - 1u;
        const uint32_t score = s_score[c0 + one], list = s_list[c0 + one];
        uint32_t before      = 0;
        for (uint32_t o = lane; o < n; o += 32u) { before += s_score[o] == score && s_list[o] < list ? 1u : 0u; }
        before = __reduce_add_sync(kFullMask, before);
        if (lane == one) { rank += before; }
      }
      if (rank < n_probes) { probes[size_t(q) * n_probes + rank] = s_list[c]; }
    }
    return;
  }
  for (uint32_t r = lane; r < n_probes; r += 32u) { probes[size_t(q) * n_probes + r] = s_list[s_place[r]]; }
}
// Lists within reach that a query can have.
uint32_t probe_cap(uint32_t n_probes) { return round_up(2u * n_probes + 48u, 8u); }

// Lists per unit: as many as leave six times as many units as wanted lists, so that the maxima select sharply (8% more lists
// reach the threshold than are wanted, the lists of a unit being chosen at random: list_at); no fewer than a warp can hold the maxima of.
uint32_t probe_unit(uint32_t n_lists, uint32_t n_probes)
{
  for (uint32_t unit : {128u, 64u, 32u}) {
    if (n_lists / unit >= 6u * n_probes && n_lists <= unit * 2048u) { return unit; }
  }
  return n_lists <= 16384u ? 8u : (n_lists <= 65536u ? 32u : 64u);
}

struct probe_layout {
  uint32_t unit, n_units, max_stride, splits, tiles_per_split, found_cap;
  size_t o_a, o_factor, o_eps, o_maxima, o_threshold, o_found, o_n_found, o_redo, o_words, o_scratch, total;
  probe_layout(uint32_t n_queries, uint32_t n_lists, uint32_t n_probes, uint32_t dim, int sm_count)
  {
    const uint32_t row_tiles = ceildiv(n_queries, kTileRows), n_tiles = ceildiv(n_lists, kLists);
    unit       = probe_unit(n_lists, n_probes);
    n_units    = n_tiles * (kLists / unit);
    max_stride = round_up(n_units, 4u);
    // the split of the lists whose last wave is fullest: clocks of a list tile (products, or the epilogue) and of an item's
    // start (its row tile)
    const uint64_t tile = std::max(2u * 140u * (operand_width(dim) / 16u), 2600u), start = 4000;
    uint64_t best       = ~0ull;
    splits = tiles_per_split = 1;
    for (uint32_t s = 1; s <= std::min(n_tiles, kMaxSegments / 2u); s++) {
      const uint32_t per = ceildiv(n_tiles, s), n = ceildiv(n_tiles, per);
      const uint64_t cost = ceildiv<uint64_t>(uint64_t(row_tiles) * n, uint64_t(sm_count)) * (per * tile + start);
      if (cost < best) {
        best            = cost;
        splits          = n;
        tiles_per_split = per;
      }
    }
    found_cap = round_up(std::min(n_probes + n_probes / 4u + 32u, tiles_per_split * 128u), 4u);
    ws_layout lay;
    o_a         = lay.add(size_t(n_queries) * operand_width(dim) * 2);
    o_factor    = lay.add(size_t(n_queries) * 4);
    o_eps       = lay.add(size_t(n_queries) * 16);
    o_maxima    = lay.add(size_t(n_queries) * max_stride * 4);
    o_threshold = lay.add(size_t(n_queries) * 4);
    o_found     = lay.add(size_t(n_queries) * splits * 2 * found_cap * 4);
    o_n_found   = lay.add(size_t(n_queries) * splits * 2 * 4);
    o_redo      = lay.add(size_t(n_queries) * 4);
    o_words     = lay.add(256);
    o_scratch   = lay.add(probe_redo_bytes(n_queries, n_lists));
    total       = lay.total();
  }
};

}  // namespace

// From 2 M (query, list) pairs on, and more where a query has many probes for the lists: what the passes save grows with the pairs, what
// they cost beside with the probes (the finish) and where the maxima select less sharply.  Whole calls, 96 dimensions, by coarse_tc.cu or
// the exact product / so (us):
// - 20 probes: 1,000 x 4,096 146 / 122, 500 x 10,000 121 / 107, 4,000 x 10,000 378 / 214;
// - 1,000 lists: 32 probes, 2,200 queries 153 / 161, 4,500 231 / 231, 9,000 378 / 353; 48 probes 175 / 187, 274 / 280, 462 / 444;
// - 2,048 lists: 64 probes, 1,074 queries 157 / 165, 2,197 220 / 215; 128 probes, 4,394 502 / 518, 8,789 914 / 910, 19,531 1,943 / 1,910;
// - 4,096 lists: 128 probes, 1,098 queries 244 / 261, 2,197 351 / 345, 4,394 581 / 536; 256 probes, 2,197 511 / 558, 9,765 1,858 / 1,880
//   (512 dimensions: 1,100 queries 706 / 851, 4,400 2,112 / 2,329);
// - 8,192 lists: 256 probes, 549 queries 268 / 289, 1,098 425 / 444, 2,197 614 / 590; 16,384 lists: 549 288 / 297, 1,098 545 / 480.
// Beyond 16,384 lists, few queries are a matter of latency, where coarse_tc.cu has fewer steps, but not with many probes of many lists:
// 110 x 20,000, 20 probes 58 / 64, 100 probes 134 / 142, 300 queries, 20 probes 102 / 100; 100 x 32,768, 10 probes 49 / 59, 32 probes 64 /
// 75, 64 probes 135 / 132; 256 queries, 10 probes 61 / 68, 700 queries 140 / 130.
bool probes_tc_usable(uint32_t n_queries, uint32_t n_lists, uint32_t n_probes, uint32_t dim)
{
  const uint32_t unit = probe_unit(n_lists, n_probes);
  const double share  = double(n_probes) / n_lists;
  return n_lists >= 256 && n_lists <= 131072 && n_probes <= 256 && n_lists / unit >= 2 * n_probes && dim <= 4096 &&
         uint64_t(n_queries) * n_lists >= (1ull << 21) && n_queries >= 2.5e6 * share * share &&
         (n_lists <= 16384 || (n_lists < 32768 ? n_queries > 128 : n_queries > 256 || n_probes >= 64));
}

size_t probes_workspace_bytes(const raft::resources& res, uint32_t n_queries, uint32_t n_lists, uint32_t n_probes, uint32_t dim)
{
  return probe_layout(n_queries, n_lists, n_probes, dim, res.sm_count).total;
}

void select_probes_tc(raft::resources& res, const float* centers, const void* model, uint32_t n_lists, uint32_t dim, uint32_t dim_ext,
                      float alpha, const float* fq, uint32_t n_queries, uint32_t max_queries, uint32_t n_probes, uint32_t* probes,
                      void* workspace)
{
  const probe_layout y(max_queries, n_lists, n_probes, dim, res.sm_count);
  const uint32_t width = operand_width(dim);
  char* ws             = static_cast<char*>(workspace);
  auto* a              = reinterpret_cast<__half*>(ws + y.o_a);
  auto* factor         = reinterpret_cast<float*>(ws + y.o_factor);
  auto* eps            = reinterpret_cast<float4*>(ws + y.o_eps);
  auto* maxima         = reinterpret_cast<float*>(ws + y.o_maxima);
  auto* threshold      = reinterpret_cast<float*>(ws + y.o_threshold);
  auto* found          = reinterpret_cast<uint32_t*>(ws + y.o_found);
  auto* n_found        = reinterpret_cast<uint32_t*>(ws + y.o_n_found);
  auto* redo           = reinterpret_cast<uint32_t*>(ws + y.o_redo);
  auto* words          = reinterpret_cast<uint32_t*>(ws + y.o_words);  // error, queries redone, queries to redo
  const auto* sum      = reinterpret_cast<const float*>(static_cast<const char*>(model) + kMeanAt);
  const auto* norms    = reinterpret_cast<const float*>(static_cast<const char*>(model) + norms_at(dim));
  const auto* b        = reinterpret_cast<const __half*>(static_cast<const char*>(model) + operand_at(n_lists, dim));
  cudaStream_t stream  = res.stream;
  auto operand = [&](auto kernel) {
    launch_chained(kernel, ceildiv<uint32_t>(n_queries, 32u), 256, 0, stream, fq, n_queries, n_lists, dim, dim_ext, width, sum,
                   static_cast<const uint32_t*>(model), 0.0f, a, factor, eps, reinterpret_cast<uint4*>(words));
  };
  if (width <= 128) {
    operand(row_operand_kernel<true>);
  } else {
    operand(row_operand_kernel<false>);
  }
  label_params p{};
  p.n_rows = n_queries;
  p.k_steps = width / 16;
  p.k_blocks = ceildiv(width, kBlockK);
  p.n_tiles = ceildiv(n_lists, kLists);
  p.tiles_per_split = y.tiles_per_split;
  p.splits = y.splits;
  p.norms = norms;
  p.factor = factor;
  p.maxima = maxima;
  p.unit = y.unit;
  p.max_stride = y.max_stride;
  p.threshold = threshold;
  p.found = found;
  p.n_found = n_found;
  p.found_cap = y.found_cap;
  p.error = words;
  const wait_limits wl = tc_wait_limits();
  p.spin_limit = wl.spin_limit;
  p.skip_kb = wl.skip_kb;
  const CUtensorMap ma = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a, n_queries, width, kRows, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  const CUtensorMap mb = make_map_2d(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, b, n_lists, width, kLists, kBlockK, CU_TENSOR_MAP_SWIZZLE_128B);
  const uint32_t items = ceildiv(n_queries, kTileRows) * y.splits;
  launch_row_list<kMaxima>(p, ma, mb, items, res.sm_count, stream);
  auto threshold_of = [&](auto kernel) {
    launch_chained(kernel, ceildiv(n_queries, 8u), 256, 0, stream, maxima, y.n_units, y.max_stride, n_queries, n_probes, eps, threshold, redo, words + 2);
  };
  if (y.n_units <= 256) {
    threshold_of(probe_threshold_kernel<8>);
  } else if (y.n_units <= 512) {
    threshold_of(probe_threshold_kernel<16>);
  } else if (y.n_units <= 1024) {
    threshold_of(probe_threshold_kernel<32>);
  } else {
    threshold_of(probe_threshold_kernel<64>);
  }
  launch_row_list<kEmit>(p, ma, mb, items, res.sm_count, stream);
  const size_t finish_smem = kProbeWarps * probe_warp_bytes(probe_cap(n_probes));
  ensure_dynamic_smem(reinterpret_cast<const void*>(probe_finish_kernel), finish_smem);
  launch_chained(probe_finish_kernel, ceildiv(n_queries, kProbeWarps), kProbeWarps * 32, finish_smem, stream, found, n_found,
                 2u * y.splits, y.found_cap, fq, centers, n_lists, dim_ext, alpha, n_queries, n_probes, probe_cap(n_probes), threshold, words,
                 res.pinned + 13, probes, redo, words + 2);
  CUDA_TRY(cudaGetLastError());
  // how many: looked at before a later batch, which may then go to the exact product
  uint32_t* host_words = res.tc_redo_record(n_queries, n_probes, n_lists, true);
  launch_probe_redo(res, redo, words, centers, fq, n_queries, max_queries, n_lists, dim_ext, alpha, n_probes,
                    reinterpret_cast<float*>(ws + y.o_scratch), probes, nullptr, host_words, res.tc_redo_seq);
  res.launches += 5;
}

}  // namespace cuvs::neighbors::ivf_pq
