// Coarse stage: choose, for every query, the n_probes nearest inverted lists.
//
// Reference: select_clusters, cpp/src/neighbors/ivf_pq/ivf_pq_search.cuh:61-168 -- one fp32 GEMM
// (queries x centers over dim_ext, the squared norm of each center riding in column `dim` against a
// query entry of -0.5) followed by select_k.  Here the exact score of a (query, list) pair is
// defined as the fp32 FMA chain over ascending k, scaled by alpha, and probes are ordered by
// (score, list id), which makes the selection deterministic.
//
// This file holds the exact SIMT path: a register-tiled fp32 product (each output accumulated by
// one thread in ascending k, so it equals the defining chain bit for bit) and a per-query radix
// select.  It is the general path (any n_probes up to 4096, any shape).
#include "common.hpp"
#include "packed.cuh"
#include "row_select.cuh"
#include "search_internal.hpp"
#include "topk.cuh"

#include <algorithm>

namespace cuvs::neighbors::ivf_pq {

using namespace cuvs_b200;

namespace {

constexpr uint32_t kMaxProbes = 4096;



// out[i, j] = alpha * sum over ascending k of b[j, k] * a[i, k], one fused multiply-add chain per output (the chain that
// defines a coarse score, a rotation, a label).  kArgmin: instead of storing, best[i] = min over j of
// (ordered score << 32 | j), "lowest score, then lowest id".
// What bounds it: the FMA pipe, and shared-memory wavefronts close behind.  128 x 128 outputs per block, 8 x 8 per thread
// as packed pairs of columns (fma.rn.f32x2: two chains per instruction), a warp 4 x 8 threads so that its loads are
// 64 and 128 distinct bytes; the next eight k are on their way while eight are used.
// 10,000 x 4,000 x 136: 487 us with 64 x 64 outputs per block and scalar FMAs, 238 us so.  kVec: rows of both operands are
// 16-byte aligned and k is a multiple of four.  kListed: the rows of `a` (and of `best`) named by row_list, *n_listed of them.
constexpr uint32_t kTile = 128, kTileK = 8, kListedBlocks = 2368;
template <bool kVec, bool kArgmin, bool kListed>
__global__ void __launch_bounds__(256, 2)
exact_gemm_kernel(const float* __restrict__ b, uint32_t n_cols, const float* __restrict__ a, uint32_t n_rows, uint32_t a_stride,
                  uint32_t kdim, float alpha, int half_scores, float* __restrict__ out, unsigned long long* __restrict__ best,
                  const uint32_t* __restrict__ row_list, const uint32_t* __restrict__ n_listed)
{
  chain_begin();
  __shared__ __align__(16) float s_a[2][kTileK][kTile + 4];
  __shared__ __align__(16) float s_b[2][kTileK][kTile + 4];
  const uint32_t tid = threadIdx.x;
  const uint32_t tx = ((tid >> 5) & 1u) * 8u + (tid & 7u), ty = (tid >> 6) * 4u + ((tid >> 3) & 3u);
  if constexpr (kListed) { n_rows = min(n_rows, __ldg(n_listed)); }
  // (listed rows: sixteen blocks per SM take the tiles in turn, since the host does not know how many there are; else each
  // block has one)
  uint32_t j0 = blockIdx.x * kTile, i0 = blockIdx.y * kTile, tile = blockIdx.x;
  [[maybe_unused]] const uint32_t across = (n_cols + kTile - 1u) / kTile;
  auto place = [&] {
    j0 = tile % across * kTile;
    i0 = tile / across * kTile;
  };
  if constexpr (kListed) {
    place();
    if (i0 >= n_rows) { return; }
  }
  // one row and four k of either operand per thread
  const uint32_t lrow = tid >> 1, lk = (tid & 1u) * 4u;
  bool in_a, in_b;
  const float *pa, *pb;
  float ra[4], rb[4];
  auto rows_of_tile = [&] {
    in_a = i0 + lrow < n_rows;
    in_b = j0 + lrow < n_cols;
    pa   = a + size_t(kListed && in_a ? __ldg(row_list + i0 + lrow) : i0 + lrow) * a_stride + lk;
    pb   = b + size_t(j0 + lrow) * kdim + lk;
  };
  rows_of_tile();
  auto load = [&](uint32_t k0) {
    if constexpr (kVec) {
      const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float4 x = in_a && k0 + lk < kdim ? __ldg(reinterpret_cast<const float4*>(pa + k0)) : z;
      const float4 y = in_b && k0 + lk < kdim ? __ldg(reinterpret_cast<const float4*>(pb + k0)) : z;
      ra[0] = x.x; ra[1] = x.y; ra[2] = x.z; ra[3] = x.w;
      rb[0] = y.x; rb[1] = y.y; rb[2] = y.z; rb[3] = y.w;
    } else {
#pragma unroll
      for (uint32_t e = 0; e < 4; e++) {
        const bool in = k0 + lk + e < kdim;
        ra[e]         = in && in_a ? __ldg(pa + k0 + e) : 0.0f;
        rb[e]         = in && in_b ? __ldg(pb + k0 + e) : 0.0f;
      }
    }
  };
  auto store = [&](uint32_t buf) {
#pragma unroll
    for (uint32_t e = 0; e < 4; e++) {
      s_a[buf][lk + e][lrow] = ra[e];
      s_b[buf][lk + e][lrow] = rb[e];
    }
  };
  load(0);
  do {
    // rows ty * 4 + {0..3} and 64 + ..., columns tx * 4 + {0..3} and 64 + ...
    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++) {
#pragma unroll
      for (int j = 0; j < 4; j++) { acc[i][j] = 0ull; }
    }
    store(0);
    __syncthreads();
    uint32_t buf = 0;
    for (uint32_t k0 = 0; k0 < kdim; k0 += kTileK, buf ^= 1u) {
      const bool more = k0 + kTileK < kdim;
      if (more) { load(k0 + kTileK); }
      // (a partial last tile stops at kdim: a product with zero would leave the chain's value alone, except for -0 and
      // infinities)
      const uint32_t kn = min(kTileK, kdim - k0);
      auto step = [&](uint32_t k) {
        const float4 x0 = *reinterpret_cast<const float4*>(&s_a[buf][k][ty * 4u]);
        const float4 x1 = *reinterpret_cast<const float4*>(&s_a[buf][k][64u + ty * 4u]);
        const ulonglong2 c0 = *reinterpret_cast<const ulonglong2*>(&s_b[buf][k][tx * 4u]);
        const ulonglong2 c1 = *reinterpret_cast<const ulonglong2*>(&s_b[buf][k][64u + tx * 4u]);
        const uint64_t x[8] = {dup2(x0.x), dup2(x0.y), dup2(x0.z), dup2(x0.w), dup2(x1.x), dup2(x1.y), dup2(x1.z), dup2(x1.w)};
        const uint64_t c[4] = {c0.x, c0.y, c1.x, c1.y};
#pragma unroll
        for (int i = 0; i < 8; i++) {
#pragma unroll
          for (int j = 0; j < 4; j++) { acc[i][j] = fma2(c[j], x[i], acc[i][j]); }
        }
      };
      if (kn == kTileK) {
#pragma unroll
        for (uint32_t k = 0; k < kTileK; k++) { step(k); }
      } else {
        for (uint32_t k = 0; k < kn; k++) { step(k); }
      }
      if (more) {
        store(buf ^ 1u);
        __syncthreads();
      }
    }
    [[maybe_unused]] const uint32_t row0 = i0, col0 = j0;
    if constexpr (kListed) {
      // the next tile's first columns are on their way while this one's results are handed over
      tile += gridDim.x;
      place();
      if (i0 < n_rows) {
        rows_of_tile();
        load(0);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t row = row0 + (i < 4 ? ty * 4u + i : 64u + ty * 4u + (i - 4));
      [[maybe_unused]] unsigned long long m = ~0ull;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t col = col0 + h * 64u + tx * 4u;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const uint64_t pair = acc[i][h * 2 + (e >> 1)];
          v[e] = __fmul_rn(alpha, __uint_as_float(uint32_t((e & 1) ? (pair >> 32) : pair)));
          // fp16 coarse search: the score is a half-precision number
          if (half_scores) { v[e] = __half2float(__float2half_rn(v[e])); }
        }
        if constexpr (kArgmin) {
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const unsigned long long key = ((unsigned long long)float_to_ordered(v[e]) << 32) | (col + e);
            if (col + e < n_cols) { m = key < m ? key : m; }
          }
        } else if (row < n_rows) {
          float* o = out + size_t(row) * n_cols + col;
          if (n_cols % 4 == 0 && col < n_cols) {
            *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; e++) {
              if (col + e < n_cols) { o[e] = v[e]; }
            }
          }
        }
      }
      if constexpr (kArgmin) {
        // eight lanes of a warp share a row: reduce before touching memory
#pragma unroll
        for (int d = 4; d > 0; d >>= 1) {
          const unsigned long long o = __shfl_xor_sync(kFullMask, m, d);
          m = o < m ? o : m;
        }
        if ((tid & 7u) == 0 && row < n_rows) { atomicMin(best + (kListed ? __ldg(row_list + row) : row), m); }
      }
    }
    if constexpr (kListed) { __syncthreads(); }
  } while (kListed && i0 < n_rows);
}

// The same product for a few rows (at most kFewRows), where the tiles above would leave the chip empty and the time is
// the latency of one block (1 x 1,024 x 136: 16 us so, 5.4 us here): 32 columns per block, their rows of `b` staged whole
// in shared memory (every load in flight at once; odd row length against bank conflicts), warp = up to kFewRows / 4
// rows of `a`, lane = column.
constexpr uint32_t kFewRows = 16;
__global__ void __launch_bounds__(128)
few_rows_kernel(const float* __restrict__ b, uint32_t n_cols, const float* __restrict__ a, uint32_t n_rows, uint32_t a_stride,
                uint32_t kdim, float alpha, int half_scores, float* __restrict__ out)
{
  chain_begin();
  extern __shared__ float s_few[];  // [32][kdim | 1], then [n_rows][kdim]
  constexpr uint32_t kPer = kFewRows / 4;
  const uint32_t j0 = blockIdx.x * 32u, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t ld = kdim | 1u;
  float* s_a        = s_few + 32u * ld;
  const uint32_t nc = min(32u, n_cols - j0);
  const float* src  = b + size_t(j0) * kdim;
#pragma unroll 8
  for (uint32_t i = tid; i < nc * kdim; i += 128u) {
    const uint32_t r = i / kdim;
    s_few[r * ld + (i - r * kdim)] = __ldg(src + i);
  }
  for (uint32_t i = tid; i < n_rows * kdim; i += 128u) {
    const uint32_t r = i / kdim;
    s_a[i]           = __ldg(a + size_t(r) * a_stride + (i - r * kdim));
  }
  __syncthreads();
  float acc[kPer] = {};
  const float* c  = s_few + lane * ld;
  if (warp < n_rows) {
#pragma unroll 4
    for (uint32_t k = 0; k < kdim; k++) {
      const float cv = c[k];
#pragma unroll
      for (uint32_t r = 0; r < kPer; r++) {
        if (warp + 4u * r < n_rows) { acc[r] = __fmaf_rn(cv, s_a[(warp + 4u * r) * kdim + k], acc[r]); }
      }
    }
  }
  if (lane < nc) {
#pragma unroll
    for (uint32_t r = 0; r < kPer; r++) {
      if (warp + 4u * r < n_rows) {
        float v = __fmul_rn(alpha, acc[r]);
        if (half_scores) { v = __half2float(__float2half_rn(v)); }
        out[size_t(warp + 4u * r) * n_cols + j0 + lane] = v;
      }
    }
  }
}

template <bool kArgmin, bool kListed = false>
void launch_exact_gemm(const float* b, uint32_t n_cols, const float* a, uint32_t n_rows, uint32_t a_stride, uint32_t kdim, float alpha,
                       bool half_scores, float* out, unsigned long long* best, cudaStream_t stream,
                       const uint32_t* row_list = nullptr, const uint32_t* n_listed = nullptr)
{
  if constexpr (!kArgmin) {
    const size_t smem = (size_t(32) * (kdim | 1u) + size_t(n_rows) * kdim) * 4;
    if (n_rows <= kFewRows && smem <= 200 * 1024) {
      ensure_dynamic_smem(reinterpret_cast<const void*>(few_rows_kernel), smem);
      launch_chained(few_rows_kernel, ceildiv(n_cols, 32u), 128, smem, stream, b, n_cols, a, n_rows, a_stride, kdim,
                     alpha, half_scores, out);
      CUDA_TRY(cudaGetLastError());
      return;
    }
  }
  // grid.y is limited to 65535 blocks of rows
  const uint32_t most = 65535u * kTile;
  for (uint32_t r0 = 0; r0 < n_rows; r0 += most) {
    const uint32_t nr = std::min(most, n_rows - r0);
    dim3 grid(ceildiv(n_cols, kTile), ceildiv(nr, kTile));
    // A block per tile: 4,096 x 128 blocks that find nothing to do take 0.6 ms, these 3 us.  As many as are resident run out
    // unevenly, and so did some eight per SM whose last wave was a sixth full.  100,000 rows labelled against 50,000 lists,
    // all redone: 25.5 ms with a block per tile, 27.1 with 1,564 blocks, 26.4 with 296, 25.6 with 1,184, 25.35 so, 25.1 with 9,472.
    if (kListed) { grid = dim3(uint32_t(std::min<uint64_t>(uint64_t(grid.x) * grid.y, kListedBlocks))); }
    const float* ar = a + size_t(r0) * a_stride;
    float* o        = out ? out + size_t(r0) * n_cols : nullptr;
    unsigned long long* bs = best ? best + r0 : nullptr;
    const bool vec = kdim % 4 == 0 && a_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(ar)) & 15u) == 0;
    auto go = [&](auto kernel) {
      launch_chained(kernel, grid, 256, 0, stream, b, n_cols, ar, nr, a_stride, kdim, alpha, half_scores, o, bs, row_list, n_listed);
    };
    if (vec) {
      go(exact_gemm_kernel<true, kArgmin, kListed>);
    } else {
      go(exact_gemm_kernel<false, kArgmin, kListed>);
    }
    CUDA_TRY(cudaGetLastError());
  }
}

// One block per row.  A row holds row_len scores, or row_ends[(row + 1) * ends_stride - 1] of them.
template <uint32_t kThreads, uint32_t kTops>
__global__ void __launch_bounds__(kThreads)
select_kernel(const float* __restrict__ scores, uint32_t row_stride, uint32_t row_len, const uint32_t* __restrict__ row_ends,
              uint32_t ends_stride, uint32_t want, uint32_t cap /* keys of shared memory */, uint32_t* __restrict__ out_idx,
              float* __restrict__ out_scores)
{
  chain_begin();
  extern __shared__ uint64_t s_keys[];  // [cap]
  __shared__ select_mem s_mem;
  const uint32_t q = blockIdx.x;
  select_row<kThreads, kTops>(scores + size_t(q) * row_stride, row_ends ? row_ends[size_t(q + 1) * ends_stride - 1] : row_len,
                              row_stride % 4 == 0, want, cap, s_keys, s_mem, [](auto* p) { return __ldg(p); },
                              out_idx + size_t(q) * want, out_scores ? out_scores + size_t(q) * want : nullptr);
}

// Threads and scores kept per thread: `want` stays below two thirds of what the block keeps, where the scores taken beyond
// the wanted ones are few.
void launch_select(const float* scores, uint32_t n_rows, uint32_t row_stride, uint32_t row_len, const uint32_t* row_ends,
                   uint32_t ends_stride, uint32_t want, uint32_t* out_idx, float* out_scores, cudaStream_t stream)
{
  const uint32_t cap = select_cap(want);
  auto go = [&](auto kernel, int threads) {
    const size_t smem = size_t(cap) * 8;
    if (smem > 48 * 1024) { ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem); }
    launch_chained(kernel, n_rows, threads, smem, stream, scores, row_stride, row_len, row_ends, ends_stride, want, cap,
                   out_idx, out_scores);
    CUDA_TRY(cudaGetLastError());
  };
  if (want <= 160) {
    go(select_kernel<256, 1>, 256);
  } else if (want <= 384) {
    go(select_kernel<256, 2>, 256);
  } else if (want <= 1200) {
    go(select_kernel<1024, 2>, 1024);
  } else {
    go(select_kernel<1024, 8>, 1024);
  }
}

__global__ void unpack_labels_kernel(const unsigned long long* __restrict__ best, uint32_t n,
                                     const uint32_t* __restrict__ row_list, const uint32_t* __restrict__ n_listed,
                                     uint32_t* __restrict__ labels, unsigned long long* __restrict__ listed)
{
  chain_begin();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (row_list != nullptr) { n = min(n, __ldg(n_listed)); }
  if (i >= n) { return; }
  if (i == 0 && listed != nullptr) { atomicAdd(listed, static_cast<unsigned long long>(n)); }
  const uint32_t r = row_list != nullptr ? __ldg(row_list + i) : i;
  labels[r]        = uint32_t(best[r]);
}

// Most queries of a chunk: its scores stay around 64 MB, so that the select passes read them from L2.
uint64_t most_queries(uint32_t n_lists)
{
  const uint64_t target = 64ull << 20;
  return std::max<uint64_t>(kTile, target / (uint64_t(n_lists) * 4)) / kTile * kTile;
}

uint32_t chunk_queries(uint32_t n_queries, uint32_t n_lists)
{
  const uint64_t c = most_queries(n_lists);
  // equal chunks: a short last one would be a nearly empty wave
  const uint32_t n = uint32_t(ceildiv<uint64_t>(n_queries, c));
  return round_up<uint32_t>(ceildiv(n_queries, n), kTile);
}

}  // namespace

size_t coarse_workspace_bytes(uint32_t n_queries, uint32_t n_lists, uint32_t n_probes)
{
  (void)n_probes;
  // (enough for fewer queries too, whose chunks may be larger: two of 8,192 for 16,384 queries x 1,100 lists, one of 12,032
  // for 12,000)
  return size_t(std::min<uint64_t>(round_up(n_queries, kTile), most_queries(n_lists))) * n_lists * 4;
}

void select_clusters(raft::resources& res, const float* centers, uint32_t n_lists, uint32_t dim_ext,
                     float alpha, const float* fq, uint32_t n_queries, uint32_t n_probes,
                     uint32_t* probes, float* scores_out, void* workspace, size_t workspace_bytes,
                     bool half_scores)
{
  CUVS_EXPECTS(n_probes <= kMaxProbes, "n_probes = %u: this engine supports n_probes <= %u", n_probes,
               kMaxProbes);
  CUVS_EXPECTS(n_probes <= n_lists, "n_probes must not exceed n_lists");
  const uint32_t chunk = chunk_queries(n_queries, n_lists);
  CUVS_EXPECTS(workspace_bytes >= size_t(chunk) * n_lists * 4, "coarse workspace too small");
  float* scores = static_cast<float*>(workspace);
  for (uint32_t q0 = 0; q0 < n_queries; q0 += chunk) {
    const uint32_t nq = std::min(chunk, n_queries - q0);
    launch_exact_gemm<false>(centers, n_lists, fq + size_t(q0) * dim_ext, nq, dim_ext, dim_ext, alpha, half_scores, scores, nullptr,
                             res.stream);
    launch_select(scores, nq, n_lists, n_lists, nullptr, 0, n_probes, probes + size_t(q0) * n_probes,
                  scores_out ? scores_out + size_t(q0) * n_probes : nullptr, res.stream);
    CUDA_TRY(cudaGetLastError());
    res.launches += 2;
  }
}

void select_rows(raft::resources& res, const float* rows, uint32_t n_rows, uint32_t row_len, uint32_t k,
                 uint32_t* out_idx, float* out_scores, const uint32_t* row_ends, uint32_t ends_stride)
{
  CUVS_EXPECTS(k <= kMaxProbes && k <= row_len, "select_rows: k = %u out of range", k);
  if (n_rows == 0) { return; }
  launch_select(rows, n_rows, row_len, row_len, row_ends, ends_stride, k, out_idx, out_scores, res.stream);
  res.launches++;
}

void exact_rows_product(raft::resources& res, const float* b, uint32_t n_cols, const float* a, uint32_t n_rows, uint32_t a_stride,
                        uint32_t k, float alpha, float* out)
{
  if (n_rows == 0) { return; }
  launch_exact_gemm<false>(b, n_cols, a, n_rows, a_stride, k, alpha, false, out, nullptr, res.stream);
  res.launches++;
}

void assign_nearest(raft::resources& res, const float* centers, uint32_t n_lists, uint32_t dim_ext,
                    float alpha, const float* x_ext, uint32_t n_rows, uint32_t* labels,
                    unsigned long long* best)
{
  if (n_rows == 0) { return; }
  CUDA_TRY(cudaMemsetAsync(best, 0xFF, size_t(n_rows) * 8, res.stream));
  launch_exact_gemm<true>(centers, n_lists, x_ext, n_rows, dim_ext, dim_ext, alpha, false, nullptr, best, res.stream);
  unpack_labels_kernel<<<ceildiv<uint32_t>(n_rows, 256), 256, 0, res.stream>>>(best, n_rows, nullptr, nullptr, labels, nullptr);
  CUDA_TRY(cudaGetLastError());
  res.launches += 2;
}

void assign_nearest_listed(raft::resources& res, const float* centers, uint32_t n_lists, uint32_t dim_ext, float alpha,
                           const float* x_ext, uint32_t n_rows, const uint32_t* row_list, const uint32_t* n_listed,
                           uint32_t* labels, unsigned long long* best)
{
  CUVS_EXPECTS(n_rows <= 65535u * kTile, "too many rows");
  launch_exact_gemm<true, true>(centers, n_lists, x_ext, n_rows, dim_ext, dim_ext, alpha, false, nullptr, best, res.stream, row_list,
                                n_listed);
  launch_chained(unpack_labels_kernel, ceildiv<uint32_t>(n_rows, 256), 256, 0, res.stream, best, n_rows, row_list, n_listed, labels,
                 res.redo_counts + raft::resources::LABELS_REDONE);
  CUDA_TRY(cudaGetLastError());
  res.launches += 2;
}

}  // namespace cuvs::neighbors::ivf_pq
