// Refinement: re-rank candidate neighbours with exact distances on the original vectors.
//
// Reference: cuvs::neighbors::refine (cpp/src/neighbors/refine/refine_device.cuh:30-138, C entry
// c/src/neighbors/refine.cpp) -- there an IVF-Flat scan over a fake one-list-per-query index; here
// one to eight warps per query: groups of 1 to 32 lanes read a candidate's row with the widest loads its
// alignment allows, a shuffle tree sums the partial distances and every warp keeps its k best in its
// register top-k (merged through shared memory where a query has several warps).
// Candidates equal to INT64_MAX (the search's "no such neighbour" marker) or outside the dataset
// are ignored.  Results are sorted best first.
//   L2Expanded / L2Unexpanded : sum (q - x)^2        L2Sqrt*: its square root
//   InnerProduct              : sum q * x (largest first)
//   CosineExpanded            : 1 - q.x / (|q| |x|)
#include "common.hpp"
#include "ivf_pq.hpp"
#include "topk.cuh"

#include <algorithm>

namespace cuvs::neighbors {

using namespace cuvs_b200;
using ivf_pq::elem_t;

namespace {

enum { REF_L2 = 0, REF_L2SQRT = 1, REF_IP = 2, REF_COS = 3 };

// How a row is read: 16-byte loads where every row starts on a 16-byte boundary, 4-byte loads where every
// row starts on a 4-byte boundary, else (16- and 8-bit elements in odd row lengths) aligned 4-byte words
// shifted into place.
enum { ROW_VEC16 = 0, ROW_WORD = 1, ROW_SHIFT = 2 };

template <typename T>
__device__ __forceinline__ void word_to_floats(uint32_t w, float* f);
template <> __device__ __forceinline__ void word_to_floats<float>(uint32_t w, float* f) { f[0] = __uint_as_float(w); }
template <> __device__ __forceinline__ void word_to_floats<__half>(uint32_t w, float* f)
{
  const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w));
  f[0]           = v.x;
  f[1]           = v.y;
}
template <> __device__ __forceinline__ void word_to_floats<int8_t>(uint32_t w, float* f)
{
#pragma unroll
  for (int i = 0; i < 4; i++) { f[i] = float(int8_t((w >> (8 * i)) & 0xFFu)); }
}
template <> __device__ __forceinline__ void word_to_floats<uint8_t>(uint32_t w, float* f)
{
#pragma unroll
  for (int i = 0; i < 4; i++) { f[i] = float((w >> (8 * i)) & 0xFFu); }
}
__device__ __forceinline__ float elem_to_float(float x) { return x; }
__device__ __forceinline__ float elem_to_float(__half x) { return __half2float(x); }
__device__ __forceinline__ float elem_to_float(int8_t x) { return float(x); }
__device__ __forceinline__ float elem_to_float(uint8_t x) { return float(x); }

// Step v of a row's words: four words (ROW_VEC16) or one.
template <typename T, int ROW>
__device__ __forceinline__ void load_step(const T* row, uint32_t v, uint32_t row_bytes, uint32_t* w)
{
  if constexpr (ROW == ROW_VEC16) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(row) + v);
    w[0] = x.x;
    w[1] = x.y;
    w[2] = x.z;
    w[3] = x.w;
  } else if constexpr (ROW == ROW_WORD) {
    w[0] = __ldg(reinterpret_cast<const uint32_t*>(row) + v);
  } else {
    // bytes [4v, 4v + 4) of a row that starts anywhere: the aligned word that holds the first of them and,
    // if the row reaches into it, the next one
    const uintptr_t a  = reinterpret_cast<uintptr_t>(row) + 4u * v;
    const uint32_t mis = uint32_t(a & 3u);
    const uint32_t* p  = reinterpret_cast<const uint32_t*>(a - mis);
    const uint32_t lo  = __ldg(p);
    const uint32_t hi  = mis != 0u && 4u * v + 4u - mis < row_bytes ? __ldg(p + 1) : 0u;
    w[0]               = __funnelshift_r(lo, hi, 8u * mis);
  }
}

// What bounds it: latency of rows of a few hundred bytes at random places, i.e. bytes in flight.  One warp
// per query with element-wise loads moved 0.65 TB/s on 4,000 x 200 candidates of 768 halves (1.32 ms);
// 16-byte loads, four rows per group of lanes in flight and several warps per query: 2.6 TB/s (0.33 ms).
template <typename T, int KPL, int ROW>
__global__ void __launch_bounds__(256, 4)
refine_kernel(const T* __restrict__ dataset, int64_t n_rows, uint32_t dim,
              const T* __restrict__ queries, uint32_t n_queries,
              const int64_t* __restrict__ candidates, uint32_t n_cand, uint32_t k,
              int mode, uint32_t log_lanes, uint32_t log_wpq, uint32_t q_floats,
              int64_t* __restrict__ indices, float* __restrict__ distances)
{
  chain_begin();
  constexpr uint32_t kWords = ROW == ROW_VEC16 ? 4u : 1u;          // 4-byte words per load step
  constexpr uint32_t kPerWord = 4u / uint32_t(sizeof(T));
  constexpr uint32_t kElems = kWords * kPerWord;
  constexpr int kRows       = 4;
  // [queries per block][q_floats] queries, zero-padded to whole load steps, then the merge buffers
  extern __shared__ __align__(16) float s_query[];
  const uint32_t wib  = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t wpq  = 1u << log_wpq;                               // warps per query
  const uint32_t qib  = wib >> log_wpq, part = wib & (wpq - 1u);
  const uint32_t qpb  = (blockDim.x >> 5) >> log_wpq;
  const uint32_t q    = blockIdx.x * qpb + qib;
  const bool active   = q < n_queries;
  float* sq           = s_query + size_t(qib) * q_floats;
  if (active) {
    const T* qrow = queries + size_t(q) * dim;
    for (uint32_t d = part * 32u + lane; d < q_floats; d += wpq * 32u) {
      sq[d] = d < dim ? elem_to_float(qrow[d]) : 0.0f;
    }
  }
  __syncthreads();
  warp_topk<KPL> queue;
  queue.init(int(k));
  const int64_t* cand      = candidates + size_t(active ? q : 0u) * n_cand;
  const uint32_t lanes     = 1u << log_lanes;                        // lanes that share a row
  const uint32_t rows      = 32u >> log_lanes;                       // rows a warp reads at a time
  const uint32_t group     = lane >> log_lanes, gl = lane & (lanes - 1u);
  const uint32_t row_bytes = dim * uint32_t(sizeof(T));
  const uint32_t n_steps   = (dim + kElems - 1u) / kElems;
  if (active) {
    float qn = 0.0f;
    if (mode == REF_COS) {
      for (uint32_t d = lane; d < dim; d += 32) { qn = __fmaf_rn(sq[d], sq[d], qn); }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) { qn += __shfl_xor_sync(kFullMask, qn, o); }
    }
    for (uint32_t c0 = part * 32u; c0 < n_cand; c0 += wpq * 32u) {
      const uint32_t n_here = min(32u, n_cand - c0);
      int64_t my_id         = -1;
      if (lane < n_here) { my_id = cand[c0 + lane]; }
      if (my_id >= n_rows) { my_id = -1; }
      float my_score = INFINITY;
      // four rows per group of lanes at a time, so that their loads are in flight together
      for (uint32_t j = 0; j < n_here; j += kRows * rows) {
        const T* x[kRows];
        bool ok[kRows];
        float acc[kRows] = {}, xn[kRows] = {};
#pragma unroll
        for (int u = 0; u < kRows; u++) {
          const uint32_t c = j + uint32_t(u) * rows + group;         // may pass 31: the shuffle wraps, ok[] masks
          const int64_t id = int64_t(shfl_u64(uint64_t(my_id), int(c & 31u)));
          ok[u]            = c < n_here && id >= 0;
          x[u]             = dataset + size_t(ok[u] ? id : 0) * dim;
        }
#pragma unroll 3
        for (uint32_t v = gl; v < n_steps; v += lanes) {
          uint32_t w[kRows][kWords];
#pragma unroll
          for (int u = 0; u < kRows; u++) {
            if (ok[u]) {
              load_step<T, ROW>(x[u], v, row_bytes, w[u]);
            } else {
#pragma unroll
              for (uint32_t i = 0; i < kWords; i++) { w[u][i] = 0u; }
            }
          }
          float qv[kElems];
          if constexpr (kElems % 4 == 0) {
#pragma unroll
            for (uint32_t e = 0; e < kElems; e += 4) {
              const float4 t = *reinterpret_cast<const float4*>(sq + v * kElems + e);
              qv[e] = t.x;
              qv[e + 1] = t.y;
              qv[e + 2] = t.z;
              qv[e + 3] = t.w;
            }
          } else {
#pragma unroll
            for (uint32_t e = 0; e < kElems; e++) { qv[e] = sq[v * kElems + e]; }
          }
#pragma unroll
          for (int u = 0; u < kRows; u++) {
            float xv[kElems];
#pragma unroll
            for (uint32_t i = 0; i < kWords; i++) { word_to_floats<T>(w[u][i], xv + i * kPerWord); }
            if constexpr (ROW == ROW_SHIFT) {
              // the last word of a row may carry bytes of the next one
#pragma unroll
              for (uint32_t e = 0; e < kElems; e++) {
                if (v * kElems + e >= dim) { xv[e] = 0.0f; }
              }
            }
            if (mode == REF_IP) {
#pragma unroll
              for (uint32_t e = 0; e < kElems; e++) { acc[u] = __fmaf_rn(qv[e], xv[e], acc[u]); }
            } else if (mode == REF_COS) {
#pragma unroll
              for (uint32_t e = 0; e < kElems; e++) {
                acc[u] = __fmaf_rn(qv[e], xv[e], acc[u]);
                xn[u]  = __fmaf_rn(xv[e], xv[e], xn[u]);
              }
            } else {
#pragma unroll
              for (uint32_t e = 0; e < kElems; e++) {
                const float t = qv[e] - xv[e];
                acc[u]        = __fmaf_rn(t, t, acc[u]);
              }
            }
          }
        }
#pragma unroll
        for (int u = 0; u < kRows; u++) {
          float a = acc[u], b = xn[u];
          for (uint32_t o = lanes >> 1; o > 0; o >>= 1) {
            a += __shfl_xor_sync(kFullMask, a, int(o));
            if (mode == REF_COS) { b += __shfl_xor_sync(kFullMask, b, int(o)); }
          }
          float score = a;                       // smaller is better
          if (mode == REF_IP) { score = -a; }
          if (mode == REF_COS) { score = 1.0f - a / (sqrtf(qn) * sqrtf(b) + 1e-30f); }
          // candidate j + u * rows + g was summed by group g: hand it to the lane of that number
          const uint32_t first = j + uint32_t(u) * rows;
          const float mine     = __shfl_sync(kFullMask, score, int(((lane - first) & (rows - 1u)) << log_lanes));
          if (lane >= first && lane < first + rows) { my_score = mine; }
        }
      }
      queue.offer(make_key(my_score, c0 + lane), my_id >= 0);
    }
  }
  if (wpq > 1u) {
    uint64_t* s_merge = reinterpret_cast<uint64_t*>(s_query + size_t(qpb) * q_floats) + size_t(qib) * wpq * k;
    if (part != 0u) { queue.store(s_merge + size_t(part) * k, int(k)); }
    __syncthreads();
    if (part != 0u) { return; }
    for (uint32_t t0 = k; t0 < wpq * k; t0 += 32) {
      const uint32_t t = t0 + lane;
      queue.offer(t < wpq * k ? s_merge[t] : kEmptyKey, t < wpq * k);
    }
  }
  if (!active) { return; }
#pragma unroll
  for (int r = 0; r < KPL; r++) {
    const uint32_t pos = uint32_t(r) * 32u + lane;
    if (pos >= k) { continue; }
    const uint64_t key = queue.a[r];
    int64_t id         = ivf_pq::kOutOfBoundsRecord;
    float d            = mode == REF_IP ? -INFINITY : INFINITY;
    if (uint32_t(key >> 32) != kEmptyScore) {
      id = cand[uint32_t(key)];
      d  = ordered_to_float(uint32_t(key >> 32));
      if (mode == REF_IP) { d = -d; }
      if (mode == REF_L2SQRT) { d = sqrtf(d); }
    }
    indices[size_t(q) * k + pos]   = id;
    distances[size_t(q) * k + pos] = d;
  }
}

template <typename T, int ROW>
void launch_refine_rows(raft::resources& res, const T* dataset, int64_t n_rows, uint32_t dim,
                        const T* queries, uint32_t n_queries, const int64_t* candidates, uint32_t n_cand,
                        uint32_t k, int mode, int64_t* indices, float* distances)
{
  constexpr uint32_t kElems = (ROW == ROW_VEC16 ? 16u : 4u) / uint32_t(sizeof(T));
  const uint32_t n_steps    = ceildiv(dim, kElems);
  // Lanes per row: as few as still leave a lane at most eight loads of the row, so that a warp reads
  // several rows at a time (a 128-byte row: one lane, 32 rows; 768 halves: 16 lanes, 2 rows: 332 us against
  // 355 us with the whole warp on a row).
  uint32_t log_lanes = 0;
  while (log_lanes < 5 && (8u << log_lanes) < n_steps) { log_lanes++; }
  // Warps per query: enough for 64 per SM (24 and 200: 15-25% slower), at most one per 32 candidates.
  uint32_t log_wpq = 0;
  while (log_wpq < 3 && (size_t(n_queries) << log_wpq) < size_t(res.sm_count) * 64 && (32u << log_wpq) < n_cand) {
    log_wpq++;
  }
  const uint32_t warps    = std::max(4u, 1u << log_wpq);
  const uint32_t qpb      = warps >> log_wpq;
  const uint32_t q_floats = round_up(n_steps * kElems, 4u);
  size_t smem             = size_t(qpb) * q_floats * 4 + (log_wpq > 0 ? size_t(warps) * k * 8 : 0);
  auto go = [&](auto kernel) {
    if (smem > 48 * 1024) {
      CUVS_EXPECTS(smem <= size_t(res.smem_optin) - 1024, "refine: dim = %u is too large", dim);
      ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    }
    launch_chained(kernel, ceildiv(n_queries, qpb), warps * 32, smem, res.stream, dataset, n_rows, dim, queries,
                   n_queries, candidates, n_cand, k, mode, log_lanes, log_wpq, q_floats, indices, distances);
    CUDA_TRY(cudaGetLastError());
  };
  if (k <= 32) {
    go(refine_kernel<T, 1, ROW>);
  } else if (k <= 64) {
    go(refine_kernel<T, 2, ROW>);
  } else {
    go(refine_kernel<T, 4, ROW>);
  }
  res.launches++;
}

template <typename T>
void launch_refine(raft::resources& res, const void* dataset, int64_t n_rows, uint32_t dim,
                   const void* queries, uint32_t n_queries, const int64_t* candidates, uint32_t n_cand,
                   uint32_t k, int mode, int64_t* indices, float* distances)
{
  const T* ds          = static_cast<const T*>(dataset);
  const T* qs          = static_cast<const T*>(queries);
  const uintptr_t bits = reinterpret_cast<uintptr_t>(dataset) | (size_t(dim) * sizeof(T));
  if ((bits & 15u) == 0) {
    launch_refine_rows<T, ROW_VEC16>(res, ds, n_rows, dim, qs, n_queries, candidates, n_cand, k, mode, indices, distances);
  } else if (sizeof(T) == 4 || (bits & 3u) == 0) {
    launch_refine_rows<T, ROW_WORD>(res, ds, n_rows, dim, qs, n_queries, candidates, n_cand, k, mode, indices, distances);
  } else if constexpr (sizeof(T) < 4) {
    launch_refine_rows<T, ROW_SHIFT>(res, ds, n_rows, dim, qs, n_queries, candidates, n_cand, k, mode, indices, distances);
  }
}

}  // namespace

void refine_any(raft::resources& res, const void* dataset, elem_t dtype, int64_t n_rows, uint32_t dim,
                const void* queries, uint32_t n_queries, const int64_t* candidates, uint32_t n_cand,
                ivf_pq::DistanceType metric, int64_t* indices, float* distances, uint32_t k)
{
  // refine_check_input of the reference (cpp/src/neighbors/refine/refine_common.hpp)
  CUVS_EXPECTS(k > 0 && k <= n_cand,
               "Number of neighbors cannot be smaller than k (candidates %u, k %u)", n_cand, k);
  CUVS_EXPECTS(k <= 128, "k must be less than topk::kMaxCapacity (%d).", 128);
  int mode;
  switch (metric) {
    case ivf_pq::DistanceType::L2Expanded:
    case ivf_pq::DistanceType::L2Unexpanded: mode = REF_L2; break;
    case ivf_pq::DistanceType::L2SqrtExpanded:
    case ivf_pq::DistanceType::L2SqrtUnexpanded: mode = REF_L2SQRT; break;
    case ivf_pq::DistanceType::InnerProduct: mode = REF_IP; break;
    case ivf_pq::DistanceType::CosineExpanded: mode = REF_COS; break;
    default: fail("refine: unsupported metric %d", int(metric));
  }
  if (n_queries == 0) { return; }
  switch (dtype) {
    case elem_t::f32:
      launch_refine<float>(res, dataset, n_rows, dim, queries, n_queries, candidates, n_cand, k, mode, indices, distances);
      break;
    case elem_t::f16:
      launch_refine<__half>(res, dataset, n_rows, dim, queries, n_queries, candidates, n_cand, k, mode, indices, distances);
      break;
    case elem_t::i8:
      launch_refine<int8_t>(res, dataset, n_rows, dim, queries, n_queries, candidates, n_cand, k, mode, indices, distances);
      break;
    default:
      launch_refine<uint8_t>(res, dataset, n_rows, dim, queries, n_queries, candidates, n_cand, k, mode, indices, distances);
  }
}

}  // namespace cuvs::neighbors
